// Device code shared by the 3D vote kernels (vote3.cu, vote3_sep.cu): input
// layouts, the voters' eigensolve and scales, and the outputs of a receiver.
#pragma once
#include "tvgb_internal.cuh"
#include "eig_device.cuh"

namespace tvgb {

template <int LAYOUT>
__device__ __forceinline__ void read_tensor(const float* __restrict__ in, size_t n, size_t i, float& a, float& b,
                                            float& c, float& d, float& e, float& f) {
    if (LAYOUT == 9) {
        const float* m = in + i * 9;
        a = __ldg(m); b = __ldg(m + 1); d = __ldg(m + 2); c = __ldg(m + 4); e = __ldg(m + 5); f = __ldg(m + 8);
    } else if (LAYOUT == 6) {
        const float* m = in + i * 6;
        a = __ldg(m); b = __ldg(m + 1); d = __ldg(m + 2); c = __ldg(m + 3); e = __ldg(m + 4); f = __ldg(m + 5);
    } else {
        a = __ldg(in + i); b = __ldg(in + n + i); d = __ldg(in + 2 * n + i);
        c = __ldg(in + 3 * n + i); e = __ldg(in + 4 * n + i); f = __ldg(in + 5 * n + i);
    }
}

// One voter's eigenpairs, ascending.
template <int LAYOUT>
__device__ __forceinline__ void solve_voter(const float* __restrict__ in, size_t n, size_t i, int parity, float (&ev)[3],
                                            float (&v0)[3], float (&v1)[3], float (&v2)[3]) {
    float a, b, c, d, e, f;
    read_tensor<LAYOUT>(in, n, i, a, b, c, d, e, f);
    if (parity) {
        eval3_d(a, b, c, d, e, f, ev[0], ev[1], ev[2]);
        evec3_d(a, b, c, d, e, f, ev, v0, v1, v2);
        // cpu::tensorvote3 / cuda::tensorvote3 pass the eigenvectors through
        // float (theta, phi) and back (tensorvote.h:1831-1849, 2831-2858)
        float th, ph;
        to_spherical_d(v0, th, ph); from_spherical_d(th, ph, v0);
        to_spherical_d(v1, th, ph); from_spherical_d(th, ph, v1);
        to_spherical_d(v2, th, ph); from_spherical_d(th, ph, v2);
    } else {
        eig3_precise_d(a, b, c, d, e, f, ev, v0, v1, v2);
    }
}

// TK: tensorvote.h:1537; ATV: atv_H's s1 = lambda2 - lambda1 (:660), no normaliser
__device__ __forceinline__ float stick_scale(const float (&ev)[3], int atv, float sticknorm) {
    return atv ? ev[2] - ev[1] : copysignf(fabsf(ev[2]) - fabsf(ev[1]), ev[2]) * sticknorm;
}

// (unit plate normal, plate scale); plate3_numerical_device normalises the
// normal and skips a zero one (:2461-2465).  TK: :2616; ATV: atv_H's
// s2 = lambda1 - lambda0 on the plane normal to n (:661)
__device__ __forceinline__ float4 plate_record(const float (&ev)[3], const float (&v0)[3], int atv) {
    const float nn = v0[0] * v0[0] + v0[1] * v0[1] + v0[2] * v0[2];
    float sp = atv ? ev[1] - ev[0] : copysignf(fabsf(ev[1]) - fabsf(ev[0]), ev[1]);
    float inv = 0.0f;
    if (nn > 1e-12f) inv = rsqrtf(nn); else sp = 0.0f;
    return make_float4(v0[0] * inv, v0[1] * inv, v0[2] * inv, sp);
}

struct FastArgs {
    const float4* A;
    const float4* B;
    const float* C;
    int s0, s1, s2, hw, rows;   // rows: voter rows (offsets) staged per stage
    float sig1, sig2;
    float* out;
    int out_layout;
    float* evals;
    float* evecs;
    int evec_fmt;
    int precise_eig;
    int zr0, zr1;               // receivers voted: planes [zr0, zr1) (launch_fast: [0, s0) if empty)
    int atv;                    // ATV weights (radial_entry_atv, sigma = sig1) instead of TK's
};

__device__ __forceinline__ void write_receiver(const FastArgs& a, size_t idx, size_t n, const float* m6) {
    float* out = a.out;
    if (out) {
        if (a.out_layout == TVGB_LAYOUT_MAT3) {
            float* o = out + idx * 9;
            o[0] = m6[0]; o[1] = m6[1]; o[2] = m6[2];
            o[3] = m6[1]; o[4] = m6[3]; o[5] = m6[4];
            o[6] = m6[2]; o[7] = m6[4]; o[8] = m6[5];
        } else if (a.out_layout == TVGB_LAYOUT_SYM6) {
            float* o = out + idx * 6;
            for (int k = 0; k < 6; ++k) o[k] = m6[k];
        } else {
            for (int k = 0; k < 6; ++k) out[k * n + idx] = m6[k];
        }
    }
    if (a.evals || a.evecs) {
        float ev[3], v[9];
        if (a.precise_eig) {
            eig3_precise_d(m6[0], m6[1], m6[3], m6[2], m6[4], m6[5], ev, v, v + 3, v + 6);
        } else {
            eval3_d(m6[0], m6[1], m6[3], m6[2], m6[4], m6[5], ev[0], ev[1], ev[2]);
            if (a.evecs) evec3_d(m6[0], m6[1], m6[3], m6[2], m6[4], m6[5], ev, v, v + 3, v + 6);
        }
        if (a.evals) { a.evals[idx * 3] = ev[0]; a.evals[idx * 3 + 1] = ev[1]; a.evals[idx * 3 + 2] = ev[2]; }
        if (a.evecs) {
            if (a.evec_fmt == TVGB_EVEC_CARTESIAN) {
                for (int k = 0; k < 9; ++k) a.evecs[idx * 9 + k] = v[k];
            } else {
                float th, ph;
                to_spherical_d(v, th, ph); a.evecs[idx * 6] = th; a.evecs[idx * 6 + 1] = ph;
                to_spherical_d(v + 3, th, ph); a.evecs[idx * 6 + 2] = th; a.evecs[idx * 6 + 3] = ph;
                to_spherical_d(v + 6, th, ph); a.evecs[idx * 6 + 4] = th; a.evecs[idx * 6 + 5] = ph;
            }
        }
    }
}

// A volume of few groups of 32 x 8 x 4 receivers, the pair-by-pair kernel's
// CTA, leaves SMs without one: there it takes one receiver plane per CTA (24 x
// 20 x 28, sigma 1.5: 76 us instead of 215).  114 groups are three CTAs of a
// plane for every SM.  Four planes' time over one's, windows 7 .. 61, with and
// without the ball: 24 groups 2.6 .. 3.4, 72 1.6 .. 2.0, 100 1.1 .. 1.6, 120
// 0.99 .. 1.2, 150 0.80 .. 1.10.
inline bool vote3_small(unsigned planes, unsigned s1, unsigned s2) {
    return size_t(ceil_div(s2, 32u)) * ceil_div(s1, 8u) * ceil_div(planes, 4u) <= 114;
}

}  // namespace tvgb
