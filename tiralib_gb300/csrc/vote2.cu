// 2D tensor voting (TK and ATV) on sm_103a and its C ABI.
//
// Reference path replaced (tira/functions/tensorvote.h):
//   tira::cuda::tensorvote :2201 -> evals2_symmetric / evecs2polar_symmetric
//   (eigen.h:769,828, each with host round trips) -> tensorvote_tk :2126
//   (cpu::build_neighbors2d :1223 on the host, upload, global_tensorvote_tk
//   :2072 with threadIdx.x on the SLOW axis, so every load is strided, and a
//   cos/sin of the voter angle per pair) or tensorvote_atv :2029.
//
// Here: one prep kernel solves every pixel's 2x2 once (eigen.h semantics) and
// stores the voter record (cos th1, sin th1, stick scale, lambda0); the vote
// kernel maps x (fast axis) to threadIdx.x so voter loads coalesce, and
// streams the Neighbor2D table through shared memory so each entry is a
// broadcast read.  The table itself is built on the host with the
// reference's float arithmetic (it is O(w^2 samples) and tiny).
#include "tvgb_internal.cuh"
#include "eig_device.cuh"
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <vector>

namespace tvgb {

struct Nb2 {             // tira::Neighbor2D, 48 bytes (tensorvote.h:776)
    int du, dv;
    float dx, dy, c1, c2, Ra, Rb, Rc, Va, Vb, Vc;
};
static_assert(sizeof(Nb2) == 48, "Neighbor2D must be 48 bytes");

// ---------------------------------------------------------------- host table (float steps of the reference)
static float atten_h(float dist, float sigma) {            // atv_attenuation, :35
    if (sigma == 0.0f) return (double(dist) > 1e-12) ? 0.0f : 1.0f;
    return std::exp(-(dist * dist) / (sigma * sigma));
}
static float stick_norm_2d_h(float s1, float s2, unsigned p) {   // tk_stick_norm_2d, :843
    if (p < 1) p = 1;
    float r = 1.0f;
    for (unsigned k = 1; k <= p; ++k) r *= float(2 * k) / float(2 * k - 1);
    return r / (float(3.14159265358979323846) * (s1 * s1 + s2 * s2));
}
static void stickvote_2d_h(float rx, float ry, float s1, float s2, unsigned power, float theta, float& Va, float& Vb,
                           float& Vc) {                     // tk_stickvote_2d, :872
    const float qx = std::cos(theta), qy = std::sin(theta);
    const float dist = std::sqrt(rx * rx + ry * ry);
    float dx = 0.0f, dy = 0.0f;
    if (dist != 0.0f) { dx = rx / dist; dy = ry / dist; }
    const float qTd = qx * dx + qy * dy;
    unsigned p = power < 1 ? 1 : power;
    const float c1 = atten_h(dist, s1), c2 = atten_h(dist, s2);
    const float q2 = qTd * qTd, t1 = 1.0f - q2, t2 = q2;
    float D;
    if (p == 1) D = c1 * t1 + c2 * t2;
    else { float e1 = t1, e2 = t2; for (unsigned i = 1; i < p; ++i) { e1 *= t1; e2 *= t2; } D = c1 * e1 + c2 * e2; }
    const float factor = D * stick_norm_2d_h(s1, s2, power);
    const float Ra = 1 - 2 * dx * dx, Rb = -2 * dx * dy, Rc = 1 - 2 * dy * dy;
    const float Rqx = Ra * qx + Rb * qy, Rqy = Rb * qx + Rc * qy;
    Va = Rqx * Rqx * factor; Vb = Rqx * Rqy * factor; Vc = Rqy * Rqy * factor;
}

static int build_table(int w, float s1, float s2, unsigned power, unsigned samples, bool stick, bool plate, Nb2* out) {
    if (w <= 0) return 0;
    const int hw = w / 2;
    const float inv1 = s1 > 0 ? 1.0f / (s1 * s1) : 0.0f, inv2 = s2 > 0 ? 1.0f / (s2 * s2) : 0.0f;
    int k = 0;
    for (int dv = -hw; dv <= hw; dv++)
        for (int du = -hw; du <= hw; du++) {
            Nb2 e{};
            e.du = du; e.dv = dv;
            const float l2 = float(du * du + dv * dv);
            if (stick) {
                if (l2 != 0.0f) { const float il = 1.0f / std::sqrt(l2); e.dx = float(du) * il; e.dy = float(dv) * il; }
                e.c1 = s1 == 0.0f ? (l2 > 1e-12f ? 0.0f : 1.0f) : std::exp(-l2 * inv1);
                e.c2 = s2 == 0.0f ? (l2 > 1e-12f ? 0.0f : 1.0f) : std::exp(-l2 * inv2);
                e.Ra = 1.0f - 2.0f * e.dx * e.dx; e.Rb = 0.0f - 2.0f * e.dx * e.dy; e.Rc = 1.0f - 2.0f * e.dy * e.dy;
            }
            if (plate && samples > 0) {      // tk_plate_numerical (2D), :1048
                const float dth = float(3.14159265358979323846 / double(float(samples)));
                float a = 0, b = 0, c = 0;
                for (unsigned i = 0; i < samples; ++i) {
                    float va, vb, vc;
                    stickvote_2d_h(float(du), float(dv), s1, s2, power, dth * float(i), va, vb, vc);
                    a += va; b += vb; c += vc;
                }
                const float wb = float(3.14159265358979323846) / float(samples);
                e.Va = a * wb; e.Vb = b * wb; e.Vc = c * wb;
            }
            if (out) out[k] = e;
            k++;
        }
    return k;
}

// ---------------------------------------------------------------- kernels
// voter record: (cos th1, sin th1, stick scale, lambda0); ATV adds (l1, cos th0, sin th0)
__global__ void k_prep2(const float4* __restrict__ in, size_t n, float4* __restrict__ V, float4* __restrict__ W) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        const float4 m = __ldg(in + i);
        float l0, l1, t0, t1;
        eval2_d(m.x, m.y, m.w, l0, l1);
        evec2polar_d(m.x, m.y, m.w, l0, t0, t1);
        float scale = fabsf(l1) - fabsf(l0);
        if (l1 < 0.0f) scale = -scale;                     // tk_stick_window, :996-997
        V[i] = make_float4(cosf(t1), sinf(t1), scale, l0);
        if (W) W[i] = make_float4(l1, cosf(t0), sinf(t0), 0.0f);
    }
}

constexpr int V2X = 32, V2Y = 8, NB_CHUNK = 512;

template <bool STICK, bool PLATE>
__global__ void __launch_bounds__(V2X * V2Y) k_vote2_tk(const float4* __restrict__ V, const Nb2* __restrict__ nb, int nbc,
                                                         int s0, int s1, float eta_s, unsigned power, float4* __restrict__ out) {
    __shared__ Nb2 snb[NB_CHUNK];
    const int x = blockIdx.x * V2X + threadIdx.x;    // fast axis (x1)
    const int y = blockIdx.y * V2Y + threadIdx.y;    // slow axis (x0)
    const int tid = threadIdx.y * V2X + threadIdx.x;
    float sa = 0, sb = 0, sc = 0, pa = 0, pb = 0, pc = 0;
    for (int c0 = 0; c0 < nbc; c0 += NB_CHUNK) {
        const int cn = min(NB_CHUNK, nbc - c0);
        __syncthreads();
        for (int i = tid; i < cn; i += V2X * V2Y) snb[i] = nb[c0 + i];
        __syncthreads();
        for (int k = 0; k < cn; ++k) {
            const Nb2& e = snb[k];
            const int r0 = y + e.dv, r1 = x + e.du;
            if ((unsigned)r0 >= (unsigned)s0 || (unsigned)r1 >= (unsigned)s1) continue;
            const float4 v = __ldg(V + size_t(r0) * s1 + r1);
            if (STICK) {
                const float qTd = v.x * e.dx + v.y * e.dy;
                const float q2 = qTd * qTd, t1 = 1.0f - q2, t2 = q2;
                float D;
                if (power == 1) D = e.c1 * t1 + e.c2 * t2;
                else { float e1 = t1, e2 = t2; for (unsigned i = 1; i < power; ++i) { e1 *= t1; e2 *= t2; } D = e.c1 * e1 + e.c2 * e2; }
                const float Rqx = e.Ra * v.x + e.Rb * v.y, Rqy = e.Rb * v.x + e.Rc * v.y;
                const float f = D * eta_s * v.z;
                sa = fmaf(f * Rqx, Rqx, sa); sb = fmaf(f * Rqx, Rqy, sb); sc = fmaf(f * Rqy, Rqy, sc);
            }
            if (PLATE && v.w != 0.0f) {
                pa = fmaf(v.w, e.Va, pa); pb = fmaf(v.w, e.Vb, pb); pc = fmaf(v.w, e.Vc, pc);
            }
        }
    }
    if (x < s1 && y < s0) out[size_t(y) * s1 + x] = make_float4(sa + pa, sb + pb, sb + pb, sc + pc);
}

// Staged variant for windows whose voter tile fits in shared memory: a CTA
// of 32 x TY threads owns 32 x (TY V2R) receivers (V2R rows per thread, TY
// apart) and reads their voters from a (32 + 2 h) x (TY V2R + 2 h) tile
// staged once, zero outside the image, so the table loop has no bounds checks
// and each table entry (a warp-uniform broadcast) serves V2R receivers.  h
// bounds |du|, |dv| over the table.  The table streams through shared memory
// in chunks of NBC entries.  Measured at 512^2 (C1, 20-step bench): TY = 8
// (256 CTAs, 0.56 of a wave) 0.083 ms, TY = 4 0.092 ms, TY = 2 (1024 CTAs,
// all resident) 0.094 ms: the kernel runs at the pace its warps' dependent
// chains allow, and smaller CTAs buy no more warps per SM.
//
// Per pair, FP32 operations (the pipe that bounds the kernel): the stick
// weight D = c1 (1 - q^2)^p + c2 (q^2)^p is, for p = 1, c1 + (c2 - c1) q^2
// (one FMA with c2 - c1 formed once per entry); the reflected orientation
// R q = q - 2 (q.d) d costs a multiply and two FMAs instead of the four
// operations of the entry's (Ra, Rb, Rc) matrix product.  16 operations per
// pair with the plate, against 19 for the reference's literal expressions;
// both agree to FP32 rounding (0.092 -> 0.083 ms at C1).  A packed form
// (two receiver rows per FFMA2 from a paired-row tile, pre-broadcast table
// entries) measured 0.092 ms: a packed instruction holds the FP32 pipe as
// long as two scalar ones, and its larger tile and entry loads cost more than
// the issue slots it saves.
template <int V2R, int TY, int NBC, bool STICK, bool PLATE, bool P1>
__global__ void __launch_bounds__(V2X * TY) k_vote2_tks(const float4* __restrict__ V, const Nb2* __restrict__ nb,
                                                        int nbc, int s0, int s1, int h, float eta_s, unsigned power,
                                                        float4* __restrict__ out) {
    extern __shared__ __align__(16) float4 sm2[];
    Nb2* snb = reinterpret_cast<Nb2*>(sm2);                       // NBC entries
    float4* tile = sm2 + NBC * sizeof(Nb2) / sizeof(float4);      // TW x TH voters
    constexpr int NT = V2X * TY;
    const int TW = V2X + 2 * h, TH = TY * V2R + 2 * h;
    const int x0 = blockIdx.x * V2X, y0 = blockIdx.y * (TY * V2R);
    const int tid = threadIdx.y * V2X + threadIdx.x;
    for (int e = tid; e < TW * TH; e += NT) {
        const int r = e / TW, c = e - r * TW;
        const int gy = y0 - h + r, gx = x0 - h + c;
        tile[e] = ((unsigned)gy < (unsigned)s0 && (unsigned)gx < (unsigned)s1) ? __ldg(V + size_t(gy) * s1 + gx)
                                                                               : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float sa[V2R], sb[V2R], sc[V2R], pa[V2R], pb[V2R], pc[V2R];
#pragma unroll
    for (int j = 0; j < V2R; ++j) { sa[j] = sb[j] = sc[j] = pa[j] = pb[j] = pc[j] = 0.0f; }
    // receiver j of this thread: (x0 + tx, y0 + ty + TY j); its voter at (du, dv) is tile[ty + TY j + h + dv][tx + h + du]
    const float4* base = tile + (threadIdx.y + h) * TW + threadIdx.x + h;
    for (int c0 = 0; c0 < nbc; c0 += NBC) {
        const int cn = min(NBC, nbc - c0);
        __syncthreads();
        for (int i = tid; i < cn; i += NT) snb[i] = nb[c0 + i];
        __syncthreads();
#pragma unroll 2
        for (int k = 0; k < cn; ++k) {
            const Nb2& e = snb[k];
            const float4* vp = base + e.dv * TW + e.du;
            const float dc = e.c2 - e.c1;
#pragma unroll
            for (int j = 0; j < V2R; ++j) {
                const float4 v = vp[j * TY * TW];
                if (STICK) {
                    const float qTd = fmaf(v.x, e.dx, v.y * e.dy);
                    const float q2 = qTd * qTd;
                    float D;
                    if (P1) D = fmaf(dc, q2, e.c1);
                    else {
                        const float t1 = 1.0f - q2, t2 = q2;
                        float e1 = t1, e2 = t2;
                        for (unsigned i = 1; i < power; ++i) { e1 *= t1; e2 *= t2; }
                        D = e.c1 * e1 + e.c2 * e2;
                    }
                    const float k2 = -2.0f * qTd;
                    const float Rqx = fmaf(k2, e.dx, v.x), Rqy = fmaf(k2, e.dy, v.y);
                    const float f = D * v.z;
                    const float fx = f * Rqx;
                    sa[j] = fmaf(fx, Rqx, sa[j]); sb[j] = fmaf(fx, Rqy, sb[j]); sc[j] = fmaf(f * Rqy, Rqy, sc[j]);
                }
                if (PLATE) {   // v.w = 0 outside the image and for zero plates
                    pa[j] = fmaf(v.w, e.Va, pa[j]); pb[j] = fmaf(v.w, e.Vb, pb[j]); pc[j] = fmaf(v.w, e.Vc, pc[j]);
                }
            }
        }
    }
    const int x = x0 + threadIdx.x;
    if (x >= s1) return;
#pragma unroll
    for (int j = 0; j < V2R; ++j) {
        const int y = y0 + threadIdx.y + TY * j;
        if (y >= s0) break;
        const float a = fmaf(eta_s, sa[j], pa[j]), b = fmaf(eta_s, sb[j], pb[j]), c = fmaf(eta_s, sc[j], pc[j]);
        out[size_t(y) * s1 + x] = make_float4(a, b, b, c);
    }
}

// ---------------------------------------------------------------- a batch of votes
// K parameter sets voted on one field in one launch (grid.z: the set), for the
// parameter sweep.  A first launch computes every set's Neighbor2D entries
// (the steps of build_table) on the device, where the host took ~5 ms for a
// 121^2 table and the stream waited for its upload.  A CTA of 32 x 8 threads
// owns 32 x 32 receivers of a set (4 per thread).  It works through the window
// in bands of offset rows: the band's entries and the voters that the band
// reaches are staged side by side, so any window up to 347 pixels runs from
// shared memory.  One launch of all sets fills the SMs that a set of a 160^2
// field alone leaves idle (25 CTAs).  45 sets on 160^2, sigma <= 20, powers <=
// 20: 10.2 ms against 118 ms for a launch and, past the kept tables, a host
// table per set (10.8 with the entries computed by each CTA).  One set of power
// 1 on 2048^2, sigma 10, 20 and 200 samples: 9.8 ms both, against 12.0 from a
// kept table, and 12.4 and 16.3 with entries computed by each CTA and one kernel
// for all powers; sigma 2: 0.86 against 0.88, and 1.02 and 1.27.  The window
// loop unrolled by 1, 2 and 4, that set: 11.5, 10.5 and 9.8 ms.
struct SweepSet {
    float s1, s2, eta;
    int h, power, out;        // out: position of the set's field and SIMF
    int entries;              // position of its first entry
};
constexpr int SWEEP_SETS = 128;
struct SweepArgs {
    const float4* V;
    float4* out;              // + set.out * n
    float4* entries;          // + 2 set.entries
    int s0, s1, samples;
    SweepSet set[SWEEP_SETS];
};

struct SweepEntry { float4 a, b; };   // (dx, dy, c1, c2), (Va, Vb, Vc, c2 - c1)

// x^p, p >= 1, by squaring
__device__ __forceinline__ float powi(float x, int p) {
    float r = 1.0f;
    for (; p > 1; p >>= 1) {
        if (p & 1) r *= x;
        x *= x;
    }
    return r * x;
}

__device__ __forceinline__ SweepEntry sweep_entry(const SweepSet& s, int samples, bool plate, int du, int dv) {
    SweepEntry e;
    const float x = float(du), y = float(dv), l2 = x * x + y * y;
    const float inv1 = 1.0f / (s.s1 * s.s1), inv2 = s.s2 > 0.0f ? 1.0f / (s.s2 * s.s2) : 0.0f;
    float dx = 0.0f, dy = 0.0f;
    if (l2 != 0.0f) { const float il = 1.0f / sqrtf(l2); dx = x * il; dy = y * il; }
    const float c1 = expf(-l2 * inv1), c2 = s.s2 == 0.0f ? (l2 > 1e-12f ? 0.0f : 1.0f) : expf(-l2 * inv2);
    float va = 0.0f, vb = 0.0f, vc = 0.0f;
    if (plate) {                          // tk_plate_numerical (2D), tensorvote.h:1048
        const float dth = float(3.14159265358979323846 / double(float(samples)));
        for (int i = 0; i < samples; ++i) {
            float qy, qx;
            sincosf(dth * float(i), &qy, &qx);
            const float u = qx * dx + qy * dy, q2 = u * u;
            const float f = (c1 * powi(1.0f - q2, s.power) + c2 * powi(q2, s.power)) * s.eta;
            const float rx = fmaf(-2.0f * u, dx, qx), ry = fmaf(-2.0f * u, dy, qy);
            va = fmaf(f * rx, rx, va); vb = fmaf(f * rx, ry, vb); vc = fmaf(f * ry, ry, vc);
        }
        const float wb = float(3.14159265358979323846) / float(samples);
        va *= wb; vb *= wb; vc *= wb;
    }
    e.a = make_float4(dx, dy, c1, c2);
    e.b = make_float4(va, vb, vc, c2 - c1);
    return e;
}

template <bool PLATE>
__global__ void __launch_bounds__(256) k_sweep_entries(const __grid_constant__ SweepArgs a) {
    const SweepSet& s = a.set[blockIdx.y];
    const int w = 2 * s.h + 1, i = blockIdx.x * 256 + threadIdx.x;
    if (i >= w * w) return;
    const SweepEntry e = sweep_entry(s, a.samples, PLATE, i % w - s.h, i / w - s.h);
    a.entries[2 * (size_t(s.entries) + i)] = e.a;
    a.entries[2 * (size_t(s.entries) + i) + 1] = e.b;
}

template <bool PLATE, bool P1>
__device__ __forceinline__ void sweep_body(const SweepArgs& a, const SweepSet& s, float4* smem,
                                           int stage_floats4) {
    constexpr int VR = 4, TYS = 8, NT = V2X * TYS;
    const int h = s.h, w = 2 * h + 1, TW = V2X + 2 * h;
    const int tid = threadIdx.y * V2X + threadIdx.x;
    const int x0 = blockIdx.x * V2X, y0 = blockIdx.y * (TYS * VR);
    // offset rows per band: entries (2 float4 each) and the voters of TYS VR + rows - 1 rows
    const int band = min(w, (stage_floats4 - (TYS * VR - 1) * TW) / (TW + 2 * w));
    float4* ent = smem;
    float4* tile = smem + 2 * w * band;
    float sa[VR], sb[VR], sc[VR], pa[VR], pb[VR], pc[VR];
#pragma unroll
    for (int j = 0; j < VR; ++j) sa[j] = sb[j] = sc[j] = pa[j] = pb[j] = pc[j] = 0.0f;
    for (int v0 = -h; v0 <= h; v0 += band) {
        const int nb = min(band, h - v0 + 1);
        __syncthreads();                  // the previous band is done with
        const float4* src = a.entries + 2 * (size_t(s.entries) + size_t(v0 + h) * w);
        for (int i = tid; i < 2 * nb * w; i += NT) ent[i] = __ldg(src + i);
        for (int i = tid; i < (TYS * VR + nb - 1) * TW; i += NT) {
            const int r = i / TW, c = i - r * TW;
            const int gy = y0 + v0 + r, gx = x0 - h + c;
            tile[i] = unsigned(gy) < unsigned(a.s0) && unsigned(gx) < unsigned(a.s1)
                          ? __ldg(a.V + size_t(gy) * a.s1 + gx) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        for (int dv = 0; dv < nb; ++dv) {
            const float4* vrow = tile + (int(threadIdx.y) + dv) * TW + threadIdx.x;
            const float4* erow = ent + 2 * dv * w;
#pragma unroll 4
            for (int k = 0; k < w; ++k) {
                const float4 ea = erow[2 * k], eb = erow[2 * k + 1];
                float4 v[VR];
                float u[VR], D[VR];
#pragma unroll
                for (int j = 0; j < VR; ++j) {
                    v[j] = vrow[j * TYS * TW + k];
                    u[j] = fmaf(v[j].x, ea.x, v[j].y * ea.y);
                }
                if (P1) {
#pragma unroll
                    for (int j = 0; j < VR; ++j) D[j] = fmaf(eb.w, u[j] * u[j], ea.z);
                } else {                  // both powers of the four receivers by squaring, side by side
                    float t1[VR], t2[VR], r1[VR], r2[VR];
#pragma unroll
                    for (int j = 0; j < VR; ++j) {
                        t2[j] = u[j] * u[j];
                        t1[j] = 1.0f - t2[j];
                        r1[j] = ea.z;
                        r2[j] = ea.w;
                    }
                    for (int p = s.power; p > 1; p >>= 1) {
                        if (p & 1) {
#pragma unroll
                            for (int j = 0; j < VR; ++j) { r1[j] *= t1[j]; r2[j] *= t2[j]; }
                        }
#pragma unroll
                        for (int j = 0; j < VR; ++j) { t1[j] *= t1[j]; t2[j] *= t2[j]; }
                    }
#pragma unroll
                    for (int j = 0; j < VR; ++j) D[j] = fmaf(r1[j], t1[j], r2[j] * t2[j]);
                }
#pragma unroll
                for (int j = 0; j < VR; ++j) {
                    const float k2 = -2.0f * u[j];
                    const float rx = fmaf(k2, ea.x, v[j].x), ry = fmaf(k2, ea.y, v[j].y);
                    const float f = D[j] * v[j].z, fx = f * rx;
                    sa[j] = fmaf(fx, rx, sa[j]); sb[j] = fmaf(fx, ry, sb[j]); sc[j] = fmaf(f * ry, ry, sc[j]);
                    if (PLATE) {
                        pa[j] = fmaf(v[j].w, eb.x, pa[j]);
                        pb[j] = fmaf(v[j].w, eb.y, pb[j]);
                        pc[j] = fmaf(v[j].w, eb.z, pc[j]);
                    }
                }
            }
        }
    }
    const int x = x0 + threadIdx.x;
    if (x >= a.s1) return;
    float4* out = a.out + size_t(s.out) * a.s0 * a.s1;
#pragma unroll
    for (int j = 0; j < VR; ++j) {
        const int y = y0 + threadIdx.y + TYS * j;
        if (y >= a.s0) break;
        const float va = fmaf(s.eta, sa[j], pa[j]), vb = fmaf(s.eta, sb[j], pb[j]), vc = fmaf(s.eta, sc[j], pc[j]);
        out[size_t(y) * a.s1 + x] = make_float4(va, vb, vb, vc);
    }
}

// sets first .. first + gridDim.z - 1, all of power 1 (ALL1: 3 CTAs per SM, which the powers' registers do not allow)
// or of any power
template <bool PLATE, bool ALL1>
__global__ void __launch_bounds__(V2X * 8, ALL1 ? 3 : 2) k_vote2_sweep(const __grid_constant__ SweepArgs a, int first,
                                                                      int stage_floats4) {
    extern __shared__ __align__(16) float4 sm2[];
    const SweepSet& s = a.set[first + blockIdx.z];
    if (ALL1 || s.power == 1) sweep_body<PLATE, true>(a, s, sm2, stage_floats4);
    else sweep_body<PLATE, false>(a, s, sm2, stage_floats4);
}

// float4s that a band of `rows` window rows needs; the rows that fit are taken
static size_t sweep_smem(int h, int rows) {
    return size_t(31 + rows) * (V2X + 2 * h) + 2 * (2 * size_t(h) + 1) * rows;
}
constexpr size_t SWEEP_SMEM = 200 * 1024, SWEEP_SMEM2 = 110 * 1024;   // one CTA per SM; two
constexpr size_t SWEEP_ENTRIES = size_t(8) << 20;                     // of a launch: 256 MB (one set has at most 120409)

// atv (2D, tensorvote.h:225) with atv_H (:161); out [a, b, c]
__device__ __forceinline__ void atv2_pair(float l0, float l1, float e0x, float e0y, float e1x, float e1y, float rx,
                                          float ry, float sigma, float& Va, float& Vb, float& Vc) {
    const float dist = sqrtf(rx * rx + ry * ry);
    const float c = sigma == 0.0f ? (dist > 1e-12f ? 0.0f : 1.0f) : expf(-(dist * dist) / (sigma * sigma));
    float dx = 0.0f, dy = 0.0f;
    if (dist != 0.0f) { dx = rx / dist; dy = ry / dist; }
    const float Ra = 1 - 2 * dx * dx, Rb = -2 * dx * dy, Rc = 1 - 2 * dy * dy;
    const float T1a = e1x * e1x, T1b = e1x * e1y, T1c = e1y * e1y;
    const float T0a = e0x * e0x + T1a, T0b = e0x * e0y + T1b, T0c = e0y * e0y + T1c;
    const float v0 = dx * (dx * T0a + dy * T0b) + dy * (dx * T0b + dy * T0c);
    const float v1 = dx * (dx * T1a + dy * T1b) + dy * (dx * T1b + dy * T1c);
    const float t0x = T0a * dx + T0b * dy, t0y = T0b * dx + T0c * dy;
    const float t1x = T1a * dx + T1b * dy, t1y = T1b * dx + T1c * dy;
    const float s1 = l1 - l0, i3 = 1.0f / 3.0f, i4 = 1.0f / 4.0f;
    float Ha = s1 * (T1a - i3 * (T1a * v1 + 2 * (t1x * t1x)));
    float Hb = s1 * (T1b - i3 * (T1b * v1 + 2 * (t1x * t1y)));
    float Hc = s1 * (T1c - i3 * (T1c * v1 + 2 * (t1y * t1y)));
    Ha += l0 * (T0a - i4 * (T0a * v0 + 2 * (t0x * t0x)));
    Hb += l0 * (T0b - i4 * (T0b * v0 + 2 * (t0x * t0y)));
    Hc += l0 * (T0c - i4 * (T0c * v0 + 2 * (t0y * t0y)));
    const float Ra2 = Ra * Ra, Rb2 = Rb * Rb, Rc2 = Rc * Rc, Rab = Ra * Rb, Rbc = Rb * Rc, Rac = Ra * Rc;
    Va = c * (Ra2 * Ha + 2 * Rab * Hb + Rb2 * Hc);
    Vb = c * (Rb2 * Hb + Rab * Ha + Rac * Hb + Rbc * Hc);
    Vc = c * (Rb2 * Ha + 2 * Rbc * Hb + Rc2 * Hc);
}

__global__ void __launch_bounds__(V2X * V2Y) k_vote2_atv(const float4* __restrict__ V, const float4* __restrict__ W,
                                                          int s0, int s1, int hw, float sigma, float4* __restrict__ out) {
    const int x = blockIdx.x * V2X + threadIdx.x, y = blockIdx.y * V2Y + threadIdx.y;
    if (x >= s1 || y >= s0) return;
    float oa = 0, ob = 0, oc = 0;
    for (int v = -hw; v <= hw; ++v) {
        const int r0 = y + v;
        if (r0 < 0 || r0 >= s0) continue;
        for (int u = -hw; u <= hw; ++u) {
            const int r1 = x + u;
            if (r1 < 0 || r1 >= s1) continue;
            const size_t i = size_t(r0) * s1 + r1;
            const float4 a = __ldg(V + i), b = __ldg(W + i);
            float va, vb, vc;
            atv2_pair(a.w, b.x, b.y, b.z, a.x, a.y, float(u), float(v), sigma, va, vb, vc);
            oa += va; ob += vb; oc += vc;
        }
    }
    out[size_t(y) * s1 + x] = make_float4(oa, ob, ob, oc);
}

// Tables the library builds itself stay on the device, one per (device,
// window, sigmas, power, samples, terms), so a repeated vote neither copies
// nor waits for its table.  At most kTableCache tables are kept (a parameter
// sweep beyond that builds and uploads the extra ones per call).
struct TableEntry {
    int dev, w, power, samples, stick, plate, nbc, h;
    float s1, s2;
    Nb2* table;
};
constexpr int kTableCache = 128;
static std::mutex g_tab_mu;
static std::vector<TableEntry> g_tabs;

static int cached_table(int w, float s1, float s2, unsigned power, unsigned samples, bool stick, bool plate,
                        const TableEntry*& hit) {
    hit = nullptr;
    int dev = 0;
    TVGB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(g_tab_mu);
    for (const TableEntry& e : g_tabs)
        if (e.dev == dev && e.w == w && e.s1 == s1 && e.s2 == s2 && e.power == int(power) &&
            e.samples == int(samples) && e.stick == int(stick) && e.plate == int(plate)) {
            hit = &e;
            return TVGB_OK;
        }
    if (int(g_tabs.size()) >= kTableCache) return TVGB_OK;
    std::vector<Nb2> t(size_t(w) * w);
    const int nbc = build_table(w, s1, s2, power, samples, stick, plate, t.data());
    int h = 0;
    for (int i = 0; i < nbc; ++i) h = std::max(h, std::max(std::abs(t[i].du), std::abs(t[i].dv)));
    Nb2* d = nullptr;
    if (nbc > 0) {
        TVGB_CUDA(cudaMalloc(&d, size_t(nbc) * sizeof(Nb2)));
        const cudaError_t e = cudaMemcpy(d, t.data(), size_t(nbc) * sizeof(Nb2), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaFree(d);
            set_error("table upload failed: %s", cudaGetErrorString(e));
            return TVGB_ERR_CUDA;
        }
    }
    g_tabs.reserve(kTableCache);   // entries never move: hit stays valid
    g_tabs.push_back(TableEntry{dev, w, int(power), int(samples), int(stick), int(plate), nbc, h, s1, s2, d});
    hit = &g_tabs.back();
    return TVGB_OK;
}

// One TK vote of prepared voter records V (k_prep2) into out: the
// Neighbor2D table is the caller's (host or device) or the library's own
// (cached on the device); the staged kernel runs whenever the table's extent
// is known and its voter tile fits in shared memory.
static int vote2_tk_launch(const float4* V, const Nb2* host_or_dev_nb, int nbc, float s1, float s2, int power,
                           unsigned w, unsigned S0, unsigned S1, bool stick, bool plate, unsigned samples, float4* out,
                           cudaStream_t st) {
    const bool use_plate = plate && samples > 0;
    std::vector<Nb2> table;
    const Nb2* nbp = host_or_dev_nb;
    const TableEntry* cached = nullptr;
    if (!nbp) {
        TVGB_TRY(cached_table(int(w), s1, s2, unsigned(power), samples, stick, use_plate, cached));
        if (cached) {
            nbp = cached->table;
            nbc = cached->nbc;
        } else {
            table.resize(size_t(w) * w);
            nbc = build_table(int(w), s1, s2, unsigned(power), samples, stick, use_plate, table.data());
            nbp = table.data();
        }
    }
    DevArray dnb;
    TVGB_TRY(dnb.in(nbp, size_t(nbc) * sizeof(Nb2), st));
    const unsigned p = power < 1 ? 1u : unsigned(power);
    const float eta_s = stick_norm_2d_h(s1, s2, p);
    int h = -1;
    if (cached) {
        h = cached->h;
    } else if (!is_device_ptr(nbp)) {
        h = 0;
        for (int i = 0; i < nbc; ++i) h = std::max(h, std::max(std::abs(nbp[i].du), std::abs(nbp[i].dv)));
    }
    // staged kernel: 4 receivers per thread (each table entry serves 4), 32 x 8 threads per CTA
    constexpr int V2R = 4, TY = 8, V2NBC = 128;
    const size_t hh = size_t(h < 0 ? 0 : h);
    const size_t smem_s = V2NBC * sizeof(Nb2) + (V2X + 2 * hh) * (size_t(TY) * V2R + 2 * hh) * sizeof(float4);
    dim3 grid(ceil_div(S1, V2X), ceil_div(S0, V2Y)), blk(V2X, V2Y);
    {
        KernelTimer kt_("k_vote2_tk", st);
        if (h >= 0 && smem_s <= 200 * 1024) {
            const void* fn = nullptr;
            if (stick && use_plate) fn = p == 1 ? (const void*)k_vote2_tks<V2R, TY, V2NBC, true, true, true>
                                                : (const void*)k_vote2_tks<V2R, TY, V2NBC, true, true, false>;
            else if (stick) fn = p == 1 ? (const void*)k_vote2_tks<V2R, TY, V2NBC, true, false, true>
                                        : (const void*)k_vote2_tks<V2R, TY, V2NBC, true, false, false>;
            else fn = (const void*)k_vote2_tks<V2R, TY, V2NBC, false, true, true>;
            TVGB_CUDA(allow_smem(fn, smem_s));
            dim3 gs(ceil_div(S1, V2X), ceil_div(S0, unsigned(TY * V2R))), bs(V2X, TY);
            const float4* vp = V;
            const Nb2* tp = dnb.get<Nb2>();
            int nbc_ = nbc, s0_ = int(S0), s1_ = int(S1), h_ = h;
            float eta_ = eta_s;
            unsigned p_ = p;
            float4* op = out;
            void* args[] = {&vp, &tp, &nbc_, &s0_, &s1_, &h_, &eta_, &p_, &op};
            TVGB_CUDA(cudaLaunchKernel(fn, gs, bs, args, smem_s, st));
        } else if (stick && use_plate) {
            k_vote2_tk<true, true><<<grid, blk, 0, st>>>(V, dnb.get<Nb2>(), nbc, int(S0), int(S1), eta_s, p, out);
        } else if (stick) {
            k_vote2_tk<true, false><<<grid, blk, 0, st>>>(V, dnb.get<Nb2>(), nbc, int(S0), int(S1), eta_s, p, out);
        } else {
            k_vote2_tk<false, true><<<grid, blk, 0, st>>>(V, dnb.get<Nb2>(), nbc, int(S0), int(S1), eta_s, p, out);
        }
        kt_.stop();
    }
    TVGB_LAUNCHED();
    if (!host_or_dev_nb && !cached) TVGB_CUDA(cudaStreamSynchronize(st));   // the host table must outlive its copy
    return TVGB_OK;
}

static int vote2_impl(float* t_out, const float* t_in, const Nb2* host_or_dev_nb, int nbc, float s1, float s2,
                      int power, unsigned w, unsigned S0, unsigned S1, bool stick, bool plate, unsigned samples,
                      bool is_atv, cudaStream_t st) {
    const size_t n = size_t(S0) * S1;
    DevArray din, dout;
    TVGB_TRY(din.in(t_in, n * 16, st));
    TVGB_TRY(dout.out(t_out, n * 16, st));
    TVGB_CHECK_ARG(reinterpret_cast<uintptr_t>(din.dev) % 16 == 0 && reinterpret_cast<uintptr_t>(dout.dev) % 16 == 0,
                   "2D tensor fields must be 16-byte aligned");
    if (!is_atv && !stick && !plate) {      // global_tensorvote_tk writes zeros (:2079-2085)
        TVGB_CUDA(cudaMemsetAsync(dout.dev, 0, n * 16, st));
        TVGB_TRY(dout.finish());
        return sync_if(din.owned || dout.owned, st);
    }
    Scratch sv, sw;
    TVGB_TRY(sv.alloc(n * 16, st));
    if (is_atv) TVGB_TRY(sw.alloc(n * 16, st));
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    size_t blocks = (n + 255) / 256;
    if (blocks > size_t(sms) * 16) blocks = size_t(sms) * 16;
    {
        KernelTimer kt_("k_prep2", st);
        k_prep2<<<unsigned(blocks ? blocks : 1), 256, 0, st>>>(din.get<float4>(), n, sv.get<float4>(),
                                                              is_atv ? sw.get<float4>() : nullptr);
        kt_.stop();
    }
    TVGB_LAUNCHED();
    dim3 grid(ceil_div(S1, V2X), ceil_div(S0, V2Y)), blk(V2X, V2Y);
    if (is_atv) {
        {
            KernelTimer kt_("k_vote2_atv", st);
            k_vote2_atv<<<grid, blk, 0, st>>>(sv.get<float4>(), sw.get<float4>(), int(S0), int(S1), int(w / 2), s1,
                                              dout.get<float4>());
            kt_.stop();
        }
        TVGB_LAUNCHED();
    } else {
        TVGB_TRY(vote2_tk_launch(sv.get<float4>(), host_or_dev_nb, nbc, s1, s2, power, w, S0, S1, stick, plate, samples,
                                 dout.get<float4>(), st));
    }
    TVGB_TRY(dout.finish());
    return sync_if(din.owned || dout.owned, st);
}

}  // namespace tvgb

using namespace tvgb;

extern "C" {

int tvgb_build_neighbors2d(int w, float sigma1, float sigma2, unsigned power, unsigned samples, int stick, int plate,
                           void* out, int* count) {
    TVGB_CHECK_ARG(count, "tvgb_build_neighbors2d: count is NULL");
    TVGB_CHECK_ARG(w >= 0, "tvgb_build_neighbors2d: w must be >= 0");
    *count = build_table(w, sigma1, sigma2, power, samples, stick != 0, plate != 0, static_cast<Nb2*>(out));
    return TVGB_OK;
}

static int check2(const float* t_out, const float* t_in, float s1, unsigned w, const char* fn) {
    TVGB_CHECK_ARG(t_out && t_in, "%s: NULL field pointer", fn);
    TVGB_CHECK_ARG(s1 > 0.0f, "%s: sigma1 must be > 0", fn);
    TVGB_CHECK_ARG(w >= 1 && (w % 2) == 1, "%s: window w must be a positive odd integer (got %u)", fn, w);
    TVGB_CHECK_ARG(w <= 1025, "%s: window w = %u too large", fn, w);
    return TVGB_OK;
}

int tvgb_tensorvote(float* t_out, const float* t_in, float sigma1, float sigma2, int power, unsigned w, unsigned shape0,
                    unsigned shape1, int stick, int plate, unsigned samples, int is_atv, void* stream) {
    TVGB_TRY(check2(t_out, t_in, sigma1, w, "tvgb_tensorvote"));
    if (size_t(shape0) * shape1 == 0) return TVGB_OK;
    return vote2_impl(t_out, t_in, nullptr, 0, sigma1, sigma2, power, w, shape0, shape1, stick != 0, plate != 0,
                      samples, is_atv != 0, as_stream(stream));
}

int tvgb_tensorvote_prebuilt(float* t_out, const float* t_in, const void* host_nb, int nb_count, float sigma1,
                             float sigma2, int power, unsigned w, unsigned shape0, unsigned shape1, int stick, int plate,
                             unsigned samples, void* stream) {
    TVGB_TRY(check2(t_out, t_in, sigma1, w, "tvgb_tensorvote_prebuilt"));
    TVGB_CHECK_ARG(nb_count >= 0 && (nb_count == 0 || host_nb), "tvgb_tensorvote_prebuilt: bad neighbour table");
    if (size_t(shape0) * shape1 == 0) return TVGB_OK;
    if (nb_count == 0) {   // nothing to vote with: zeros, like a kernel with nb_count = 0
        const size_t n = size_t(shape0) * shape1;
        cudaStream_t st = as_stream(stream);
        DevArray dout;
        TVGB_TRY(dout.out(t_out, n * 16, st, true));
        TVGB_TRY(dout.finish());
        return sync_if(dout.owned, st);
    }
    return vote2_impl(t_out, t_in, static_cast<const Nb2*>(host_nb), nb_count, sigma1, sigma2, power, w, shape0, shape1,
                      stick != 0, plate != 0, samples, false, as_stream(stream));
}

// Parameter sweep of the TK vote (the objective evaluations of tiralib's
// optimize_tk, python/tira/tensors_lib/optimize.py:256-279): K parameter
// sets (sigma1, sigma2, power) against one input field and one target field
// G.  The input is solved once; the sets, each with its window
// (optimize.py:_w_from_sigma), are voted in one launch (k_vote2_sweep) and
// scored in two, by the SIMF of G against the voted field (metrics.py:37).  simf[k] receives it; t_out, if
// given, receives the K voted fields.
int tvgb_tensorvote_sweep(const float* t_in, const float* G, unsigned shape0, unsigned shape1, const double* params,
                          int K, unsigned samples, int plate, double* simf, float* t_out, void* stream) {
    TVGB_CHECK_ARG(t_in && G && params && simf, "tvgb_tensorvote_sweep: NULL pointer");
    TVGB_CHECK_ARG(K >= 0, "tvgb_tensorvote_sweep: K must be >= 0");
    for (int k = 0; k < K; ++k) {
        TVGB_CHECK_ARG(params[3 * k] > 0.0 && params[3 * k + 1] >= 0.0 && params[3 * k + 2] >= 1.0 &&
                           params[3 * k] < 1e4 && params[3 * k + 1] < 1e4 && params[3 * k + 2] < 1e4,
                       "tvgb_tensorvote_sweep: parameter set %d out of range", k);
    }
    const size_t n = size_t(shape0) * shape1;
    if (K == 0) return TVGB_OK;
    if (n == 0) { for (int k = 0; k < K; ++k) simf[k] = 0.0; return TVGB_OK; }
    cudaStream_t st = as_stream(stream);
    DevArray din, dG, dout;
    TVGB_TRY(din.in(t_in, n * 16, st));
    TVGB_TRY(dG.in(G, n * 16, st));
    if (t_out) TVGB_TRY(dout.out(t_out, size_t(K) * n * 16, st));
    TVGB_CHECK_ARG(reinterpret_cast<uintptr_t>(din.dev) % 16 == 0 && reinterpret_cast<uintptr_t>(dG.dev) % 16 == 0 &&
                       reinterpret_cast<uintptr_t>(dout.dev) % 16 == 0,
                   "tvgb_tensorvote_sweep: fields must be 16-byte aligned");
    Scratch sv, sacc;
    TVGB_TRY(sv.alloc(n * 16, st));
    TVGB_TRY(sacc.alloc(size_t(K) * 3 * sizeof(double), st));
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    size_t blocks = (n + 255) / 256;
    if (blocks > size_t(sms) * 16) blocks = size_t(sms) * 16;
    {
        KernelTimer kt_("k_prep2", st);
        k_prep2<<<unsigned(blocks ? blocks : 1), 256, 0, st>>>(din.get<float4>(), n, sv.get<float4>(), nullptr);
        kt_.stop();
    }
    TVGB_LAUNCHED();
    std::vector<SweepSet> sets(K);
    for (int k = 0; k < K; ++k) {
        const double s1d = params[3 * k], s2d = params[3 * k + 1];
        const int pw = std::max(1, int(params[3 * k + 2]));
        const double sm = std::max(s1d, s2d);
        int w = 2 * int(3.0 * sm) + 1;        // optimize.py:9-15
        if (w < 3) w = 3;
        if (w % 2 == 0) w += 1;
        sets[k] = SweepSet{float(s1d), float(s2d), stick_norm_2d_h(float(s1d), float(s2d), unsigned(pw)), w / 2, pw, k, 0};
    }
    // widest windows first: they are the longest CTAs
    std::stable_sort(sets.begin(), sets.end(), [](const SweepSet& a, const SweepSet& b) { return a.h > b.h; });
    std::vector<int> row(K);                  // set k's SIMF sums
    const bool use_plate = plate != 0 && samples > 0;
    auto entries_of = [](const SweepSet& s) {  // of a set whose window is staged; 0: too wide
        const size_t w = 2 * size_t(s.h) + 1;
        return sweep_smem(s.h, 1) * sizeof(float4) <= SWEEP_SMEM ? w * w : size_t(0);
    };
    // sets and entries per launch: fields that the caller does not take within 1 GiB, and less of both, down to a set's,
    // where the device has no more
    size_t widest = 0, share = 0;
    for (const SweepSet& s : sets) {
        widest = std::max(widest, entries_of(s));
        share = std::min(share + entries_of(s), SWEEP_ENTRIES);
    }
    int per = std::min(K, SWEEP_SETS);
    if (!t_out) per = int(std::max<size_t>(1, std::min<size_t>(per, (size_t(1) << 30) / (n * 16))));
    Scratch sb, se;
    for (;; per = (per + 1) / 2, share = std::max(widest, share / 2)) {
        int rc = t_out ? TVGB_OK : sb.alloc(size_t(per) * n * 16, st);
        if (rc == TVGB_OK) rc = se.alloc(share * sizeof(SweepEntry), st);
        if (rc == TVGB_OK) break;
        sb.release();
        if (rc != TVGB_ERR_NOMEM || (per == 1 && share == widest)) return rc;
        cudaGetLastError();
    }
    float4* fields = t_out ? dout.get<float4>() : sb.get<float4>();
    for (int k0 = 0, m = 0; k0 < K; k0 += m) {
        SweepArgs a{};
        a.V = sv.get<float4>(); a.out = fields; a.entries = se.get<float4>(); a.s0 = int(shape0); a.s1 = int(shape1); a.samples = int(samples);
        int staged = 0;
        size_t entries = 0;
        for (m = 0; m < per && k0 + m < K; ++m) {
            SweepSet s = sets[k0 + m];
            const size_t ne = entries_of(s);
            if (entries + ne > share) break;
            row[s.out] = t_out ? s.out : k0 + m;
            if (!t_out) s.out = m;
            if (ne) {
                s.entries = int(entries);
                entries += ne;
                a.set[staged++] = s;
            } else {                          // a window too wide to stage: a vote by itself, from a table
                TVGB_TRY(vote2_tk_launch(sv.get<float4>(), nullptr, 0, s.s1, s.s2, s.power, unsigned(2 * s.h + 1), shape0,
                                         shape1, true, plate != 0, samples, fields + size_t(s.out) * n, st));
            }
        }
        if (staged > 0) {
            const int wmax = 2 * a.set[0].h + 1;
            // a set that fills the SMs by itself votes with those of its kind: power 1, or above
            const unsigned gx = ceil_div(shape1, V2X), gy = ceil_div(shape0, 32u);
            const auto one = [](const SweepSet& s) { return s.power == 1; };
            int ones = int(std::count_if(a.set, a.set + staged, one));
            if (size_t(gx) * gy >= 304) std::stable_partition(a.set, a.set + staged, one);
            else if (ones < staged) ones = 0;
            {
                KernelTimer kt_("k_sweep_entries", st);
                auto tab = use_plate ? k_sweep_entries<true> : k_sweep_entries<false>;
                tab<<<dim3(ceil_div(size_t(wmax) * wmax, 256u), unsigned(staged)), 256, 0, st>>>(a);
                kt_.stop();
            }
            TVGB_LAUNCHED();
            auto vote = [&](int first, int count, auto kern) -> int {
                if (count == 0) return TVGB_OK;
                // what the widest set's window takes whole, or two CTAs per SM where that holds an offset row of it
                const int h = a.set[first].h;
                size_t smem = sweep_smem(h, 2 * h + 1) * sizeof(float4);
                if (smem > SWEEP_SMEM2) smem = sweep_smem(h, 1) * sizeof(float4) <= SWEEP_SMEM2 ? SWEEP_SMEM2 : SWEEP_SMEM;
                TVGB_CUDA(allow_smem(kern, smem));
                {
                    KernelTimer kt_("k_vote2_sweep", st);
                    kern<<<dim3(gx, gy, unsigned(count)), dim3(V2X, 8), smem, st>>>(a, first, int(smem / sizeof(float4)));
                    kt_.stop();
                }
                TVGB_LAUNCHED();
                return TVGB_OK;
            };
            TVGB_TRY(vote(0, ones, use_plate ? k_vote2_sweep<true, true> : k_vote2_sweep<false, true>));
            TVGB_TRY(vote(ones, staged - ones, use_plate ? k_vote2_sweep<true, false> : k_vote2_sweep<false, false>));
        }
        if (!t_out) TVGB_TRY(simf2_device(dG.get<float4>(), fields, n, m, sacc.get<double>() + 3 * size_t(k0), st));
    }
    if (t_out) TVGB_TRY(simf2_device(dG.get<float4>(), fields, n, K, sacc.get<double>(), st));
    std::vector<double> acc(size_t(K) * 3);
    TVGB_CUDA(cudaMemcpyAsync(acc.data(), sacc.get<double>(), acc.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    TVGB_TRY(dout.finish());
    TVGB_CUDA(cudaStreamSynchronize(st));
    for (int k = 0; k < K; ++k) simf[k] = acc[3 * size_t(row[k]) + 2] / double(n);
    return TVGB_OK;
}

}  // extern "C"
