// The 3D TK vote with power p > 1 and an exact plate (samples 0 or >= p + 2),
// stick, plate and ball, in closed form per pair (reference: the pair rules of
// tira/functions/tensorvote.h:1184, :2457 with their powers).
//
// At offset o = |o| d, with f(u) = c1 (1 - u^2)^p + c2 u^2p, R = I - 2 d d^T:
//   stick  f(q.d) (R q)(R q)^T
//   plate  the mean of sticks over the circle normal to n.  With y = (n.d)^2,
//          x = 1 - y, the part of d in the circle's plane p = d - (n.d) n,
//          m = R n and the means W(i, k) of cos^2i sin^2k over the circle:
//            B (I - m m^T) + D (R p)(R p)^T,
//            B = c1 sum_j C(p,j) W(j, p-j+1) y^j + c2 W(p, 1) x^p
//            D = c1 sum_j e_j y^j + c2 (W(p+1, 0) - W(p, 1)) x^(p-1),
//          e_j the sums up to j of C(p,i) (W(i+1, p-i) - W(i, p-i+1)): the
//          (1 - u^2)^p = (sin^2 + y cos^2)^p of the circle's u^2 = x cos^2,
//          divided by x.  All terms of a sum have one sign, so the sums lose
//          nothing to cancellation at any p.
//   ball   the mean over the sphere: a I + b d d^T with a, b linear in c1, c2.
// 40 x 48 x 56, sigma 2, p = 3: 0.8 ms against 6.6 ms for one receiver per
// thread with expf, sqrtf and p + 2 = 5 sticks with sincosf per pair.
#include "vote3_pow.cuh"
#include <algorithm>
#include <cmath>

namespace tvgb {

constexpr int PX = 32, PY = 8;             // receivers per CTA: one per thread
constexpr int POW_MAX = 32;

struct PowArgs {
    FastArgs f;
    int power;
    float b1[POW_MAX + 1], d1[POW_MAX + 1];   // B's and D's coefficients of y^j for c1
    float b2, d2;                             // of x^p and x^(p-1) for c2
    float ball_a1, ball_a2, ball_b1, ball_b2; // ball: I and d d^T, for c1 and c2
    float ball_0;                             // at the voter itself (c1 = 1, d = 0)
};

// table entry for integer |o|^2 = L2: (c1, c2, g = 1 / |o|^2, y at n.o = 0: 0, or 1 at the voter itself)
__device__ __forceinline__ float4 pow_entry(int L2, float s1, float s2) {
    const float l2 = float(L2);
    const float inv1 = s1 > 0.0f ? 1.0f / (s1 * s1) : 0.0f, inv2 = s2 > 0.0f ? 1.0f / (s2 * s2) : 0.0f;
    const float c1 = s1 == 0.0f ? (l2 > 1e-12f ? 0.0f : 1.0f) : expf(-l2 * inv1);
    const float c2 = s2 == 0.0f ? (l2 > 1e-12f ? 0.0f : 1.0f) : expf(-l2 * inv2);
    return make_float4(c1, c2, L2 > 0 ? 1.0f / l2 : 0.0f, L2 > 0 ? 0.0f : 1.0f);
}

// POW: the power, 0 for any
template <int POW, bool STICK, bool PLATE, bool BALL>
__device__ __forceinline__ void pow_pair(const PowArgs& a, const float4& A, const float4& B, float lb, float ox,
                                         float oy, float oz, const float4& t, float (&P)[7]) {
    const int p = POW ? POW : a.power;
    if (STICK) {
        const float u = fmaf(A.x, ox, fmaf(A.y, oy, A.z * oz));
        const float k = u * t.z;
        const float rx = fmaf(-2.0f * k, ox, A.x), ry = fmaf(-2.0f * k, oy, A.y), rz = fmaf(-2.0f * k, oz, A.z);
        const float t2 = u * k, t1 = 1.0f - t2;
        float e1 = t1, e2 = t2;
#pragma unroll
        for (int i = 1; i < p; ++i) { e1 *= t1; e2 *= t2; }
        const float term = A.w * fmaf(t.x, e1, t.y * e2);
        const float t0 = term * rx, tt1 = term * ry, tt2 = term * rz;
        P[0] = fmaf(t0, rx, P[0]); P[1] = fmaf(t0, ry, P[1]); P[2] = fmaf(t0, rz, P[2]);
        P[3] = fmaf(tt1, ry, P[3]); P[4] = fmaf(tt1, rz, P[4]); P[5] = fmaf(tt2, rz, P[5]);
    }
    if (PLATE) {
        const float v = fmaf(B.x, ox, fmaf(B.y, oy, B.z * oz));
        const float k = v * t.z;
        const float mx = fmaf(-2.0f * k, ox, B.x), my = fmaf(-2.0f * k, oy, B.y), mz = fmaf(-2.0f * k, oz, B.z);
        const float hx = fmaf(v, mx, ox), hy = fmaf(v, my, oy), hz = fmaf(v, mz, oz);   // h = -|o| R p
        const float y = fmaf(v, k, t.w), x = 1.0f - y;
        float b = a.b1[p], d = a.d1[p - 1], xp = 1.0f;
#pragma unroll
        for (int j = p - 1; j >= 0; --j) b = fmaf(b, y, a.b1[j]);
#pragma unroll
        for (int j = p - 2; j >= 0; --j) d = fmaf(d, y, a.d1[j]);
#pragma unroll
        for (int j = 1; j < p; ++j) xp *= x;
        const float c2x = t.y * xp;                                        // c2 x^(p-1)
        const float sA = B.w * fmaf(t.x, b, a.b2 * c2x * x), sB = B.w * t.z * fmaf(t.x, d, a.d2 * c2x);
        P[6] += sA;
        const float ax = sA * mx, ay = sA * my, az = sA * mz, bx = sB * hx, by = sB * hy, bz = sB * hz;
        P[0] = fmaf(bx, hx, fmaf(-ax, mx, P[0])); P[1] = fmaf(bx, hy, fmaf(-ax, my, P[1]));
        P[2] = fmaf(bx, hz, fmaf(-ax, mz, P[2])); P[3] = fmaf(by, hy, fmaf(-ay, my, P[3]));
        P[4] = fmaf(by, hz, fmaf(-ay, mz, P[4])); P[5] = fmaf(bz, hz, fmaf(-az, mz, P[5]));
    }
    if (BALL) {
        P[6] = fmaf(lb, fmaf(t.x, a.ball_a1, t.y * a.ball_a2) + t.w * a.ball_0, P[6]);
        const float wb = lb * t.z * fmaf(t.x, a.ball_b1, t.y * a.ball_b2);
        const float wx = wb * ox, wy = wb * oy, wz = wb * oz;
        P[0] = fmaf(wx, ox, P[0]); P[1] = fmaf(wx, oy, P[1]); P[2] = fmaf(wx, oz, P[2]);
        P[3] = fmaf(wy, oy, P[3]); P[4] = fmaf(wy, oz, P[4]); P[5] = fmaf(wz, oz, P[5]);
    }
}

// One receiver per thread: the windows are small here (the pairs' arithmetic,
// not the voters' loads, bounds the kernel), and small fields get CTAs for
// every SM.  Voter rows with their halo are staged in shared memory as many at
// a time as fit; sums run over a voter plane before they join the receiver's.
template <int POW, bool STICK, bool PLATE, bool BALL>
__global__ void __launch_bounds__(PX * PY) k_vote3_pow(const __grid_constant__ PowArgs a) {
    extern __shared__ __align__(16) float4 smem[];
    const FastArgs& f = a.f;
    const int hw = f.hw, nt = 3 * hw * hw + 1, SW = PX + 2 * hw, SR = PY + f.rows - 1;
    float4* tbl = smem;
    float4* sA = tbl + nt;
    float4* sB = sA + (STICK ? SR * SW : 0);
    float* sC = reinterpret_cast<float*>(sB + (PLATE ? SR * SW : 0));
    const int tid = threadIdx.y * PX + threadIdx.x;
    for (int L2 = tid; L2 < nt; L2 += PX * PY) tbl[L2] = pow_entry(L2, f.sig1, f.sig2);
    const int x0 = blockIdx.x * PX, y0 = blockIdx.y * PY, z = blockIdx.z;
    const size_t plane = size_t(f.s1) * f.s2;
    float tot[6] = {0, 0, 0, 0, 0, 0};
    for (int vz = max(0, z - hw); vz <= min(f.s0 - 1, z + hw); ++vz) {
        const int oz = vz - z;
        float P[7] = {0, 0, 0, 0, 0, 0, 0};
        for (int oy0 = -hw; oy0 <= hw; oy0 += f.rows) {
            const int oy1 = min(hw, oy0 + f.rows - 1);
            __syncthreads();
            for (int e = tid; e < (PY + oy1 - oy0) * SW; e += PX * PY) {
                const int r = e / SW, c = e - r * SW;
                const int gy = y0 + oy0 + r, gx = x0 - hw + c;
                const bool in = unsigned(gy) < unsigned(f.s1) && unsigned(gx) < unsigned(f.s2);
                const size_t gi = size_t(vz) * plane + size_t(gy) * f.s2 + gx;
                if (STICK) sA[e] = in ? __ldg(f.A + gi) : make_float4(0, 0, 0, 0);
                if (PLATE) sB[e] = in ? __ldg(f.B + gi) : make_float4(0, 0, 0, 0);
                if (BALL) sC[e] = in ? __ldg(f.C + gi) : 0.0f;
            }
            __syncthreads();
            for (int oy = oy0; oy <= oy1; ++oy) {
                if (unsigned(y0 + int(threadIdx.y) + oy) >= unsigned(f.s1)) continue;   // warp-uniform
                const int base = (int(threadIdx.y) + oy - oy0) * SW + int(threadIdx.x) + hw;
                const int Lyz = oy * oy + oz * oz;
                const float4 Z4 = make_float4(0, 0, 0, 0);
                const float oyf = float(oy), ozf = float(oz);
                for (int ox = -hw; ox <= hw; ++ox)
                    pow_pair<POW, STICK, PLATE, BALL>(a, STICK ? sA[base + ox] : Z4, PLATE ? sB[base + ox] : Z4,
                                                      BALL ? sC[base + ox] : 0.0f, float(ox), oyf, ozf,
                                                      tbl[Lyz + ox * ox], P);
            }
        }
        tot[0] += P[0] + P[6]; tot[1] += P[1]; tot[2] += P[2];
        tot[3] += P[3] + P[6]; tot[4] += P[4]; tot[5] += P[5] + P[6];
    }
    const int x = x0 + threadIdx.x, y = y0 + threadIdx.y;
    if (x < f.s2 && y < f.s1)
        write_receiver(f, size_t(z) * plane + size_t(y) * f.s2 + x, size_t(f.s0) * plane, tot);
}

static size_t pow_smem(int hw, int rows, bool S, bool P, bool B) {
    return (size_t(3) * hw * hw + 1) * 16 + size_t(PY + rows - 1) * (PX + 2 * hw) * ((S ? 16 : 0) + (P ? 16 : 0) + (B ? 4 : 0));
}

bool vote3_pow_fits(int hw, bool S, bool P, bool B) { return pow_smem(hw, 1, S, P, B) <= 200 * 1024; }

// mean over the circle of cos^2i sin^2k: (2i-1)!! (2k-1)!! / (2i+2k)!!
static double circle_mean(int i, int k) {
    double v = 1.0;
    for (int j = 1; j <= i; ++j) v *= (2.0 * j - 1.0) / (2.0 * j);
    for (int j = 1; j <= k; ++j) v *= (2.0 * j - 1.0) / (2.0 * (i + j));
    return v;
}

int vote3_pow_launch(FastArgs f, unsigned power, bool S, bool P, bool B, cudaStream_t st) {
    PowArgs a{};
    const int p = int(power);
    a.power = p;
    double c = 1.0, e = 0.0;                               // C(p, j), the running sum e_j
    for (int j = 0; j <= p; ++j) {
        a.b1[j] = float(c * circle_mean(j, p - j + 1));
        e += c * (circle_mean(j + 1, p - j) - circle_mean(j, p - j + 1));
        a.d1[j] = j < p ? float(e) : 0.0f;
        c = c * (p - j) / (j + 1);
    }
    a.b2 = float(circle_mean(p, 1));
    a.d2 = float(circle_mean(p + 1, 0) - circle_mean(p, 1));
    // ball: u uniform on [-1, 1]; d d^T gets the mean of f u^2, I - d d^T that of f (1 - u^2) / 2
    double q = 1.0;                                        // mean of (1 - u^2)^p
    for (int j = 1; j <= p; ++j) q *= 2.0 * j / (2.0 * j + 1.0);
    const double q1 = q * (2.0 * p + 2.0) / (2.0 * p + 3.0);   // of (1 - u^2)^(p+1)
    const double u0 = 1.0 / (2.0 * p + 1.0), u1 = 1.0 / (2.0 * p + 3.0);
    a.ball_a1 = float(0.5 * q1);
    a.ball_b1 = float((q - q1) - 0.5 * q1);
    a.ball_a2 = float(0.5 * (u0 - u1));
    a.ball_b2 = float(u1 - 0.5 * (u0 - u1));
    a.ball_0 = float(1.0 / 3.0 - 0.5 * q1 - 0.5 * (u0 - u1));  // d = 0 (c1 = c2 = 1): every stick votes q q^T, mean I / 3
    int rows = 2 * f.hw + 1;                               // at most 75 KB, for three CTAs per SM, where that holds a row
    while (rows > 1 && pow_smem(f.hw, rows, S, P, B) > 75 * 1024) rows = (rows + 1) / 2;
    f.rows = rows;
    a.f = f;
    const size_t smem = pow_smem(f.hw, rows, S, P, B);
    const dim3 grid(ceil_div(f.s2, PX), ceil_div(f.s1, PY), f.s0), block(PX, PY);
    auto run = [&](auto kern) -> int {
        TVGB_CUDA(allow_smem(kern, smem));
        {
            KernelTimer kt_("k_vote3_pow", st);
            kern<<<grid, block, smem, st>>>(a);
            kt_.stop();
        }
        TVGB_LAUNCHED();
        return TVGB_OK;
    };
    // powers 2 and 3 unrolled; the rest, and votes with the ball, by the loops
    if (B) {
        if (S && P) return run(k_vote3_pow<0, true, true, true>);
        if (S) return run(k_vote3_pow<0, true, false, true>);
        if (P) return run(k_vote3_pow<0, false, true, true>);
        return run(k_vote3_pow<0, false, false, true>);
    }
    if (S && P) return p == 2 ? run(k_vote3_pow<2, true, true, false>) : p == 3 ? run(k_vote3_pow<3, true, true, false>)
                                                                                : run(k_vote3_pow<0, true, true, false>);
    if (S) return p == 2 ? run(k_vote3_pow<2, true, false, false>) : p == 3 ? run(k_vote3_pow<3, true, false, false>)
                                                                            : run(k_vote3_pow<0, true, false, false>);
    if (P) return p == 2 ? run(k_vote3_pow<2, false, true, false>) : p == 3 ? run(k_vote3_pow<3, false, true, false>)
                                                                            : run(k_vote3_pow<0, false, true, false>);
    return TVGB_OK;
}

}  // namespace tvgb
