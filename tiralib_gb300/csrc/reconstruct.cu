// Consumers of a voted 2D field on sm_103a: stick saliency, Otsu's
// threshold, saliency thresholding with optional closing + hole filling, and
// the scale-invariant mean Frobenius distance (SIMF) used as the objective
// of tiralib's parameter sweeps.
//
// Reference (python/tira/tensors_lib):
//   reconstruct.py:14  stick_saliency      |lambda|max - |lambda|min per pixel
//   reconstruct.py:34  _otsu_threshold     256-bin histogram over [0, max], between-class variance
//   reconstruct.py:66  saliency_threshold  s > thr, optionally binary_closing + binary_fill_holes
//   metrics.py:37      simf                mean || A - alpha B ||_F, alpha = <A,B> / <B,B>
// Fields are (H, W) pixels of [a, b, b, c] (float4), as the 2D vote writes them.
#include "tvgb_internal.cuh"
#include <algorithm>
#include <cmath>

namespace tvgb {

// |lambda|max - |lambda|min of [[a, b], [b, c]]: with d = lambda+ - lambda- =
// 2 hypot((a - c)/2, b) >= 0 and t = lambda+ + lambda- = a + c, it is d when
// both eigenvalues share a sign and |t| otherwise, i.e. min(d, |t|).
__device__ __forceinline__ float saliency2(float4 m) {
    const float d = 2.0f * hypotf(0.5f * (m.x - m.w), m.y);
    return fminf(d, fabsf(m.x + m.w));
}

// Block maximum of values >= 0 into *vmax_bits (their bits order as values).
// One atomic per block of a grid of a few blocks per SM: with one per warp of
// one pixel per thread the atomics to the one address took most of the time
// (1024^2: 16 us, 10.5 so).
__device__ __forceinline__ void block_vmax(float mx, unsigned* __restrict__ vmax_bits) {
    __shared__ unsigned part[32];
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned b = __reduce_max_sync(0xffffffffu, threadIdx.x < blockDim.x / 32 ? part[threadIdx.x] : 0u);
        if (threadIdx.x == 0) atomicMax(vmax_bits, b);
    }
}

__global__ void k_saliency2(const float4* __restrict__ in, size_t n, float* __restrict__ sal,
                            unsigned* __restrict__ vmax_bits) {
    float mx = 0.0f;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        const float s = saliency2(__ldg(in + i));
        if (sal) sal[i] = s;
        mx = fmaxf(mx, s);
    }
    if (vmax_bits) block_vmax(mx, vmax_bits);
}

__global__ void k_vmax(const float* __restrict__ v, size_t n, unsigned* __restrict__ vmax_bits) {
    float mx = 0.0f;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        mx = fmaxf(mx, v[i]);
    block_vmax(mx, vmax_bits);
}

// np.histogram(values, bins=256, range=(0, vmax)) bin of v for float32
// values: NumPy builds the edges in the values' type, float32 here
// (linspace(0, vmax, 257): i * (vmax / 256) rounded to float, the last edge
// vmax), takes int(v / vmax * 256) in FP64 as the first guess and corrects
// it against the float32 edges.
__device__ __forceinline__ float hist_edge(int i, double vmax) {
    return i >= 256 ? float(vmax) : float(double(i) * (vmax / 256.0));
}
__device__ __forceinline__ int hist_bin(float v, double vmax) {
    int i = int((double(v) / vmax) * 256.0);
    if (i >= 256) i = 255;
    if (i < 0) i = 0;
    if (v < hist_edge(i, vmax)) --i;
    else if (i != 255 && v >= hist_edge(i + 1, vmax)) ++i;
    return i;
}

// The edges decide the bin, so any first guess within one bin of it will do:
// an FP32 one (GB300 divides in FP64 at 1/64 of the FP32 rate).  Below 1e-30
// the edges themselves may coincide, and the FP64 steps are taken as they are.
// Two blocks per SM: each computes the edges and adds its 256 counts to the
// global ones once (1024^2: 10.5 us, 15 with a block per 256 values).
__global__ void k_hist256(const float* __restrict__ v, size_t n, const unsigned* __restrict__ vmax_bits,
                          unsigned long long* __restrict__ hist) {
    __shared__ unsigned h[256];
    __shared__ float edge[257];
    const double vmax = double(__uint_as_float(*vmax_bits));
    for (int i = threadIdx.x; i < 257; i += blockDim.x) {
        if (i < 256) h[i] = 0;
        edge[i] = hist_edge(i, vmax);
    }
    __syncthreads();
    if (vmax > 0.0) {
        const float vf = float(vmax), scale = 256.0f / vf;
        const bool wide = vf > 1e-30f && vf < 1e30f;
        for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
            const float x = v[i];
            if (!(x >= 0.0f && x <= vf)) continue;
            int b;
            if (wide) {
                b = min(int(x * scale), 255);
                if (x < edge[b]) --b;
                else if (b != 255 && x >= edge[b + 1]) ++b;
            } else {
                b = hist_bin(x, vmax);
            }
            atomicAdd(&h[b], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
        if (h[i]) atomicAdd(hist + i, (unsigned long long)h[i]);
}

// Otsu on the histogram, one block of 256 threads, one per bin
// (reconstruct.py:44-63): bin centres are float32 like the edges, the class
// weights and means FP64, the first maximum of the between-class variance
// wins.  Thread 0 adds the 256 products up in order, as NumPy's cumsum does;
// the FP64 divisions, 512 in a row for one thread before, run side by side.
__global__ void __launch_bounds__(256) k_otsu(const unsigned long long* __restrict__ hist,
                                              const unsigned* __restrict__ vmax_bits, double* __restrict__ thr) {
    __shared__ double cnt[256], prod[256], var[256];
    __shared__ int at[256];
    const int i = threadIdx.x;
    const double vmax = double(__uint_as_float(*vmax_bits));
    if (!(vmax > 0.0)) { if (i == 0) *thr = 0.0; return; }
    const double c = double((hist_edge(i, vmax) + hist_edge(i + 1, vmax)) / 2.0f);
    const double m = double(hist[i]);
    cnt[i] = m;
    prod[i] = m * c;
    __syncthreads();
    if (i == 0) {
        double w = 0.0, s = 0.0;
        for (int k = 0; k < 256; ++k) {
            w += cnt[k];
            s += prod[k];
            cnt[k] = w;
            prod[k] = s;
        }
    }
    __syncthreads();
    const double total = cnt[255], cum_all = prod[255];
    if (total == 0.0) { if (i == 0) *thr = 0.0; return; }
    const double w0 = cnt[i], w1 = total - w0;
    const double mu0 = w0 > 0.0 ? prod[i] / w0 : 0.0;
    const double mu1 = w1 > 0.0 ? (cum_all - prod[i]) / w1 : 0.0;
    const double dm = mu0 - mu1;
    const double bv = (w0 * w1) * (dm * dm);
    var[i] = bv > -1.0 ? bv : -1.0;                        // an infinite range makes it NaN, which never wins
    at[i] = i;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (i < o) {
            const double a = var[i], b = var[i + o];
            if (b > a || (b == a && at[i + o] < at[i])) { var[i] = b; at[i] = at[i + o]; }
        }
        __syncthreads();
    }
    if (i == at[0]) *thr = var[0] > -1.0 ? c : 0.0;
}

// s > thr with the threshold in FP64, as NumPy compares a float32 map with a Python float
__global__ void k_threshold(const float* __restrict__ s, size_t n, const double* __restrict__ thr,
                            unsigned char* __restrict__ mask) {
    const double t = *thr;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        mask[i] = double(s[i]) > t ? 1 : 0;
}

// square (2 r + 1) structuring element, one axis at a time; pixels outside
// the image count as 0 (scipy's border_value = 0): dilation ORs, erosion ANDs
template <bool DILATE, bool ALONG_X>
__global__ void k_morph(const unsigned char* __restrict__ in, unsigned char* __restrict__ out, int H, int W, int r) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    unsigned char acc = DILATE ? 0 : 1;
    for (int k = -r; k <= r; ++k) {
        const int xx = ALONG_X ? x + k : x, yy = ALONG_X ? y : y + k;
        const unsigned char v = (xx >= 0 && xx < W && yy >= 0 && yy < H) ? in[size_t(yy) * W + xx] : 0;
        if (DILATE) acc |= v; else acc &= v;
    }
    out[size_t(y) * W + x] = acc;
}

// Closing by a small square in one pass: a 32 x 32 tile with twice the radius
// around it in shared memory, dilated and eroded along x and y there.  Pixels
// outside the image are 0 before the dilation and again before the erosion.
constexpr int CT = 32, CLOSE_MAX = 8;
__global__ void __launch_bounds__(CT * 8) k_close(const unsigned char* __restrict__ in, unsigned char* __restrict__ out,
                                                 int H, int W, int r) {
    __shared__ unsigned char a[CT + 4 * CLOSE_MAX][CT + 4 * CLOSE_MAX], b[CT + 4 * CLOSE_MAX][CT + 4 * CLOSE_MAX];
    const int x0 = blockIdx.x * CT, y0 = blockIdx.y * CT, tid = threadIdx.y * CT + threadIdx.x;
    const int S = CT + 4 * r, D = CT + 2 * r;             // tile of the input; of the dilated image
    for (int e = tid; e < S * S; e += CT * 8) {
        const int y = e / S, x = e - y * S, gy = y0 - 2 * r + y, gx = x0 - 2 * r + x;
        a[y][x] = gy >= 0 && gy < H && gx >= 0 && gx < W ? in[size_t(gy) * W + gx] : 0;
    }
    __syncthreads();
    for (int e = tid; e < S * D; e += CT * 8) {           // dilate along x
        const int y = e / D, x = e - y * D;
        unsigned char v = 0;
        for (int k = 0; k <= 2 * r; ++k) v |= a[y][x + k];
        b[y][x] = v;
    }
    __syncthreads();
    for (int e = tid; e < D * D; e += CT * 8) {           // and along y: pixels (x0 - r + x, y0 - r + y)
        const int y = e / D, x = e - y * D, gy = y0 - r + y, gx = x0 - r + x;
        unsigned char v = 0;
        for (int k = 0; k <= 2 * r; ++k) v |= b[y + k][x];
        a[y][x] = gy >= 0 && gy < H && gx >= 0 && gx < W ? v : 0;
    }
    __syncthreads();
    for (int e = tid; e < D * CT; e += CT * 8) {          // erode along x
        const int y = e / CT, x = e - y * CT;
        unsigned char v = 1;
        for (int k = 0; k <= 2 * r; ++k) v &= a[y][x + k];
        b[y][x] = v;
    }
    __syncthreads();
    for (int y = threadIdx.y; y < CT; y += 8) {
        const int gy = y0 + y, gx = x0 + threadIdx.x;
        unsigned char v = 1;
        for (int k = 0; k <= 2 * r; ++k) v &= b[y + k][threadIdx.x];
        if (gy < H && gx < W) out[size_t(gy) * W + gx] = v;
    }
}

// Hole filling (binary_fill_holes): background 4-connected to the border stays
// background, the rest becomes foreground.  Connected components by union-find
// over all background pixels at once: pixel i is node i + 1, node 0 stands for
// the outside and takes the border's pixels.  A node's parent is never larger
// than itself and only roots are linked (compare-and-swap), so every chain and
// every retry ends.  Three launches and no word from the host; tiles that
// propagated by rounds, with a synchronisation after each, took 1.2 of the
// 1.43 ms of a 1024^2 mask.
//
// The root of x by path halving (Tarjan and van Leeuwen, 1984): each node on
// the way is hung on its grandparent.  Other threads write the same nodes, but
// only ever one of a node's ancestors, and only to nodes that are no roots.
template <class I>
__device__ __forceinline__ I uf_find(I* __restrict__ p, I x) {
    volatile I* parent = p;
    for (;;) {
        const I up = parent[x];
        if (up == x) return x;
        const I top = parent[up];
        if (top == up) return up;
        parent[x] = top;
        x = top;
    }
}
__device__ __forceinline__ unsigned uf_cas(unsigned* a, unsigned c, unsigned v) { return atomicCAS(a, c, v); }
__device__ __forceinline__ unsigned long long uf_cas(unsigned long long* a, unsigned long long c, unsigned long long v) {
    return atomicCAS(a, c, v);
}
template <class I>
__device__ __forceinline__ void uf_link(I* __restrict__ p, I x, I y) {
    I a = uf_find(p, x), b = uf_find(p, y);
    while (a != b) {
        const I hi = a > b ? a : b, lo = a > b ? b : a;
        const I old = uf_cas(p + hi, hi, lo);
        if (old == hi) break;
        a = uf_find(p, old);                               // hi was linked meanwhile: go on from its parent
        b = uf_find(p, lo);
    }
}

// a background pixel's first parent: the outside on the border, else the start of its run within the warp's 32 pixels
template <class I>
__global__ void __launch_bounds__(256) k_uf_init(const unsigned char* __restrict__ fg, I* __restrict__ p, int H, int W) {
    const int lane = threadIdx.x, x = blockIdx.x * 32 + lane;
    if (blockIdx.x == 0 && blockIdx.y == 0 && lane == 0 && threadIdx.y == 0) p[0] = 0;
    for (int y = blockIdx.y * 8 + threadIdx.y; y < H; y += gridDim.y * 8) {   // the same rows for a whole warp
        const bool bg = x < W && !fg[size_t(y) * W + x];
        const unsigned runs = __ballot_sync(0xffffffffu, bg);
        if (x >= W) continue;
        const size_t i = size_t(y) * W + x;
        const unsigned below = ~runs & ((1u << lane) - 1u);   // foreground to the left, within the warp
        const int start = below ? 32 - __clz(below) : 0;
        const bool border = x == 0 || y == 0 || x == W - 1 || y == H - 1;
        p[i + 1] = I(bg ? (border ? 0 : i + 1 - (lane - start)) : i + 1);
    }
}
template <class I>
__global__ void __launch_bounds__(256) k_uf_link(const unsigned char* __restrict__ fg, I* __restrict__ p, int H, int W) {
    const int x = blockIdx.x * 32 + threadIdx.x;
    if (x >= W) return;
    for (int y = blockIdx.y * 8 + threadIdx.y; y < H; y += gridDim.y * 8) {
        const size_t i = size_t(y) * W + x;
        if (fg[i]) continue;
        const bool left = x > 0 && !fg[i - 1], up = y > 0 && !fg[i - W];
        const bool border = x == 0 || y == 0 || x == W - 1 || y == H - 1;
        // runs meet across warps; a border pixel's parent is the outside, so its run is linked here too
        if (left && ((x & 31) == 0 || border || x == 1 || y == 0 || y == H - 1)) uf_link(p, I(i + 1), I(i));
        // one link per stretch of pixels whose upper neighbours are background too
        if (up && !(left && !fg[i - W - 1])) uf_link(p, I(i + 1), I(i + 1 - W));
    }
}
template <class I>
__global__ void __launch_bounds__(256) k_uf_finish(const unsigned char* __restrict__ fg, I* __restrict__ p, size_t n,
                                                   unsigned char* __restrict__ mask) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        mask[i] = fg[i] || uf_find(p, I(i + 1)) != 0 ? 1 : 0;
}

// SIMF passes: <A,B>, <B,B> (pass 1) and sum_p || A_p - alpha B_p ||_F (pass 2), FP64 accumulation
__device__ __forceinline__ void block_add(double v, double* dst) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(dst, v);
}

// blockIdx.y: one of several fields B, n apart, each with its three sums in acc
__global__ void k_simf_dots(const float4* __restrict__ A, const float4* __restrict__ B, size_t n, double* acc) {
    B += blockIdx.y * n;
    acc += 3 * blockIdx.y;
    double ab = 0.0, bb = 0.0;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        const float4 a = __ldg(A + i), b = __ldg(B + i);
        ab += double(a.x) * b.x + double(a.y) * b.y + double(a.z) * b.z + double(a.w) * b.w;
        bb += double(b.x) * b.x + double(b.y) * b.y + double(b.z) * b.z + double(b.w) * b.w;
    }
    block_add(ab, acc);
    block_add(bb, acc + 1);
}

__global__ void k_simf_norms(const float4* __restrict__ A, const float4* __restrict__ B, size_t n, double* sums) {
    B += blockIdx.y * n;
    const double* dots = sums + 3 * blockIdx.y;
    double* acc = sums + 3 * blockIdx.y + 2;
    const double alpha = dots[1] < 1e-8 ? 0.0 : dots[0] / dots[1];   // metrics.py:137-146
    const float al = float(alpha);
    double s = 0.0;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        const float4 a = __ldg(A + i), b = __ldg(B + i);
        const float d0 = fmaf(-al, b.x, a.x), d1 = fmaf(-al, b.y, a.y), d2 = fmaf(-al, b.z, a.z),
                    d3 = fmaf(-al, b.w, a.w);
        s += sqrt(double(d0) * d0 + double(d1) * d1 + double(d2) * d2 + double(d3) * d3);
    }
    block_add(s, acc);
}

static unsigned grid1(size_t n) {
    size_t b = (n + 255) / 256;
    if (b > 152 * 8) b = 152 * 8;
    return unsigned(b ? b : 1);
}

int simf2_device(const float4* A, const float4* B, size_t n, int K, double* dev_acc3, cudaStream_t st) {
    TVGB_CUDA(cudaMemsetAsync(dev_acc3, 0, size_t(K) * 3 * sizeof(double), st));
    for (int k = 0; k < K; k += 65535) {                   // grid.y
        const unsigned m = unsigned(K - k < 65535 ? K - k : 65535);
        const float4* b = B + size_t(k) * n;
        k_simf_dots<<<dim3(grid1(n), m), 256, 0, st>>>(A, b, n, dev_acc3 + 3 * size_t(k));
        TVGB_LAUNCHED();
        k_simf_norms<<<dim3(grid1(n), m), 256, 0, st>>>(A, b, n, dev_acc3 + 3 * size_t(k));
        TVGB_LAUNCHED();
    }
    return TVGB_OK;
}

}  // namespace tvgb

using namespace tvgb;

extern "C" {

int tvgb_stick_saliency2(const float* field, size_t n, float* saliency, void* stream) {
    TVGB_CHECK_ARG(field && saliency, "tvgb_stick_saliency2: NULL pointer");
    if (n == 0) return TVGB_OK;
    cudaStream_t st = as_stream(stream);
    DevArray din, dout;
    TVGB_TRY(din.in(field, n * 16, st));
    TVGB_TRY(dout.out(saliency, n * 4, st));
    TVGB_CHECK_ARG(reinterpret_cast<uintptr_t>(din.dev) % 16 == 0, "tvgb_stick_saliency2: field must be 16-byte aligned");
    {
        KernelTimer kt_("k_saliency2", st);
        k_saliency2<<<grid1(n), 256, 0, st>>>(din.get<float4>(), n, dout.get<float>(), nullptr);
        kt_.stop();
    }
    TVGB_LAUNCHED();
    TVGB_TRY(dout.finish());
    return sync_if(din.owned || dout.owned, st);
}

static int otsu_device(const float* v, size_t n, unsigned* vmax_bits, bool have_max, unsigned long long* hist,
                       double* thr, cudaStream_t st) {
    if (!have_max) {
        TVGB_CUDA(cudaMemsetAsync(vmax_bits, 0, sizeof(unsigned), st));
        k_vmax<<<std::min(grid1(n), 1216u), 256, 0, st>>>(v, n, vmax_bits);
        TVGB_LAUNCHED();
    }
    TVGB_CUDA(cudaMemsetAsync(hist, 0, 256 * sizeof(unsigned long long), st));
    {
        KernelTimer kt_("k_hist256", st);
        k_hist256<<<std::min(grid1(n), 304u), 512, 0, st>>>(v, n, vmax_bits, hist);
        kt_.stop();
    }
    TVGB_LAUNCHED();
    k_otsu<<<1, 256, 0, st>>>(hist, vmax_bits, thr);
    TVGB_LAUNCHED();
    return TVGB_OK;
}

int tvgb_otsu_threshold(const float* values, size_t n, double* threshold, void* stream) {
    TVGB_CHECK_ARG(values && threshold, "tvgb_otsu_threshold: NULL pointer");
    cudaStream_t st = as_stream(stream);
    if (n == 0) { *threshold = 0.0; return TVGB_OK; }
    DevArray din;
    TVGB_TRY(din.in(values, n * 4, st));
    Scratch sc;
    TVGB_TRY(sc.alloc(256 * 8 + 16 + 8, st));
    unsigned long long* hist = sc.get<unsigned long long>();
    double* thr = reinterpret_cast<double*>(hist + 256);
    unsigned* vmax = reinterpret_cast<unsigned*>(thr + 1);
    TVGB_TRY(otsu_device(din.get<float>(), n, vmax, false, hist, thr, st));
    TVGB_CUDA(cudaMemcpyAsync(threshold, thr, sizeof(double), cudaMemcpyDeviceToHost, st));
    TVGB_CUDA(cudaStreamSynchronize(st));
    return TVGB_OK;
}

int tvgb_saliency_threshold2(const float* field, unsigned s0, unsigned s1, int fill, int use_otsu, double threshold,
                             int close_radius, unsigned char* mask, double* threshold_used, void* stream) {
    TVGB_CHECK_ARG(field && mask, "tvgb_saliency_threshold2: NULL pointer");
    TVGB_CHECK_ARG(close_radius >= 0 && close_radius <= 4096, "tvgb_saliency_threshold2: bad close_radius %d",
                   close_radius);
    const size_t n = size_t(s0) * s1;
    if (n == 0) return TVGB_OK;
    cudaStream_t st = as_stream(stream);
    DevArray din, dmask;
    TVGB_TRY(din.in(field, n * 16, st));
    TVGB_TRY(dmask.out(mask, n, st));
    TVGB_CHECK_ARG(reinterpret_cast<uintptr_t>(din.dev) % 16 == 0,
                   "tvgb_saliency_threshold2: field must be 16-byte aligned");
    Scratch sc;
    // saliency, later the fill's parents (n + 1, 64-bit from 2^32 - 1 pixels on), and two masks
    const bool wide = fill && n >= 0xffffffffull;
    const size_t words = (n + 2) * (wide ? 8 : 4);
    TVGB_TRY(sc.alloc(words + 2 * n + 256 * 8 + 64, st));
    unsigned long long* hist = sc.get<unsigned long long>();
    double* thr = reinterpret_cast<double*>(hist + 256);
    unsigned* vmax = reinterpret_cast<unsigned*>(thr + 1);
    float* sal = reinterpret_cast<float*>(reinterpret_cast<char*>(hist) + 256 * 8 + 64);
    unsigned char* b0 = reinterpret_cast<unsigned char*>(sal) + words;
    unsigned char* b1 = b0 + n;
    TVGB_CUDA(cudaMemsetAsync(vmax, 0, sizeof(unsigned), st));
    {
        KernelTimer kt_("k_saliency2", st);
        k_saliency2<<<std::min(grid1(n), 1216u), 256, 0, st>>>(din.get<float4>(), n, sal, vmax);
        kt_.stop();
    }
    TVGB_LAUNCHED();
    if (use_otsu) {
        TVGB_TRY(otsu_device(sal, n, vmax, true, hist, thr, st));
    } else {
        TVGB_CUDA(cudaMemcpyAsync(thr, &threshold, sizeof(double), cudaMemcpyHostToDevice, st));
    }
    unsigned char* out = dmask.get<unsigned char>();
    k_threshold<<<grid1(n), 256, 0, st>>>(sal, n, thr, fill ? b0 : out);
    TVGB_LAUNCHED();
    if (fill) {
        const int H = int(s0), W = int(s1);
        dim3 blk(32, 8), g(ceil_div(s1, 32u), ceil_div(s0, 8u));
        unsigned char* cur = b0;
        if (close_radius > 0 && close_radius <= CLOSE_MAX) {   // binary_closing: dilation then erosion, border value 0
            KernelTimer kt_("k_close", st);
            k_close<<<dim3(ceil_div(s1, unsigned(CT)), ceil_div(s0, unsigned(CT))), blk, 0, st>>>(b0, b1, H, W,
                                                                                                 close_radius);
            kt_.stop();
            TVGB_LAUNCHED();
            cur = b1;
        } else if (close_radius > 0) {
            k_morph<true, true><<<g, blk, 0, st>>>(b0, b1, H, W, close_radius);
            k_morph<true, false><<<g, blk, 0, st>>>(b1, out, H, W, close_radius);
            k_morph<false, true><<<g, blk, 0, st>>>(out, b1, H, W, close_radius);
            k_morph<false, false><<<g, blk, 0, st>>>(b1, b0, H, W, close_radius);
            for (int i = 0; i < 4; ++i) TVGB_LAUNCHED();
        }
        auto fill_holes = [&](auto* parent) -> int {
            KernelTimer kt_("k_fill", st);
            const dim3 gu(g.x, std::min(g.y, 65535u));        // taller images: several rows per thread
            k_uf_init<<<gu, blk, 0, st>>>(cur, parent, H, W);
            TVGB_LAUNCHED();
            k_uf_link<<<gu, blk, 0, st>>>(cur, parent, H, W);
            TVGB_LAUNCHED();
            k_uf_finish<<<grid1(n), 256, 0, st>>>(cur, parent, n, out);
            kt_.stop();
            TVGB_LAUNCHED();
            return TVGB_OK;
        };
        // the saliency's place is free by now
        if (wide) TVGB_TRY(fill_holes(reinterpret_cast<unsigned long long*>(sal)));
        else TVGB_TRY(fill_holes(reinterpret_cast<unsigned*>(sal)));
    }
    if (threshold_used) {
        TVGB_CUDA(cudaMemcpyAsync(threshold_used, thr, sizeof(double), cudaMemcpyDeviceToHost, st));
        TVGB_CUDA(cudaStreamSynchronize(st));
    }
    TVGB_TRY(dmask.finish());
    return sync_if(din.owned || dmask.owned, st);
}

int tvgb_simf2(const float* A, const float* B, size_t n, double* simf, void* stream) {
    TVGB_CHECK_ARG(A && B && simf, "tvgb_simf2: NULL pointer");
    if (n == 0) { *simf = 0.0; return TVGB_OK; }
    cudaStream_t st = as_stream(stream);
    DevArray da, db;
    TVGB_TRY(da.in(A, n * 16, st));
    TVGB_TRY(db.in(B, n * 16, st));
    TVGB_CHECK_ARG(reinterpret_cast<uintptr_t>(da.dev) % 16 == 0 && reinterpret_cast<uintptr_t>(db.dev) % 16 == 0,
                   "tvgb_simf2: fields must be 16-byte aligned");
    Scratch sc;
    TVGB_TRY(sc.alloc(3 * sizeof(double), st));
    TVGB_TRY(simf2_device(da.get<float4>(), db.get<float4>(), n, 1, sc.get<double>(), st));
    double h[3];
    TVGB_CUDA(cudaMemcpyAsync(h, sc.get<double>(), sizeof(h), cudaMemcpyDeviceToHost, st));
    TVGB_CUDA(cudaStreamSynchronize(st));
    *simf = h[2] / double(n);
    return TVGB_OK;
}

}  // extern "C"
