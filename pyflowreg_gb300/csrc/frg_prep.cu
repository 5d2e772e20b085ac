// Per-frame work before and after the flow: input preprocessing and
// post-registration statistics, on the device.
//
// Preprocessing (motion_correction/compensate_recording.py:521-561,
// util/image_processing.py:12-165): normalisation by the raw reference's
// min/max ((x - lo) / (hi - lo + 1e-8), jointly or per channel), then a
// Gaussian filter per channel as scipy.ndimage.gaussian_filter applies it:
// one 1-D correlation per axis in axis order (time, rows, columns), mode
// "reflect" (d c b a | a b c d | d c b a), each output sum formed in double
// as scipy's symmetric correlation forms it (outermost pair first):
//   acc = x[i] * w[0];  for j = r .. 1:  acc += (x[i - j] + x[i + j]) * w[j]
// and stored in the input's precision after each pass: float32 when numpy
// keeps the normalised frames float32 (float32 frames and reference), float64
// otherwise.  The taps (w[0 .. r], normalised in float64 by the host) come
// from the caller.  The result is stored as float32, the type the flow path's
// resize consumes.
//
// Post-registration (motion_correction/compensate_recording.py:808-821,
// core/warping.py:14-60, 128-157): per frame the valid mask of the backward
// warp (x + u in [0, W), y + v in [0, H); 0 or 255), and the partial sums of
// |w|, max |w|, the divergence du/dx + dv/dy (np.gradient: central inside,
// one-sided at the edges), u and v, reduced per frame by a second kernel.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/flowreg_gb300.h"
#include "frg_dfsum.cuh"
#include "frg_internal.h"

namespace frg {

namespace {

__device__ __forceinline__ int reflect_scipy(int i, int n)
{
    // scipy.ndimage mode "reflect": the edge sample is repeated
    if (n == 1) return 0;
    const int period = 2 * n;
    i %= period;
    if (i < 0) i += period;
    return i < n ? i : period - 1 - i;
}

struct PrepArgs {
    const float* raw;   // (T, H, W, K) float32 frames, or
    const double* raw64;  // the same in float64 (then raw is NULL and numpy normalises in float64)
    int T, H, W, K;
    double lo[kMaxK], den[kMaxK];  // normalisation per channel (same value for all channels when joint)
    const double* wt;   // temporal taps [K][rt + 1] (channel k uses its first rtk[k] + 1)
    const double* wy;   // row taps [K][ry + 1]
    const double* wx;   // column taps [K][rx + 1]
    int rt, ry, rx;     // tap strides - 1 (the largest radius per axis)
    int rtk[kMaxK], ryk[kMaxK], rxk[kMaxK];  // radius per channel
};

// N: the precision numpy normalises in (float32 for float32 frames and
// reference, else float64); S: the storage of the normalised values and of
// every pass's output (N for joint normalisation; float64 for per-channel
// normalisation, which writes into a float64 array).  Sums are formed in
// double either way, as scipy's line buffers do.
template <typename S>
__device__ __forceinline__ S normed(const PrepArgs& A, int t, int y, int x, int k);
template <>
__device__ __forceinline__ float normed<float>(const PrepArgs& A, int t, int y, int x, int k)
{
    const float v = A.raw[(((long long)t * A.H + y) * A.W + x) * A.K + k];
    return __fdiv_rn(__fsub_rn(v, (float)A.lo[k]), (float)A.den[k]);
}
template <>
__device__ __forceinline__ double normed<double>(const PrepArgs& A, int t, int y, int x, int k)
{
    const long long i = (((long long)t * A.H + y) * A.W + x) * A.K + k;
    const double v = A.raw64 ? A.raw64[i] : (double)A.raw[i];
    return __ddiv_rn(__dsub_rn(v, A.lo[k]), A.den[k]);
}

// scipy's symmetric correlation of one output sample (no contraction):
// acc = c * w[0], then acc += (left_j + right_j) * w[j] for j = r .. 1
template <typename F>
__device__ __forceinline__ double corr_sym(const double* w, int r, double c, F at)
{
    double acc = __dmul_rn(c, w[0]);
    for (int j = r; j >= 1; --j) {
        double l, rr;
        at(j, l, rr);
        acc = __dadd_rn(acc, __dmul_rn(__dadd_rn(l, rr), w[j]));
    }
    return acc;
}

// value after the temporal pass, stored as S (the temporal pass is an
// identity, x * 1.0, when its radius is 0)
template <typename N, typename S>
__device__ __forceinline__ S tpass(const PrepArgs& A, int t, int y, int x, int k)
{
    const double* w = A.wt + (long long)k * (A.rt + 1);
    const double acc = corr_sym(w, A.rtk[k], (double)normed<N>(A, t, y, x, k), [&](int j, double& l, double& r) {
        l = (double)normed<N>(A, reflect_scipy(t - j, A.T), y, x, k);
        r = (double)normed<N>(A, reflect_scipy(t + j, A.T), y, x, k);
    });
    return (S)acc;
}

// pass 1: temporal and row correlation into tmp (T, K, H, W) of S
template <typename N, typename S>
__global__ void k_prep_rows(PrepArgs A, S* __restrict__ tmp)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= A.W) return;
    const int y = blockIdx.y;
    const int tk = blockIdx.z;
    const int t = tk / A.K, k = tk % A.K;
    const double* w = A.wy + (long long)k * (A.ry + 1);
    const double acc = corr_sym(w, A.ryk[k], (double)tpass<N, S>(A, t, y, x, k), [&](int j, double& l, double& r) {
        l = (double)tpass<N, S>(A, t, reflect_scipy(y - j, A.H), x, k);
        r = (double)tpass<N, S>(A, t, reflect_scipy(y + j, A.H), x, k);
    });
    tmp[((long long)tk * A.H + y) * A.W + x] = (S)acc;
}

// pass 2: column correlation; float32 output (T, H, W, K)
template <typename S>
__global__ void k_prep_cols(PrepArgs A, const S* __restrict__ tmp, float* __restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= A.W) return;
    const int y = blockIdx.y;
    const int tk = blockIdx.z;
    const int t = tk / A.K, k = tk % A.K;
    const S* row = tmp + ((long long)tk * A.H + y) * A.W;
    const double* w = A.wx + (long long)k * (A.rx + 1);
    const double acc = corr_sym(w, A.rxk[k], (double)row[x], [&](int j, double& l, double& r) {
        l = (double)row[reflect_scipy(x - j, A.W)];
        r = (double)row[reflect_scipy(x + j, A.W)];
    });
    out[(((long long)t * A.H + y) * A.W + x) * A.K + k] = (float)(S)acc;
}

// Both correlations of one 32 x 32 tile of one frame and channel, for batches
// without a temporal filter (radius 0): the tile with its halo is normalised once
// into shared memory, the rows' correlation stays there, and only the result is
// written.  The two-kernel form above normalises and converts every sample once
// per tap.  Samples stored in float32 are summed as float32 pairs (DfSum; the
// taps split into two float32s, left + right exact as a two-sum), which gives the
// bits of the float64 sum; samples stored in float64 are summed in float64.
// 200 frames of 512 x 512 x 2, sigma 1, with the flow statistics below: 19.1 ms
// before, 4.28 ms now.
constexpr int kPrepTile = 32;

template <typename S, typename F>
__device__ __forceinline__ S corr_tile(const double* w, const float2* wf, int r, F at)
{
    if constexpr (sizeof(S) == 4) {
        DfSum acc;
        const float c = at(0);
        {
            const float p = __fmul_rn(c, wf[0].x);
            acc.add_pair(c, p, __fmaf_rn(c, wf[0].y, __fmaf_rn(c, wf[0].x, -p)));
        }
        for (int j = r; j >= 1; --j) {
            const float a = at(-j), b = at(j);
            const float s = __fadd_rn(a, b), z = __fsub_rn(s, a);
            const float d = __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), __fsub_rn(b, z));  // a + b = s + d
            const float2 t = wf[j];
            const float p = __fmul_rn(s, t.x);
            acc.add_pair(s, p, __fmaf_rn(d, t.x, __fmaf_rn(s, t.y, __fmaf_rn(s, t.x, -p))));
        }
        float v;
        if (acc.value(kDfErr(4 * (r + 1)), &v)) return v;
    }
    return (S)corr_sym(w, r, (double)at(0), [&](int j, double& l, double& rr) {
        l = (double)at(-j);
        rr = (double)at(j);
    });
}

template <typename N, typename S>
__global__ void __launch_bounds__(256) k_prep_tile(PrepArgs A, float* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char prep_sm[];
    const int tk = blockIdx.z, t = tk / A.K, k = tk % A.K;
    const int ry = A.ryk[k], rx = A.rxk[k];
    const int iw = kPrepTile + 2 * rx, ih = kPrepTile + 2 * ry;
    double* wy = reinterpret_cast<double*>(prep_sm);
    double* wx = wy + A.ry + 1;
    float2* wyf = reinterpret_cast<float2*>(wx + A.rx + 1);
    float2* wxf = wyf + A.ry + 1;
    S* in = reinterpret_cast<S*>(wxf + A.rx + 1);
    S* mid = in + (kPrepTile + 2 * A.ry) * (kPrepTile + 2 * A.rx);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto taps = [&](const double* w, int r, double* d, float2* f) {
        for (int i = tid; i <= r; i += 256) {
            d[i] = w[i];
            const float h = (float)w[i];
            f[i] = make_float2(h, (float)__dsub_rn(w[i], (double)h));
        }
    };
    taps(A.wy + (long long)k * (A.ry + 1), ry, wy, wyf);
    taps(A.wx + (long long)k * (A.rx + 1), rx, wx, wxf);
    const double w0 = A.wt[(long long)k * (A.rt + 1)];  // radius 0: x * w0, an identity for w0 = 1
    const int x0 = blockIdx.x * kPrepTile - rx, y0 = blockIdx.y * kPrepTile - ry;
    for (int yy = warp; yy < ih; yy += 8) {
        const int y = reflect_scipy(y0 + yy, A.H);
        for (int xx = lane; xx < iw; xx += 32) {
            S v = normed<N>(A, t, y, reflect_scipy(x0 + xx, A.W), k);
            if (w0 != 1.0) v = (S)__dmul_rn((double)v, w0);
            in[yy * iw + xx] = v;
        }
    }
    __syncthreads();
    for (int yy = warp; yy < kPrepTile; yy += 8)
        for (int xx = lane; xx < iw; xx += 32) {
            const S* c = in + (yy + ry) * iw + xx;
            mid[yy * iw + xx] = corr_tile<S>(wy, wyf, ry, [&](int j) { return c[j * iw]; });
        }
    __syncthreads();
    const int x = blockIdx.x * kPrepTile + lane;
    for (int yy = warp; yy < kPrepTile; yy += 8) {
        const int y = blockIdx.y * kPrepTile + yy;
        if (x >= A.W || y >= A.H) continue;
        const S* c = mid + yy * iw + lane + rx;
        out[(((long long)t * A.H + y) * A.W + x) * A.K + k] = (float)corr_tile<S>(wx, wxf, rx, [&](int j) { return c[j]; });
    }
}

// sqrt(s), correctly rounded, for s >= 0: the hardware's approximation of 1 / sqrt(s)
// and two Newton corrections g += (s - g^2) / (2 sqrt(s)), the residual exact by an
// fma, bring g to within an ulp; Tuckerman's test then picks the nearest double: with
// u the spacing at g, g is too small when s - g^2 > g u and too large when
// s - g^2 <= -g u (u the spacing below g).  7 float64 operations.
__device__ __forceinline__ double sqrt_rn(double s)
{
    const int hi = __double2hiint(s);
    if (hi < 0x2c000000 || hi >= 0x54000000) return sqrt(s);  // zero, tiny, huge, infinite, NaN
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    const double h = __hiloint2double(__double2hiint(y) - 0x100000, __double2loint(y));
    double g = __dmul_rn(s, y);
    g = __fma_rn(__fma_rn(-g, g, s), h, g);
    g = __fma_rn(__fma_rn(-g, g, s), h, g);
    const long long r = __double_as_longlong(__fma_rn(-g, g, s));
    const long long b = __double_as_longlong(g), e = b >> 52;
    long long gu = b + ((e - 1075) << 52);  // the bits of g u
    const long long mag = r & 0x7fffffffffffffffll;
    if (r >= 0) return __longlong_as_double(b + (mag > gu));
    if ((b << 12) == 0) gu -= 1ll << 52;
    return __longlong_as_double(b - (mag >= gu));
}

// Post-registration pass over flows (T, H, W, 2): valid masks and per-block
// partials (sum |w|, max |w|, sum div, sum u, sum v) at part[(f, block)][5]; a
// block takes 256 columns of ROWS rows.
//
// np.gradient's divergence (central inside, one-sided at the edges) summed over a
// row telescopes: sum du/dx = -3/2 u[0] + 1/2 u[1] - 1/2 u[W-2] + 3/2 u[W-1], and
// likewise down the columns for v; a value that is not finite and has both
// neighbours makes the sum NaN, as the differences' sum is.  The mask's tests
// x + u >= 0 and x + u < W are u >= -x and u < W - x, exact in float32 (beyond 2^24
// with -x and W - x rounded up: no float32 lies between).  About 12
// float64 operations per pixel are left of about 45.
// A block of small frames takes fewer rows, since the rows are its chain (one frame of
// 256 x 256 44 us with 16 rows, 37 with four), by the frame's size alone, so that a
// frame's sums do not depend on the batch that it comes in.
constexpr int kPostRows = 16, kPostRowsSmall = 4;

// PAIRS: the flow lies on an 8-byte boundary, so (u, v) is one load.
template <bool PAIRS, int ROWS>
__global__ void __launch_bounds__(256) k_flow_post(const float* __restrict__ flow, int H, int W, uint8_t* __restrict__ valid,
                                                   double* __restrict__ part)
{
    const int x = blockIdx.x * 256 + threadIdx.x;
    const int y0 = blockIdx.y * ROWS;
    const long long f = blockIdx.z;
    double s_mag = 0, s_div = 0, s_u = 0, s_v = 0;
    long long m_mag = 0;  // the bits of the largest magnitude
    if (x < W) {
        const auto edge = [](int i, int n) {
            return n < 2 ? 0.0 : (i == 0 ? -1.5 : 0.0) + (i == 1 ? 0.5 : 0.0) + (i == n - 2 ? -0.5 : 0.0) + (i == n - 1 ? 1.5 : 0.0);
        };
        const double ex = edge(x, W);
        const bool inner_x = x > 0 && x < W - 1;
        const float xlo = -__int2float_rd(x), xhi = __int2float_ru(W - x);
        const int y1 = min(y0 + ROWS, H);
#pragma unroll 4
        for (int y = y0; y < y1; ++y) {
            const long long p = (f * H + y) * W + x;
            const float2 w = PAIRS ? reinterpret_cast<const float2*>(flow)[p] : make_float2(flow[2 * p], flow[2 * p + 1]);
            if (valid) valid[p] = (w.x >= xlo && w.x < xhi && w.y >= -(float)y && w.y < (float)(H - y)) ? 255 : 0;
            const double u = f2d(w.x), v = f2d(w.y);
            const double mag = sqrt_rn(__fma_rn(u, u, __dmul_rn(v, v)));
            s_mag = __dadd_rn(s_mag, mag);
            const long long b = __double_as_longlong(mag);
            if (b > m_mag && b <= 0x7ff0000000000000ll) m_mag = b;  // NaN is passed over, as fmax does
            s_u = __dadd_rn(s_u, u);
            s_v = __dadd_rn(s_v, v);
            if (ex != 0.0) s_div = __fma_rn(ex, u, s_div);
            if (y < 2 || y >= H - 2) {
                const double ey = edge(y, H);
                if (ey != 0.0) s_div = __fma_rn(ey, v, s_div);
            }
            const bool odd_u = (__float_as_uint(w.x) & 0x7f800000u) == 0x7f800000u;
            const bool odd_v = (__float_as_uint(w.y) & 0x7f800000u) == 0x7f800000u;
            if ((odd_u && inner_x) || (odd_v && y > 0 && y < H - 1)) s_div = __longlong_as_double(0x7ff8000000000000ll);
        }
    }
    __shared__ double red[5][8];
    const int t = threadIdx.x;
    // the warp's four sums at once: half of the lanes go on with two of them, a quarter with one (6 float64 additions
    // where one sum at a time takes 20); the maximum as integers
    for (int o = 16; o > 0; o >>= 1) m_mag = max(m_mag, __shfl_xor_sync(~0u, m_mag, o));
    const bool h16 = t & 16, h8 = t & 8;
    const double p0 = __dadd_rn(h16 ? s_u : s_mag, __shfl_xor_sync(~0u, h16 ? s_mag : s_u, 16));
    const double p1 = __dadd_rn(h16 ? s_v : s_div, __shfl_xor_sync(~0u, h16 ? s_div : s_v, 16));
    double q = __dadd_rn(h8 ? p1 : p0, __shfl_xor_sync(~0u, h8 ? p0 : p1, 8));
    for (int o = 4; o > 0; o >>= 1) q = __dadd_rn(q, __shfl_xor_sync(~0u, q, o));
    if ((t & 7) == 0) {
        const int i = (t & 31) >> 3;  // magnitude, divergence, u, v
        red[i == 0 ? 0 : i + 1][t >> 5] = q;
        if (i == 0) red[1][t >> 5] = __longlong_as_double(m_mag);
    }
    __syncthreads();
    if (t < 5) {
        double a = red[t][0];
        for (int w = 1; w < 8; ++w) a = t == 1 ? fmax(a, red[1][w]) : a + red[t][w];
        part[((f * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * 5 + t] = a;
    }
}

// stats (T, 4): mean |w|, max |w|, mean divergence, |mean w|
__global__ void k_flow_stats(const double* __restrict__ part, long long n_slots, double n_pix, double* __restrict__ stats)
{
    const long long f = blockIdx.x;
    const double* p = part + f * n_slots * 5;
    double a = 0, m = 0, d = 0, su = 0, sv = 0;
    for (long long i = threadIdx.x; i < n_slots; i += blockDim.x) {
        a += p[5 * i];
        m = fmax(m, p[5 * i + 1]);
        d += p[5 * i + 2];
        su += p[5 * i + 3];
        sv += p[5 * i + 4];
    }
    __shared__ double red[5][256];
    const int t = threadIdx.x;
    red[0][t] = a;
    red[1][t] = m;
    red[2][t] = d;
    red[3][t] = su;
    red[4][t] = sv;
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
        if (t < st) {
            red[0][t] += red[0][t + st];
            red[1][t] = fmax(red[1][t], red[1][t + st]);
            red[2][t] += red[2][t + st];
            red[3][t] += red[3][t + st];
            red[4][t] += red[4][t + st];
        }
        __syncthreads();
    }
    if (t == 0) {
        const double mu = red[3][0] / n_pix, mv = red[4][0] / n_pix;
        stats[4 * f] = red[0][0] / n_pix;
        stats[4 * f + 1] = red[1][0];
        stats[4 * f + 2] = red[2][0] / n_pix;
        stats[4 * f + 3] = sqrt(mu * mu + mv * mv);
    }
}

}  // namespace

cudaError_t launch_preprocess(const float* raw, const double* raw64, int T, int H, int W, int K, const double* lo,
                              const double* den, const double* wt, const int* rt, const double* wy, const int* ry,
                              const double* wx, const int* rx, int f32_norm, int f32_storage, void* tmp, float* out,
                              cudaStream_t st)
{
    PrepArgs A;
    A.raw = raw;
    A.raw64 = raw64;
    A.T = T;
    A.H = H;
    A.W = W;
    A.K = K;
    for (int k = 0; k < kMaxK; ++k) {
        A.lo[k] = k < K ? lo[k] : 0.0;
        A.den[k] = k < K ? den[k] : 1.0;
    }
    A.wt = wt;
    A.wy = wy;
    A.wx = wx;
    A.rt = A.ry = A.rx = 0;
    for (int k = 0; k < kMaxK; ++k) {
        A.rtk[k] = k < K ? rt[k] : 0;
        A.ryk[k] = k < K ? ry[k] : 0;
        A.rxk[k] = k < K ? rx[k] : 0;
        A.rt = A.rtk[k] > A.rt ? A.rtk[k] : A.rt;
        A.ry = A.ryk[k] > A.ry ? A.ryk[k] : A.ry;
        A.rx = A.rxk[k] > A.rx ? A.rxk[k] : A.rx;
    }
    // no temporal filter and a halo that fits the shared memory every launch has (three blocks and more per SM):
    // both correlations in one kernel; else the two-kernel form, which normalises once per tap (3.0 times the time on
    // ten frames of 512 x 512 x 4 at sigma 1) but takes any radius
    const size_t elem = f32_storage ? sizeof(float) : sizeof(double);
    const size_t cols = kPrepTile + 2 * (size_t)A.rx;
    const size_t smem = (size_t)(A.ry + A.rx + 2) * 16 + elem * cols * (2 * kPrepTile + 2 * (size_t)A.ry);
    if (A.rt == 0 && smem <= 48 * 1024) {
        const dim3 tiles((unsigned)((W + kPrepTile - 1) / kPrepTile), (unsigned)((H + kPrepTile - 1) / kPrepTile),
                         (unsigned)(T * K));
        if (f32_storage)
            k_prep_tile<float, float><<<tiles, 256, smem, st>>>(A, out);
        else if (f32_norm)
            k_prep_tile<float, double><<<tiles, 256, smem, st>>>(A, out);
        else
            k_prep_tile<double, double><<<tiles, 256, smem, st>>>(A, out);
        host_count_launches(1);
        return cudaGetLastError();
    }
    host_count_launches(2);
    const dim3 grid((unsigned)((W + 127) / 128), (unsigned)H, (unsigned)(T * K));
    if (f32_storage) {
        k_prep_rows<float, float><<<grid, 128, 0, st>>>(A, (float*)tmp);
        k_prep_cols<float><<<grid, 128, 0, st>>>(A, (const float*)tmp, out);
    } else if (f32_norm) {
        k_prep_rows<float, double><<<grid, 128, 0, st>>>(A, (double*)tmp);
        k_prep_cols<double><<<grid, 128, 0, st>>>(A, (const double*)tmp, out);
    } else {
        k_prep_rows<double, double><<<grid, 128, 0, st>>>(A, (double*)tmp);
        k_prep_cols<double><<<grid, 128, 0, st>>>(A, (const double*)tmp, out);
    }
    return cudaGetLastError();
}

cudaError_t launch_flow_post(const float* flow, int T, int H, int W, uint8_t* valid, double* part, double* stats,
                             cudaStream_t st)
{
    const int bx = (W + 255) / 256;
    const bool small = (long long)bx * ((H + kPostRows - 1) / kPostRows) < 64;
    const int rows = small ? kPostRowsSmall : kPostRows;
    const dim3 grid((unsigned)bx, (unsigned)((H + rows - 1) / rows), (unsigned)T);
    const bool pairs = ((uintptr_t)flow & 7) == 0;
    const auto kern = pairs ? (small ? k_flow_post<true, kPostRowsSmall> : k_flow_post<true, kPostRows>)
                            : (small ? k_flow_post<false, kPostRowsSmall> : k_flow_post<false, kPostRows>);
    kern<<<grid, 256, 0, st>>>(flow, H, W, valid, part);
    k_flow_stats<<<T, 256, 0, st>>>(part, (long long)grid.y * grid.x, (double)H * W, stats);
    return cudaGetLastError();
}

}  // namespace frg

extern "C" {

namespace {

int preprocess_checked(int n_frames, int height, int width, int channels, const float* raw, const double* raw64,
                       const double* lo, const double* den, const double* wt, const int* rt, const double* wy,
                       const int* ry, const double* wx, const int* rx, int f32_norm, int f32_storage, void* tmp,
                       float* out, void* stream)
{
    using namespace frg;
    if ((!raw && !raw64) || !lo || !den || !wt || !wy || !wx || !rt || !ry || !rx || !tmp || !out)
        return host_fail(FRG_EINVAL, "NULL argument");
    if (n_frames < 1 || height < 1 || width < 1 || channels < 1 || channels > kMaxK)
        return host_fail(FRG_EINVAL, "bad shape");
    if ((long long)n_frames * channels > 65535 || height > 65535) return host_fail(FRG_EINVAL, "batch too large");
    for (int k = 0; k < channels; ++k)
        if (rt[k] < 0 || ry[k] < 0 || rx[k] < 0) return host_fail(FRG_EINVAL, "negative filter radius");
    if (f32_storage && !f32_norm) return host_fail(FRG_EINVAL, "float32 storage needs float32 normalisation");
    if (raw64 && f32_norm) return host_fail(FRG_EINVAL, "float64 frames normalise in float64");
    for (int k = 0; k < channels; ++k)
        if (!(den[k] != 0.0)) return host_fail(FRG_EINVAL, "zero normalisation range");
    cudaError_t e = launch_preprocess(raw, raw64, n_frames, height, width, channels, lo, den, wt, rt, wy, ry, wx, rx,
                                      f32_norm, f32_storage, tmp, out, (cudaStream_t)stream);
    if (e != cudaSuccess) return host_fail(FRG_ECUDA, cudaGetErrorString(e));
    return FRG_OK;
}

}  // namespace

int frg_preprocess(int n_frames, int height, int width, int channels, const float* raw, const double* lo,
                   const double* den, const double* wt, const int* rt, const double* wy, const int* ry,
                   const double* wx, const int* rx, int f32_norm, int f32_storage, void* tmp, float* out, void* stream)
{
    if (!raw) return frg::host_fail(FRG_EINVAL, "NULL argument");
    return preprocess_checked(n_frames, height, width, channels, raw, nullptr, lo, den, wt, rt, wy, ry, wx, rx,
                              f32_norm, f32_storage, tmp, out, stream);
}

int frg_preprocess_f64(int n_frames, int height, int width, int channels, const double* raw, const double* lo,
                       const double* den, const double* wt, const int* rt, const double* wy, const int* ry,
                       const double* wx, const int* rx, int f32_storage, void* tmp, float* out, void* stream)
{
    if (!raw) return frg::host_fail(FRG_EINVAL, "NULL argument");
    return preprocess_checked(n_frames, height, width, channels, nullptr, raw, lo, den, wt, rt, wy, ry, wx, rx, 0,
                              f32_storage, tmp, out, stream);
}

size_t frg_flow_post_workspace(int n_frames, int height, int width)
{
    return (size_t)n_frames * height * ((width + 255) / 256) * 5 * sizeof(double);
}

int frg_flow_post(int n_frames, int height, int width, const float* flow, unsigned char* valid, void* workspace,
                  double* stats, void* stream)
{
    using namespace frg;
    if (!flow || !workspace || !stats) return host_fail(FRG_EINVAL, "NULL argument");
    if (n_frames < 1 || n_frames > 65535 || height < 1 || height > 65535 || width < 1)
        return host_fail(FRG_EINVAL, "bad shape");
    host_count_launches(2);
    cudaError_t e = launch_flow_post(flow, n_frames, height, width, valid, (double*)workspace, stats,
                                     (cudaStream_t)stream);
    if (e != cudaSuccess) return host_fail(FRG_ECUDA, cudaGetErrorString(e));
    return FRG_OK;
}

}  // extern "C"

