// Exact-order chained SOR in float64 (the parity precision).
//
// compute_flow (core/level_solver.py:158-369) sweeps columns outer, rows
// inner, in place, in float64.  Float32 arithmetic moves the flow by up to
// ~0.7 px against it: the 1/32-pixel warp of the next level turns rounding
// differences into different samples, and even last-bit differences do so at
// single pixels of a large batch.  So the pyramid keeps float64 and its
// operations in one order, and on GB300, where one float64 instruction holds a
// scheduler's float64 pipe for 64 clocks, it is bound by float64 instructions:
// 14 per pixel update and about 47 (two channels) per fold of a pixel's
// coefficients, once per pass of up to five updates.
//
// Schedule (k_sor_chain's, frg_sor.cu).  Row r's local time is tau = s - r; pass p
// occupies tau in [start_p, start_p + span_p), pixel (r, c) of pipelined
// iteration gi is updated at tau = start_p + c + 2 gi, and every neighbour value
// an update reads was produced one step earlier.
//
// A step's work is split over specialised warps.  One warp that updates all five
// iterations of 32 rows and folds the entering pixels issues 117 dependent
// float64 instructions per step, 7500 clocks, on one of the SM's four pipes.
// Here every 32 rows have an update warp per iteration (NU = 5) and FC fold
// warps, which run up to kFoldAhead steps ahead: fold warp j takes steps j, j +
// FC, ..., and writes each entering pixel's five coefficients (A12, BU, BV,
// omega/den_u, omega/den_v) and pass-start state into a ring of slots in shared
// memory, so that all four pipes work on one strip and the folds' loads are off
// the step.  An iteration writes its new values to a buffer of the last three
// steps, from which the next iteration reads the right, lower and own values and
// the row below the upper one; one barrier per step.  One more warp waits for
// the folds and for the neighbouring CTAs while the others update.  A frame's
// row strips are CTAs of a cluster and pass their edge rows by st.async with a
// transaction barrier.  Any split gives the same bits.
//
// 512 x 512 x 2, all levels, GB300: one frame 187 -> 37 ms, 24 frames 208 -> 87,
// 100 frames 423 -> 291, against one warp per 32 rows for everything (its strip
// heights chosen from the batch size).  What is left is the pipe: 117
// instructions at 64 to 76 clocks over four pipes, about 2000 clocks of a
// measured 2300 per step.
#include "frg_dpow.cuh"
#include "frg_split_sor.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <set>
#include <vector>

namespace frg {

// The tables of dpow_tab, from the host's long double log2 / exp2 (extended or
// quadruple precision), rounded to double once.  Copied on a stream of its own, so
// that the first call may come while the caller's stream is being captured.
cudaError_t upload_dpow_tables()
{
    static std::mutex mu;
    static std::set<int> done;
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    if (done.count(dev)) return cudaSuccess;
    double lt[3 * kDpowLogN], et[kDpowExpN];
    const long double two42 = 4398046511104.0L;
    for (int j = 0; j < kDpowLogN; ++j) {
        const double c = 1.0 + (2.0 * j + 1.0) / 512.0;  // exact
        const double inv = 1.0 / c;
        const long double L = -log2l((long double)inv);   // in [0, 1)
        const double Lhi = (double)(nearbyintl(L * two42) / two42);
        const double Llo = (double)(L - (long double)Lhi);
        const long long L42 = (long long)nearbyintl(L * two42);  // Lhi 2^42, below 2^42
        lt[3 * j] = inv;
        std::memcpy(&lt[3 * j + 1], &L42, sizeof(L42));
        lt[3 * j + 2] = Llo;
    }
    for (int i = 0; i < kDpowExpN; ++i) et[i] = (double)exp2l((long double)i / (long double)kDpowExpN);
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if ((e = cudaThreadExchangeStreamCaptureMode(&mode)) != cudaSuccess) return e;
    cudaStream_t own = nullptr;
    if ((e = cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking)) == cudaSuccess) {
        e = cudaMemcpyToSymbolAsync(g_dpow_log, lt, sizeof(lt), 0, cudaMemcpyHostToDevice, own);
        if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(g_dpow_exp, et, sizeof(et), 0, cudaMemcpyHostToDevice, own);
        const cudaError_t s = cudaStreamSynchronize(own);  // lt and et are this call's
        if (e == cudaSuccess) e = s;
        cudaStreamDestroy(own);
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e == cudaSuccess) done.insert(dev);
    return e;
}

// dpow_b's table for exponent b: T(e, j) = 2^(e b) (1 / inv_j)^b in long double,
// split into a double and the double of the remainder; inv_j as the device's
// log table holds it.
bool make_pow_table(double b, double2* tab, PowTab64* pt)
{
    if (!(b >= -1.0 && b <= 1.0)) return false;
    const long double lb = b;
    long double B[256];
    for (int j = 0; j < 256; ++j) {
        const double c = 1.0 + (2.0 * j + 1.0) / 512.0;  // exact
        const double inv = 1.0 / c;
        B[j] = exp2l(-lb * log2l((long double)inv));
    }
    for (int e = 0; e < kPowTabN / 256; ++e) {
        const long double A = exp2l((long double)(e + kPowEMin) * lb);
        for (int j = 0; j < 256; ++j) {
            const long double v = A * B[j];
            const double hi = (double)v;
            tab[e * 256 + j] = make_double2(hi, (double)(v - (long double)hi));
        }
    }
    // binomial coefficients C(b, n) = C(b, n - 1) (b - n + 1) / n
    long double c = lb, cn[7];
    for (int n = 2; n <= 6; ++n) cn[n] = c = c * (lb - (n - 1)) / n;
    pt->c2 = (double)cn[2];
    pt->c3 = (double)cn[3];
    pt->c4 = (float)cn[4];
    pt->c5 = (float)cn[5];
    pt->c6 = (float)cn[6];
    return true;
}

namespace {

__global__ void k_pow64(long long n, const double* __restrict__ x, double b, PowTab64 P, double* __restrict__ out)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = dpow_b(x[i], b, P);
}

}  // namespace

cudaError_t launch_pow64(long long n, const double* x, double b, double* out, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    if ((n + 255) / 256 > 0x7fffffffLL) return cudaErrorInvalidValue;
    PowTab64 P;
    std::vector<double2> tab(kPowTabN);
    double2* dt = nullptr;
    if (make_pow_table(b, tab.data(), &P)) {
        // stream-ordered: the copy from pageable memory returns once the table is staged
        cudaError_t e = cudaMallocAsync((void**)&dt, sizeof(double2) * kPowTabN, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(dt, tab.data(), sizeof(double2) * kPowTabN, cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) {
            if (dt) cudaFreeAsync(dt, st);
            return e;
        }
        P.t = dt;
    }
    k_pow64<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, x, b, P, out);
    cudaError_t e = cudaGetLastError();
    if (dt) {
        const cudaError_t f = cudaFreeAsync(dt, st);
        if (e == cudaSuccess) e = f;
    }
    return e;
}

namespace {

struct Sor64Args : SplitArgs<double> {
    double a_m1[kMaxK];  // a_data - 1
    PowTab64 pw[kMaxK];  // the power's table per channel (null table: the general power)
};

struct Coef64 {
    double A12, BU, BV, iDu, iDv;
};

// 1 / x for a normal x: the hardware approximation (rcp.approx.ftz.f64, about
// 2^-22 relative) refined by two Newton steps y += y (1 - x y), each doubling
// the correct bits, to within an ulp: 4 float64 operations where a division
// costs about 7.
__device__ __forceinline__ double rcp64(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = __fma_rn(-x, y, 1.0);
    y = __fma_rn(y, e, y);
    e = __fma_rn(-x, y, 1.0);
    return __fma_rn(y, e, y);
}

// omega / den, 0 when den is 0 (core/level_solver.py:352, 363); subnormal,
// infinite or NaN denominators take the division.  The tests look at the bits
// (integer instructions), not at the value (float64 compares).
__device__ __forceinline__ double omega_over(double omega, double den)
{
    const int hi = __double2hiint(den);
    const int ex = hi & 0x7ff00000;
    if (ex == 0 || ex == 0x7ff00000) {
        if (((hi & 0x7fffffff) | __double2loint(den)) == 0) return 0.0;
        return __ddiv_rn(omega, den);
    }
    return __dmul_rn(omega, rcp64(den));
}

// Coefficients of one pixel for a pass (core/level_solver.py:229-255, 309-364):
// with psi at a tick from the pixel's pass-start du, dv (E in nested fused
// multiply-adds; the reference adds J23 dv twice, hence 2 J23), psi = 1 on the
// first pass, or the stored coefficients of the group's first pass.  On a tick
// W psi = (W a) (E + 1e-5)^(a - 1), with W a and J33 + 1e-5 stored per pixel.
//   A12 = sum_k W psi J12,  BU = lap_u - sum_k W psi J13,  BV = lap_v - sum_k W psi J23,
//   iDu = omega / (wsum + sum_k W psi J11) (0 when the denominator is 0), iDv likewise
//   (omega times the reciprocal: within an ulp or two of the quotient).
// The tensor holds the cross terms doubled (2 J12, 2 J13, 2 J23, exact), as E
// uses them; the sums over them are then twice the sums above, exactly, and
// A12 = sum / 2, BU = fma(-1/2, sum, lap_u) give the same bits.
template <int K>
__device__ __forceinline__ Coef64 fold64(const Sor64Args& A, int pk, const FoldIn<double, K>& r, double du, double dv)
{
    Coef64 o;
    if (pk & kPkCoef) {
        o.A12 = r.j[0];
        o.BU = r.j[1];
        o.BV = r.j[2];
        o.iDu = r.j[3];
        o.iDv = r.j[4];
        return o;
    }
    const bool tick = (pk & kPkTick) != 0;
    double den_u = A.wsum, den_v = A.wsum, a12 = 0.0, c13 = 0.0, c23 = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double j11 = r.j[0 * K + k], j22 = r.j[1 * K + k], j33 = r.j[2 * K + k];
        const double j12 = r.j[3 * K + k], j13 = r.j[4 * K + k], j23 = r.j[5 * K + k];
        double wp = r.w[k];  // W, or W * a_data on a tick pass
        if (tick) {
            const double a = du, b = dv;
            // E + 1e-5 = a (J11 a + 2 J12 b + 2 J13) + b (J22 b + 2 J23) + (J33 + 1e-5):
            // 5 float64 operations; max(E, 0) + 1e-5 as max(E + 1e-5, 1e-5), compared as
            // 64-bit integers (the order of non-negative doubles; negative ones are below,
            // down to -inf: a NaN with its sign set, quiet as an operation's result is, lies
            // above that as an unsigned integer and stays)
            double t = __fma_rn(j11, a, j13);
            t = __fma_rn(j12, b, t);
            const double q = __fma_rn(j22, b, j23);
            double E = __fma_rn(t, a, __fma_rn(q, b, j33));
            if (__double_as_longlong(E) < __double_as_longlong(0.00001) && (unsigned)__double2hiint(E) <= 0xfff00000u)
                E = 0.00001;
            wp = __dmul_rn(wp, dpow_b(E, A.a_m1[k], A.pw[k]));
        }
        den_u = __fma_rn(wp, j11, den_u);
        den_v = __fma_rn(wp, j22, den_v);
        a12 = __fma_rn(wp, j12, a12);
        c13 = __fma_rn(wp, j13, c13);
        c23 = __fma_rn(wp, j23, c23);
    }
    o.A12 = __dmul_rn(0.5, a12);
    o.BU = __fma_rn(-0.5, c13, r.lu);
    o.BV = __fma_rn(-0.5, c23, r.lv);
    o.iDu = omega_over(A.omega, den_u);
    o.iDv = omega_over(A.omega, den_v);
    return o;
}

// One SOR update (core/level_solver.py:309-364, a_smooth = 1): c the pixel's
// (du, dv) before it, up/dn the rows above (new) and below (old), lf/rt the
// columns left (new) and right (old), Neumann copies already applied.  du
// first, then dv from the new du; 14 float64 operations.
__device__ __forceinline__ double2 sor_point64(double2 c, double2 up, double2 dn, double2 lf, double2 rt, double2 ca,
                                               double2 cb, double iDv, double wa, double wb, double omm)
{
    double nu = __fma_rn(wa, __dadd_rn(up.x, dn.x), ca.y);
    nu = __fma_rn(wb, __dadd_rn(lf.x, rt.x), nu);
    nu = __fma_rn(-ca.x, c.y, nu);
    const double dun = __fma_rn(nu, cb.y, __dmul_rn(omm, c.x));
    double nv = __fma_rn(wa, __dadd_rn(up.y, dn.y), cb.x);
    nv = __fma_rn(wb, __dadd_rn(lf.y, rt.y), nv);
    nv = __fma_rn(-ca.x, dun, nv);
    const double dvn = __fma_rn(nv, iDv, __dmul_rn(omm, c.y));
    return make_double2(dun, dvn);
}

template <int K_>
struct Ar64 {
    static constexpr int K = K_;
    static constexpr bool tick_weights = true, rings = true;
    using T = double;
    using T2 = double2;
    using Args = Sor64Args;
    using Coef = Coef64;
    __device__ static double2 pair(double x, double y) { return make_double2(x, y); }
    __device__ static Coef64 fold(const Args& A, int pk, const FoldIn<double, K>& r, double du, double dv)
    {
        return fold64<K>(A, pk, r, du, dv);
    }
    __device__ static double2 point(const Args& A, double2 c, double2 up, double2 dn, double2 lf, double2 rt, double2 ca,
                                    double2 cb, double iDv)
    {
        return sor_point64(c, up, dn, lf, rt, ca, cb, iDv, A.wa, A.wb, A.one_m_omega);
    }
};

// Rows per CTA and warps per 32 rows.  32 rows while the launch has at most one CTA
// per SM (all registers).  With more CTAs what counts is how a frame's cluster packs
// into the GPCs (14 to 20 SMs): 16 CTAs of 32 rows leave 40 of 152 SMs without a CTA,
// 8 CTAs of 64 rows none, while 13 CTAs of 32 rows fill 143 SMs and 7 of 64 rows,
// one strip of which is empty, 136.  So the shorter of both by `cost`; at 100 frames
// of 512 x 512 x 2: 71 ms with 64 rows against 91, and over all smaller levels 182
// against 162.  Levels over 512 and 1024 rows need 64 and 128 rows; 16 frames of
// 1024 x 1024 x 2: 222 ms with two CTAs of fewer warps per SM, 239 with one.
template <int K>
cudaError_t run_split64_m(const Sor64Args& A, const PassTable& T, int m, int n_frames, int dev, int n_sms, cudaStream_t st)
{
    using One = SplitLaunch<Ar64<K>, 1, 5, 6, 1>;
    using Two = SplitLaunch<Ar64<K>, 1, 5, 6, 2>;
    using Tall = SplitLaunch<Ar64<K>, 2, 3, 4, 2>;
    if (m == 4) return SplitLaunch<Ar64<K>, 4, 2, 4, 1>::run(A, T, n_frames, st);
    if (m == 2 && (long long)n_frames * Tall::ctas(A.g) <= n_sms) return SplitLaunch<Ar64<K>, 2, 5, 6, 1>::run(A, T, n_frames, st);
    if (m == 2) return Tall::run(A, T, n_frames, st);
    if ((long long)n_frames * One::ctas(A.g) <= n_sms) return One::run(A, T, n_frames, st);
    return Tall::cost(dev, A.g, n_frames) < Two::cost(dev, A.g, n_frames) ? Tall::run(A, T, n_frames, st)
                                                                          : Two::run(A, T, n_frames, st);
}

}  // namespace

bool sor_chain64_rows_ok(const DiagGeom& g, int rows)
{
    return (rows == 64 || rows == 128 || rows == 256) && (g.P + rows - 1) / rows <= kMaxSplitCluster;
}

bool sor_chain64_supports(int K, const DiagGeom& g, int n_passes)
{
    if (K < 1 || K > 4 || (g.P & 31) || g.w < 3 || n_passes < 1 || n_passes > kMaxChain) return false;
    // 32-bit offsets within a frame: the largest plane index read is (6K + 2) planes of D * P
    const long long plane = (long long)g.D * g.P;
    const int strips = g.P / 32;
    if (strips > kMaxSplitStrips || plane * (6 * K + 2) >= 0x7fffffffLL) return false;
    if (strips_per_cta(strips, kPortableCluster)) return true;
    // over 1024 rows: a device that takes clusters of over 8 CTAs
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const int nc = (strips + 3) / 4;
    switch (K) {
        case 1: return SplitLaunch<Ar64<1>, 4, 2, 4, 1>::frames_at_once(dev, nc, 1) > 0;
        case 2: return SplitLaunch<Ar64<2>, 4, 2, 4, 1>::frames_at_once(dev, nc, 1) > 0;
        case 3: return SplitLaunch<Ar64<3>, 4, 2, 4, 1>::frames_at_once(dev, nc, 1) > 0;
        default: return SplitLaunch<Ar64<4>, 4, 2, 4, 1>::frames_at_once(dev, nc, 1) > 0;
    }
}

cudaError_t launch_sor_chain64(const double* J, long long J_fs, const double* W, long long W_fs, const double* lap,
                               long long lap_fs, double* coef, long long coef_fs, double* du, double* dv,
                               long long st_fs, int n_frames, int K, DiagGeom g, const ChainPass* passes,
                               int n_passes, const double* a_data, double wx, double wy, double omega,
                               cudaStream_t st, double* out_du, double* out_dv, long long out_fs, int out_rs,
                               int rows, const PowTab64* pows, int ring)
{
    if (!sor_chain64_supports(K, g, n_passes) || n_frames < 1) return cudaErrorInvalidValue;
    if (rows != 0 && !sor_chain64_rows_ok(g, rows)) return cudaErrorInvalidValue;
    int dev = 0, n_sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    PassTable T;
    T.n = n_passes;
    for (int p = 0; p < n_passes; ++p) {
        const ChainPass& q = passes[p];
        if (q.G < 1 || q.G > kGMax || q.mode < -1 || q.mode > 3) return cudaErrorInvalidValue;
        const bool coef_in = q.mode < 0, store = q.mode >= 0 && q.store_coef;
        T.pk[p] = (q.G << 8) | (store ? kPkStore : 0) | (coef_in ? kPkCoef : 0) |
                  (!coef_in && (q.mode & 2) ? kPkTick : 0) | (!coef_in && (q.mode & 1) ? kPkZero : 0);
    }
    for (int p = n_passes; p < kMaxChain; ++p) T.pk[p] = 1 << 8;
    Sor64Args A;
    A.J = J;
    A.J_fs = J_fs;
    A.W = W;
    A.W_fs = W_fs;
    A.lap = lap;
    A.lap_fs = lap_fs;
    A.coef = coef;
    A.coef_fs = coef_fs;
    A.du = du;
    A.dv = dv;
    A.st_fs = st_fs;
    A.out_du = out_du;
    A.out_dv = out_dv;
    A.out_fs = out_fs;
    A.out_rs = out_rs;
    A.ring = ring;
    A.g = g;
    A.wa = wy;  // the thread index runs along rows: row neighbours carry the y weight
    A.wb = wx;
    A.wsum = ((wx + wx) + wy) + wy;
    A.omega = omega;
    A.one_m_omega = 1.0 - omega;
    for (int k = 0; k < kMaxK; ++k) {
        A.a_m1[k] = k < K ? a_data[k] - 1.0 : 0.0;
        A.pw[k] = pows && k < K ? pows[k] : PowTab64();
    }
    // rows per CTA: 32 unless the cluster would pass 16 CTAs; a caller's choice of more is taken
    const int strips = g.P / 32;
    const int asked = rows >= 128 ? 4 : (rows >= 64 ? 2 : 1);
    return launch_or_taller(strips, std::max(asked, strips_per_cta(strips, kMaxSplitCluster)), [&](int m) {
        switch (K) {
            case 1: return run_split64_m<1>(A, T, m, n_frames, dev, n_sms, st);
            case 2: return run_split64_m<2>(A, T, m, n_frames, dev, n_sms, st);
            case 3: return run_split64_m<3>(A, T, m, n_frames, dev, n_sms, st);
            default: return run_split64_m<4>(A, T, m, n_frames, dev, n_sms, st);
        }
    });
}

}  // namespace frg
