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
#include "frg_split.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <set>
#include <vector>

namespace frg {

// The tables of dpow_tab, from the host's long double log2 / exp2 (extended or
// quadruple precision), rounded to double once.
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
    if ((e = cudaMemcpyToSymbol(g_dpow_log, lt, sizeof(lt))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(g_dpow_exp, et, sizeof(et))) != cudaSuccess) return e;
    done.insert(dev);
    return cudaSuccess;
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

constexpr int kLane64 = 256;       // most rows per CTA a caller may ask for
constexpr int kG64 = kGMax;        // iterations pipelined per pass, as a template maximum
constexpr int kMaxStrips64 = 16;   // cluster size (over 8: the non-portable opt-in)
constexpr int kPortableStrips = 8;

struct Sor64Args {
    const double* J;    // [6][K][D*P] per frame: J11, J22, J33 + 1e-5, 2 J12, 2 J13, 2 J23
    long long J_fs;
    const double* W;    // [2][K][D*P] per frame, W then W * a_data (W_fs 0: shared by all frames)
    long long W_fs;
    const double* lap;  // [2][D*P]: the u- and v-parts of the smoothness numerator from u, v
    long long lap_fs;
    double* coef;       // [5][D*P]: folded coefficients of passes that continue a group
    long long coef_fs;
    double* du;         // [D*P] pass-to-pass state
    double* dv;
    long long st_fs;
    double* out_du;     // final pass: du, dv at out + r * out_rs + c (frame stride out_fs)
    double* out_dv;
    long long out_fs;
    int out_rs;
    DiagGeom g;
    double wa, wb;      // smoothness weights of the row neighbours (y) and the column neighbours (x)
    double wsum;        // ((wx + wx) + wy) + wy, the reference's order
    double omega, one_m_omega;
    double a_m1[kMaxK];  // a_data - 1
    PowTab64 pw[kMaxK];  // the power's table per channel (null table: the general power)
    int nc;              // CTAs per frame
    int ahead;           // steps a fold may run ahead: at most the columns of a row less one
    const int* marks;    // frames to compute (fx_recompute); null: all
    int ring;            // the final pass also writes the border copies around the output
};

// The fold's inputs of one pixel (J, W, lap; or the stored coefficients),
// loaded at the start of the step whose end folds them: a step of float64
// work takes several microseconds, far longer than the loads.
template <int K>
struct FoldIn64 {
    double j[6 * K];
    double w[K];
    double lu, lv;
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
__device__ __forceinline__ Coef64 fold64(const Sor64Args& A, int pk, const FoldIn64<K>& r, double du, double dv)
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
            // 64-bit integers (the order of non-negative doubles; negative ones are below)
            double t = __fma_rn(j11, a, j13);
            t = __fma_rn(j12, b, t);
            const double q = __fma_rn(j22, b, j23);
            double E = __fma_rn(t, a, __fma_rn(q, b, j33));
            if (__double_as_longlong(E) < __double_as_longlong(0.00001)) E = 0.00001;
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

// Shared memory of a CTA of M strips of 32 rows: ring double2[3][kRingSlots][32 M + 1]
// (A12, BU | BV, iDu | state, whose last row is the next strip's first) and
// double[kRingSlots][32 M + 1] (iDv) | iteration buffers double2[G][3][32 M + 2] |
// mbarriers: full[M][kRingSlots], empty[M][kRingSlots], edge[2 parities] | a word
// for waits that ran out.
template <int M>
struct Split64Smem {
    static constexpr int rows = 32 * M;
    static constexpr int plane = kRingSlots * (rows + 1);
    static constexpr int buf = rows + 2;
    static constexpr size_t bytes = ((size_t)3 * plane + (size_t)kGMax * 3 * buf) * sizeof(double2) +
                                    (size_t)plane * sizeof(double) + (size_t)(2 * M * kRingSlots + 2) * 8 + 16;
};

// The chained solver, one step of the wavefront divided among warps (see the
// file's head).  MB: CTAs per SM that the registers are to allow.
template <int K, int M, int NU, int FC, int MB>
__global__ void __launch_bounds__(32 * SplitRoles<M, NU, FC>::warps, MB) k_sor_split64(Sor64Args A, PassTable T)
{
    using SM = Split64Smem<M>;
    using Roles = SplitRoles<M, NU, FC>;
    constexpr int G = kG64;
    constexpr int S = kRingSlots;
    constexpr int ROWS = SM::rows, PL = SM::plane, SR = ROWS + 1, BUF = SM::buf, WU = Roles::WU;
    extern __shared__ __align__(16) double sm64[];
    double2* ring = reinterpret_cast<double2*>(sm64);  // planes kA, kB, kS
    constexpr int kA = 0, kB = PL, kS = 2 * PL;
    double2* bufs = ring + 3 * PL;
    double* ringd = reinterpret_cast<double*>(bufs + G * 3 * BUF);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(ringd + PL);
    int* gave_up = reinterpret_cast<int*>(bars + 2 * M * S + 2);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nc = A.nc;
    const int cta = nc > 1 ? (int)(blockIdx.x % nc) : 0;
    const int f = nc > 1 ? (int)(blockIdx.x / nc) : (int)blockIdx.x;
    if (A.marks && !fx_recompute(A.marks[f])) return;  // the same for every CTA of a cluster
    const bool update = warp < WU;
    const int strip = (update ? warp : Roles::fold(warp)) % M;
    const int row = strip * 32 + lane;  // in the CTA
    const int r = cta * ROWS + row;     // in the level
    const DiagGeom g = A.g;
    const int P = g.P, h = g.h, w = g.w;
    const int pl = g.D * P;
    const bool row_ok = r < h;
    const bool above = cta > 0, below = cta + 1 < nc;  // other CTAs of the frame
    auto full_bar = [&](int st, int slot) { return smem_addr(bars + st * S + slot); };
    auto empty_bar = [&](int st, int slot) { return smem_addr(bars + M * S + st * S + slot); };
    auto edge_bar = [&](int par) { return smem_addr(bars + 2 * M * S + par); };
    // bytes a step's edge rows bring: every iteration's from above, all but the last one's from below
    const unsigned edge_bytes = (above ? G * sizeof(double2) : 0) + (below ? (G - 1) * sizeof(double2) : 0);
    if (t == 0) {
        *gave_up = 0;
        for (int i = 0; i < 2 * M * S + 2; ++i) mbar_init(smem_addr(bars + i), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (nc > 1)
            for (int par = 0; par < 2; ++par) mbar_expect(edge_bar(par), edge_bytes);
    }
    auto sync_all = [&]() {
        if (nc > 1)
            cooperative_groups::this_cluster().sync();
        else
            __syncthreads();
    };
    sync_all();

    double* odu = A.out_du + f * A.out_fs;
    double* odv = A.out_dv + f * A.out_fs;
    int total = 0;
    for (int p = 0; p < T.n; ++p) total += pass_span(w, T.pk[p]);
    const int nsteps = total + h - 1;
    bool dead = false;
    Cursor cur;
    cur.init(T, w);

    if (!update && warp != Roles::wait && warp != Roles::idle) {
        // ------------------------------------------------------------ fold
        const int fj = Roles::fold(warp) / M;
        const double* Jr = A.J + f * A.J_fs + r;
        const double* Wr = A.W + f * A.W_fs + r;
        const double* lapr = A.lap + f * A.lap_fs + r;
        double* coefr = A.coef + f * A.coef_fs + r;
        const double* dur = A.du + f * A.st_fs + r;
        const double* dvr = A.dv + f * A.st_fs + r;
        // the first row's state also goes to the CTA above, as the row below its last one
        const bool sends = above && row == 0;
        unsigned halo = smem_addr(ring + kS + ROWS), halo_bar = full_bar(M - 1, 0);
        if (sends) {
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(halo) : "r"(cta - 1));
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(halo_bar) : "r"(cta - 1));
        }
        const bool gets = below && strip == M - 1;
        for (int s = fj; s < nsteps; s += FC) {
            const int slot = (unsigned)s % S;
            // the update has finished step s - ahead: the slot is free, and the states stored up to then can be read
            if (s >= A.ahead) mbar_wait(empty_bar(strip, slot), ((unsigned)(s - A.ahead) / S) & 1, dead);
            cur.advance(T, w, s - r);
            const int c = s - r - cur.start, pk = cur.pk, o = (r + c) * P;
            const bool in_level = row_ok && (unsigned)c < (unsigned)w;
            FoldIn64<K> in;
            double su = 0.0, sv = 0.0;
            if (in_level) {
                if (!(pk & kPkZero)) {
                    su = dur[o];
                    sv = dvr[o];
                }
                if (pk & kPkCoef) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) in.j[q] = coefr[q * pl + o];
                } else {
#pragma unroll
                    for (int q = 0; q < 6 * K; ++q) in.j[q] = __ldg(Jr + q * pl + o);
                    const double* wsrc = (pk & kPkTick) ? Wr + K * pl : Wr;  // W * a_data on a tick
#pragma unroll
                    for (int k = 0; k < K; ++k) in.w[k] = __ldg(wsrc + k * pl + o);
                    in.lu = __ldg(lapr + o);
                    in.lv = __ldg(lapr + pl + o);
                }
            }
            const int ro = slot * SR + row;
            const double2 st = make_double2(su, sv);
            ring[kS + ro] = st;
            st_async_if(sends, halo + slot * SR * 16, *reinterpret_cast<const int4*>(&st), halo_bar + slot * 8);
            if (in_level) {
                const Coef64 cf = fold64<K>(A, pk, in, su, sv);
                if (pk & kPkStore) {
                    coefr[o] = cf.A12;
                    coefr[pl + o] = cf.BU;
                    coefr[2 * pl + o] = cf.BV;
                    coefr[3 * pl + o] = cf.iDu;
                    coefr[4 * pl + o] = cf.iDv;
                }
                ring[kA + ro] = make_double2(cf.A12, cf.BU);
                ring[kB + ro] = make_double2(cf.BV, cf.iDu);
                ringd[ro] = cf.iDv;
            }
            __syncwarp();
            if (lane == 0) {
                if (gets)
                    mbar_arrive_expect(full_bar(strip, slot), sizeof(double2));
                else
                    mbar_arrive(full_bar(strip, slot));
            }
        }
    } else if (warp == Roles::wait) {
        // ------------------------------------------------------------ wait
        // What a step needs from other warps and CTAs is awaited here, beside the update of the
        // step before: the fold's slots and the neighbouring CTAs' edge rows.
        auto wait_full = [&](int s) {
            if (s < nsteps)
                for (int st = 0; st < M; ++st) mbar_wait(full_bar(st, (unsigned)s % S), ((unsigned)s / S) & 1, dead);
        };
        wait_full(0);
        wait_full(1);
        asm volatile("bar.sync 1, %0;" ::"n"(32 * (WU + 1)) : "memory");
        for (int s = 0; s < nsteps; ++s) {
            wait_full(s + 2);
            if (nc > 1 && s + 1 < nsteps) {
                mbar_wait(edge_bar(s & 1), ((unsigned)s >> 1) & 1, dead);
                if (lane == 0) mbar_expect(edge_bar(s & 1), edge_bytes);
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * (WU + 1)) : "memory");
            // step s is done by every iteration: the slot of the pixel that entered 2 (G - 1) steps ago is free
            if (lane < M) mbar_arrive(empty_bar(lane, (unsigned)(s + A.ahead) % S));
        }
    } else if (update) {
        // ---------------------------------------------------------- update
        constexpr int NG = (G + NU - 1) / NU;  // iterations of this warp: g0, g0 + NU, ...
        const int g0 = warp / M;
        const double omm = A.one_m_omega, wa = A.wa, wb = A.wb;
        const bool first_row = r == 0, last_row = r == h - 1;
        // edge rows to the neighbouring CTAs: the last row's values go below, the first row's above
        const bool send_dn = below && row == ROWS - 1, send_up = above && row == 0;
        unsigned ebuf = smem_addr(bufs + (send_dn ? 0 : ROWS + 1)), ebar = edge_bar(0);
        if (send_dn || send_up) {
            const int peer = send_dn ? cta + 1 : cta - 1;
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(ebuf) : "r"(peer));
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(ebar) : "r"(peer));
        }
        double2 lf[NG], own[NG];  // the values left of the current pixel, and the pixel's own
        double2* myring = ring + row;
        int co[NG];               // ring offset of iteration i's pixel
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            lf[i] = own[i] = make_double2(0.0, 0.0);
            co[i] = (unsigned)(-2 * (g0 + i * NU)) % S * SR;
        }
        auto next_slot = [&](int o) { return o == (S - 1) * SR ? 0 : o + SR; };
        int so = 0, so1 = SR;                // state slots of steps s and s + 1
        int b0 = 0, b1 = 2 * BUF, b2 = BUF;  // the buffers of steps s, s - 1, s - 2
        double* sdu = A.du + f * A.st_fs + r;
        double* sdv = A.dv + f * A.st_fs + r;
        asm volatile("bar.sync 1, %0;" ::"n"(32 * (WU + 1)) : "memory");
        if (g0 == 0) own[0] = myring[kS];
        for (int s = 0; s < nsteps; ++s) {
            cur.advance(T, w, s - r);
            const int Gp = cur.pk >> 8;
            const int d0 = s - cur.start;  // the diagonal of iteration 0's pixel
#pragma unroll
            for (int i = 0; i < NG; ++i) {
                const int gi = g0 + i * NU;
                if (gi >= G) break;
                const int c = d0 - r - 2 * gi;
                // where the iteration before has its values: of this pixel (before), and what it wrote
                // in the last step: the right neighbour, and in the next row the lower one (prev)
                const double2* base = gi == 0 ? myring + kS : bufs + (gi - 1) * 3 * BUF + row + 1;
                const double2* before = base + (gi == 0 ? so : b2);
                const double2* prev = base + (gi == 0 ? so1 : b1);
                double2* mybuf = bufs + gi * 3 * BUF + row + 1;
                // border copies: the neighbour outside is the pixel's own value before the update
                const double2 rt = *(c == w - 1 ? before : prev);
                double2 n = lf[i];
                const bool valid = gi < Gp && row_ok && (unsigned)c < (unsigned)w;
                if (valid) {
                    const double2 dn = *(last_row ? before : prev + 1);
                    const double2 up = *(first_row ? before : mybuf + b1 - 1);
                    const double2 ow = own[i];
                    n = sor_point64(ow, up, dn, c == 0 ? ow : lf[i], rt, myring[kA + co[i]], myring[kB + co[i]],
                                    ringd[row + co[i]], wa, wb, omm);
                    if (gi == Gp - 1) {
                        if (cur.p < T.n - 1) {
                            sdu[(d0 - 2 * gi) * P] = n.x;
                            sdv[(d0 - 2 * gi) * P] = n.y;
                        } else {
                            const long long o = (long long)r * A.out_rs + c;
                            odu[o] = n.x;
                            odv[o] = n.y;
                            if (A.ring && (c == 0 || c == w - 1 || r == 0 || r == h - 1))
                                for (int yr = r == 0 ? -1 : 0; yr <= (r == h - 1 ? 1 : 0); ++yr)
                                    for (int xc = c == 0 ? -1 : 0; xc <= (c == w - 1 ? 1 : 0); ++xc)
                                        if (yr | xc) {
                                            odu[o + (long long)yr * A.out_rs + xc] = ow.x;
                                            odv[o + (long long)yr * A.out_rs + xc] = ow.y;
                                        }
                        }
                    }
                }
                mybuf[b0] = n;
                st_async_if((send_dn || (send_up && gi + 1 < G)) && s + 1 < nsteps, ebuf + (gi * 3 * BUF + b0) * 16,
                            *reinterpret_cast<const int4*>(&n), ebar + (s & 1) * 8);
                lf[i] = n;
                own[i] = rt;
                co[i] = next_slot(co[i]);
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * (WU + 1)) : "memory");
            so = so1;
            so1 = next_slot(so1);
            const int b = b2;
            b2 = b1;
            b1 = b0;
            b0 = b;
        }
    }
    if (dead) *gave_up = 1;
    __syncthreads();
    if (*gave_up && row_ok && update)  // a wait ran out: the rows' result is void
        for (int c = warp / M; c < w; c += NU) {
            const long long o = (long long)r * A.out_rs + c;
            odu[o] = odv[o] = __longlong_as_double(0x7ff8000000000000ll);
        }
    sync_all();  // no CTA leaves while another may still write into its shared memory
}

// Row strips of a level with at most `rows` rows per CTA (256, 128 or 64).
void split64(const DiagGeom& g, int rows, int* nc, int* nt)
{
    const int n = (g.P + rows - 1) / rows;
    *nc = n;
    *nt = ((g.P + n - 1) / n + 31) / 32 * 32;
}

template <int K, int M, int NU, int FC, int MB>
cudaError_t run_split64(Sor64Args A, const PassTable& T, int n_frames, cudaStream_t st)
{
    constexpr size_t smem = Split64Smem<M>::bytes;
    A.ahead = std::min(kFoldAhead, A.g.w - 1);
    A.nc = (A.g.P / 32 + M - 1) / M;
    if (A.nc > kMaxSplitCluster || (long long)n_frames * A.nc > 0x7fffffffLL) return cudaErrorInvalidValue;
    auto kern = k_sor_split64<K, M, NU, FC, MB>;
    cudaError_t e = ensure_max_dyn_smem((const void*)kern, (int)smem);
    if (e != cudaSuccess) return e;
    if (A.nc > kPortableStrips && (e = ensure_nonportable_clusters((const void*)kern)) != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_frames * A.nc));
    cfg.blockDim = dim3(32 * SplitRoles<M, NU, FC>::warps);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)A.nc;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = A.nc > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, A, T);
}

// Warps per 32 rows by what the launch has to fill: at most one CTA per SM, all
// registers; more, two CTAs per SM (100 frames 291 ms against 364).  Levels over
// 512 and 1024 rows need 64 and 128 rows per CTA.  Other counts of update and
// fold warps measured within 3 % or worse.
template <int K>
cudaError_t run_split64_m(const Sor64Args& A, const PassTable& T, int m, int n_frames, int n_sms, cudaStream_t st)
{
    if (m == 4) return run_split64<K, 4, 3, 3, 1>(A, T, n_frames, st);
    if (m == 2) return run_split64<K, 2, 5, 6, 1>(A, T, n_frames, st);
    if ((long long)n_frames * (A.g.P / 32) <= n_sms) return run_split64<K, 1, 5, 6, 1>(A, T, n_frames, st);
    return run_split64<K, 1, 5, 6, 2>(A, T, n_frames, st);
}

}  // namespace

bool sor_chain64_rows_ok(const DiagGeom& g, int rows)
{
    if (rows != 64 && rows != 128 && rows != kLane64) return false;
    int nc, nt;
    split64(g, rows, &nc, &nt);
    return nc <= kMaxStrips64;
}

bool sor_chain64_supports(int K, const DiagGeom& g, int n_passes)
{
    if (K < 1 || K > 4 || (g.P & 31) || g.w < 3 || n_passes < 1 || n_passes > kMaxChain) return false;
    int nc, nt;
    split64(g, kLane64, &nc, &nt);
    // 32-bit offsets within a frame: the largest plane index read is (6K + 2) planes of D * P
    const long long plane = (long long)g.D * g.P;
    // the tallest strips must fit a portable cluster: the fallback of a refused larger cluster
    return nc <= kPortableStrips && plane * (6 * K + 2) < 0x7fffffffLL;
}

cudaError_t launch_sor_chain64(const double* J, long long J_fs, const double* W, long long W_fs, const double* lap,
                               long long lap_fs, double* coef, long long coef_fs, double* du, double* dv,
                               long long st_fs, int n_frames, int K, DiagGeom g, const ChainPass* passes,
                               int n_passes, const double* a_data, double wx, double wy, double omega,
                               cudaStream_t st, double* out_du, double* out_dv, long long out_fs, int out_rs,
                               int rows, const PowTab64* pows, const int* marks, int ring)
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
        if (q.G < 1 || q.G > kG64 || q.mode < -1 || q.mode > 3) return cudaErrorInvalidValue;
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
    A.marks = marks;
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
    int m = strips <= kMaxSplitCluster ? 1 : (strips <= 2 * kMaxSplitCluster ? 2 : 4);
    if (rows >= 64) m = std::max(m, rows >= 128 ? 4 : 2);
    switch (K) {
        case 1: return run_split64_m<1>(A, T, m, n_frames, n_sms, st);
        case 2: return run_split64_m<2>(A, T, m, n_frames, n_sms, st);
        case 3: return run_split64_m<3>(A, T, m, n_frames, n_sms, st);
        default: return run_split64_m<4>(A, T, m, n_frames, n_sms, st);
    }
}

}  // namespace frg
