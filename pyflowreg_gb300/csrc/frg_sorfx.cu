// Exact-order chained SOR of a single level (the level_solver seam) with the
// updates in 64-bit fixed point, as exact as float64 but not its bits.  The
// pyramid keeps k_sor_split: there a last-bit difference moves psi by up to
// 1e-7 where the residual cancels, and among the 1e8 pixels of a batch some 1/32
// px warp sample of the next level comes out another one.
//
// compute_flow (core/level_solver.py:158-369) sweeps columns outer, rows inner,
// in place, in float64.  On GB300 one float64 instruction holds a scheduler's
// float64 pipe for 64 clocks (2 lanes per clock per SM; a dependent chain sees
// the same 64 clocks), while a 32 x 32 -> 64-bit product issues every 2 clocks.
// An update of 14 float64 operations therefore costs 896 clocks per warp; the
// same update on two-limb integers costs about 60 instructions.  So the state
// (du, dv) is held in 64-bit fixed point and updated on the integer pipe, and
// only the fold of the coefficients, once per pass of up to five updates, uses
// float64.
//
// Number format.  A state value x is an integer multiple of 2^-q, split as
// x = h 2^30 + l with a balanced low limb l in [-2^29, 2^29).  Coefficients are
// multiples of 2^-60 below 1, split the same way.  With
//   c = omega w / den,  a 2^k = -omega A12 / den,  p = omega B / den
// folded per pixel and pass (k the smallest exponent with |a| < 1), an update is
//   du <- (1 - omega) du + c (up + down + left + right) + a 2^k dv + p
// (c per axis when the two smoothness weights differ).  The products h h and
// h l + l h are summed exactly in 64-bit accumulators and rounded once, to the
// nearest multiple of 2^-q; the l l products (below one unit of 2^-q for the
// sums, 2^(k - 2) units for a, with a sign that varies with both limbs) are left
// out.  Exact zeros stay zero.  The error of an update is thus about one unit of
// 2^-q (2^-56 px on the finest levels), where float64 rounds |du| ~ 1 px sums to
// 2^-53 several times.
//
// Range.  States are held below 2^lim units, |a 2^k| below 2^kmax and p below
// 2^62 units, with lim + kmax = 63: then the sum of the true terms stays below
// 2^64 - 2^lim, so a sum that wraps cannot land in the range of a state.  The
// unit follows from the caller's bound 2^reach px of |du|, |dv|: q = lim - reach.
// A coefficient or a state outside its range, or anything not finite,
// marks the frame, and so does a level whose result is nowhere above 2^42 units
// but not zero (so small that a float64 state would hold more bits).  Marked
// frames are solved again by a second launch with a wider format, and what that
// one marks by k_sor_split.
//
// Schedule: that of k_sor_split (row r's local time is tau = s - r; pixel
// (r, c) of pipelined iteration gi of a pass is updated at tau = start + c +
// 2 gi), with the work split over specialised warps.  Every 32 rows have NU
// update warps, which share the five pipelined iterations, and FC fold warps,
// which run ahead of them: fold warp j takes steps j, j + FC, ..., and writes
// each entering pixel's coefficients and pass-start state into a ring of kRingSlots
// slots in shared memory (mbarriers both ways).  The folds' float64
// instructions and loads are off the update's critical path, and the float64
// pipes of all four schedulers work on one row strip.  An update's neighbours
// come from shared memory: each iteration writes its new values to a buffer of
// the last three steps, from which the next iteration reads the right, lower
// and own values and the row below the upper one; one barrier per step.  A
// frame's strips in other CTAs of its cluster get the edge rows through
// distributed shared memory (st.async with a transaction barrier).
#include "frg_split.cuh"

#include <algorithm>
#include <cmath>

namespace frg {

namespace {

constexpr int kFxKmax = 4, kFxLim = 63 - kFxKmax;  // |omega A12 / den| stays below 16 but for rare pixels of coarse levels
constexpr int kFxWider = 3;          // bits by which the second launch widens both

struct FxArgs {
    const double* J;
    long long J_fs;
    const double* W;     // [2][K][D*P]: W / wsum, W a_data / wsum
    long long W_fs;
    const double* lap;
    long long lap_fs;
    double* wp;          // [K][D*P]: weights times psi of passes that continue a group
    long long wp_fs;
    long long* du;       // [D*P] pass-to-pass state, multiples of 2^-q
    long long* dv;
    long long st_fs;
    double* out_du;      // final pass, at out + r * out_rs + c
    double* out_dv;
    long long out_fs;
    int out_rs;
    int ring;            // also write the border copies around the output (rows -1 and h, columns -1 and w)
    DiagGeom g;
    double lap_scale;    // 2 / wsum
    long long half_omega, ca, cb;  // omega / 2, 2 wa / wsum, 2 wb / wsum: 61 fraction bits
    int oh, ol;          // 1 - omega
    FxPow pw[4];
    int *marks, *marks2;   // [n_frames] of the first and the second launch
    int lim, kmax, reach;
    int ahead;           // steps a fold may run ahead (fold_ahead)
    int second;          // second launch: frames the first one marked, format wider by kFxWider bits
    int nc;              // CTAs per frame
};

__device__ __forceinline__ long long mulw(int a, int b) { return (long long)a * b; }

// Limbs of an integer: v = h 2^30 + l, l in [-2^29, 2^29).
__device__ __forceinline__ int2 limbs(long long v)
{
    const long long u = v + (1 << 29);
    return make_int2((int)(u >> 30), (int)((unsigned)u & 0x3fffffffu) - (1 << 29));
}

// Top 64 bits of a 128-bit product, shifted left by k: a b 2^(k - 64) for
// |a|, |b| < 2^62, within about 2^(k + 1) units.
template <int k>
__device__ __forceinline__ long long mulh(long long a, long long b)
{
    const int ah = (int)(a >> 32), bh = (int)(b >> 32);
    const int al = (int)((unsigned)a >> 1), bl = (int)((unsigned)b >> 1);
    return (mulw(ah, bh) << k) + ((mulw(ah, bl) + mulw(bh, al)) >> (31 - k));
}

// Integer times 2^-q as a double, to nearest; on the integer pipe.
__device__ __forceinline__ double fx_to_double(long long v, int q)
{
    if (v == 0) return 0.0;
    const unsigned long long m = (unsigned long long)(v < 0 ? -v : v);
    const int n = __clzll((long long)m);
    const unsigned long long x = m << n, t = (x >> 11) + ((x >> 10) & 1);  // 53 bits (2^53 when it rounds up)
    const unsigned long long e = (unsigned long long)(63 - n - q + 1022);
    return __longlong_as_double((long long)(((e << 52) + t) | (v < 0 ? 0x8000000000000000ull : 0ull)));
}

// Magnitude of a double's mantissa with 61 fraction bits below its leading one
// (in [2^61, 2^62)); d = +-m 2^(e - 1084), e the biased exponent (0: d is taken
// as zero or too small to matter).
__device__ __forceinline__ long long mantissa61(double d)
{
    return (long long)(((unsigned long long)(((unsigned)__double2hiint(d) & 0xfffffu) | 0x100000u) << 41) |
                       ((unsigned long long)(unsigned)__double2loint(d) << 9));
}
__device__ __forceinline__ int exponent_of(double d) { return (__double2hiint(d) >> 20) & 0x7ff; }

// +-m 2^-n as whole units (rounded down) and a 30-bit fraction, the latter plus
// 2^29 (half a unit, for the update's rounding); m < 2^62, n >= 1.
__device__ __forceinline__ void split_units(long long m, int n, bool neg, long long& whole, int& frac)
{
    const unsigned long long v = n > 63 ? 0ull : (unsigned long long)m >> n;
    const unsigned long long lost = n > 94 ? 0ull : (n > 63 ? (unsigned long long)m >> (n - 64) : (unsigned long long)m << (64 - n));
    int f = (int)(lost >> 34);
    whole = (long long)v;
    if (neg) {
        whole = ~whole + (f == 0);
        f = (-f) & 0x3fffffff;
    }
    frac = f + (1 << 29);
}

// w x^b for 1e-5 <= x < 2^47 and |b| <= 1 on the integer pipe: x = 2^e m,
// m in [1, 2), R an integer near 2^16 / m from the top 8 bits of m's fraction,
// r = m R 2^-16 - 1 exactly (|r| < 2^-8.9; the product's low 64 bits), and
//   x^b = 2^(e b) (2^16 / R)^b (1 + r)^b
// with both factors tabulated and (1 + r)^b - 1 by its binomial series to r^6
// (the next term is below 2^-62).  All steps carry at least 2^-58 relative
// precision; the product with w is rounded once to float64.  7 float64
// operations (448 clocks of a scheduler's pipe) become about 80 integer
// instructions.
__device__ __forceinline__ double fx_wpow(double w, double x, const FxPow& P, int& bad)
{
    const int hi = __double2hiint(x);
    const unsigned e = (unsigned)((hi >> 20) - (1023 + kPowEMin));
    bad |= e >= 64u;
    const unsigned ec = e & 63u;
    const unsigned j = ((unsigned)hi >> 12) & 0xffu;
    const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
    const unsigned ml = (unsigned)__double2loint(x);
    const unsigned R = P.R[j];
    const long long B = P.B[j];
    const longlong2 Am = P.A[ec];
    // r 2^68
    const long long r = (long long)((unsigned long long)ml * R + ((unsigned long long)(mh * R) << 32));
    const int rh = (int)(r >> 29);  // r 2^39
    int t = P.c5 + ((int)(mulw(rh, P.c6) >> 32) >> 7);
    t = P.c4 + ((int)(mulw(rh, t) >> 32) >> 7);
    t = P.c3 + ((int)(mulw(rh, t) >> 32) >> 7);
    const long long p2 = P.c2 + (mulw(rh, t) >> 9);       // 2^60
    const long long p1 = P.c1 + (mulh<0>(r, p2) >> 4);    // 2^60
    const long long s = mulh<0>(r, p1);                   // 2^64
    const long long AB = mulh<3>(Am.x, B);                // 2^60, in [2^59, 2^62)
    const int ew = exponent_of(w);
    bad |= ew > 1023 + 60;
    const long long v = mulh<2>(AB + mulh<0>(AB, s), mantissa61(w));
    const double d = fx_to_double(v, 1082 - ew - (int)Am.y);
    return ew == 0 ? 0.0 : (__double2hiint(w) < 0 ? -d : d);
}

// (omega / 2) / d for d >= 1 as v 2^-(62 + ex), v in [2^60, 2^62): a float32
// reciprocal of d's mantissa, its exact error 1 - m y (the product's low 64
// bits) and y + y (e + e^2), to 2^-60; about 45 integer instructions for 4
// float64 operations (256 clocks).
__device__ __forceinline__ long long fx_half_omega_over(double d, long long half_omega, int& ex, int& bad)
{
    const int hi = __double2hiint(d);
    const unsigned lo = (unsigned)__double2loint(d);
    ex = (hi >> 20) - 1023;
    bad |= (unsigned)ex > 60u;
    float yf;
    asm("rcp.approx.ftz.f32 %0, %1;"
        : "=f"(yf)
        : "f"(__uint_as_float(0x3f800000u | ((unsigned)hi & 0xfffffu) << 3 | lo >> 29)));
    const int y0 = __float_as_int(yf + 1.0f) - 0x3f800000;  // y 2^23
    const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
    const long long e = -(long long)((unsigned long long)lo * (unsigned)y0 + ((unsigned long long)(mh * (unsigned)y0) << 32));
    const int eh = (int)(e >> 24);                           // e 2^75 before, 2^51 here; |e| < 2^-20
    const long long t = e + (mulw(eh, eh) >> 27);
    const long long tl = (long long)((unsigned long long)(unsigned)t * (unsigned)y0);
    const long long y = ((long long)y0 << 39) + ((mulw(y0, (int)(t >> 32)) + (long long)((unsigned long long)tl >> 32)) >> 4);
    return mulh<3>(y, half_omega);
}

template <int K>
struct FxIn {
    double j[6 * K];
    double w[K];
    double lu, lv;
};

// Ring planes, int4 each: (c_u, c_v), (a_u, a_v), (p_u, p_v) whole units, (k_u,
// k_v, p's fractions), state (one row more: the next strip's first row), and the
// second smoothness coefficient pair when the axes' weights differ.
constexpr int kPC = 0, kPA = 1, kPP = 2, kPK = 3, kPS = 4, kPD = 5;

// Folds one pixel's coefficients (core/level_solver.py:229-255, 309-364).  The
// weights come divided by wsum = 2 (wx + wy), so with the tensor's cross terms
// doubled and sums S over the channels
//   d = 1 + S W psi J11,  c = (2 w / wsum) D,  a 2^k = -(S W psi 2 J12) D,
//   p = (2 lap / wsum - S W psi 2 J13) D,  D = (omega / 2) / d.
// The quadratic form E and the sums are float64 (11 K + 2 operations less the
// power); the power, the reciprocals and the products with D are integers.
template <int K, bool ISO>
__device__ __forceinline__ void fx_fold(const FxArgs& A, const FxPow* pw, int pk, const FxIn<K>& in, long long su,
                                        long long sv, double* wp_io, int wp_plane, int4* slot, int plane, int q, int kmax,
                                        int& bad)
{
    const bool tick = (pk & kPkTick) != 0;
    double den[2] = {1.0, 1.0}, a12 = 0.0, c3[2] = {0.0, 0.0};
    double a = 0.0, b = 0.0;
    if (tick) {
        a = fx_to_double(su, q);
        b = fx_to_double(sv, q);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double j11 = in.j[0 * K + k], j22 = in.j[1 * K + k], j33 = in.j[2 * K + k];
        const double j12 = in.j[3 * K + k], j13 = in.j[4 * K + k], j23 = in.j[5 * K + k];
        double wp = in.w[k];
        if (tick) {
            double t = __fma_rn(j11, a, j13);
            t = __fma_rn(j12, b, t);
            const double v = __fma_rn(j22, b, j23);
            double E = __fma_rn(t, a, __fma_rn(v, b, j33));
            if (__double_as_longlong(E) < __double_as_longlong(0.00001)) E = 0.00001;
            wp = fx_wpow(wp, E, pw[k], bad);
        }
        if (pk & kPkStore) wp_io[k * wp_plane] = wp;
        den[0] = __fma_rn(wp, j11, den[0]);
        den[1] = __fma_rn(wp, j22, den[1]);
        a12 = __fma_rn(wp, j12, a12);
        c3[0] = __fma_rn(wp, j13, c3[0]);
        c3[1] = __fma_rn(wp, j23, c3[1]);
    }
    // c < 1/2 for one coefficient over four neighbours, < 1 for one per axis
    int4 vc, va, vp, vk, vd;
    int* oc = &vc.x;
    int* oa = &va.x;
    int* op = &vp.x;
    int* ok = &vk.x;
    int* od = &vd.x;
    const long long m12 = mantissa61(a12);
    const int e12 = exponent_of(a12);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        int ex;
        const long long D = fx_half_omega_over(den[i], A.half_omega, ex, bad);
        int2 x = limbs(mulh<3>(D, A.ca) >> min(2 + ex, 63));
        oc[2 * i] = x.x;
        oc[2 * i + 1] = x.y;
        if (!ISO) {
            x = limbs(mulh<3>(D, A.cb) >> min(2 + ex, 63));
            od[2 * i] = x.x;
            od[2 * i + 1] = x.y;
        }
        // |a12| D = v 2^(z - 62) with v < 2^62
        const int z = e12 - 1084 - ex + 62;
        const int k = max(0, z);
        bad |= k > kmax;
        const long long v = mulh<2>(m12, D) >> min(2 + max(0, -z), 63);
        x = limbs(__double2hiint(a12) < 0 ? v : -v);
        oa[2 * i] = x.x;
        oa[2 * i + 1] = x.y;
        ok[i] = k & 31;
        const double bb = __fma_rn(A.lap_scale, i ? in.lv : in.lu, -c3[i]);
        const int n = 1084 + ex - q - exponent_of(bb);
        bad |= n < 1;
        long long whole;
        split_units(mulh<2>(mantissa61(bb), D), max(n, 1), __double2hiint(bb) < 0, whole, ok[2 + i]);
        // 2^29 units are added so that the update's result is already offset for its split into limbs
        whole += 1 << 29;
        op[2 * i] = (int)whole;
        op[2 * i + 1] = (int)(whole >> 32);
    }
    slot[kPC * plane] = vc;
    slot[kPA * plane] = va;
    slot[kPP * plane] = vp;
    slot[kPK * plane] = vk;
    if (!ISO) slot[kPD * plane] = vd;
}

// 32 x 32 -> 64 bits.  As an instruction of its own: the fused multiply-add with
// a 64-bit addend issues at 25 lanes per clock against 63 (measured), and a
// chain of them waits 12.5 clocks a link against 9 for a product and a sum.
__device__ __forceinline__ long long mulx(int a, int b)
{
    long long r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}

// One component's update; p and the result are offset by 2^29, f holds p's
// fraction plus half a unit.
template <bool ISO>
__device__ __forceinline__ long long fx_point(int oh, int ol, int ch, int cl, int dh, int dl, int ah, int al, int k, int f,
                                              long long p, int own_h, int own_l, int oth_h, int oth_l, int s_h, int s_l,
                                              int t_h, int t_l)
{
    long long M = f + mulx(oh, own_l) + mulx(ol, own_h);
    long long H = p + mulx(oh, own_h);
    if (!ISO) {
        M += mulx(dh, t_l) + mulx(dl, t_h);
        H += mulx(dh, t_h);
    }
    M += mulx(ch, s_l) + mulx(cl, s_h);
    H += mulx(ch, s_h);
    const long long MA = mulx(ah, oth_l) + mulx(al, oth_h);
    return H + (mulx(ah, oth_h) << k) + (((M >> k) + MA) >> (30 - k));
}

__device__ __forceinline__ int4 sel4(bool c, int4 a, int4 b)
{
    return make_int4(c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z, c ? a.w : b.w);
}
__device__ __forceinline__ long long join(int h, int l) { return ((long long)h << 30) + l; }

constexpr int kFxTabBytes = 64 * 16 + 256 * 8 + 256 * 4;

// Shared memory of a CTA of M strips: ring int4[planes][kRingSlots][32 M] with the
// state plane's halo int4[kRingSlots] | iteration buffers int4[G][3][32 M + 2] |
// mbarriers: full[M][kRingSlots], empty[M][kRingSlots], edge[2 parities] | the power table where there is room.
template <int M, bool ISO>
struct FxSmem {
    static constexpr int rows = 32 * M;
    static constexpr int plane = kRingSlots * (rows + 1);  // int4 per ring plane (the halo row only used by the state)
    static constexpr int planes = ISO ? 5 : 6;
    static constexpr int buf = rows + 2;
    static constexpr size_t bytes =
        ((size_t)planes * plane + (size_t)kGMax * 3 * buf) * sizeof(int4) + (size_t)(2 * M * kRingSlots + 2) * 8;
    static constexpr bool table = bytes + kFxTabBytes <= 232448;  // room for a power table
    static constexpr size_t bytes_all = bytes + (table ? kFxTabBytes : 0);
};

// The border copies around pixel (r, c): its value before the last iteration
// (set_boundary_2d, core/level_solver.py:45-66).
__device__ __noinline__ void fx_ring(double* odu, double* odv, int rs, int r, int c, int h, int w, int4 own, int q)
{
    if (c != 0 && c != w - 1 && r != 0 && r != h - 1) return;
    const double bu = fx_to_double(join(own.x, own.y), q), bv = fx_to_double(join(own.z, own.w), q);
    for (int y = r == 0 ? -1 : r; y <= (r == h - 1 ? h : r); ++y)
        for (int x = c == 0 ? -1 : c; x <= (c == w - 1 ? w : c); ++x)
            if (y != r || x != c) {
                odu[(long long)y * rs + x] = bu;
                odv[(long long)y * rs + x] = bv;
            }
}

__host__ __device__ __forceinline__ void place_fx(const void* tab, FxPow* P)
{
    P->A = static_cast<const longlong2*>(tab);
    P->B = reinterpret_cast<const long long*>(P->A + 64);
    P->R = reinterpret_cast<const unsigned*>(P->B + 256);
}

// MB: CTAs per SM that the registers are to allow.  A fold's loads are not
// fetched ahead: the registers for that would cost the second CTA of an SM, and
// folds wait less than they run ahead.
template <int K, bool ISO, int M, int NU, int FC, int MB>
__global__ void __launch_bounds__(32 * SplitRoles<M, NU, FC>::warps, MB) k_sor_fx(FxArgs A, PassTable T)
{
    using SM = FxSmem<M, ISO>;
    constexpr int G = kGMax;
    constexpr int S = kRingSlots;
    constexpr int ROWS = SM::rows, PL = SM::plane, SR = ROWS + 1, BUF = SM::buf;
    extern __shared__ __align__(16) unsigned char fx_sm[];
    int4* ring = reinterpret_cast<int4*>(fx_sm);
    int4* bufs = ring + SM::planes * PL;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(bufs + G * 3 * BUF);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nc = A.nc;
    const int cta = nc > 1 ? (int)(blockIdx.x % nc) : 0;
    const int f = nc > 1 ? (int)(blockIdx.x / nc) : (int)blockIdx.x;
    if (A.second && !fx_recompute(A.marks[f])) return;  // the same for every CTA of a cluster
    using Roles = SplitRoles<M, NU, FC>;
    constexpr int WU = Roles::WU;
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
    const unsigned edge_bytes = (above ? G * sizeof(int4) : 0) + (below ? (G - 1) * sizeof(int4) : 0);
    // the power's table in shared memory when the channels share one: a fold's three look-ups
    // are dependent loads, about 700 clocks each from L2
    bool one = SM::table;
    for (int k = 1; k < K; ++k) one = one && A.pw[k].A == A.pw[0].A;
    int4* tab = reinterpret_cast<int4*>(bars + 2 * M * S + 2);
    if (one)
        for (int i = t; i < kFxTabBytes / 16; i += blockDim.x) tab[i] = reinterpret_cast<const int4*>(A.pw[0].A)[i];
    if (t == 0) {
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

    // the number format
    const int kmax = A.kmax + (A.second ? kFxWider : 0);
    const int lim = A.lim - (A.second ? kFxWider : 0);
    const int q = lim - A.reach - (A.second ? kFxWider : 0);

    double* odu = A.out_du + f * A.out_fs;
    double* odv = A.out_dv + f * A.out_fs;
    int total = 0;
    for (int p = 0; p < T.n; ++p) total += pass_span(w, T.pk[p]);
    const int nsteps = total + h - 1;
    bool dead = false;
    int bad = 0, big = 0, nonzero = 0, top = 0;
    Cursor cur;
    cur.init(T, w);

    if (!update && warp != Roles::wait && warp != Roles::idle) {
        // ------------------------------------------------------------ fold
        const int fj = Roles::fold(warp) / M;
        FxPow pw[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            pw[k] = A.pw[k];
            if (one) place_fx(tab, &pw[k]);
        }
        const double* Jr = A.J + f * A.J_fs + r;
        const double* Wr = A.W + f * A.W_fs + r;
        const double* lapr = A.lap + f * A.lap_fs + r;
        double* wpr = A.wp + f * A.wp_fs + r;
        const long long* dur = A.du + f * A.st_fs + r;
        const long long* dvr = A.dv + f * A.st_fs + r;
        // the first row's state also goes to the CTA above, as the row below its last one
        const bool sends = above && row == 0;
        unsigned halo = smem_addr(ring + kPS * PL + ROWS), halo_bar = full_bar(M - 1, 0);
        if (sends) {
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(halo) : "r"(cta - 1));
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(halo_bar) : "r"(cta - 1));
        }
        const bool gets = below && strip == M - 1;
        for (int s = fj; s < nsteps; s += FC) {
            const int slot = (unsigned)s % S;
            // the update has finished step s - ahead: the slot is free, and the states stored up to then can be read
            if (s >= A.ahead) mbar_wait(empty_bar(strip, slot), ((unsigned)(s - A.ahead) / S) & 1, dead);
            cur.seek(T, w, s - r);
            const int c = s - r - cur.start, pk = cur.pk, o = (r + c) * P;
            const bool in_level = row_ok && (unsigned)c < (unsigned)w;
            FxIn<K> in;
            long long su = 0, sv = 0;
            if (in_level) {
                if (!(pk & kPkZero)) {
                    su = dur[o];
                    sv = dvr[o];
                }
#pragma unroll
                for (int i = 0; i < 6 * K; ++i) in.j[i] = __ldg(Jr + i * pl + o);
                const double* wsrc = (pk & kPkCoef) ? wpr : ((pk & kPkTick) ? Wr + K * pl : Wr);
#pragma unroll
                for (int k = 0; k < K; ++k) in.w[k] = wsrc[k * pl + o];
                in.lu = __ldg(lapr + o);
                in.lv = __ldg(lapr + pl + o);
            }
            int4* sl = ring + slot * SR + row;
            const int2 lu = limbs(su), lv = limbs(sv);
            sl[kPS * PL] = make_int4(lu.x, lu.y, lv.x, lv.y);
            st_async_if(sends, halo + slot * SR * 16, make_int4(lu.x, lu.y, lv.x, lv.y), halo_bar + slot * 8);
            if (in_level) fx_fold<K, ISO>(A, pw, pk, in, su, sv, wpr + o, pl, sl, PL, q, kmax, bad);
            __syncwarp();
            if (lane == 0) {
                if (gets)
                    mbar_arrive_expect(full_bar(strip, slot), sizeof(int4));
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
        const int oh = A.oh, ol = A.ol;
        const bool first_row = r == 0, last_row = r == h - 1;
        // edge rows to the neighbouring CTAs: the last row's values go below, the first row's above
        const bool send_dn = below && row == ROWS - 1, send_up = above && row == 0;
        unsigned ebuf = smem_addr(bufs + (send_dn ? 0 : ROWS + 1)), ebar = edge_bar(0);
        if (send_dn || send_up) {
            const int peer = send_dn ? cta + 1 : cta - 1;
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(ebuf) : "r"(peer));
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(ebar) : "r"(peer));
        }
        const int limw = 1 << (lim - 32);
        int4 lf[NG], own[NG];  // the values left of the current pixel, and the pixel's own
        int4 C[NG], Ac[NG], Pc[NG], Kc[NG], D[NG];  // coefficients of the current step
        int4* myring = ring + row;
        int co[NG];            // ring offset of iteration i's pixel
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            lf[i] = own[i] = make_int4(0, 0, 0, 0);
            co[i] = (unsigned)(-2 * (g0 + i * NU)) % S * SR;
        }
        auto next_slot = [&](int o) { return o == (S - 1) * SR ? 0 : o + SR; };
        auto fetch_coef = [&]() {
#pragma unroll
            for (int i = 0; i < NG; ++i) {
                const int4* rg = myring + co[i];
                C[i] = rg[kPC * PL];
                Ac[i] = rg[kPA * PL];
                Pc[i] = rg[kPP * PL];
                Kc[i] = rg[kPK * PL];
                if (!ISO) D[i] = rg[kPD * PL];
                co[i] = next_slot(co[i]);
            }
        };
        int so = 0, so1 = SR;           // state slots of steps s and s + 1
        int b0 = 0, b1 = 2 * BUF, b2 = BUF;  // the buffers of steps s, s - 1, s - 2
        long long* sdu = A.du + f * A.st_fs + r;
        long long* sdv = A.dv + f * A.st_fs + r;
        asm volatile("bar.sync 1, %0;" ::"n"(32 * (WU + 1)) : "memory");
        if (g0 == 0) own[0] = myring[kPS * PL];
        fetch_coef();
        for (int s = 0; s < nsteps; ++s) {
            cur.advance(T, w, s - r);
            const int Gp = cur.pk >> 8;
            const int d0 = s - cur.start;  // the diagonal of iteration 0's pixel
            const int c0 = d0 - r;
#pragma unroll
            for (int i = 0; i < NG; ++i) {
                const int gi = g0 + i * NU;
                if (gi >= G) break;
                const int c = c0 - 2 * gi;
                // border copies: the neighbour outside is the pixel's own value before the update
                const int4* base = gi == 0 ? myring + kPS * PL : bufs + (gi - 1) * 3 * BUF + row + 1;
                const int4* before = base + (gi == 0 ? so : b2);
                const int4* prev = base + (gi == 0 ? so1 : b1);
                int4* mybuf = bufs + gi * 3 * BUF + row + 1;
                const int4 rt = *(c == w - 1 ? before : prev);
                const int4 dn = *(last_row ? before : prev + 1);
                const int4 up = *(first_row ? before : mybuf + b1 - 1);
                const int4 ow = own[i];
                const int4 le = sel4(c == 0, ow, lf[i]);
                const int4 Ci = C[i], Ai = Ac[i], Pi = Pc[i], Ki = Kc[i], Di = ISO ? make_int4(0, 0, 0, 0) : D[i];
                int4 su, sv;  // sums over the neighbours: (h, l) of the rows', then of the columns'
                if (ISO) {
                    su = make_int4(up.x + dn.x + le.x + rt.x, up.y + dn.y + le.y + rt.y, 0, 0);
                    sv = make_int4(up.z + dn.z + le.z + rt.z, up.w + dn.w + le.w + rt.w, 0, 0);
                } else {
                    su = make_int4(up.x + dn.x, up.y + dn.y, le.x + rt.x, le.y + rt.y);
                    sv = make_int4(up.z + dn.z, up.w + dn.w, le.z + rt.z, le.w + rt.w);
                }
                const long long pu = ((long long)Pi.y << 32) | (unsigned)Pi.x;
                const long long pv = ((long long)Pi.w << 32) | (unsigned)Pi.z;
                const long long U = fx_point<ISO>(oh, ol, Ci.x, Ci.y, Di.x, Di.y, Ai.x, Ai.y, Ki.x, Ki.z, pu, ow.x, ow.y, ow.z,
                                                  ow.w, su.x, su.y, su.z, su.w);
                int4 n;
                n.x = (int)(U >> 30);
                n.y = (int)((unsigned)U & 0x3fffffffu) - (1 << 29);
                const long long V = fx_point<ISO>(oh, ol, Ci.z, Ci.w, Di.z, Di.w, Ai.z, Ai.w, Ki.y, Ki.w, pv, ow.z, ow.w, n.x,
                                                  n.y, sv.x, sv.y, sv.z, sv.w);
                n.z = (int)(V >> 30);
                n.w = (int)((unsigned)V & 0x3fffffffu) - (1 << 29);
                mybuf[b0] = n;
                st_async_if((send_dn || (send_up && gi + 1 < G)) && s + 1 < nsteps, ebuf + (gi * 3 * BUF + b0) * 16, n,
                            ebar + (s & 1) * 8);
                const int uh = (int)(U >> 32), vh = (int)(V >> 32);
                const bool valid = gi < Gp && row_ok && (unsigned)c < (unsigned)w;
                top |= valid ? (uh ^ (uh >> 31)) | (vh ^ (vh >> 31)) : 0;
                const bool last = valid && gi == Gp - 1;
                if (__any_sync(~0u, last)) {
                    const int o = (d0 - 2 * gi) * P;
                    if (last) {
                        sdu[o] = U - (1 << 29);
                        sdv[o] = V - (1 << 29);
                        if (A.ring && cur.p == T.n - 1) fx_ring(odu, odv, A.out_rs, r, c, h, w, ow, q);
                    }
                }
                lf[i] = n;
                own[i] = rt;
            }
            fetch_coef();
            asm volatile("bar.sync 1, %0;" ::"n"(32 * (WU + 1)) : "memory");
            so = so1;
            so1 = next_slot(so1);
            const int b = b2;
            b2 = b1;
            b1 = b0;
            b0 = b;
        }
        bad |= top >= limw;
    }
    // the level's result, by all warps: states as float64, row-major
    __syncthreads();
    if (row_ok && (update || (warp != Roles::wait && warp != Roles::idle))) {
        const long long* sdu = A.du + f * A.st_fs + r;
        const long long* sdv = A.dv + f * A.st_fs + r;
        for (int c = update ? warp / M : NU + Roles::fold(warp) / M; c < w; c += NU + FC) {
            const long long nu = sdu[(r + c) * P], nv = sdv[(r + c) * P];
            const long long mag = (nu < 0 ? ~nu : nu) | (nv < 0 ? ~nv : nv);
            big |= mag >= (1ll << 42);
            nonzero |= (nu | nv) != 0;
            const long long o = (long long)r * A.out_rs + c;
            odu[o] = fx_to_double(nu, q);
            odv[o] = fx_to_double(nv, q);
        }
    }
    const int m = (bad || dead ? 1 : 0) | (big ? 2 : 0) | (nonzero ? 4 : 0);
    const int mm = __reduce_or_sync(~0u, m);
    if (lane == 0 && mm) atomicOr((A.second ? A.marks2 : A.marks) + f, mm);
    sync_all();  // no CTA leaves while another may still write into its shared memory
}

template <int K, bool ISO, int M, int NU, int FC, int MB>
cudaError_t run_fx(FxArgs A, const PassTable& T, int n_frames, cudaStream_t st)
{
    constexpr size_t smem = FxSmem<M, ISO>::bytes_all;
    A.ahead = fold_ahead(A.g.w);
    A.nc = (A.g.P / 32 + M - 1) / M;
    if (A.nc > kMaxSplitCluster) return cudaErrorInvalidValue;
    auto kern = k_sor_fx<K, ISO, M, NU, FC, MB>;
    cudaError_t e = ensure_max_dyn_smem((const void*)kern, (int)smem);
    if (e != cudaSuccess) return e;
    if (A.nc > 8 && (e = ensure_nonportable_clusters((const void*)kern)) != cudaSuccess) return e;
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

// 32 rows per CTA, five update and eight fold warps each with all registers, up to
// the 512 rows that a cluster of 16 CTAs covers (the level of 410 x 410 x 2 in
// seam_chain64).  Levels over 512 and 1024 rows need 64 and 128 rows per CTA.
template <int K, bool ISO>
cudaError_t run_fx_m(const FxArgs& A, const PassTable& T, int m, int n_frames, cudaStream_t st)
{
    if (m == 4) return run_fx<K, ISO, 4, 3, 3, 1>(A, T, n_frames, st);
    if (m == 2) return run_fx<K, ISO, 2, 5, 6, 1>(A, T, n_frames, st);
    return run_fx<K, ISO, 1, 5, 8, 1>(A, T, n_frames, st);
}

template <int K>
cudaError_t run_fx_k(const FxArgs& A, const PassTable& T, int m, int n_frames, cudaStream_t st)
{
    return A.ca == A.cb ? run_fx_m<K, true>(A, T, m, n_frames, st) : run_fx_m<K, false>(A, T, m, n_frames, st);
}

}  // namespace

size_t fx_pow_bytes() { return kFxTabBytes; }

bool make_fx_pow(double b, void* host, FxPow* P)
{
    if (!(b >= -1.0 && b <= 1.0)) return false;
    longlong2* A = static_cast<longlong2*>(host);
    long long* B = reinterpret_cast<long long*>(A + 64);
    unsigned* R = reinterpret_cast<unsigned*>(B + 256);
    const long double lb = b;
    for (int e = 0; e < 64; ++e) {
        const long double y = (e + kPowEMin) * lb;
        const long double fl = std::floor(y);
        A[e].x = (long long)std::rint(exp2l(y - fl) * 2305843009213693952.0L);  // 2^61
        A[e].y = (long long)fl;
    }
    for (int j = 0; j < 256; ++j) {
        R[j] = (unsigned)std::rint(65536.0 / (1.0 + (2.0 * j + 1.0) / 512.0));
        B[j] = (long long)std::rint(exp2l(lb * (16.0L - log2l((long double)R[j]))) * 1152921504606846976.0L);  // 2^60
    }
    long double c = lb, cn[7];
    for (int n = 2; n <= 6; ++n) cn[n] = c = c * (lb - (n - 1)) / n;
    P->c1 = (long long)std::rint(lb * 1152921504606846976.0L);
    P->c2 = (long long)std::rint(cn[2] * 1152921504606846976.0L);
    P->c3 = (int)std::rint(cn[3] * 1073741824.0L);
    P->c4 = (int)std::rint(cn[4] * 1073741824.0L);
    P->c5 = (int)std::rint(cn[5] * 1073741824.0L);
    P->c6 = (int)std::rint(cn[6] * 1073741824.0L);
    return true;
}

void place_fx_pow(void* dev, FxPow* P) { place_fx(dev, P); }

bool sor_fx_supports(int K, const DiagGeom& g, int n_passes, double omega)
{
    // three columns or more: the least a fold runs ahead (fold_ahead); omega in [1, 2) keeps |1 - omega| < 1 and c < 1/2
    return K >= 1 && K <= 4 && (g.P & 31) == 0 && g.w >= 3 && n_passes >= 1 && n_passes <= kMaxChain &&
           g.P / 32 <= kMaxSplitStrips && omega >= 1.0 && omega < 2.0 &&
           (long long)g.D * g.P * (6 * K + 2) < 0x7fffffffLL;
}

cudaError_t launch_sor_fx(const double* J, long long J_fs, const double* W, long long W_fs, const double* lap,
                          long long lap_fs, double* wp, long long wp_fs, double* du, double* dv, long long st_fs,
                          int n_frames, int K, DiagGeom g, const ChainPass* passes, int n_passes, double wx, double wy,
                          double omega, cudaStream_t st, double* out_du, double* out_dv, long long out_fs, int out_rs,
                          int ring, const FxPow* pows, int reach, int second, int* marks, int* marks2)
{
    if (!sor_fx_supports(K, g, n_passes, omega) || n_frames < 1 || !out_du || !out_dv || !marks || !marks2)
        return cudaErrorInvalidValue;
    // rows per CTA: 32, the most CTAs per frame, unless the cluster would pass 16 CTAs
    const int strips = g.P / 32;
    const int m = strips <= kMaxSplitCluster ? 1 : (strips <= 2 * kMaxSplitCluster ? 2 : 4);
    PassTable T;
    T.n = n_passes;
    for (int p = 0; p < n_passes; ++p) {
        const ChainPass& c = passes[p];
        if (c.G < 1 || c.G > kGMax || c.mode < -1 || c.mode > 3) return cudaErrorInvalidValue;
        const bool coef_in = c.mode < 0, store = c.mode >= 0 && c.store_coef;
        T.pk[p] = (c.G << 8) | (store ? kPkStore : 0) | (coef_in ? kPkCoef : 0) |
                  (!coef_in && (c.mode & 2) ? kPkTick : 0) | (!coef_in && (c.mode & 1) ? kPkZero : 0);
    }
    for (int p = n_passes; p < kMaxChain; ++p) T.pk[p] = 1 << 8;
    FxArgs A;
    A.J = J;
    A.J_fs = J_fs;
    A.W = W;
    A.W_fs = W_fs;
    A.lap = lap;
    A.lap_fs = lap_fs;
    A.wp = wp;
    A.wp_fs = wp_fs;
    A.du = reinterpret_cast<long long*>(du);
    A.dv = reinterpret_cast<long long*>(dv);
    A.st_fs = st_fs;
    A.out_du = out_du;
    A.out_dv = out_dv;
    A.out_fs = out_fs;
    A.out_rs = out_rs;
    A.ring = ring;
    A.g = g;
    // the row neighbours (above and below) carry the y weight
    const double wsum = ((wx + wx) + wy) + wy, two61 = 2305843009213693952.0;
    A.lap_scale = 2.0 / wsum;
    A.half_omega = (long long)std::rint(0.5 * omega * two61);
    A.ca = (long long)std::rint(2.0 * wy / wsum * two61);
    A.cb = (long long)std::rint(2.0 * wx / wsum * two61);
    // 1 - omega as float64 holds it, in limbs
    const long long om = (long long)std::rint((1.0 - omega) * 1152921504606846976.0);
    A.oh = (int)((om + (1 << 29)) >> 30);
    A.ol = (int)(om - ((long long)A.oh << 30));
    for (int k = 0; k < 4; ++k) A.pw[k] = k < K ? pows[k] : FxPow();
    A.lim = kFxLim;
    A.kmax = kFxKmax;
    A.reach = reach;
    A.second = second;
    A.marks = marks;
    A.marks2 = marks2;
    switch (K) {
        case 1: return run_fx_k<1>(A, T, m, n_frames, st);
        case 2: return run_fx_k<2>(A, T, m, n_frames, st);
        case 3: return run_fx_k<3>(A, T, m, n_frames, st);
        default: return run_fx_k<4>(A, T, m, n_frames, st);
    }
}

}  // namespace frg
