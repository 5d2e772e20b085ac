// The strip kernel of the exact-order chained SOR, for the float64 solver
// (frg_sor64.cu, whose head describes it) and the float32 one (frg_sor.cu).
#pragma once

#include "frg_split.cuh"

#include <atomic>
#include <cstdint>

namespace frg {

namespace {

template <typename T>
struct SplitArgs {
    const T* J;    // [6][K][D*P] per frame
    long long J_fs;
    const T* W;    // [K][D*P] per frame, or [2][K][D*P] (Ar::tick_weights; W_fs 0: shared by all frames)
    long long W_fs;
    const T* lap;  // [2][D*P]: the u- and v-parts of the smoothness numerator from u, v
    long long lap_fs;
    T* coef;       // [5][D*P]: folded coefficients of passes that continue a group
    long long coef_fs;
    T* du;         // [D*P] pass-to-pass state
    T* dv;
    long long st_fs;
    T* out_du;     // final pass: du, dv at out + r * out_rs + c (frame stride out_fs); null: into du, dv
    T* out_dv;
    long long out_fs;
    int out_rs;
    DiagGeom g;
    T wa, wb;      // smoothness weights of the row neighbours (y) and the column neighbours (x)
    T wsum;        // ((wx + wx) + wy) + wy, the reference's order
    T omega, one_m_omega;
    int nc;              // CTAs per frame
    int ahead;           // steps a fold may run ahead (fold_ahead)
    int ring;            // the final pass also writes the border copies around the output
};

// The fold's inputs of one pixel (J, W, lap; or the stored coefficients).
template <typename T, int K>
struct FoldIn {
    T j[6 * K];
    T w[K];
    T lu, lv;
};

// Shared memory of a CTA of M strips of 32 rows, T float or R, T2 a pair: ring
// T2[3][kRingSlots][32 M + 1] (A12, BU | BV, iDu | state, whose last row is the next
// strip's first) and T[kRingSlots][32 M + 1] (iDv) | iteration buffers T2[G][3][32 M + 2] |
// mbarriers: full[M][kRingSlots], empty[M][kRingSlots], edge[2 parities] | a word
// for waits that ran out.
template <typename T, int M>
struct SplitSmem {
    static constexpr int rows = 32 * M;
    static constexpr int plane = kRingSlots * (rows + 1);
    static constexpr int buf = rows + 2;
    static constexpr size_t bytes = ((size_t)3 * plane + (size_t)kGMax * 3 * buf) * 2 * sizeof(T) +
                                    (size_t)plane * sizeof(T) + (size_t)(2 * M * kRingSlots + 2) * 8 + 16;
};

// NaN in place of this CTA's rows of the result, the border copies included.  Its place
// is read anew: values kept for it through the solve would cost registers there.
template <class Ar, int M, int NU>
__device__ __forceinline__ void void_rows(const typename Ar::Args& A)
{
    using R = typename Ar::T;
    int t, block;
    asm volatile("mov.u32 %0, %%tid.x;\n\tmov.u32 %1, %%ctaid.x;" : "=r"(t), "=r"(block));
    const int warp = t >> 5, h = A.g.h, w = A.g.w;
    const long long f = block / A.nc;
    const int r = (block % A.nc * M + warp % M) * 32 + (t & 31);
    if (r >= h || warp >= M * NU) return;
    const R nan = (R)__int_as_float(0x7fc00000);
    const int b = Ar::rings && A.out_du && A.ring ? 1 : 0;
    for (int y = r == 0 ? -b : r; y <= (r == h - 1 ? r + b : r); ++y)
        for (int c = warp / M - b; c < w + b; c += NU) {
            const long long o = A.out_du ? f * A.out_fs + (long long)y * A.out_rs + c : f * A.st_fs + r + (long long)(r + c) * A.g.P;
            (A.out_du ? A.out_du : A.du)[o] = nan;
            (A.out_du ? A.out_dv : A.dv)[o] = nan;
        }
}

// The chained solver, one step of the wavefront divided among warps (see the
// head of frg_sor64.cu).  MB: CTAs per SM that the registers are to allow.
// Ar: the arithmetic (types, the fold of a pixel's coefficients, a pixel's update).
template <class Ar, int M, int NU, int FC, int MB>
__global__ void __launch_bounds__(32 * SplitRoles<M, NU, FC>::warps, MB) k_sor_split(typename Ar::Args A, PassTable T)
{
    using R = typename Ar::T;
    using R2 = typename Ar::T2;
    using SM = SplitSmem<R, M>;
    constexpr int K = Ar::K;
    using Roles = SplitRoles<M, NU, FC>;
    constexpr int G = kGMax;
    constexpr int S = kRingSlots;
    constexpr int ROWS = SM::rows, PL = SM::plane, SR = ROWS + 1, BUF = SM::buf, WU = Roles::WU;
    extern __shared__ __align__(16) unsigned char split_sm[];
    R2* ring = reinterpret_cast<R2*>(split_sm);  // planes kA, kB, kS
    constexpr int kA = 0, kB = PL, kS = 2 * PL;
    R2* bufs = ring + 3 * PL;
    R* ringd = reinterpret_cast<R*>(bufs + G * 3 * BUF);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(ringd + PL);
    int* gave_up = reinterpret_cast<int*>(bars + 2 * M * S + 2);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nc = A.nc;
    const int cta = (int)(blockIdx.x % nc);
    const int f = (int)(blockIdx.x / nc);
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
    const unsigned edge_bytes = (above ? G * sizeof(R2) : 0) + (below ? (G - 1) * sizeof(R2) : 0);
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

    R* odu = A.out_du ? A.out_du + f * A.out_fs : nullptr;
    R* odv = A.out_du ? A.out_dv + f * A.out_fs : nullptr;
    int total = 0;
    for (int p = 0; p < T.n; ++p) total += pass_span(w, T.pk[p]);
    const int nsteps = total + h - 1;
    bool dead = false;
    Cursor cur;
    cur.init(T, w);

    if (!update && warp != Roles::wait && warp != Roles::idle) {
        // ------------------------------------------------------------ fold
        const int fj = Roles::fold(warp) / M;
        const R* Jr = A.J + f * A.J_fs;
        const R* Wr = A.W + f * A.W_fs;
        const R* lapr = A.lap + f * A.lap_fs;
        R* coefr = A.coef + f * A.coef_fs;
        const R* dur = A.du + f * A.st_fs + r;
        const R* dvr = A.dv + f * A.st_fs + r;
        // a plane's start is the same for the whole CTA, the byte offset in it (below 2^32) the lane's own
        auto at = [](auto* plane, unsigned bytes) { return reinterpret_cast<decltype(plane)>((uintptr_t)plane + bytes); };
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
            cur.seek(T, w, s - r);
            const int c = s - r - cur.start, pk = cur.pk, o = (r + c) * P;
            const bool in_level = row_ok && (unsigned)c < (unsigned)w;
            FoldIn<R, K> in;
            R su = 0, sv = 0;
            if (in_level) {
                if (!(pk & kPkZero)) {
                    su = dur[o];
                    sv = dvr[o];
                }
                const unsigned b = (unsigned)(r + o) * (unsigned)sizeof(R);  // byte offset in a plane
                if (pk & kPkCoef) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) in.j[q] = *at(coefr + q * pl, b);
                } else {
#pragma unroll
                    for (int q = 0; q < 6 * K; ++q) in.j[q] = __ldg(at(Jr + q * pl, b));
                    const R* wsrc = Ar::tick_weights && (pk & kPkTick) ? Wr + K * pl : Wr;  // W * a_data on a tick
#pragma unroll
                    for (int k = 0; k < K; ++k) in.w[k] = __ldg(at(wsrc + k * pl, b));
                    in.lu = __ldg(at(lapr, b));
                    in.lv = __ldg(at(lapr + pl, b));
                }
            }
            const int ro = slot * SR + row;
            const R2 st = Ar::pair(su, sv);
            ring[kS + ro] = st;
            st_async_if(sends, halo + slot * SR * (int)sizeof(R2), st, halo_bar + slot * 8);
            if (in_level) {
                const typename Ar::Coef cf = Ar::fold(A, pk, in, su, sv);
                if (pk & kPkStore) {
                    R* cw = coefr + r + o;
                    cw[0] = cf.A12;
                    cw[pl] = cf.BU;
                    cw[2 * pl] = cf.BV;
                    cw[3 * pl] = cf.iDu;
                    cw[4 * pl] = cf.iDv;
                }
                ring[kA + ro] = Ar::pair(cf.A12, cf.BU);
                ring[kB + ro] = Ar::pair(cf.BV, cf.iDu);
                ringd[ro] = cf.iDv;
            }
            __syncwarp();
            if (lane == 0) {
                if (gets)
                    mbar_arrive_expect(full_bar(strip, slot), sizeof(R2));
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
        const bool first_row = r == 0, last_row = r == h - 1;
        const unsigned columns = row_ok ? (unsigned)w : 0u;
        // edge rows to the neighbouring CTAs: the last row's values go below, the first row's above
        const bool send_dn = below && row == ROWS - 1, send_up = above && row == 0;
        unsigned ebuf = smem_addr(bufs + (send_dn ? 0 : ROWS + 1)), ebar = edge_bar(0);
        if (send_dn || send_up) {
            const int peer = send_dn ? cta + 1 : cta - 1;
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(ebuf) : "r"(peer));
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(ebar) : "r"(peer));
        }
        R2 lf[NG], own[NG];  // the values left of the current pixel, and the pixel's own
        R2* myring = ring + row;
        int co[NG];               // ring offset of iteration i's pixel
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            lf[i] = own[i] = Ar::pair(0, 0);
            co[i] = (unsigned)(-2 * (g0 + i * NU)) % S * SR;
        }
        auto next_slot = [&](int o) { return o == (S - 1) * SR ? 0 : o + SR; };
        int so = 0, so1 = SR;                // state slots of steps s and s + 1
        int b0 = 0, b1 = 2 * BUF, b2 = BUF;  // the buffers of steps s, s - 1, s - 2
        R* sdu = A.du + f * A.st_fs + r;
        R* sdv = A.dv + f * A.st_fs + r;
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
                const R2* base = gi == 0 ? myring + kS : bufs + (gi - 1) * 3 * BUF + row + 1;
                const R2* before = base + (gi == 0 ? so : b2);
                const R2* prev = base + (gi == 0 ? so1 : b1);
                R2* mybuf = bufs + gi * 3 * BUF + row + 1;
                // border copies: the neighbour outside is the pixel's own value before the update
                const R2 rt = *(c == w - 1 ? before : prev);
                const bool valid = gi < Gp && (unsigned)c < columns;
                R2 n = lf[i];
                if (valid) {
                    const R2 dn = *(last_row ? before : prev + 1);
                    const R2 up = *(first_row ? before : mybuf + b1 - 1);
                    const R2 ow = own[i];
                    n = Ar::point(A, ow, up, dn, c == 0 ? ow : lf[i], rt, myring[kA + co[i]], myring[kB + co[i]],
                                  ringd[row + co[i]]);
                    if (gi == Gp - 1) {
                        if (cur.p < T.n - 1 || !odu) {
                            sdu[(d0 - 2 * gi) * P] = n.x;
                            sdv[(d0 - 2 * gi) * P] = n.y;
                        } else {
                            const long long o = (long long)r * A.out_rs + c;
                            odu[o] = n.x;
                            odv[o] = n.y;
                            if (Ar::rings && A.ring && (c == 0 || c == w - 1 || r == 0 || r == h - 1))
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
                st_async_if((send_dn || (send_up && gi + 1 < G)) && s + 1 < nsteps, ebuf + (gi * 3 * BUF + b0) * (int)sizeof(R2), n, ebar + (s & 1) * 8);
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
    // A wait ran out: this CTA's rows are void, and with them what the neighbouring CTAs made of its edge rows.
    if (dead)
        for (int i = 0; i < nc; ++i) st_cluster(smem_addr(gave_up), i, 1);
    sync_all();  // no CTA leaves while another may still write into its shared memory
    if (*gave_up) void_rows<Ar, M, NU>(A);
}

constexpr int kMaxDevices = 64;

template <class Ar, int M, int NU, int FC, int MB>
struct SplitLaunch {
    static constexpr size_t smem = SplitSmem<typename Ar::T, M>::bytes;
    static const void* kernel() { return (const void*)k_sor_split<Ar, M, NU, FC, MB>; }
    static int ctas(const DiagGeom& g) { return (g.P / 32 + M - 1) / M; }
    static cudaError_t prepare(int nc)
    {
        const cudaError_t e = ensure_max_dyn_smem(kernel(), 232448);
        return e == cudaSuccess && nc > 8 ? ensure_nonportable_clusters(kernel()) : e;
    }
    static void config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, unsigned grid, int nc, size_t bytes)
    {
        *cfg = cudaLaunchConfig_t{};
        cfg->gridDim = dim3(grid);
        cfg->blockDim = dim3(32 * SplitRoles<M, NU, FC>::warps);
        cfg->dynamicSmemBytes = bytes;
        at->id = cudaLaunchAttributeClusterDimension;
        at->val.clusterDim.x = (unsigned)nc;
        at->val.clusterDim.y = 1;
        at->val.clusterDim.z = 1;
        cfg->attrs = at;
        cfg->numAttrs = nc > 1 ? 1 : 0;
    }
    // Frames the device holds at a time with `per_sm` CTAs per SM (1 or MB), as the driver counts them; a device
    // property, asked for once per device and cluster size.  0: cannot tell.
    static int frames_at_once(int dev, int nc, int per_sm)
    {
        static std::atomic<int> known[kMaxDevices][2][kMaxSplitCluster + 1];
        if (dev < 0 || dev >= kMaxDevices || nc < 1 || nc > kMaxSplitCluster) return 0;
        std::atomic<int>& k = known[dev][per_sm == 1][nc];
        int v = k.load(std::memory_order_relaxed);
        if (v == 0 && prepare(nc) == cudaSuccess) {
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute at;
            // one CTA per SM: as much shared memory as no two can have
            config(&cfg, &at, (unsigned)(nc * 1024), nc, per_sm == 1 ? std::max<size_t>(smem, 120 * 1024) : smem);
            if (nc == 1) {
                int per = 0, n = 0;
                if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel(), (int)cfg.blockDim.x, cfg.dynamicSmemBytes) ==
                        cudaSuccess &&
                    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
                    v = per * n;
            } else if (cudaOccupancyMaxActiveClusters(&v, kernel(), &cfg) != cudaSuccess) {
                v = 0;
                cudaGetLastError();  // the caller's next check is for its own launches
            }
            k.store(v, std::memory_order_relaxed);
        }
        return v;
    }
    // The launch's time in 32-row strips per SM: full rounds of CTAs, then what is left of the frames.
    static int cost(int dev, const DiagGeom& g, int n_frames)
    {
        const int nc = ctas(g), all = frames_at_once(dev, nc, MB), one = frames_at_once(dev, nc, 1);
        if (all < 1 || one < 1) return 0x7fffffff;
        const int rest = n_frames % all;
        return n_frames / all * M * MB + (rest == 0 ? 0 : M * (rest <= one ? 1 : MB));
    }
    static cudaError_t run(typename Ar::Args A, const PassTable& T, int n_frames, cudaStream_t st)
    {
        A.ahead = fold_ahead(A.g.w);
        A.nc = ctas(A.g);
        if (A.nc > kMaxSplitCluster || (long long)n_frames * A.nc > 0x7fffffffLL) return cudaErrorInvalidValue;
        const cudaError_t e = prepare(A.nc);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        config(&cfg, &at, (unsigned)(n_frames * A.nc), A.nc, smem);
        cfg.stream = st;
        return cudaLaunchKernelEx(&cfg, k_sor_split<Ar, M, NU, FC, MB>, A, T);
    }
};

// launch(m) with m strips per CTA.  A device that cannot schedule a cluster of over 8
// CTAs refuses the launch (nothing ran, and the error is not sticky): taller CTAs give
// the same bits in at most 8, up to 1024 rows.
template <class Launch>
cudaError_t launch_or_taller(int strips, int m, Launch launch)
{
    cudaError_t e = launch(m);
    const int taller = strips_per_cta(strips, kPortableCluster);
    if (e != cudaSuccess && (strips + m - 1) / m > kPortableCluster && taller > m) {
        cudaGetLastError();
        e = launch(taller);
    }
    return e;
}

}  // namespace

}  // namespace frg
