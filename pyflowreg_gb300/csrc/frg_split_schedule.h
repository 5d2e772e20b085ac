// The schedule of the split chained SOR: which pass and pixel a step of a row is,
// and how far its fold may run ahead of its update.  Plain integer rules, without
// device code: tests/split_model.cpp replays the kernels' waits with them on the CPU.
#pragma once

#ifdef __CUDACC__
#define FRG_HD __host__ __device__ __forceinline__
#else
#define FRG_HD inline
#endif

namespace frg {

constexpr int kGMax = 5;       // SOR iterations pipelined per wavefront pass
constexpr int kMaxChain = 64;  // passes of a level

constexpr int kRingSlots = 16;  // ring slots: a pixel's coefficients are read for 2 (G - 1) + 1 = 9 steps
constexpr int kRingUse = 2 * (kGMax - 1);
constexpr int kFoldAhead = kRingSlots - kRingUse;  // most steps a fold may run ahead of the update

constexpr int kMaxSplitStrips = 64;   // strips of 32 rows of a level
constexpr int kMaxSplitCluster = 16;  // CTAs of a frame (over 8: the non-portable opt-in)
constexpr int kPortableCluster = 8;

// Strips per CTA (1, 2 or 4), the fewest with which a level's CTAs are a cluster of at
// most `most`; 0: none is enough.
FRG_HD int strips_per_cta(int strips, int most)
{
    for (int m = 1; m <= 4; m *= 2)
        if ((strips + m - 1) / m <= most) return m;
    return 0;
}

struct PassTable {
    int n;
    int pk[kMaxChain];  // G << 8 | store << 3 | coef << 2 | tick << 1 | zero
};

// Steps a row spends in a pass.  After a single iteration one step more, so that
// the step before a row's first pixel of the next pass (which takes that
// pixel's value as its right neighbour) is free.
FRG_HD int pass_span(int w, int pk)
{
    const int n = pk >> 8;
    return w + (n > 1 ? 2 * (n - 1) : 1);
}

// Steps the fold of a row of w columns may run ahead of the update.  A pixel's state
// is stored w steps (w + 1 after a single iteration) before the next pass's fold
// reads it, so at most w.  And at least three: the end of step s waits for the fold
// of step s + 2, which must not wait for the end of step s in turn (so w >= 3).
FRG_HD int fold_ahead(int w) { return w < kFoldAhead ? w : kFoldAhead; }

// A row's place in the chain of passes at local time tau.
struct Cursor {
    int p, start, end, pk;
    FRG_HD void init(const PassTable& T, int w)
    {
        p = 0;
        start = 0;
        pk = T.pk[0];
        end = pass_span(w, pk);
    }
    FRG_HD void next(const PassTable& T, int w)
    {
        ++p;
        start = end;
        pk = T.pk[p];
        end = start + pass_span(w, pk);
    }
    // For a caller that comes by every step: no pass is shorter than that.
    FRG_HD void advance(const PassTable& T, int w, int tau)
    {
        if (tau >= end && p < T.n - 1) next(T, w);
    }
    // For a fold warp, whose steps lie FC apart: a pass of few columns may lie between two of them.
    FRG_HD void seek(const PassTable& T, int w, int tau)
    {
        while (tau >= end && p < T.n - 1) next(T, w);
    }
};

}  // namespace frg
