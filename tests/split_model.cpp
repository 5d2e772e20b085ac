// A CPU model of the split chained SOR (k_sor_split) over the kernels' own schedule
// rules: who waits for whom, and which pixel each fold takes.
//
// Waits of a CTA.  The fold of step s waits for the end of step s - ahead.  A strip's
// slot of step s is full once its fold is done (the last strip's also needs the first
// row's state from the CTA below, which that CTA's fold of step s sends).  The end of
// step s waits for the slots of step s + 2 and for the rows that the neighbouring CTAs
// send in step s, which they do once their step s - 1 has ended.  Every condition
// stays true once it holds, so running whatever can run until nothing can decides
// whether any order gets stuck.
#include "frg_split_schedule.h"

#include <vector>

using namespace frg;

namespace {

struct Run {
    int h, w, M, FC;
    PassTable T;
    int start[kMaxChain + 1];
    int G(int p) const { return T.pk[p] >> 8; }
    int nsteps() const { return start[T.n] + h - 1; }
};

void make_starts(Run& R)
{
    R.start[0] = 0;
    for (int p = 0; p < R.T.n; ++p) R.start[p + 1] = R.start[p] + pass_span(R.w, R.T.pk[p]);
}

bool finishes(const Run& R, int ahead)
{
    const int nc = (R.h + 32 * R.M - 1) / (32 * R.M), N = R.nsteps();
    std::vector<std::vector<char>> folded((size_t)nc * R.M, std::vector<char>(N, 0));
    std::vector<int> next((size_t)nc * R.M * R.FC), done(nc, -1);
    for (size_t i = 0; i < next.size(); ++i) next[i] = (int)(i % R.FC);
    auto full = [&](int cta, int s) {
        if (s >= N) return true;
        for (int st = 0; st < R.M; ++st)
            if (!folded[cta * R.M + st][s]) return false;
        return cta + 1 == nc || folded[(cta + 1) * R.M][s] != 0;
    };
    for (bool moved = true; moved;) {
        moved = false;
        for (size_t i = 0; i < next.size(); ++i) {
            const int strip = (int)(i / R.FC), cta = strip / R.M;
            while (next[i] < N && (next[i] < ahead || done[cta] >= next[i] - ahead)) {
                folded[strip][next[i]] = 1;
                next[i] += R.FC;
                moved = true;
            }
        }
        for (int c = 0; c < nc; ++c)
            while (done[c] + 1 < N) {
                const int s = done[c] + 1;
                if (s == 0 && !(full(c, 0) && full(c, 1))) break;
                if (!full(c, s + 2)) break;
                if (s + 1 < N && ((c > 0 && done[c - 1] < s - 1) || (c + 1 < nc && done[c + 1] < s - 1))) break;
                ++done[c];
                moved = true;
            }
    }
    for (int c = 0; c < nc; ++c)
        if (done[c] != N - 1) return false;
    return true;
}

}  // namespace

extern "C" int split_strips_per_cta(int strips, int most) { return strips_per_cta(strips, most); }

// 0: sound; 1: a wait never ends; 2: a fold takes another pixel than the one that
// enters; 3: a state or stored coefficients are read before they are surely written;
// 4: a ring slot is written while its last contents may still be read.
extern "C" int split_model(int h, int w, int M, int FC, int n, const int* G, const int* continues)
{
    Run R{h, w, M, FC, {}, {}};
    R.T.n = n;
    for (int p = 0; p < n; ++p) R.T.pk[p] = G[p] << 8 | (continues[p] ? 4 : 0);
    make_starts(R);
    const int ahead = fold_ahead(w), N = R.nsteps();
    // the slot of step s is written once step s - ahead has ended; step s - kRingSlots's coefficients are read until
    // step s - kRingSlots + 2 (kGMax - 1), its states until step s - kRingSlots
    if (-kRingSlots + 2 * (kGMax - 1) > -ahead) return 4;
    for (int r = 0; r < h; r = r + 1 < h && r + 33 >= h ? h - 1 : r + 1 + 31 * (r > 0))
        for (int j = 0; j < FC; ++j) {
            Cursor cur;
            cur.init(R.T, w);
            for (int s = j; s < N; s += FC) {
                const int tau = s - r;
                cur.seek(R.T, w, tau);
                int p = 0;
                while (p + 1 < n && tau >= R.start[p + 1]) ++p;
                const int c = tau - R.start[p];
                const bool in = tau >= 0 && c < w;
                const int cc = tau - cur.start;
                if (in != (cc >= 0 && cc < w) || (in && (cur.p != p || cc != c))) return 2;
                if (!in) continue;
                // surely done by now: the end of step s - ahead, and what it waited for
                if (p > 0 && r + R.start[p - 1] + c + 2 * (R.G(p - 1) - 1) > s - ahead) return 3;
                if (continues[p]) {
                    int q = p;
                    while (q > 0 && continues[q]) --q;
                    if (r + R.start[q] + c > s - ahead + 2) return 3;
                }
            }
        }
    return finishes(R, ahead) ? 0 : 1;
}
