// Replays a sweep schedule (phenlei_b200/csrc/phx_schedule.cpp) on the host:
// warps take turns, one row at a time, a row runs when its polled neighbours are
// done, and the shared-memory slots are kept as the kernels keep them.  Returns
// 0, or the number of the first rule that does not hold.
#include <algorithm>
#include <vector>

#include "../phenlei_b200/csrc/phx_internal.h"
#include "../phenlei_b200/csrc/phx_schedule.h"

extern "C" int replay(int nc, int nb, const int *off, const int *c2f, const int *left, const int *right, int forward,
                      int maxWarps, int *nWarps)
{
    using namespace phx;
    const SweepGraph g{nc, nb, off, c2f, left, right};
    const SweepRows s = build_sweep(g, forward != 0, maxWarps);
    *nWarps = s.nWarps;
    if (s.nWarps < 1 || s.nWarps > maxWarps || (int)s.rowOff.size() != s.nWarps + 1) return 1;
    std::vector<int> done(nc, 0), seen(nc, 0), row(s.rowOff.begin(), s.rowOff.end() - 1);
    std::vector<int> held((size_t)s.nWarps * kSweepLocal * kSweepSlots, -1);
    std::vector<int> last((size_t)s.nWarps * kSweepSlots, -1);   // cell continued by the slot's next row
    for (int left_rows = s.rowOff[s.nWarps]; left_rows > 0;) {
        int ran = 0;
        for (int w = 0; w < s.nWarps; ++w) {
            if (row[w] == s.rowOff[w + 1]) continue;
            const size_t r = row[w];
            int *h = &held[(size_t)w * kSweepLocal * kSweepSlots];
            bool ready = true;
            for (int i = 0; i < kSweepSlots; ++i) {
                const size_t at = r * kSweepSlots + i;
                const int c = s.cell[at], n = s.flags[at] & 7;
                if (c < 0) continue;
                if (n > kSweepLanes) return 2;
                if (((s.flags[at] & kSweepFirst) == 0) != (last[w * kSweepSlots + i] == c)) return 3;
                for (int k = 0; k < kSweepLanes; ++k) {
                    const int e = s.ent[at * kSweepLanes + k], q = s.loc[at * kSweepLanes + k];
                    if ((e >= 0) != (k < n)) return 4;
                    if (e < 0) continue;
                    const int f = c2f[off[c] + e], o = left[f] == c ? right[f] : left[f];
                    if (f < nb || (forward ? o >= c : o <= c)) return 5;
                    if (q >= 0) {
                        if (q >= kSweepLocal * kSweepSlots || h[q] != o) return 6;
                    } else if (!done[o]) {
                        ready = false;
                    }
                }
            }
            if (!ready) continue;
            for (int i = 0; i < kSweepSlots; ++i) {
                const size_t at = r * kSweepSlots + i;
                const int c = s.cell[at];
                if (c < 0) continue;
                seen[c] += s.flags[at] & 7;
                const bool end = (s.flags[at] & kSweepLast) != 0;
                last[w * kSweepSlots + i] = end ? -1 : c;
                if (!end) continue;
                if (done[c]++) return 7;
                if (s.store[r] < 0 || s.store[r] >= kSweepLocal) return 8;
                h[s.store[r] * kSweepSlots + i] = c;
            }
            ++row[w];
            ++ran;
            --left_rows;
        }
        if (!ran) return 9;   // no row can run
    }
    for (int c = 0; c < nc; ++c) {
        int n = 0;
        for (int j = off[c]; j < off[c + 1]; ++j) {
            const int f = c2f[j];
            if (f >= nb) n += forward ? (left[f] == c ? right[f] : left[f]) < c : (left[f] == c ? right[f] : left[f]) > c;
        }
        if (done[c] != 1 || seen[c] != n) return 10;
    }
    return 0;
}

// Rows of the schedule, warps, rows of the longest warp, and the share of the neighbours
// that a warp's shared memory holds.
extern "C" void shape(int nc, int nb, const int *off, const int *c2f, const int *left, const int *right, int forward,
                      int maxWarps, double *out)
{
    using namespace phx;
    const SweepRows s = build_sweep(SweepGraph{nc, nb, off, c2f, left, right}, forward != 0, maxWarps);
    int longest = 0;
    for (int w = 0; w < s.nWarps; ++w) longest = std::max(longest, s.rowOff[w + 1] - s.rowOff[w]);
    long long held = 0, all = 0;
    for (size_t e = 0; e < s.ent.size(); ++e)
        if (s.ent[e] >= 0) { ++all; held += s.loc[e] >= 0; }
    out[0] = s.rowOff[s.nWarps];
    out[1] = s.nWarps;
    out[2] = longest;
    out[3] = all ? (double)held / all : 1.0;
}
