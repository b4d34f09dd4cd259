// Schedule of the LU-SGS dataflow sweeps (kernels: phx_kernels.cu, phx_sa.cu).
//
// A sweep is a triangular solve in the reference's cell order: a cell needs the
// results of its neighbours on the sweep's side.  A result that travels from
// one SM to another through L2 takes several times as long as a cell's
// arithmetic, so the schedule keeps dependent cells on the warp that computed
// their neighbour: every cell follows one of its neighbours in that
// neighbour's slot (a chain; on a mesh numbered along i, the pencils along i),
// and eight chains make a warp, which hands the results of its last eight rows on
// in shared memory (chains of a warp are often two or three levels apart; with
// one row a chain kept, the 1M-cell bump's warps read their own results through
// L2, and its sweeps took 754 and 537 us, NS and SA, instead of 608 and 441).
// A chain that begins joins the warp of its nearest neighbour in the numbering,
// or the warp that this one's chains spill into, where the distance is at most 1.5
// times that of the chains already there (on the same mesh: eight pencils next to
// one another in j, none from another plane; at twice the distance the prism
// layers' warps mix and the backward sweep of the 1M-cell bump takes 318 us
// instead of 245, below 1.5 grown numberings fill their warps half), so that warps mostly depend on one
// another in one direction: a warp that has fallen behind the ones it reads from
// finds their results already there and runs at the speed of its arithmetic.
// The latency between SMs is then paid once per warp boundary on the way through
// the mesh and not once per level.
//
// Order: every cell has a level above those of its neighbours on the sweep's
// side, a row holds cells of one level, and a warp's rows ascend in level, so
// the unfinished row of the lowest level can always run and the waits cannot
// cycle, as long as all warps are resident.
#include "phx_schedule.h"

#include <algorithm>
#include <cstdlib>

#include "phx_internal.h"

namespace phx {

SweepRows build_sweep(const SweepGraph &g, bool forward, int maxWarps)
{
    const int nc = g.nCell;
    SweepRows out;
    // per cell: its neighbours on the sweep's side, in the cell's face order,
    // with their positions in the cell's face list; levels
    std::vector<int> noff(nc + 1, 0), nbr, pos, lev(nc, 0);
    nbr.reserve(g.off[nc] / 2);
    pos.reserve(g.off[nc] / 2);
    for (int c = 0; c < nc; ++c) {
        for (int j = g.off[c]; j < g.off[c + 1]; ++j) {
            const int f = g.c2f[j];
            if (f < g.nBFace) continue;
            const int o = g.left[f] == c ? g.right[f] : g.left[f];
            if (forward ? o < c : o > c) { nbr.push_back(o); pos.push_back(j - g.off[c]); }
        }
        noff[c + 1] = (int)nbr.size();
    }
    int nlev = 0;
    for (int i = 0; i < nc; ++i) {
        const int c = forward ? i : nc - 1 - i;
        int l = 0;
        for (int j = noff[c]; j < noff[c + 1]; ++j) l = std::max(l, lev[nbr[j]] + 1);
        lev[c] = l;
        nlev = std::max(nlev, l + 1);
    }
    std::vector<int> loff(nlev + 1, 0), cells(nc);
    for (int c = 0; c < nc; ++c) loff[lev[c] + 1]++;
    for (int l = 0; l < nlev; ++l) loff[l + 1] += loff[l];
    {
        std::vector<int> fill(loff.begin(), loff.end() - 1);
        for (int i = 0; i < nc; ++i) {
            const int c = forward ? i : nc - 1 - i;
            cells[fill[lev[c]]++] = c;
        }
    }

    // chains: the slot of every cell (chain warp * kSweepSlots + slot), level by level
    std::vector<int> slot(nc, -1), endCell, endLev, claim;   // per slot: last cell, its level, claimant at this level
    std::vector<int> spill, reach;   // per chain warp: the one its chains spill into (-1: none); distance of its chains
    int root = -1;                   // the warp of chains without a neighbour
    std::vector<int> waits(nc, 0);   // cells that still wait for a cell
    for (int o : nbr) ++waits[o];
    // a slot whose chain nothing follows any more, or has not for two levels
    auto free_slot = [&](int v, int l) {
        for (int s = v * kSweepSlots; s < (v + 1) * kSweepSlots; ++s)
            if (endLev[s] < 0 || (endLev[s] < l && (waits[endCell[s]] == 0 || endLev[s] < l - 2))) return s;
        return -1;
    };
    // the slot of the neighbour nearest in the numbering that ends its chain
    auto follow = [&](int c, int l) {
        int b = -1;
        for (int j = noff[c]; j < noff[c + 1]; ++j) {
            const int s = slot[nbr[j]];
            if (endCell[s] == nbr[j] && endLev[s] < l &&
                (b < 0 || std::abs(nbr[j] - c) < std::abs(endCell[b] - c)))
                b = s;
        }
        return b;
    };
    std::vector<int> rest, put;
    for (int l = 0; l < nlev; ++l) {
        // of several cells that would follow the same neighbour the nearest does
        rest.clear();
        put.clear();
        for (int i = loff[l]; i < loff[l + 1]; ++i) {
            const int c = cells[i], s = follow(c, l);
            slot[c] = s;
            if (s >= 0 && (claim[s] < 0 || std::abs(endCell[s] - c) < std::abs(endCell[s] - claim[s]))) claim[s] = c;
        }
        for (int i = loff[l]; i < loff[l + 1]; ++i) {
            const int c = cells[i], s = slot[c];
            if (s >= 0 && claim[s] == c) put.push_back(c);
            else rest.push_back(c);
        }
        for (int c : put) { endLev[slot[c]] = l; claim[slot[c]] = -1; }
        for (int c : rest) {
            int s = follow(c, l);
            if (s < 0) {
                int near = -1;
                for (int j = noff[c]; j < noff[c + 1]; ++j)
                    if (near < 0 || std::abs(nbr[j] - c) < std::abs(near - c)) near = nbr[j];
                const int d = near < 0 ? 0 : std::abs(near - c), from = near < 0 ? -1 : slot[near] / kSweepSlots;
                const bool like = from < 0 || reach[from] == 0 || 2LL * d <= 3LL * reach[from];
                if (like && from >= 0) {
                    s = free_slot(from, l);
                    if (s >= 0 && reach[from] == 0) reach[from] = d;
                }
                const int next = from < 0 ? root : spill[from];
                if (s < 0 && like && next >= 0) s = free_slot(next, l);
                if (s < 0) {
                    const int v = (int)spill.size();
                    if (like) (from < 0 ? root : spill[from]) = v;
                    reach.push_back(like && from >= 0 ? reach[from] : 0);
                    spill.push_back(-1);
                    endCell.resize(endCell.size() + kSweepSlots, -1);
                    endLev.resize(endLev.size() + kSweepSlots, -1);
                    claim.resize(claim.size() + kSweepSlots, -1);
                    s = v * kSweepSlots;
                }
            }
            slot[c] = s;
            endLev[s] = l;
        }
        for (int i = loff[l]; i < loff[l + 1]; ++i) {
            const int c = cells[i];
            endCell[slot[c]] = c;
            for (int j = noff[c]; j < noff[c + 1]; ++j) --waits[nbr[j]];
        }
    }

    auto parts = [&](int c) { return std::max(1, (noff[c + 1] - noff[c] + kSweepLanes - 1) / kSweepLanes); };
    // the cells of a level by chain warp
    auto order = [&]() {
        for (int l = 0; l < nlev; ++l)
            std::sort(cells.begin() + loff[l], cells.begin() + loff[l + 1], [&](int a, int b) { return slot[a] < slot[b]; });
    };
    // calls fn(chain warp, first, last, rows) for every chain warp with cells at a level, in the order of the levels
    auto groups = [&](auto &&fn) {
        for (int l = 0; l < nlev; ++l)
            for (int a = loff[l], b; a < loff[l + 1]; a = b) {
                const int v = slot[cells[a]] / kSweepSlots;
                int need = 1;
                for (b = a; b < loff[l + 1] && slot[cells[b]] / kSweepSlots == v; ++b)
                    need = std::max(need, parts(cells[b]));
                fn(v, a, b, need);
            }
    };
    order();
    // Where a numbering has no chains to follow they leave most slots idle, and the
    // warps run many more rows than there are levels: full rows of each level then,
    // dealt out over the warps.  Both have to hold.  With at most about a row a level
    // on the longest warp, idle slots cost nothing: each level then takes a row's
    // time, and dealt out a hop through L2 as well.  Both NS sweeps, mixed, chains
    // against dealt-out rows, with rows of the longest warp a level:
    //   ducts of 4000x1x1 (1.0) 2489 and 3723 us, 200x3x2 (1.0) 159 and 217,
    //   300x4x4 (1.0) 231 and 334, a block of 16x8x2 (1.0) 40 and 49;
    //   numbered at random: 8k hexahedra (1.6) 43 and 49, 48k tetrahedra (1.2) 42
    //   and 44, 162k tetrahedra (2.3) 65 and 56, 524k hexahedra (8) 249 and 124;
    //   66k hexahedra, FP64: forward (1.9) 54 and 45, backward (1.7) 42 and 42.
    const int chainWarps = std::max(1, std::min(maxWarps, (int)spill.size()));
    std::vector<int> warpRows(chainWarps, 0);
    size_t rows = 0;
    groups([&](int v, int, int, int need) { rows += need; warpRows[v % chainWarps] += need; });
    const int longest = *std::max_element(warpRows.begin(), warpRows.end());
    if (rows * kSweepSlots > 2 * (size_t)nc && 4LL * longest > 7LL * nlev) {
        spill.clear();
        for (int l = 0; l < nlev; ++l) {
            std::sort(cells.begin() + loff[l], cells.begin() + loff[l + 1],
                      [&](int a, int b) { return parts(a) != parts(b) ? parts(a) > parts(b) : a < b; });
            for (int i = loff[l]; i < loff[l + 1]; ++i) {
                if ((i - loff[l]) % kSweepSlots == 0) spill.push_back(-1);
                slot[cells[i]] = ((int)spill.size() - 1) * kSweepSlots + (i - loff[l]) % kSweepSlots;
            }
        }
        order();
    }

    // rows: chain warp v runs on warp v % nWarps; a warp's shared memory holds the
    // results of its last kSweepLocal rows
    const int nv = (int)spill.size(), nw = std::max(1, std::min(maxWarps, nv));
    out.nWarps = nw;
    out.rowOff.assign(nw + 1, 0);
    groups([&](int v, int, int, int need) { out.rowOff[v % nw + 1] += need; });
    for (int w = 0; w < nw; ++w) out.rowOff[w + 1] += out.rowOff[w];
    const size_t nrow = out.rowOff[nw];
    out.store.assign(nrow, 0);
    out.cell.assign(nrow * kSweepSlots, -1);
    out.flags.assign(nrow * kSweepSlots, 0);
    out.ent.assign(nrow * kSweepSlots * kSweepLanes, -1);
    out.loc.assign(nrow * kSweepSlots * kSweepLanes, -1);
    std::vector<int> next(out.rowOff.begin(), out.rowOff.end() - 1);
    std::vector<int> held((size_t)nw * kSweepLocal * kSweepSlots, -1);   // cell whose result a shared-memory slot holds
    std::vector<int> place(nc, -1);                                      // shared-memory slot of a cell's result
    groups([&](int v, int a, int b, int need) {
        const int w = v % nw, r0 = next[w];
        int *h = &held[(size_t)w * kSweepLocal * kSweepSlots];
        next[w] += need;
        for (int p = 0; p < need; ++p) {
            const int lr = (r0 + p - out.rowOff[w]) % kSweepLocal;
            out.store[r0 + p] = lr;
            for (int i = a; i < b; ++i) {
                const int c = cells[i], np = parts(c);
                if (p >= np) continue;
                const size_t at = (size_t)(r0 + p) * kSweepSlots + slot[c] % kSweepSlots;
                const int j0 = noff[c] + p * kSweepLanes, j1 = std::min(noff[c + 1], j0 + kSweepLanes);
                out.cell[at] = c;
                out.flags[at] = std::max(0, j1 - j0) | (p == 0 ? kSweepFirst : 0) | (p == np - 1 ? kSweepLast : 0);
                for (int j = j0; j < j1; ++j) {
                    out.ent[at * kSweepLanes + (j - j0)] = pos[j];
                    const int q = place[nbr[j]];
                    if (slot[nbr[j]] / kSweepSlots % nw == w && h[q] == nbr[j]) out.loc[at * kSweepLanes + (j - j0)] = q;
                }
            }
            for (int i = a; i < b; ++i)   // results are stored after the row's reads
                if (parts(cells[i]) == p + 1) {
                    place[cells[i]] = lr * kSweepSlots + slot[cells[i]] % kSweepSlots;
                    h[place[cells[i]]] = cells[i];
                }
        }
    });
    return out;
}

}  // namespace phx
