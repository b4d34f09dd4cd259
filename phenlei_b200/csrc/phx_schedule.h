// Host-side schedule of the LU-SGS dataflow sweeps (phx_schedule.cpp).
#pragma once
#include <vector>

namespace phx {

// The cells' faces in the reference's numbering: faces of cell c in the
// reference's face order are c2f[off[c] .. off[c + 1]); faces below nBFace are
// boundary faces.
struct SweepGraph {
    int nCell, nBFace;
    const int *off, *c2f;
    const int *left, *right;
};

// One sweep as rows of kSweepSlots cells per warp.  Warp w runs rows
// [rowOff[w], rowOff[w + 1]) in order; slot s of row r holds cell[r * kSweepSlots
// + s] (reference number, -1: idle) with flags: number of entries served by this
// row (0..kSweepLanes) | kSweepFirst | kSweepLast (a cell with more neighbours
// than lanes takes consecutive rows of its slot).  Lane k of the slot serves
// ent[(r * kSweepSlots + s) * kSweepLanes + k]: the neighbour's position in the
// cell's face list (-1: none), and loc: the slot of the warp's shared memory
// that holds the neighbour's result (-1: its record in memory is polled).  The
// row's own results go to shared-memory slots store[r] * kSweepSlots + s.
struct SweepRows {
    int nWarps = 0;
    std::vector<int> rowOff, store;
    std::vector<int> cell, flags, ent, loc;
};

SweepRows build_sweep(const SweepGraph &g, bool forward, int maxWarps);

}  // namespace phx
