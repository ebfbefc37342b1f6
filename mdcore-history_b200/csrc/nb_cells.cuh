// Interface of the cell sweep (nb_cells.cu): its launch parameters, shared-memory sizes and
// unit bound.
#pragma once
#include "nb_device.cuh"

namespace nb {

constexpr int kCellTasks = 31;           // tasks of one cell at most (one lane each)
constexpr int kCellSlotBits = 27;        // bits of a slot number in a list entry, its task above

struct CellParams {
    Params p;
    const int2* units;          // cell, strip | strips << 8 | share << 16 | shares << 24
    const int* nunits;          // may exceed units_cap (a status bit is set then)
    int units_cap;              // room in units
    int* head;                  // queue head
    const int* toff;            // tasks of cell c (as its ci): [toff[c], toff[c + 1])
    const TaskRec* tasks;
    const float4* tshift;
    const float2* cscale;       // sort scale and bias per cell (candidate counts)
    const int* count_cand;      // nonzero: count the sorted sweep's candidates
    int copies;                 // interleaved copies of the tables in shared memory
    float axes[13][3];          // sort axes (candidate counts)
    float neg_zero = -0.0f;     // square2's addend, a value the assembler does not know
};

// Most units of nslots particle slots in ncells cells of at most cap particles and maxtasks
// tasks each.
size_t cell_units_bound(size_t nslots, int ncells, int cap, int maxtasks);
// Worker warps per block, interleaved table copies and shared memory for tables of ncoef floats
// (0: read from global memory), npots tables and mt types; false when they do not fit.
bool cell_sweep_shape(int rows, int ncoef, int npots, int mt, int* nw, int* copies, size_t* smem);

// Clears the queue words (queue head, number of units), lists the units of the cells' current
// counts and sweeps them: nw warps per block, one block per SM.  rows: i particles of a unit at
// most, 24 or 32.  tab: table mode (kTabShared, kTabOne, kTabGlobal).  units: C.units, with room
// for C.units_cap; units past it are dropped with kStatusCellOverflow.  The kernels' attributes
// are set unless the stream is being captured.
cudaError_t launch_cell_sweep(const CellParams& C, int ncells, int rows, int2* units, bool has_excl, int tab, int nw,
                              size_t smem, int grid, bool capturing, cudaStream_t s);

// Counts the sorted sweep's candidates when *C.count_cand (one block per SM).
cudaError_t launch_cell_count(const CellParams& C, int grid, cudaStream_t s);

}  // namespace nb
