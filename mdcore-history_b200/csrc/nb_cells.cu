// Cell sweep (sm_100a): the nonbonded forces of one evaluation by units of up to 32 i
// particles of one cell against the j particles of all the cell's tasks at once.  No sort
// keys and no per-task work: what sweep_tuned and sweep_tiled do once per cell pair (queue
// pop, staging, j list, prefix searches, j and i force output) is done once per unit.
//
// A warp takes a unit (cell, strip of up to 24 or 32 of its particles, share of its j
// particles) and
//  1. holds the strip's rows in its shared-memory slice and clears a force accumulator per
//     row and lane;
//  2. walks the j particles of the cell's tasks as one list, 32 per pass, drops those farther
//     than the cutoff from the strip's bounding box and packs the rest;
//  3. tests 32 of those, one per lane, against every row by r^2 = |xi|^2 - 2 xi.xj + |xj|^2
//     (three packed multiply-adds for two rows), with the cutoff widened by the rounding of
//     that form: a bit mask of rows per j.  j with a row left go to one of two lists, by
//     the number of their rows, so that lanes evaluated together have about equally many;
//  4. evaluates 32 list entries, one per lane: every lane walks the rows of its own mask, two
//     at a time in packed FP32 pairs (add/mul/fma.rn.f32x2).  The exact test of the pair
//     (displacement, r^2 and cutoff rounded as in the other sweeps) decides, so the pair set
//     is the same bit for bit.  The j force stays in the lane's registers, the i forces go
//     to the lane's own accumulator of the row: no shuffles and no atomics per pair;
//  5. adds each j's force once per list entry and each row's force once per unit to the
//     fixed-point accumulators.
// The partial sums of a unit depend only on the cells' contents, so forces, energies and
// virials do not depend on the order in which units run.
//
// What bounds it: instruction latency and issue.  512 argon replicas (1.45 M atoms, cells of
// 18-45, 58.8 M pairs): 10.2 warp instructions per pair against the queue form's 19.4, issue
// slots 60 % busy with 2.75 warps per scheduler (the accumulators limit an SM to 12 or 13
// warps), shared-memory pipe 50 %, DRAM idle (95 MB per launch); 0.86 ms per sweep against 1.19
// and no sort (0.13); a resident step 1.47 -> 0.95 ms (0.6 % of it for non-finite rows).  About
// half of the instructions evaluate pairs (two per lane and iteration, 52 % of the lane slots
// carrying one, counted on the CPU: the two lists by number of rows give that, one list gives
// 40 %), a quarter tests rows.  Solvated chains, 12,400 atoms, tables in global memory, charges:
// an evaluation with its candidate count 0.71 -> 0.42 ms.  On cells of 135 particles (water) it
// loses, 0.45 against 0.28 ms per step: every strip walks the whole neighbourhood again.
//
// Precision: a row's force is summed in FP32 over all tasks of its cell, in 32 sums (one per
// lane) that are added pairwise, and converted to fixed point once per unit; the queue form
// converts after every cell pair and strip.  Error of the forces against 64 bits, 2-norm, queue
// (32 i) / queue (8 x 4) / cells / cells24, mean of two seeds in 1e-7: argon 32,000 5.79 / 5.77 /
// 5.76 / 5.77, water 24,000 6.54 / 6.33 / 6.27 / 6.27, slab 1.25 / 1.25 / 1.23 / 1.23, chains of
// 12,400 1.52 / 1.58 / 1.38 / 1.44, of 3,720 1.48 / 1.34 / 1.44 / 1.41: never above the larger of
// the queue form's own two layouts.
// The tables are held in 8 interleaved copies, one per lane of a quarter warp, so that the
// 16-byte reads at random intervals meet no bank conflicts.
#include <algorithm>
#include "nb_tuned.cuh"
#include "nb_cells.cuh"

namespace nb {

constexpr int kCellWarps = 13;           // worker warps of a block at most, one block per SM
constexpr int kCellShare = 16384;        // row tests of a unit before a cell's j list is split
constexpr int kCellRing = 64;            // near list
constexpr int kCellList = 96;            // evaluation lists: up to 31 left of each class and 32 new

// One worker warp's slice of shared memory; ROWS (24 or 32): i particles of a unit at most.
// The accumulators are most of it: 24 rows leave room for 13 warps instead of 12, 32 need fewer
// units for cells of 25 to 32 particles (resident steps with 24 / 32 rows: slab 0.92 / 0.99 ms,
// replicas 1.04 / 0.94; the autotuner times both).
template <int ROWS>
struct CellWarp {
    float acc[3][ROWS][32];         // i force by component, row, lane
    float4 rt[32];                       // row pairs of the test: {-2x, -2x', -2y, -2y'}, {-2z, -2z', |x|^2, |x'|^2}
    float4 sh[kCellTasks + 1];           // per task with particles: shift of cell j, cutoff^2
    int tslot[kCellTasks + 1];           // first slot of its particles less their place in the list
    int tplace[kCellTasks + 1];          // their place in the list
    float4 bx[kCellRing];                // j near the strip: position and type
    float4 ex[kCellList];                // j with rows to evaluate: class 0 from the front, 1 from the back
    float rx[32], ry[32], rz[32], rq[32];
    int rtype[32], rpid[32];
    unsigned bm[kCellRing];              // slot | task << kCellSlotBits
    unsigned em[kCellList], emask[kCellList];
    int epid[kCellList];
};

// ---------------------------------------------------------------- packed FP32 pairs
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// Each component rounded to nearest on its own.
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
// a * a rounded on its own: the assembler was seen to contract mul.rn.f32x2 with a following
// add.rn.f32x2 (a pair at r^2 = 1 + 2^-23 was accepted at a cutoff of 1), so the square is a
// multiply-add with a -0 that it cannot see.
__device__ __forceinline__ f32x2 square2(f32x2 a, f32x2 neg_zero) { return fma2(a, a, neg_zero); }
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// ---------------------------------------------------------------- units
// Strips of at most `rows` particles and shares of the j list of one cell: a function of
// the counts of the cell and its neighbours alone, so an engine has the same units alone and
// in a batch.  Shares: one per kCellShare row tests (large cells: several warps per strip).
__device__ __forceinline__ void cell_split(int n, int nj, int rows, int& strips, int& shares) {
    strips = (n + rows - 1) / rows;
    const long long tests = (long long)((n + strips - 1) / strips) * nj;
    shares = (int)min(255ll, max(1ll, (tests + kCellShare / 2) / kCellShare));
}

__global__ void __launch_bounds__(256) cell_units(const int* __restrict__ ccount, const int* __restrict__ toff,
                                                  const TaskRec* __restrict__ tasks, int ncells, int rows,
                                                  int2* __restrict__ units,
                                                  int* __restrict__ nunits, int cap, unsigned long long* __restrict__ acc,
                                                  const unsigned long long* __restrict__ abort) {
    if (step_aborted(abort)) return;
    const int c = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const int n = c < ncells ? ccount[c] : 0;
    int strips = 0, shares = 0;
    if (n > 0) {
        int nj = 0;
        bool self = false;
        for (int t = toff[c]; t < toff[c + 1]; ++t) {
            if (tasks[t].sid >= 0) nj += ccount[tasks[t].cj];
            else self = true;
        }
        if (nj > 0 || (self && n > 1)) cell_split(n, nj + n, rows, strips, shares);
    }
    const int mine = strips * shares;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    int base = 0;
    if (lane == 31 && incl > 0) base = atomicAdd(nunits, incl);
    base = __shfl_sync(0xffffffffu, base, 31) + incl - mine;
    for (int k = 0; k < mine; ++k) {
        if (base + k >= cap) {           // never within cell_units_bound
            atomicOr(&acc[kAccStatus], (unsigned long long)kStatusCellOverflow);
            return;
        }
        units[base + k] = make_int2(c, (k / shares) | (strips << 8) | ((k % shares) << 16) | (shares << 24));
    }
}

// ---------------------------------------------------------------- pair evaluation
// The tables as the block holds them: chunk k of copy r at 16-byte units k * 2 copies + r
// (centre, 1/halfwidth, c5, c4) and + copies (c3..c0).
struct CellTables {
    const float4* chunk;        // shared: this lane's copy; global tables: unused
    const float4* info;
    const int* potidx;
    int copies;
    float4 one;
};

template <int TAB>
__device__ __forceinline__ void cell_eval_table(const Params& P, const CellTables& S, int pot, float r, float rinv,
                                                float& e, float& f) {
    if (TAB == kTabGlobal) {
        const float4 info = P.potinfo[pot];
        eval_table_fast(P.coef, info, __float_as_int(info.w) >> 20, r, rinv, e, f);
        return;
    }
    const float4 info = TAB == kTabOne ? S.one : S.info[pot];
    const float t = fmaf(r, fmaf(r, info.z, info.y), info.x);
    const int w = __float_as_int(info.w);
    // the unsigned conversion takes negative values and NaN to 0
    const int ind = (int)min(__float2uint_rz(t), (unsigned)(w >> 20)) + ((w & 0xfffff) >> 3);
    const float4* c = S.chunk + ind * (2 * S.copies);
    const float4 c0 = c[0], c1 = c[S.copies];
    const float x = (r - c0.x) * c0.y;
    float ee = fmaf(c0.z, x, c0.w);
    float eff = c0.z;
    eff = fmaf(eff, x, ee); ee = fmaf(ee, x, c1.x);
    eff = fmaf(eff, x, ee); ee = fmaf(ee, x, c1.y);
    eff = fmaf(eff, x, ee); ee = fmaf(ee, x, c1.z);
    eff = fmaf(eff, x, ee); ee = fmaf(ee, x, c1.w);
    e = ee;
    f = eff * c0.y * rinv;
}

__device__ __forceinline__ bool cell_excluded(const Params& P, const IExcl& jx, int ipid) {
    const int d = ipid - jx.pid;
    if ((unsigned)(d - jx.lo) <= (unsigned)jx.span) return (jx.emask >> (d + 16 - (d > 0))) & 1u;
    bool ex = false;
    for (int q = jx.exlo; q < jx.exhi; ++q) ex |= P.exlist[q] == ipid;
    return ex;
}

struct CellSums {
    double e = 0.0, v = 0.0;
    unsigned npairs = 0, nexcl = 0, status = 0;
};

// 32 list entries, one per lane (mask 0: none): all accepted pairs of the lane's j with the
// rows of its mask (row r at bit top - r).
template <bool EX, int TAB, int ROWS>
__device__ __forceinline__ void cell_window(const Params& P, CellWarp<ROWS>& W, const CellTables& S, float4 xj, unsigned meta,
                                            unsigned mask, int jpid, int top, f32x2 nz2, CellSums& R, int lane) {
    const bool live = mask != 0;
    const size_t slot = meta & ((1u << kCellSlotBits) - 1u);
    const float4 sh = W.sh[meta >> kCellSlotBits];
    const float cut2 = sh.w;
    IExcl jx = no_iexcl();
    if (EX && live) jx = load_iexcl(P, jpid);
    float qj = 0.f;
    if (TAB == kTabGlobal && P.ep_pot >= 0 && live) qj = P.qid[jpid];
    // lanes without an entry hold whatever the ring held: neither a type to index a table with
    // nor a position to multiply a zero force by
    if (!live) xj = make_float4(0.f, 0.f, 0.f, 0.f);
    const int prow = TAB == kTabOne ? 0 : __float_as_int(xj.w) * P.max_type;
    const int* potidx = TAB == kTabGlobal ? P.potidx : S.potidx;
    const f32x2 sx = pack2(-sh.x, -sh.x), sy = pack2(-sh.y, -sh.y), sz = pack2(-sh.z, -sh.z);
    const f32x2 jx2 = pack2(-xj.x, -xj.x), jy2 = pack2(-xj.y, -xj.y), jz2 = pack2(-xj.z, -xj.z);
    const f32x2 half = pack2(0.5f, 0.5f), nhalf = pack2(-0.5f, -0.5f), none = pack2(-1.0f, -1.0f);
    f32x2 fx = 0ull, fy = 0ull, fz = 0ull;       // minus the force on j, by row parity
    float* __restrict__ acc = &W.acc[0][0][lane];
    const int iters = ((int)__reduce_max_sync(0xffffffffu, (unsigned)__popc(mask)) + 1) >> 1;
    // the next two rows of the lane's mask (row 0 where there is none) and their positions,
    // read one iteration ahead
    bool nA, nB;
    int qA, qB;
    f32x2 px, py, pz;
    auto next_rows = [&]() {
        nA = mask != 0;
        const int bA = nA ? 31 - __clz(mask) : top;
        mask &= ~(1u << bA);
        nB = mask != 0;
        const int bB = nB ? 31 - __clz(mask) : bA;
        mask &= ~(1u << bB);
        qA = top - bA;
        qB = top - bB;
        px = pack2(W.rx[qA], W.rx[qB]);
        py = pack2(W.ry[qA], W.ry[qB]);
        pz = pack2(W.rz[qA], W.rz[qB]);
    };
    next_rows();
    for (int it = 0; it < iters; ++it) {
        const bool actA = nA, actB = nB;
        const int rA = qA, rB = qB;
        const f32x2 dx = add2(add2(px, sx), jx2);
        const f32x2 dy = add2(add2(py, sy), jy2);
        const f32x2 dz = add2(add2(pz, sz), jz2);
        float* a = acc + rA * 32;
        float* b = acc + rB * 32;
        constexpr int C = ROWS * 32;
        const float a0 = a[0], a1 = a[C], a2 = a[2 * C], b0 = b[0], b1 = b[C], b2 = b[2 * C];
        next_rows();
        const f32x2 r2 = add2(add2(square2(dx, nz2), square2(dy, nz2)), square2(dz, nz2));
        float r2A, r2B;
        unpack2(r2, r2A, r2B);
        bool okA = actA && r2A <= cut2, okB = actB && r2B <= cut2;
        int potA = 0, potB = 0;
        if (TAB != kTabOne) {
            potA = potidx[prow + W.rtype[rA]];
            potB = potidx[prow + W.rtype[rB]];
            const bool ep = TAB == kTabGlobal && P.ep_pot >= 0;
            okA = okA && (potA >= 0 || ep);
            okB = okB && (potB >= 0 || ep);
        }
        if (EX) {
            if (okA && cell_excluded(P, jx, W.rpid[rA])) { okA = false; ++R.nexcl; }
            if (okB && cell_excluded(P, jx, W.rpid[rB])) { okB = false; ++R.nexcl; }
        }
        // 1/r: rsqrt plus one Newton step; r: r2/r corrected by one residual step, the
        // correctly rounded square root (as pair_force)
        f32x2 ri = pack2(rsqrt_approx(r2A), rsqrt_approx(r2B));
        ri = fma2(mul2(nhalf, ri), fma2(mul2(r2, ri), ri, none), ri);
        f32x2 r = mul2(r2, ri);
        r = fma2(fma2(mul2(none, r), r, r2), mul2(half, ri), r);
        float rA_, rB_, iA, iB;
        unpack2(r, rA_, rB_);
        unpack2(ri, iA, iB);
        float eA = 0.f, eB = 0.f, fA = 0.f, fB = 0.f;
        if (TAB == kTabGlobal) {
            if (okA && potA >= 0) cell_eval_table<TAB>(P, S, potA, rA_, iA, eA, fA);
            if (okB && potB >= 0) cell_eval_table<TAB>(P, S, potB, rB_, iB, eB, fB);
            if (P.ep_pot >= 0) {                  // + q_i q_j ep(r)
                float ee, fe;
                if (okA) {
                    cell_eval_table<TAB>(P, S, P.ep_pot, rA_, iA, ee, fe);
                    const float qq = W.rq[rA] * qj;
                    eA = fmaf(qq, ee, eA);
                    fA = fmaf(qq, fe, fA);
                }
                if (okB) {
                    cell_eval_table<TAB>(P, S, P.ep_pot, rB_, iB, ee, fe);
                    const float qq = W.rq[rB] * qj;
                    eB = fmaf(qq, ee, eB);
                    fB = fmaf(qq, fe, fB);
                }
            }
        } else {
            cell_eval_table<TAB>(P, S, TAB == kTabOne ? 0 : max(potA, 0), rA_, iA, eA, fA);
            cell_eval_table<TAB>(P, S, TAB == kTabOne ? 0 : max(potB, 0), rB_, iB, eB, fB);
            eA = okA ? eA : 0.f;
            fA = okA ? fA : 0.f;
            eB = okB ? eB : 0.f;
            fB = okB ? fB : 0.f;
        }
        const f32x2 f = pack2(-fA, -fB);         // 0 for a rejected pair; positions are finite
        const f32x2 wx = mul2(f, dx), wy = mul2(f, dy), wz = mul2(f, dz);
        fx = add2(fx, wx);
        fy = add2(fy, wy);
        fz = add2(fz, wz);
        float ax, ay, az, bx, by, bz;
        unpack2(wx, ax, bx);
        unpack2(wy, ay, by);
        unpack2(wz, az, bz);
        a[0] = a0 + ax;
        a[C] = a1 + ay;
        a[2 * C] = a2 + az;
        if (actB) {                              // else row B is row A again
            b[0] = b0 + bx;
            b[C] = b1 + by;
            b[2 * C] = b2 + bz;
        }
        R.e += (double)eA;
        R.e += (double)eB;
        R.npairs += (okA ? 1u : 0u) + (okB ? 1u : 0u);
    }
    if (live) {
        float a, b;
        unpack2(fx, a, b);
        const float gx = -(a + b);
        unpack2(fy, a, b);
        const float gy = -(a + b);
        unpack2(fz, a, b);
        const float gz = -(a + b);
        // virial: sum over pairs of r_ij.F_ij = sum_i x_i.F_i + sum_j (x_j + shift).F_j
        R.v += ((double)xj.x + sh.x) * gx + ((double)xj.y + sh.y) * gy + ((double)xj.z + sh.z) * gz;
        unsigned long long* fp = P.force + 3 * slot;
        atomic_add_fixed(fp + 0, to_fixed(gx, R.status));
        atomic_add_fixed(fp + 1, to_fixed(gy, R.status));
        atomic_add_fixed(fp + 2, to_fixed(gz, R.status));
    }
}

// ---------------------------------------------------------------- candidate counts
// Candidates of the sorted sweep (Params::acc[kAccCand]), which this form does not sweep:
// pairs of a pair task whose projections on the task's axis, in key units, pass its bound
// (sorted_prefix: dist_j < dmaxdist - dnshift + dist_i), every pair of a self task.  A warp
// takes 32 tasks: their records and counts one per lane, pairs of at most kCountLane
// candidates by the lane itself (a vapour's), the others one by one by the whole warp: 32
// rows' bounds in shared memory as packed 16-bit pairs, one j per lane, two rows per min/max
// instruction: clamp(bound - dist_j, 0, 1).  Runs beside the sweep, whose one block per SM
// leaves warps, registers and issue slots for one of these blocks (the bounds of both kernels
// are chosen so that they fit an SM together; one that does not waits for the other).
constexpr int kCountWarps = 8;
constexpr int kCountLane = 12;

__global__ void __launch_bounds__(kCountWarps * 32) count_candidates(CellParams C) {
    __shared__ uint4 bounds[kCountWarps][4];
    constexpr unsigned FULL = 0xffffffffu;
    const Params& P = C.p;
    if (*C.count_cand == 0 || step_aborted(P.abort)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned count = 0;
    for (int t0 = (blockIdx.x * kCountWarps + warp) * 32; t0 < P.ntasks; t0 += gridDim.x * kCountWarps * 32) {
        TaskRec mine = TaskRec{0, 0, -1, 0};
        int my_ni = 0, my_nj = 0, my_si = 0, my_sj = 0;
        float2 my_ci = make_float2(0.f, 0.f), my_cj = my_ci;
        if (t0 + lane < P.ntasks) {
            mine = P.tasks[t0 + lane];
            my_ni = P.ccount[mine.ci];
            my_nj = P.ccount[mine.cj];
            if (mine.sid < 0) {
                count += (unsigned)(my_ni * (my_ni - 1) / 2);
                my_ni = 0;
            }
        }
        const bool some = my_ni > 0 && my_nj > 0, alone = some && my_ni * my_nj <= kCountLane;
        if (some) {
            my_si = P.cstart[mine.ci];
            my_sj = P.cstart[mine.cj];
            my_ci = C.cscale[mine.ci];
            my_cj = C.cscale[mine.cj];
        }
        const int my_bound = task_dmax(mine) - task_dnshift(mine);
        if (alone) {
            const float nx = C.axes[mine.sid][0], ny = C.axes[mine.sid][1], nz = C.axes[mine.sid][2];
            for (int i = 0; i < my_ni; ++i) {
                const int lim = my_bound + (int)sort_dist(P.xq[my_si + i], nx, ny, nz, my_ci.x, my_ci.y);
                for (int j = 0; j < my_nj; ++j)
                    count += (int)sort_dist(P.xq[my_sj + j], nx, ny, nz, my_cj.x, my_cj.y) < lim ? 1u : 0u;
            }
        }
        for (unsigned left = __ballot_sync(FULL, some && !alone); left; left &= left - 1) {
            const int b = __ffs(left) - 1;
            const int ni = __shfl_sync(FULL, my_ni, b), nj = __shfl_sync(FULL, my_nj, b);
            const int si = __shfl_sync(FULL, my_si, b), sj = __shfl_sync(FULL, my_sj, b);
            const int sid = __shfl_sync(FULL, mine.sid, b), bound = __shfl_sync(FULL, my_bound, b);
            const float2 sci = make_float2(__shfl_sync(FULL, my_ci.x, b), __shfl_sync(FULL, my_ci.y, b));
            const float2 scj = make_float2(__shfl_sync(FULL, my_cj.x, b), __shfl_sync(FULL, my_cj.y, b));
            const float nx = C.axes[sid][0], ny = C.axes[sid][1], nz = C.axes[sid][2];
            for (int r0 = 0; r0 < ni; r0 += 32) {
                const int nr = min(32, ni - r0);
                float4 xj = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < nj) xj = P.xq[sj + lane];
                // rows past the last: a bound that no distance is below
                const int lim = lane < nr ? bound + (int)sort_dist(P.xq[si + r0 + lane], nx, ny, nz, sci.x, sci.y) : 0;
                __syncwarp();
                reinterpret_cast<short*>(bounds[warp])[lane] = (short)(min(max(lim, 0), 32767) - 16384);
                __syncwarp();
                for (int k = 0; k < nj; k += 32) {
                    const bool on = k + lane < nj;
                    if (k > 0 && on) xj = P.xq[sj + k + lane];
                    // lanes past the last: a distance that no bound is above
                    const int dj = on ? (int)sort_dist(xj, nx, ny, nz, scj.x, scj.y) : 32767;
                    if (__any_sync(FULL, on && dj > 32766)) {
                        // a particle far outside its cell: distances past 15 bits, one by one
                        for (int r = 0; r < nr; ++r) {
                            const int lr = __shfl_sync(FULL, lim, r);
                            count += on && dj < lr ? 1u : 0u;
                        }
                        continue;
                    }
                    // 16384 - dj in both halves; bound - 16384 + that = bound - dj, in 16 bits
                    const unsigned nd = (unsigned)((16384 - dj) & 0xffff) * 0x10001u;
                    unsigned sum = 0;
                    for (int q = 0; q < nr; q += 8) {
                        const uint4 v = bounds[warp][q >> 3];
                        sum += __viaddmin_s16x2_relu(v.x, nd, 0x10001u) + __viaddmin_s16x2_relu(v.y, nd, 0x10001u) +
                               __viaddmin_s16x2_relu(v.z, nd, 0x10001u) + __viaddmin_s16x2_relu(v.w, nd, 0x10001u);
                    }
                    count += (sum & 0xffffu) + (sum >> 16);
                }
            }
        }
    }
    count = __reduce_add_sync(FULL, count);
    if (lane == 0 && count) atomicAdd(&P.acc[kAccCand], (unsigned long long)count);
}

// The bound of 32 threads more than a block has keeps the registers of kCountWarps warps free.
template <bool EX, int TAB, int ROWS>
__global__ void __launch_bounds__(kCellWarps * 32 + 32, 1) sweep_cells(CellParams C) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr unsigned FULL = 0xffffffffu;
    const Params& P = C.p;
    if (step_aborted(P.abort)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    CellWarp<ROWS>& W = reinterpret_cast<CellWarp<ROWS>*>(smem_raw)[warp];
    CellTables S;
    S.one = TAB == kTabOne ? P.potinfo[0] : make_float4(0.f, 0.f, 0.f, 0.f);
    S.copies = C.copies;
    S.chunk = nullptr;
    S.info = nullptr;
    S.potidx = nullptr;
    if (TAB != kTabGlobal) {
        float4* tab = reinterpret_cast<float4*>(smem_raw + (size_t)nw * sizeof(CellWarp<ROWS>));
        const float4* coef = reinterpret_cast<const float4*>(P.coef);
        for (int k = threadIdx.x; k < P.ncoef / 4 * C.copies; k += blockDim.x) tab[k] = coef[k / C.copies];
        float4* info = tab + (size_t)(P.ncoef / 4) * C.copies;
        for (int k = threadIdx.x; k < P.npots; k += blockDim.x) info[k] = P.potinfo[k];
        int* potidx = reinterpret_cast<int*>(info + P.npots);
        for (int k = threadIdx.x; k < P.max_type * P.max_type; k += blockDim.x) potidx[k] = P.potidx[k];
        S.chunk = tab + lane % C.copies;
        S.info = info;
        S.potidx = potidx;
    }
    __syncthreads();

    const bool need_pid = EX || (TAB == kTabGlobal && P.ep_pot >= 0);
    const int nu = min(*C.nunits, C.units_cap);
    const int batch = max(1, min(4, nu / (8 * (int)gridDim.x * nw)));
    const f32x2 nz2 = pack2(C.neg_zero, C.neg_zero);
    CellSums R;
    // the next unit, its cell's particles and tasks are read while the current one runs
    int u = 0, uend = 0;
    auto pop = [&]() {
        if (u >= uend) {
            int q = 0;
            if (lane == 0) q = atomicAdd(C.head, batch);
            u = __shfl_sync(FULL, q, 0);
            uend = min(u + batch, nu);
        }
        return u < nu ? C.units[u++] : make_int2(-1, 0);
    };
    int2 next = pop();
    int nn = 0, nstart = 0, nt0 = 0, nt1 = 0;
    if (next.x >= 0) {
        nn = P.ccount[next.x];
        nstart = P.cstart[next.x];
        nt0 = C.toff[next.x];
        nt1 = C.toff[next.x + 1];
    }
    while (next.x >= 0) {
        const int2 unit = next;
        const int c = unit.x, n = nn, start = nstart, t0 = nt0, ntask = nt1 - nt0;
        next = pop();
        if (next.x >= 0) {
            nn = P.ccount[next.x];
            nstart = P.cstart[next.x];
            nt0 = C.toff[next.x];
            nt1 = C.toff[next.x + 1];
        }
        const int strip = unit.y & 0xff, strips = (unit.y >> 8) & 0xff, share = (unit.y >> 16) & 0xff,
                  shares = (unsigned)unit.y >> 24;
        const int r0 = n * strip / strips, r1 = n * (strip + 1) / strips;
        const int nr = r1 - r0, top = ((nr + 1) & ~1) - 1;
        R.e = 0.0;
        R.v = 0.0;

        // the tasks with particles (self: below the last row), one per lane: their j particles
        // form one list, task after task
        int total;
        unsigned selfs;
        {
            int tn = 0, tself = 0, tstart = 0;
            float4 sh = make_float4(0.f, 0.f, 0.f, 0.f);
            if (lane < ntask) {
                const TaskRec tr = C.tasks[t0 + lane];
                tself = tr.sid < 0;
                if (!tself) sh = C.tshift[t0 + lane];
                tstart = P.cstart[tr.cj];
                tn = tself ? r1 - 1 : P.ccount[tr.cj];
                sh.w = tself ? P.cutoff2s : P.cutoff2;
            }
            int incl = tn;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += v;
            }
            total = __shfl_sync(FULL, incl, 31);
            const unsigned some = __ballot_sync(FULL, tn > 0);
            const int k = __popc(some & ((1u << lane) - 1u));
            if (tn > 0) {
                W.sh[k] = sh;
                W.tslot[k] = tstart - (incl - tn);
            }
            selfs = __reduce_or_sync(FULL, tself && tn > 0 ? 1u << k : 0u);
            W.tplace[lane] = 0x7fffffff;
            __syncwarp();
            if (tn > 0) W.tplace[k] = incl - tn;
        }
        const int lo = total * share / shares, hi = total * (share + 1) / shares;

        // the rows
        float4 xi = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane < nr) xi = P.xq[start + r0 + lane];
        float ni = lane < nr ? fmaf(xi.z, xi.z, fmaf(xi.y, xi.y, xi.x * xi.x)) : INFINITY;
        // A non-finite position (or one whose square overflows: beyond 1e19 nm) has no pairs: such
        // a row is treated as those past the last (no test passes it, and its position in W is
        // finite, since rejected pairs multiply their displacement by 0), such a j is dropped by
        // the box test.
        const bool in = ni < INFINITY;
        if (!in) {
            xi.x = xi.y = xi.z = 0.f;
            ni = INFINITY;
        }
        W.rx[lane] = xi.x;
        W.ry[lane] = xi.y;
        W.rz[lane] = xi.z;
        W.rtype[lane] = __float_as_int(xi.w);
        if (need_pid) {
            const int id = lane < nr ? P.pid[start + r0 + lane] : 0;
            W.rpid[lane] = id;
            if (TAB == kTabGlobal && P.ep_pot >= 0) W.rq[lane] = P.qid[id];
        }
        {
            float* rt = reinterpret_cast<float*>(W.rt) + (lane >> 1) * 8 + (lane & 1);
            rt[0] = -2.f * xi.x;
            rt[2] = -2.f * xi.y;
            rt[4] = -2.f * xi.z;
            rt[6] = ni;
        }
        const float lox = warp_min(in ? xi.x : INFINITY), hix = warp_max(in ? xi.x : -INFINITY);
        const float loy = warp_min(in ? xi.y : INFINITY), hiy = warp_max(in ? xi.y : -INFINITY);
        const float loz = warp_min(in ? xi.z : INFINITY), hiz = warp_max(in ? xi.z : -INFINITY);
        const float nimax = warp_max(in ? ni : 0.f);
        // Rounding of the test's form of r^2 and of the box distance, and of the exact one: below
        // 24 roundings of 2^-24 relative to |xi|^2 + |xj|^2 (1.5e-6); 4e-6 is taken.
        constexpr float kSlack = 4e-6f;
        {
            float4* z = reinterpret_cast<float4*>(&W.acc[0][0][0]);
            constexpr int Q = ROWS * 8;
            for (int k = lane; k < nr * 8; k += 32)
                z[k] = z[k + Q] = z[k + 2 * Q] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();

        // the 32 list places from `at` on (ascending calls): slot, task and position of this
        // lane's.  tb: the last task that starts before `at`
        const int pre = W.tplace[lane];
        int tb = __popc(__ballot_sync(FULL, pre < lo)) - 1;
        auto fetch = [&](int at, float4& x, unsigned& meta) {
            const unsigned d = (unsigned)(pre - at);
            const unsigned starts = __reduce_or_sync(FULL, d < 32u ? 1u << d : 0u);
            const int t = tb + __popc(starts & ((2u << lane) - 1u));
            tb += __popc(starts);
            if (at + lane < hi) {
                const int slot = W.tslot[t] + at + lane;
                x = P.xq[slot];
                meta = (unsigned)slot | ((unsigned)t << kCellSlotBits);
            }
        };
        int b0 = 0, nb = 0;                    // near list: ring head and length
        int ne0 = 0, ne1 = 0;                  // evaluation lists
        // tests m <= 32 entries of the near list against the rows
        auto test_rows = [&](int m) {
            const int q = (b0 + lane) & (kCellRing - 1);
            const bool on = lane < m;
            const float4 xj = W.bx[q];
            const unsigned meta = on ? W.bm[q] : 0u;
            const int t = meta >> kCellSlotBits;
            int jpid = 0;
            if (need_pid && on) jpid = P.pid[meta & ((1u << kCellSlotBits) - 1u)];
            const float4 sh = W.sh[t];
            const float x = xj.x + sh.x, y = xj.y + sh.y, z = xj.z + sh.z;
            const float nj = fmaf(z, z, fmaf(y, y, x * x));
            const float thr = fmaf(kSlack, nj + nimax, sh.w) - nj;
            const f32x2 x2 = pack2(x, x), y2 = pack2(y, y), z2 = pack2(z, z), n2 = pack2(-thr, -thr);
            unsigned near = 0;
#pragma unroll 4
            for (int k = 0; k <= top; k += 2) {
                const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(&W.rt[k]);
                const ulonglong2 s = *reinterpret_cast<const ulonglong2*>(&W.rt[k + 1]);
                const f32x2 d = add2(fma2(p.x, x2, fma2(p.y, y2, fma2(s.x, z2, s.y))), n2);
                // r^2 - cutoff^2: negative when near
                float dA, dB;
                unpack2(d, dA, dB);
                near = __funnelshift_l(__float_as_uint(dA), near, 1);
                near = __funnelshift_l(__float_as_uint(dB), near, 1);
            }
            unsigned mask = on ? near & (0xffffffffu >> (31 - top)) : 0u;
            // a self task's j meets the rows after it only
            if ((selfs >> t) & 1u) {
                const int m0 = (int)(meta & ((1u << kCellSlotBits) - 1u)) - start - r0 + 1;   // first row
                if (m0 > top) mask = 0u;
                else if (m0 > 0) mask &= (2u << (top - m0)) - 1u;
            }
            b0 = (b0 + m) & (kCellRing - 1);
            nb -= m;
            const bool many = __popc(mask) * 10 >= 3 * nr;
            const unsigned p0 = __ballot_sync(FULL, mask != 0 && many), p1 = __ballot_sync(FULL, mask != 0 && !many);
            const unsigned below = (1u << lane) - 1u;
            if (mask != 0) {
                const int o = many ? ne0 + __popc(p0 & below) : kCellList - 1 - ne1 - __popc(p1 & below);
                W.ex[o] = xj;
                W.em[o] = meta;
                W.emask[o] = mask;
                if (need_pid) W.epid[o] = jpid;
            }
            ne0 += __popc(p0);
            ne1 += __popc(p1);
            __syncwarp();
        };

        // two passes of positions in flight
        float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0;
        unsigned m0_ = 0, m1_ = 0;
        int base = lo;
        bool any = false;
        if (base < hi) fetch(base, x0, m0_);
        if (base + 32 < hi) fetch(base + 32, x1, m1_);
        for (;;) {
            while (nb < 32 && base < hi) {
                const float4 xj = x0;
                const unsigned meta = m0_;
                const bool on = base + lane < hi;
                x0 = x1;
                m0_ = m1_;
                if (base + 64 < hi) fetch(base + 64, x1, m1_);
                base += 32;
                const float4 sh = W.sh[on ? meta >> kCellSlotBits : 0];
                const float x = xj.x + sh.x, y = xj.y + sh.y, z = xj.z + sh.z;
                const float gx = fmaxf(fmaxf(lox - x, x - hix), 0.f), gy = fmaxf(fmaxf(loy - y, y - hiy), 0.f),
                            gz = fmaxf(fmaxf(loz - z, z - hiz), 0.f);
                const float nj = fmaf(z, z, fmaf(y, y, x * x));
                // no less than: the slack covers equality, and neither side of a non-finite position
                // (both infinite, or the right one NaN) is less than the other
                const bool close = on && fmaf(gz, gz, fmaf(gy, gy, gx * gx)) < fmaf(kSlack, nj + nimax, sh.w);
                const unsigned ball = __ballot_sync(FULL, close);
                if (close) {
                    const int o = (b0 + nb + __popc(ball & ((1u << lane) - 1u))) & (kCellRing - 1);
                    W.bx[o] = xj;
                    W.bm[o] = meta;
                }
                nb += __popc(ball);
                __syncwarp();
            }
            if (nb > 0) test_rows(min(nb, 32));
            const bool last = nb == 0 && base >= hi;
            // full windows of one class; at the end what is left of both, many rows first
            while (ne0 >= 32 || ne1 >= 32 || (last && ne0 + ne1 > 0)) {
                const int m0 = ne0 >= 32 ? 32 : ne1 >= 32 ? 0 : ne0;
                const int m1 = ne0 >= 32 ? 0 : min(ne1, 32 - m0);
                const bool on = lane < m0 + m1;
                const int q = lane < m0 ? ne0 - m0 + lane : kCellList - 1 - (ne1 - m1 + lane - m0);
                const int o = on ? q : 0;
                cell_window<EX, TAB, ROWS>(P, W, S, W.ex[o], on ? W.em[o] : 0u, on ? W.emask[o] : 0u,
                                     need_pid && on ? W.epid[o] : 0, top, nz2, R, lane);
                ne0 -= m0;
                ne1 -= m1;
                any = true;
                __syncwarp();
            }
            if (last) break;
        }
        if (!any) continue;

        // i forces: lane r sums its row over the lanes' accumulators
        __syncwarp();
        if (lane < nr) {
            float f[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float s = 0.f, s1 = 0.f;
#pragma unroll 8
                for (int k = 0; k < 32; k += 2) {
                    s += W.acc[d][lane][(lane + k) & 31];
                    s1 += W.acc[d][lane][(lane + k + 1) & 31];
                }
                f[d] = s + s1;
            }
            R.v += (double)xi.x * f[0] + (double)xi.y * f[1] + (double)xi.z * f[2];
            unsigned long long* fp = P.force + 3 * (size_t)(start + r0 + lane);
#pragma unroll
            for (int d = 0; d < 3; ++d) atomic_add_fixed(fp + d, to_fixed(f[d], R.status));
        }
        const long long e_fix = warp_sum_fixed(__double2ll_rn(R.e * kEnergyScale));
        const long long v_fix = warp_sum_fixed(__double2ll_rn(-R.v * kEnergyScale));
        if (lane == 0) {
            atomicAdd(&P.cell_epot[c], (unsigned long long)e_fix);
            atomicAdd(P.cell_vir ? &P.cell_vir[c] : &P.acc[kAccVirial], (unsigned long long)v_fix);
        }
        __syncwarp();
    }
    flush_counters(P, R.npairs, R.nexcl, 0u, R.status, lane);
}

namespace {
// Shared memory of a block at most (the attribute of all launches, as kSweepSmem).
constexpr size_t kCellSmem = 227 * 1024;

template <bool EX, int TAB, int ROWS>
cudaError_t launch_k(const CellParams& C, int nw, size_t smem, int grid, bool capturing, cudaStream_t s) {
    auto kern = sweep_cells<EX, TAB, ROWS>;
    if (!capturing) {
        const cudaError_t err =
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCellSmem);
        if (err != cudaSuccess) return err;
    }
    kern<<<grid, nw * 32, smem, s>>>(C);
    return cudaGetLastError();
}

template <int ROWS>
cudaError_t launch_rows(const CellParams& C, bool has_excl, int tab, int nw, size_t smem, int grid, bool capturing,
                        cudaStream_t s) {
    if (tab == kTabGlobal)
        return has_excl ? launch_k<true, kTabGlobal, ROWS>(C, nw, smem, grid, capturing, s)
                        : launch_k<false, kTabGlobal, ROWS>(C, nw, smem, grid, capturing, s);
    if (tab == kTabOne)
        return has_excl ? launch_k<true, kTabOne, ROWS>(C, nw, smem, grid, capturing, s)
                        : launch_k<false, kTabOne, ROWS>(C, nw, smem, grid, capturing, s);
    return has_excl ? launch_k<true, kTabShared, ROWS>(C, nw, smem, grid, capturing, s)
                    : launch_k<false, kTabShared, ROWS>(C, nw, smem, grid, capturing, s);
}
}  // namespace

// Shares are at most 1 + tests / kCellShare per strip (cell_split).
size_t cell_units_bound(size_t nslots, int ncells, int cap, int maxtasks) {
    const size_t strips = nslots / 24 + (size_t)ncells;      // of 24 rows, the more of the two
    return 2 * strips + (nslots + strips) * (size_t)maxtasks * (size_t)cap / kCellShare + 64;
}

// 8 copies (no bank conflicts) up to 32 KB of tables, fewer for larger ones; as many warps, up
// to kCellWarps, as the rest of an SM's 227 KB holds.
bool cell_sweep_shape(int rows, int ncoef, int npots, int mt, int* nw, int* copies, size_t* smem) {
    const size_t room = kCellSmem, slice = rows == 24 ? sizeof(CellWarp<24>) : sizeof(CellWarp<32>);
    auto tables = [&](int n) { return (size_t)ncoef * 4 * n + (size_t)npots * 16 + (size_t)((mt * mt + 3) & ~3) * 4; };
    *copies = 8;
    while (*copies > 1 && tables(*copies) > 32 * 1024) *copies /= 2;
    if (tables(*copies) + slice > room) return false;
    *nw = (int)std::min<size_t>(kCellWarps, (room - tables(*copies)) / slice);
    *smem = (size_t)*nw * slice + tables(*copies);
    return true;
}

cudaError_t launch_cell_count(const CellParams& C, int grid, cudaStream_t s) {
    count_candidates<<<grid, kCountWarps * 32, 0, s>>>(C);
    return cudaGetLastError();
}

cudaError_t launch_cell_sweep(const CellParams& C, int ncells, int rows, int2* units, bool has_excl, int tab, int nw,
                              size_t smem, int grid, bool capturing, cudaStream_t s) {
    cudaError_t err = cudaMemsetAsync(C.head, 0, 2 * sizeof(int), s);
    if (err != cudaSuccess) return err;
    const Params& P = C.p;
    cell_units<<<(ncells + 255) / 256, 256, 0, s>>>(P.ccount, C.toff, C.tasks, ncells, rows, units, C.head + 1,
                                                    C.units_cap, P.acc, P.abort);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    return rows == 24 ? launch_rows<24>(C, has_excl, tab, nw, smem, grid, capturing, s)
                      : launch_rows<32>(C, has_excl, tab, nw, smem, grid, capturing, s);
}

}  // namespace nb
