// k_coop.cuh -- a whole run of a small or medium system in one cooperative
// launch (both force modes).
//
// One graph unit of the plain path (step kernel, conditional rebuild) costs
// 15-25 us whatever the system's size: launches, the IF node, and the drain
// of each kernel.  Up to about 100,000 particles the arithmetic of a
// step takes less than that, so k_coop advances the run inside one launch:
// every block owns fixed tiles of particles, a step is the triangle pass, the
// particle pass and a grid-wide exchange, and every block takes the rebuild
// decision of NeighborList::update (femmd2D/src/nn.cpp:114-134) from the same
// exchanged maximum.  A system of one tile runs in one block, where an
// exchange is a block barrier.
//
// Every block works all the triangles of its own particles (CoopArgs::triOwn)
// and keeps their forces in shared memory: the few with particles of two blocks
// are worked twice, and the particle pass needs no exchange before it.  Of a
// triangle's blocks one stores its energy, which is added up a step later.
// Where a particle has too many incidences or shared memory is short, the
// triangles are shared out and an exchange follows the triangle pass: 256 disks
// run(100) 1034 us against 849, 144 disks in solvent (fast mode) run(50) 1211
// against 1137, the adjoint of 64 disks 7729 against 7034 (its reverse steps by two
// kernels each).
//
// At these sizes a step is bound by latency: dependent L2 accesses (about
// 0.4 us each: an exchange invalidates L1) and, with a warp or two per
// scheduler, dependent instructions (7 cycles each: a thread that works its 20
// pairs one after another takes 12,000 cycles).  So a particle is worked by
// four lanes: each gathers and works every fourth list entry and puts the
// pair's four terms (force x, y, energy, virial) into shared memory, and then
// each adds up one of the four sums over the entries in list order; lanes 0
// and 1 integrate one axis each.  The lists, the bond and triangle
// incidences and the triangles' vertices stay in shared memory for the whole
// launch, loads that do not depend on each other are issued together, and the
// energy sums are reduced while the exchange is waited for.
//
// Measured against the plain kernels in CUDA graphs (a whole set_state, run,
// get_state; us): LJ fluid 400 particles run(20) 659 -> 207, 10,201 run(50)
// 1390 -> 407; 256-disk suspension (32,512) run(100) 1842 -> 849; adjoint of 64
// disks over 200 steps 14,260 -> 5200; fast mode, run(50): LJ fluid 90,000 1408
// -> 1112, 144 disks in solvent (68,288) 1778 -> 1137, run(100) of 4096 1275 -> 749
// (1060 by a kernel of its own for small fluids, a thread per particle, with
// five launches around it).  The particle pass of the 10,201
// particles takes 4.1 us; a thread per particle instead of a quad took 7.7.
//
// The per-particle and per-triangle arithmetic and the list order are those
// of the plain kernels (step_body.cuh, nn_body.cuh), and so is the grouping
// of the energy sums: FP32 over the 32 lanes and the 4 (8) warps of a tile of
// 128 particles (256 triangles), then 64-bit fixed point, which is exact in
// any order.  Positions, velocities, forces, energies and rebuild steps are
// therefore the plain path's bit for bit.
//
// FAST: the fast force mode's arithmetic (k_fast.cu) instead, bit for bit as
// to positions, velocities and forces.  Its pair sums run over the even and the
// odd list entries apart (one type: the two lanes of fast_pairs_x2) or in list
// order (several types: fast_pairs) by fused multiply-adds, so a lane puts a
// pair's factors into shared memory and the sums are formed there.  The
// launch keeps the particles in id order: the lists' order does not depend on
// the storage order, and it leaves lists without windows behind (storage
// slots, padded with the ghost's).  Small systems' energies are grouped by the
// storage slot the step kernels would have the particle in (coop_by_slot): a
// particle's go to its slot in memory and are added up a step later.
//
// Exchanges are grid_exchange's (grid_sync.cuh), bounded: a wait that gives
// up sets the timeout flag, and the block leaves the kernel.  They are numbered
// over the life of the context (DevScalars::runTag).  A step's energy sums are
// added into one of four rotating sets after its exchange (the triangles' by
// block after the next step's) and are therefore complete to a block that has
// completed the following one; block 0 takes them during the exchange after
// that.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>
#include "femmd_internal.h"
#include "launch.h"
#include "device_common.cuh"
#include "fast_body.cuh"
#include "grid_sync.cuh"
#include "nn_body.cuh"
#include "step_body.cuh"

namespace femmd {

namespace {

constexpr int kCoopThreads = 512;
constexpr int kCoopTimeout = 8;     // DevScalars::overflow bit: a bounded wait expired
constexpr int kCoopCrowded = 16;    // DevScalars::overflow bit: a cell holds more than cell_cap particles
constexpr int kCoopLeft = 32;       // DevScalars::overflow bit: a rebuild could not be made (kRebuildLeft)
constexpr int kCoopMaxTiles = 32;   // tiles of one block (one lane of a warp sums each)
constexpr int kTriTile = 256;       // triangles per energy group (k_tri_forces' block)
constexpr int kListLanes = 8;       // lanes that build one particle's list
// Incidences of one bonded particle kept in shared memory: a count word, up
// to kIncTri triangle entries and kIncBond bond entries of two words.
constexpr int kIncTri = kCoopIncTri, kIncBond = kCoopIncBond, kIncWords = 1 + kIncTri + 2 * kIncBond;
constexpr int kQuadPairs = 6;                // list entries per lane and round
constexpr int kQuadRows = 4 * kQuadPairs;    // entries per particle and round
// One round's terms in shared memory: component c of entry k of the tile's
// particle p at c kTermComp + k kTermRow + p.  The pads put the four entries
// a quad writes together, and the four components it reads together, into
// different banks.
constexpr int kTermRow = kStepBlock + 8, kTermComp = kQuadRows * kTermRow + 8;
// components of a term: the four sums' own, or the fast mode's factors
__host__ __device__ constexpr int coop_terms(bool fast) { return fast ? 6 : 4; }
constexpr int kListRow = kStepBlock + 8;     // a list row in shared memory (padded as kTermRow)

// Loads that stay where they are written, ahead of what uses them (a plain
// load is moved down to its use when registers are short).
__device__ __forceinline__ float2 ld_early(const float2 *p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_early(const float4 *p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ int ld_early(const int *p) {
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
struct CoopDue {
    unsigned x;  // the exchange (modulo 2^32) after which the last of the step's sums were stored
    unsigned set;  // their set
    int mode, row, reb;
    float vm, d;
};

struct CoopShared {
    PairEntry tab[kMaxTypes * kMaxTypes];
    float vmax[kCoopThreads / 32];    // per warp: its particles' largest v^2
    float tred[kCoopMaxTiles][8];     // per triangle tile and warp: energy
    unsigned long long acc[3];        // the step's energy sums of this block (U, W, K)
    unsigned long long accTri;        // triangles by block: the previous step's triangle energy
    CoopDue due[4];                   // block 0: steps whose totals have still to be added up
    int wsum[kCoopThreads / 32];
    unsigned ok, maxBits;             // of the last exchange
    int before;                       // particles in the earlier blocks' cells
};

// What every block carries through the launch (the same on each).
struct CoopRun {
    unsigned long long made;  // exchanges over the life of the context
    unsigned dueIn, dueOut;  // entries pushed to and taken from CoopShared::due (one per step)
    unsigned dueOk;          // entries whose sums are all stored
    float dispHi;
    int row, stepNow, updates;
    int cnt;  // which of the two cell-count arrays the last rebuild filled
};

// Step 'n' of a launch adds its energies (U, W, K as fixed point, every block by
// integer atomics: exact in any order) into set n mod 4; zero when it starts.
__device__ __forceinline__ unsigned long long *coop_sums(const DevSys &s, unsigned n) {
    return s.runRec + kGridSlots * kGridSlotWords + 4 * (size_t)(n % 4u);
}
// a word per block
__device__ __forceinline__ unsigned long long *coop_words(const DevSys &s) {
    return s.runRec + kGridSlots * kGridSlotWords + 16;
}

// One thread: the totals of a step into the scalars and, for the modes that
// complete a step, its observable row; the set is zero again.  (Summed up by
// block 0 from a record per block instead, this took longer than the exchange
// beside it: 256 disks on 152 blocks, 1053 us a run(100), 849 so.)
__device__ __noinline__ void coop_totals(const DevSys &s, const CoopDue &d) {
    unsigned long long *set = coop_sums(s, d.set);
    const unsigned long long u = __ldcg(set), w = __ldcg(set + 1), k = __ldcg(set + 2);
    set[0] = set[1] = set[2] = 0ull;
    {
        DevScalars *sc = s.sc;
        const double U = from_fixed(u), W = from_fixed(w), KE = from_fixed(k);
        sc->U = U;
        sc->W = W;
        if (d.mode == MODE_MID || d.mode == MODE_LAST) {
            sc->KE = KE;
            sc->vvMax = d.vm;
            if (s.obs && d.row < s.obsCap) {
                double *o = s.obs + (size_t)d.row * kObsCols;
                o[0] = U;
                o[1] = W;
                o[2] = KE;
                o[3] = (double)d.vm;
                o[4] = (double)d.d;
                o[5] = (double)d.reb;
            }
        }
    }
}

// An exchange: maxBits = the largest value as a float (the values' bits).
// Block 0's warp 2 meanwhile adds up the totals that are due (all: every one
// left), and 'meanwhile' runs on the warps from 3 on.  withhold: this block
// does not count (femmd_test_expire_next_exchange).  False when the wait gave
// up.  Call it after a block barrier that follows the block's stores; it ends
// with one.
struct Nothing {
    __device__ void operator()() const {}
};
template <class Work = Nothing>
__device__ __forceinline__ bool coop_exchange(const DevSys &s, CoopShared &sh, CoopRun &r, unsigned value,
                                              bool withhold = false, bool all = false, Work meanwhile = {}) {
    if (threadIdx.x == 0) {
        unsigned m = value;
        sh.ok = (gridDim.x == 1 && !withhold) ||
                grid_exchange(s.runRec, r.made, gridDim.x, value, withhold, m);
        sh.maxBits = m;
    }
    // a step's sums are visible once the exchange after its own is complete
    while (r.dueOut != r.dueOk && !all) {
        const CoopDue &d = sh.due[r.dueOut & 3u];
        if ((int)((unsigned)r.made - d.x) < 2) break;
        if (blockIdx.x == 0 && threadIdx.x == 64) coop_totals(s, d);
        r.dueOut++;
    }
    r.made++;
    if (threadIdx.x >> 5 >= 3) meanwhile();
    __syncthreads();
    if (sh.ok) return true;
    if (threadIdx.x == 0) atomicOr(&s.sc->overflow, kCoopTimeout);
    return false;
}

// Exclusive scan of v over the block (every thread calls it); 'total' is the
// block's sum.
__device__ __forceinline__ int block_scan(CoopShared &sh, int v, int &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();  // wsum may still be read
    if (lane == 31) sh.wsum[warp] = x;
    __syncthreads();
    const int w = lane < nw ? sh.wsum[lane] : 0;
    int z = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, z, o);
        if (lane >= o) z += y;
    }
    total = __shfl_sync(0xffffffffu, z, 31);
    return __shfl_sync(0xffffffffu, z - w, warp) + x - v;
}

// The launch's shared-memory arrays beside CoopShared.
struct CoopMem {
    float *term;  // a round's terms (kTermComp)
    float *part;  // [tile of the block][3][kStepBlock]: the particles' U, W, m v^2 of the step
    int *list;    // [tile][rows][kListRow]: the first 'rows' list entries of every particle
    int rows;     // (a multiple of 4)
    int *count;  // [tile][kStepBlock]: list lengths
    int *inc;    // [tile][kIncWords][kStepBlock], or null
    // triangles by tile: [triangle tile][kTriTile], the vertices, or null; by
    // block: the block's, vertices and CoopArgs::triOwn's word, and their forces
    int4 *tri;
    float2 *triF;
    int tiles, first, stride;  // the block's tiles of particles: first, first + stride, ...
    // by slot: the storage slot of the block's particles [tile][kStepBlock], and where the step's U, W, m v^2 go ([3][engRow], by slot)
    int *slot;
    float *eng;
    size_t engRow;
};

// The tiles of block b.  Tile j is b + j grid, so that bonded and free particles
// (and their rebuilds) are shared out.  With triangles by block and two tiles a
// block (pair), they are neighbours: fewer triangles have particles of two
// blocks (256 disks of 216 triangles on 152 blocks: at most 504 a block, 562
// with tiles apart, where 512 threads want at most 512).
__host__ __device__ inline bool coop_pairs(int ntiles, int grid) { return (ntiles + grid - 1) / grid == 2; }
__host__ __device__ inline int coop_tiles(int ntiles, int grid, int b, bool pair, int &first, int &stride) {
    pair = pair && coop_pairs(ntiles, grid);
    first = pair ? 2 * b : b;
    stride = pair ? 1 : grid;
    if (first >= ntiles) return 0;
    return pair ? (ntiles - first < 2 ? ntiles - first : 2) : (ntiles - 1 - first) / stride + 1;
}

// Particles that a cell of the launch's table holds (a multiple of 8).
template <bool SLOT>
__device__ __forceinline__ int cell_cap(const DevSys &s) {
    return SLOT ? s.cellCap : kCellCap;
}

// The list of particle i (slot 'col' of the block's tile j) by kListLanes
// lanes: the 3 x 3 cells in the reference's order (dx outer, dy inner, each
// cell's particles by ascending id, cell indices wrapped as applyCellBC,
// nnCuda.cu:26-36), kListLanes candidates of a cell at a time, a ballot
// placing the hits.  FAST: fast_walk_ok, the image shift is the cell's; else
// the minimum image per pair.  The first candidates of all nine cells are in
// flight together.  Entries go to shared memory (from entry mem.rows on, to
// the list itself; the others are copied there at the end of the launch).  All lanes of the warp call it; returns the list length.
template <bool FAST, bool SLOT>
__device__ __forceinline__ int coop_list(const DevSys &s, const CoopMem &mem, const int *cnt, const float2 *pos, int i,
                                         int j, int col, bool valid) {
    const int lane = threadIdx.x & 31, sub = lane & (kListLanes - 1), shift = lane & ~(kListLanes - 1);
    const int ncx = s.ncx, ncy = s.ncy, cap = s.nbrCap;
    const float R2 = s.nnRadiusSq;
    const float Lx = s.wrapx ? s.Lx : 0.0f, Ly = s.wrapy ? s.Ly : 0.0f;
    const float2 p = valid ? pos[i] : make_float2(0.0f, 0.0f);
    const int gi = valid ? s.excl[i] : -1;
    int ix, iy;
    cell_xy(p.x, p.y, ncx, ncy, s.Lx, s.Ly, ix, iy);
    const int cx[3] = {(ix == 0 ? ncx : ix) - 1, ix, ix == ncx - 1 ? 0 : ix + 1};
    const int cy[3] = {(iy == 0 ? ncy : iy) - 1, iy, iy == ncy - 1 ? 0 : iy + 1};
    const float sx[3] = {ix == 0 ? -Lx : 0.0f, 0.0f, ix == ncx - 1 ? Lx : 0.0f};
    const float sy[3] = {iy == 0 ? -Ly : 0.0f, 0.0f, iy == ncy - 1 ? Ly : 0.0f};
    const int cells = cell_cap<SLOT>(s);
    int n[9];
    float4 c0[9];
#pragma unroll
    for (int q = 0; q < 9; q++) {
        const int cell = cx[q / 3] * ncy + cy[q % 3];
        n[q] = ld_early(cnt + cell);
        if constexpr (SLOT) c0[q] = ld_early(s.cellCand + (size_t)cell * cells + sub);
        else c0[q] = ld_early(s.cellCand + (size_t)cell * kCellCap + sub);  // (by 'cells' the kernel spills)
    }
    int *lst = mem.list + (size_t)j * mem.rows * kListRow + col;
    int k = 0;
    auto test = [&](float4 c, bool on, int q) {
        float dr2;
        if (FAST) {
            const float dx = (p.x - c.x) - sx[q / 3], dy = (p.y - c.y) - sy[q % 3];
            dr2 = dx * dx + dy * dy;
        } else {
            float dxr, dxo, dyr, dyo;
            image_axis(p.x, c.x, s.Lx, s.wrapx, false, dxr, dxo);
            image_axis(p.y, c.y, s.Ly, s.wrapy, false, dyr, dyo);
            dr2 = dxr * dxr + dyr * dyr;
        }
        const int tag = __float_as_int(c.z);
        const bool hit = on && dr2 <= R2 && (tag & kIdMask) != i && (gi == -1 || gi != __float_as_int(c.w));
        const unsigned hits = (__ballot_sync(0xffffffffu, hit) >> shift) & ((1u << kListLanes) - 1u);
        if (hit) {
            const int at = k + __popc(hits & ((1u << sub) - 1u));
            if (at < mem.rows) lst[at * kListRow] = tag;
            else if (at < cap) s.nbr[nbr_at(at, i, s.Ncap)] = tag;
        }
        k += __popc(hits);
    };
    bool more = false;
#pragma unroll
    for (int q = 0; q < 9; q++) {
        n[q] = valid ? min(n[q], cells) : 0;
        more = more || n[q] > kListLanes;
    }
    if (!__any_sync(0xffffffffu, more)) {
#pragma unroll
        for (int q = 0; q < 9; q++) test(c0[q], sub < n[q], q);
    } else {
#pragma unroll
        for (int q = 0; q < 9; q++) {
            test(c0[q], sub < n[q], q);
            const int most = __reduce_max_sync(0xffffffffu, n[q]);
            const int cell = cx[q / 3] * ncy + cy[q % 3];
            for (int o = kListLanes; o < most; o += kListLanes) {
                const bool on = o + sub < n[q];
                test(s.cellCand[(size_t)cell * cells + (on ? o + sub : 0)], on, q);
            }
        }
    }
    if (valid && sub == 0) {
        s.nbrCount[i] = k;
        mem.count[j * kStepBlock + col] = min(k, cap);
    }
    return k;
}

// NeighborList::update's taken branch for the positions of buffer p: cells of
// at most cell_cap particles by counting atomics, the in-cell order by id,
// and the lists of the block's own particles.  Two exchanges.  A non-finite
// position or a crowded cell ends the launch here, on every block alike
// (kRebuildLeft): there are no lists to go on with (before a run's first rebuild
// not even old ones), and the host repeats the run from its start by the plain kernels.
enum CoopRebuild { kRebuildLost, kRebuildLeft, kRebuildDone };  // lost: an exchange gave up

template <bool SLOT>
__device__ __forceinline__ CoopRebuild coop_rebuild(const DevSys &s, CoopShared &sh, const CoopMem &mem, CoopRun &r,
                                                    int p, bool withhold) {
    const float2 *pos = p ? s.pos1 : s.pos0;
    DevScalars *sc = s.sc;
    const int groups = blockDim.x / kStepBlock;
    const int grp = threadIdx.x / kStepBlock, gt = threadIdx.x % kStepBlock, lane = threadIdx.x & 31;
    r.updates += 1;
    r.dispHi = 0.0f;
    r.cnt ^= 1;
    int *cnt = s.cellFill + (size_t)r.cnt * s.ncells, *other = s.cellFill + (size_t)(r.cnt ^ 1) * s.ncells;
    const int cap = cell_cap<SLOT>(s);
    // 1: cells, and the ids into them in any order
    for (int j = grp; j < mem.tiles; j += groups) {
        const int i = (mem.first + j * mem.stride) * kStepBlock + gt;
        if (i >= s.N) continue;
        const float2 x = pos[i];
        if (!(isfinite(x.x) && isfinite(x.y))) atomicOr(&sc->nonfinite, 1);
        if (outside_box(s, x)) atomicOr(&sc->outside, 1);
        const int c = cell_col(x.x, x.y, s.ncx, s.ncy, s.Lx, s.Ly);
        s.cellOf[i] = c;
        const int k = atomicAdd(cnt + c, 1);
        if (k < cap) s.cellIds[(size_t)c * cap + k] = i;
        else atomicOr(&sc->overflow, kCoopCrowded);
        if (SLOT && k >= cap) atomicMax(&sc->maxCell, k + 1);
    }
    __syncthreads();
    if (!coop_exchange(s, sh, r, 0u, withhold)) return kRebuildLost;
    // the same on every block: what is tested was stored before its block's part
    // of the exchange above, and nothing sets it again before the next one, which no
    // block completes without this one
    if (__ldcg(&sc->nonfinite) != 0 || (__ldcg(&sc->overflow) & kCoopCrowded)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            atomicOr(&sc->overflow, kCoopLeft);
            sc->builds -= (unsigned long long)(r.updates - 1);  // the run's lists are built again by its repeat
        }
        return kRebuildLeft;
    }
    // 2: ascending id inside each cell; the other counts cleared for the next
    // rebuild (their last readers were the lists before this rebuild)
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < s.ncells; c += gridDim.x * blockDim.x) other[c] = 0;
    // by slot: the cells' starts (no terms there now; at most 16,384 particles)
    [[maybe_unused]] unsigned short *start = reinterpret_cast<unsigned short *>(mem.term);
    if constexpr (SLOT) {
        const int chunk = (s.ncells + blockDim.x - 1) / blockDim.x;
        const int c0 = min((int)threadIdx.x * chunk, s.ncells), c1 = min(c0 + chunk, s.ncells);
        int sum = 0, tot;
        for (int c = c0; c < c1; c++) {
            const int n = min(__ldcg(cnt + c), cap);
            start[c] = (unsigned short)n;
            sum += n;
        }
        int at = block_scan(sh, sum, tot);
        for (int c = c0; c < c1; c++) {
            const int n = start[c];
            start[c] = (unsigned short)at;
            at += n;
        }
        __syncthreads();
    }
    for (int j = grp; j < mem.tiles; j += groups) {
        const int i = (mem.first + j * mem.stride) * kStepBlock + gt;
        if (i >= s.N) continue;
        const int c = s.cellOf[i], n = min(__ldcg(cnt + c), cap);
        const int4 *ids = reinterpret_cast<const int4 *>(s.cellIds + (size_t)c * cap);
        const float2 x = pos[i];
        const int tag = own_tag(s, i), gi = s.excl[i];
        int k = 0;
        for (int q = 0; q < n; q += 8) {
            const int4 a = __ldcg(ids + q / 4), b = __ldcg(ids + q / 4 + 1);
            const int id[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int u = 0; u < 8; u++) k += q + u < n && id[u] < i;
        }
        if constexpr (SLOT) mem.slot[j * kStepBlock + gt] = min(start[c] + k, s.N - 1);
        s.cellCand[(size_t)c * cap + k] = make_float4(x.x, x.y, __int_as_float(tag), __int_as_float(gi));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->nbrSum = 0ull;
        sc->maxCount = 0;
        sc->builds += 1ull;
    }
    __syncthreads();
    if (!coop_exchange(s, sh, r, 0u)) return kRebuildLost;
    // 3: the lists of the block's own particles
    {
        const bool fast = (s.wrapx ? s.ncx >= 5 : s.ncx >= 3) && (s.wrapy ? s.ncy >= 5 : s.ncy >= 3) &&
                          !__ldcg(&sc->outside);  // fast_walk_ok
        constexpr int per = 32 / kListLanes;      // particles per warp
        int kmax = 0, ksum = 0;
        for (int b = (threadIdx.x >> 5) * per; b < mem.tiles * kStepBlock; b += (blockDim.x >> 5) * per) {
            const int q = b + lane / kListLanes, j = q / kStepBlock, col = q % kStepBlock;
            const int i = (mem.first + j * mem.stride) * kStepBlock + col;
            const int k = fast ? coop_list<true, SLOT>(s, mem, cnt, pos, i, j, col, i < s.N)
                               : coop_list<false, SLOT>(s, mem, cnt, pos, i, j, col, i < s.N);
            if (i < s.N && (lane & (kListLanes - 1)) == 0) {
                kmax = max(kmax, k);
                ksum += k;
            }
        }
        __syncwarp();
        kmax = __reduce_max_sync(0xffffffffu, kmax);
        ksum = __reduce_add_sync(0xffffffffu, ksum);
        if (lane == 0) {
            if (ksum) atomicAdd(&sc->nbrSum, (unsigned long long)ksum);
            if (kmax > 0) atomicMax(&sc->maxCount, kmax);
            if (kmax > s.nbrCap) atomicOr(&sc->overflow, 1);
        }
    }
    __syncthreads();
    return kRebuildDone;
}

// The lists of the last rebuild where the getters and the kernels that follow
// read them, a 16-byte group per store; unused words of a particle's last group
// are zero (FAST: the ghost slot's number; and the records of the step blocks,
// which are kStepBlock slots each, say that they have no window and how many
// groups their longest list has).
template <bool FAST>
__device__ __forceinline__ void coop_write_lists(const DevSys &s, const CoopMem &mem) {
    const int tiles = mem.tiles;
    for (int q = threadIdx.x; q < tiles * kStepBlock; q += blockDim.x) {
        const int j = q / kStepBlock, col = q % kStepBlock, i = (mem.first + j * mem.stride) * kStepBlock + col;
        if (i >= s.N) continue;
        const int k = min(mem.count[q], mem.rows);
        const int *lst = mem.list + (size_t)j * mem.rows * kListRow + col;
        for (int g = 0; 4 * g < k; g++) {
            int v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = 4 * g + u < k ? lst[(4 * g + u) * kListRow] : (FAST ? s.N : 0);
            reinterpret_cast<int4 *>(s.nbr)[(size_t)g * s.Ncap + i] = make_int4(v[0], v[1], v[2], v[3]);
        }
        const int all = mem.count[q];
        if (FAST && all > mem.rows)
            for (int e = all; e & 3; e++) s.nbr[nbr_at(e, i, s.Ncap)] = s.N;
    }
    if (FAST) {
        static_assert(kStepBlock == kFastBlock, "a tile is a step block");
        const int lane = threadIdx.x & 31;
        for (int j = threadIdx.x >> 5; j < tiles; j += blockDim.x >> 5) {
            const int b = mem.first + j * mem.stride;
            int most = 0;
            for (int c = lane; c < kStepBlock; c += 32)
                if (b * kStepBlock + c < s.N) most = max(most, mem.count[j * kStepBlock + c]);
            most = __reduce_max_sync(0xffffffffu, most);
            int *w = s.blockWin + kWinInts * (size_t)b;
            for (int c = lane; c < kWinInts; c += 32) w[c] = c == kWLen ? -1 : (c == kWGroups ? (most + 3) >> 2 : 0);
        }
    }
}

// The cell arrays of the last rebuild as the plain kernels leave them:
// cellStart (the exclusive scan of the counts, a contiguous chunk of cells per
// block), sortedIds and cellSorted.
template <bool SLOT>
__device__ __forceinline__ bool coop_cells(const DevSys &s, CoopShared &sh, CoopRun &r) {
    const int cap = cell_cap<SLOT>(s);
    const int *cnt = s.cellFill + (size_t)r.cnt * s.ncells;
    const int chunk = (s.ncells + gridDim.x - 1) / gridDim.x;
    const int c0 = min((int)blockIdx.x * chunk, s.ncells), c1 = min(c0 + chunk, s.ncells);
    int sum = 0, tot = 0;
    for (int cb = c0; cb < c1; cb += blockDim.x) {
        const int c = cb + threadIdx.x;
        block_scan(sh, c < c1 ? min(__ldcg(cnt + c), cap) : 0, tot);
        sum += tot;
    }
    unsigned long long *counts = coop_words(s);
    if (threadIdx.x == 0) counts[blockIdx.x] = (unsigned long long)sum;
    __syncthreads();
    if (!coop_exchange(s, sh, r, 0u)) return false;
    if (threadIdx.x < 32) {
        int before = 0;
        for (int b = threadIdx.x; b < (int)blockIdx.x; b += 32) before += (int)__ldcg(counts + b);
        before = __reduce_add_sync(0xffffffffu, before);
        if (threadIdx.x == 0) sh.before = before;
    }
    __syncthreads();
    int carry = sh.before;
    for (int cb = c0; cb < c1; cb += blockDim.x) {
        const int c = cb + threadIdx.x;
        const int n = c < c1 ? min(__ldcg(cnt + c), cap) : 0;
        const int at = carry + block_scan(sh, n, tot);
        carry += tot;
        if (c < c1) s.cellStart[c] = at;
        for (int q = 0; q < n && at + q < s.N; q++) {
            const float4 e = __ldcg(s.cellCand + (size_t)c * cap + q);
            s.cellSorted[at + q] = e;
            s.sortedIds[at + q] = __float_as_int(e.z) & kIdMask;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) s.cellStart[s.ncells] = s.N;
    return true;
}

// The four terms of one pair as lj_pair (step_body.cuh) adds them: force x and
// y, doubled energy and virial, or zeros outside the cutoff.
template <bool MT, bool SG, bool WX, bool WY, bool SIG1>
__device__ __forceinline__ float4 coop_pair(const DevSys &s, const PairEntry *tab, int ti, float si, float sj,
                                            float2 pi, int tag, float2 pj) {
    float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const PairEntry pe0 = tab[0];
    lj_pair_sig<MT, SG, WX, WY, SIG1>(s, tab, pe0, ti, si, sj, pi, tag, pj, o.x, o.y, o.z, o.w);
    return o;
}

// finish_particle (FAST: fast_finish), an axis per lane (lanes 2 and 3 along
// with 0 and 1).  f: lanes 0 and 1, the axis' force; e2: lanes 2 and 3, the
// doubled energy and virial.
template <bool WX, bool WY, bool FAST, bool SLOT>
__device__ __forceinline__ void coop_finish(const DevSys &s, const CoopMem &mem, int i, bool on, int j, int col, int q,
                                            int mode, int stepNow, float2 pi, float m, float2 v2, float f, float e2,
                                            float uwall, float2 *pout, float2 *slot, float &vvm, bool &bad) {
    const bool y = q & 1;
    float e = e2 * 0.5f;
    if (q == 2) e += uwall;
    if (s.wallOn && on) {
        const float yw = wall_y(s, stepNow);
        const float dl = s.wallDelta[i];
        const float ht = (pi.y + dl) - yw;
        if (ht > 0.0f) {
            if (q == 1) f -= s.wallK * ht;
            if (q == 2) e += 0.5f * s.wallK * ht * ht;
        }
        const float hb = dl - pi.y;
        if (hb > 0.0f) {
            if (q == 1) f += s.wallK * hb;
            if (q == 2) e += 0.5f * s.wallK * hb * hb;
        }
    }
    bad = bad || (on && !isfinite(f));
    const float a = FAST ? f * rcp_approx(m) : f / m;
    float v = y ? v2.y : v2.x, vv = 0.0f;
    if (mode != MODE_FIRST) {
        v = FAST ? __fmaf_rn(s.hdt, a, v) : v + s.hdt * a;
        const float sq = v * v, other = __shfl_xor_sync(0xffffffffu, sq, 1);
        vv = sq + other;
        if (FAST) {
            vv = __fmaf_rn(v, v, other);  // on the lanes of the x axis
            vv = __shfl_sync(0xffffffffu, vv, threadIdx.x & 30);
        }
    }
    if constexpr (SLOT) {
        if (on && q != 1) {
            const int at = mem.slot[j * kStepBlock + col];
            mem.eng[(q == 0 ? 2 : q - 2) * mem.engRow + at] = q == 0 ? m * vv : e;
        }
    } else {
        float *part = mem.part + (size_t)j * 3 * kStepBlock + col;
        if (q == 2) part[0] = on ? e : 0.0f;
        if (q == 3) part[kStepBlock] = on ? e : 0.0f;
        if (q == 0) part[2 * kStepBlock] = on ? m * vv : 0.0f;
    }
    if (on && q < 2) {
        vvm = fmaxf(vvm, vv);
        float *vel = reinterpret_cast<float *>(s.vel + i) + q;
        if (mode == MODE_LAST) {
            *vel = v;
            reinterpret_cast<float *>(s.acc + i)[q] = a;
            reinterpret_cast<float *>(s.forceOut + i)[q] = f;
        } else {
            const float p = y ? pi.y : pi.x, L = y ? s.Ly : s.Lx;
            v = FAST ? __fmaf_rn(s.hdt, a, v) : v + s.hdt * a;
            float x = FAST ? __fmaf_rn(s.dt, v, p) : p + s.dt * v;
            if (y ? WY : WX) x = FAST ? fast_wrap(x, L) : wrap_near(x, L);
            reinterpret_cast<float *>(pout + i)[q] = x;
            *vel = v;
            if (slot) reinterpret_cast<float *>(slot + i)[q] = x;
        }
    }
}

// The pair sums of the fast mode and the rest of the step.  Components of the
// terms: one type fc, dx, dy, ir6, ir2, r2; several types fc, dx, dy, u, r2.
// Lane 0 forms sum fc dx, lane 1 sum fc dy; one type: lane 2 sum ir6^2 and sum
// ir6, lane 3 sum ir2 r2 (the pairs inside the cutoff), each over the even and
// the odd entries apart; several types: lane 2 sum u, lane 3 sum fc r2.
template <bool MT, bool WX, bool WY, bool SIG1, bool SLOT, class Gather>
__device__ __forceinline__ void fast_sums(const DevSys &s, const CoopMem &mem, const PairEntry *tab, Gather &gather,
                                          int most, int cnt, int q, int col, int ti, const int *tag, const float2 *pj,
                                          float2 pi, bool near, float fx, float fy, float ue, float uwall, float m,
                                          float2 v2, int i, bool on, int j, int mode, int stepNow, float2 *pout,
                                          float2 *slot, float &vvm, bool &bad) {
    const int ca = MT ? (q == 2 ? 3 : 0) : (q < 2 ? 0 : q + 1);
    const int cb = q < 2 ? q + 1 : (MT ? 4 : (q == 2 ? 3 : 5));
    const float *pa = mem.term + ca * kTermComp + col, *pb = mem.term + cb * kTermComp + col;
    float s0 = MT ? (q == 0 ? fx : (q == 1 ? fy : 0.0f)) : 0.0f, s1 = 0.0f, t0 = 0.0f, t1 = 0.0f;
    const PairEntry pe0 = tab[0];
    for (int base = 0; base < most; base += kQuadRows) {
        if (base > 0) gather(base);
#pragma unroll
        for (int u = 0; u < kQuadPairs; u++) {
            const PairEntry pe = MT ? tab[ti * s.numTypes + ((unsigned)tag[u] >> kIdBits)] : pe0;
            float dx, dy;
            if (near) {
                dx = fdiff<WX, true>(pi.x, pj[u].x, s.Lx);
                dy = fdiff<WY, true>(pi.y, pj[u].y, s.Ly);
            } else {
                dx = pi.x - pj[u].x;
                dy = pi.y - pj[u].y;
            }
            const float r2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
            const bool in = base + 4 * u + q < cnt && r2 < pe.rcut2;
            const float ir2 = in ? ((SIG1 && !MT) ? rcp_approx(r2) : pe.sig2 * rcp_approx(r2)) : 0.0f;
            const float ir4 = ir2 * ir2, ir6 = ir4 * ir2, ir8 = ir4 * ir4;
            const float fc = ir8 * __fmaf_rn(pe.c, ir6, -0.5f * pe.c);
            float *w = mem.term + (4 * u + q) * kTermRow + col;
            w[0] = fc;
            w[kTermComp] = dx;
            w[2 * kTermComp] = dy;
            if (MT) {
                w[3 * kTermComp] = in ? __fmaf_rn(pe.eps4, __fmaf_rn(ir6, ir6, -ir6), pe.us) : 0.0f;
                w[4 * kTermComp] = r2;
            } else {
                w[3 * kTermComp] = ir6;
                w[4 * kTermComp] = ir2;
                w[5 * kTermComp] = r2;
            }
        }
        __syncwarp();
        const int rows = (min(most - base, kQuadRows) + 1) & ~1;
        if (MT) {
#pragma unroll 4
            for (int k = 0; k < rows; k++) s0 = __fmaf_rn(pa[k * kTermRow], q == 2 ? 1.0f : pb[k * kTermRow], s0);
        } else {
#pragma unroll 4
            for (int k = 0; k < rows; k += 2) {
                const float a0 = pa[k * kTermRow], a1 = pa[(k + 1) * kTermRow];
                s0 = __fmaf_rn(a0, pb[k * kTermRow], s0);
                s1 = __fmaf_rn(a1, pb[(k + 1) * kTermRow], s1);
                t0 += a0;
                t1 += a1;
            }
        }
        __syncwarp();
    }
    float f = 0.0f, e2;
    if (MT) {
        if (q < 2) f = s0;
        e2 = q == 2 ? ue + s0 : s0;
    } else {
        const float S = s0 + s1, T = t0 + t1;
        const int lane = threadIdx.x & 31, l2 = (lane & ~3) + 2;
        const float A = __shfl_sync(0xffffffffu, S, l2), B = __shfl_sync(0xffffffffu, T, l2);
        float n = __shfl_sync(0xffffffffu, S, l2 + 1);
        if (!SIG1) n = n / pe0.sig2;
        if (q == 0) f = fx + S;
        if (q == 1) f = fy + S;
        e2 = q == 2 ? ue + __fmaf_rn(pe0.eps4, A - B, pe0.us * n) : pe0.eps48 * __fmaf_rn(-0.5f, B, A);
    }
    coop_finish<WX, WY, true, SLOT>(s, mem, i, on, j, col, q, mode, stepNow, pi, m, v2, f, e2, uwall, pout, slot, vvm, bad);
}

// particle_step for one particle by the four lanes of a quad (lane 'q' of 0 ..
// 3; particle i, slot 'col' of the block's tile j; on: i < N).  All lanes of
// the warp call it.
template <bool MT, bool SG, bool WX, bool WY, bool SIG1, bool FAST, bool SLOT>
__device__ __forceinline__ void coop_particle(const DevSys &s, const CoopMem &mem, const PairEntry *tab, int i, bool on,
                                              int j, int col, int q, int mode, int stepNow, const float2 *pin,
                                              float2 *pout, float2 *slot, float &vvm, bool &bad) {
    const int ic = on ? i : 0;
    const int cnt = on ? mem.count[j * kStepBlock + col] : 0;
    const int *lst = mem.list + (size_t)j * mem.rows * kListRow + col;
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    // the lane's entries base + q, base + q + 4, ... and their positions
    int tag[kQuadPairs];
    float2 pj[kQuadPairs];
    auto gather = [&](int base) {
#pragma unroll
        for (int u = 0; u < kQuadPairs; u++) {
            const int k = base + 4 * u + q;
            tag[u] = ic;  // an unused place: the particle itself, no term is taken from it
            if (k < cnt) tag[u] = k < mem.rows ? lst[k * kListRow] : s.nbr[nbr_at(k, i, s.Ncap)];
        }
#pragma unroll
        for (int u = 0; u < kQuadPairs; u++) pj[u] = ld_early(pin + (tag[u] & kIdMask));
    };
    const float2 pi = ld_early(pin + ic);
    gather(0);
    const float m = s.mass[ic];
    const float2 v2 = ld_early(s.vel + ic);
    const int ti = MT ? s.typeId[ic] : 0;
    const float si = SG ? s.sigma[ic] : 0.0f;
    // what comes before the pair forces (bonded_forces), on every lane
    float ue = 0.0f, utri = 0.0f, uwall = 0.0f, fx = 0.0f, fy = 0.0f;
    const int *inc = mem.inc ? mem.inc + (size_t)j * kIncWords * kStepBlock + col : nullptr;
    const int head = (inc && on && i < s.nBonded) ? inc[0] : -1;
    if (head >= 0) {
        // with the incidences at hand: the triangles' forces and the first
        // two partners in flight, then the terms in order
        const int nT = head & 0xff, nB = head >> 8;
        auto bond = [&](int k) {
            return make_int2(inc[(1 + kIncTri + 2 * k) * kStepBlock], inc[(2 + kIncTri + 2 * k) * kStepBlock]);
        };
        float2 tf[kIncTri], pb[2];
#pragma unroll
        for (int k = 0; k < kIncTri; k++)
            if (k < nT) {
                const int e = inc[(1 + k) * kStepBlock];
                tf[k] = mem.triF ? mem.triF[e] : ld_early(s.triF + e);
            }
#pragma unroll
        for (int k = 0; k < 2; k++)
            if (k < nB) pb[k] = ld_early(pin + (bond(k).x & 0x7fffffff));
        if (s.refWalls) ref_walls(s, i, pi, fx, fy, uwall);
        if (s.gravity > 0.0f) fy -= m * s.gravity;
#pragma unroll
        for (int k = 0; k < 2; k++)
            if (k < nB) bond_term<WX, WY>(s, bond(k), pi, pb[k], fx, fy, ue);
        for (int k = 2; k < nB; k++) {
            const int2 en = bond(k);
            bond_term<WX, WY>(s, en, pi, pin[en.x & 0x7fffffff], fx, fy, ue);
        }
#pragma unroll
        for (int k = 0; k < kIncTri; k++)
            if (k < nT) {
                fx += tf[k].x;
                fy += tf[k].y;
            }
    } else if (on) {
        bonded_forces<WX, WY, false>(s, i, mode, pin, pi, fx, fy, ue, utri, uwall);
    }
    const bool near = __any_sync(0xffffffffu, on && near_edge<WX, WY>(s, pi));
    if constexpr (FAST) {
        fast_sums<MT, WX, WY, SIG1, SLOT>(s, mem, tab, gather, most, cnt, q, col, ti, tag, pj, pi, near, fx, fy, ue, uwall,
                                    m, v2, i, on, j, mode, stepNow, pout, slot, vvm, bad);
        return;
    }
    // the pairs: the lane's sum is force x, force y, energy or virial
    float sum = q == 0 ? fx : (q == 1 ? fy : (q == 2 ? ue : 0.0f));
    const float *mine = mem.term + q * kTermComp + col;
    for (int base = 0; base < most; base += kQuadRows) {
        if (base > 0) gather(base);
        float4 o[kQuadPairs];
        bool done = false;
        if (SIG1 && !SG) {
            // the packed terms, with the images where a lane of the warp is
            // near an edge; the scalar ones where they do not stand
            float far = 0.0f, close = 1.0f, w = 0.0f;
            auto packed = [&](auto edge) {
#pragma unroll
                for (int u = 0; u < kQuadPairs; u++) {
                    const bool in = base + 4 * u + q < cnt;
                    const float4 e = *reinterpret_cast<const float4 *>(
                        tab + (MT ? ti * s.numTypes + ((unsigned)tag[u] >> kIdBits) : 0));
                    o[u] = lj_terms_x2<decltype(edge)::value, WX, WY>(s, pi, pj[u], make_float2(e.x, e.y), e.z, e.w,
                                                                     in, far, close);
                    w += o[u].w;
                }
            };
            if (near) packed(std::true_type{});
            else packed(std::false_type{});
            done = !__any_sync(0xffffffffu, !lj_sums_ok<WX, WY>(s, far, close, w));
        }
        if (!done) {
#pragma unroll
            for (int u = 0; u < kQuadPairs; u++) {
                o[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (base + 4 * u + q < cnt)
                    o[u] = coop_pair<MT, SG, WX, WY, SIG1>(s, tab, ti, si, SG ? s.sigma[tag[u] & kIdMask] : 0.0f, pi,
                                                           tag[u], pj[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < kQuadPairs; u++) {
            float *w = mem.term + (4 * u + q) * kTermRow + col;
            w[0] = o[u].x;
            w[kTermComp] = o[u].y;
            w[2 * kTermComp] = o[u].z;
            w[3 * kTermComp] = o[u].w;
        }
        __syncwarp();
        const int rows = min(most - base, kQuadRows);
#pragma unroll 8
        for (int k = 0; k < rows; k++) sum += mine[k * kTermRow];
        __syncwarp();
    }
    coop_finish<WX, WY, false, false>(s, mem, i, on, j, col, q, mode, stepNow, pi, m, v2, q < 2 ? sum : 0.0f, sum, uwall, pout,
                               slot, vvm, bad);
}

// One warp: the block's energy sums of a step.  A tile's 128 particles in the
// plain kernels' grouping: FP32 over 32 lanes (warp_sum_f), over the four
// warps in order, then fixed point; a triangle tile's eight warp sums alike.
// Warps 'w0', w0 + 1, ... of the block share the tiles.
__device__ __forceinline__ void coop_block_sums(const DevSys &s, CoopShared &sh, const CoopMem &mem, int ttiles,
                                                int w0) {
    const int tiles = mem.tiles;
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) - w0, nw = (blockDim.x >> 5) - w0;
    bool ob = false;
    for (int j = w; j < tiles; j += nw) {
        const float *part = mem.part + (size_t)j * 3 * kStepBlock + lane;
        float t[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int g = 0; g < kStepBlock / 32; g++)
#pragma unroll
            for (int c = 0; c < 3; c++) t[c] += warp_sum_f(part[c * kStepBlock + 32 * g]);
        if (lane == 0)
#pragma unroll
            for (int c = 0; c < 3; c++) atomicAdd(&sh.acc[c], to_fixed(t[c], ob));
    }
    for (int j = w * 32 + lane; j < ttiles; j += nw * 32) {
        float x = 0.0f;
#pragma unroll
        for (int g = 0; g < kTriTile / 32; g++) x += sh.tred[j][g];
        atomicAdd(&sh.acc[0], to_fixed(x, ob));
    }
    if (ob) atomicOr(&s.sc->nonfinite, 2);
}

// By slot: the energies of a step (e) over the block's tiles of slots, as
// coop_block_sums.  Warps w0, w0 + 1, w0 + 2 take U, W, K.
__device__ __forceinline__ void coop_slot_sums(const DevSys &s, CoopShared &sh, const CoopMem &mem, const float *e, int w0) {
    const int lane = threadIdx.x & 31, c = (int)(threadIdx.x >> 5) - w0;
    if (c < 0 || c >= 3) return;
    bool ob = false;
    for (int j = 0; j < mem.tiles; j++) {
        const int t = (mem.first + j * mem.stride) * kStepBlock + lane;
        float v[kStepBlock / 32], x = 0.0f;
#pragma unroll
        for (int g = 0; g < kStepBlock / 32; g++) v[g] = t + 32 * g < s.N ? __ldcg(e + c * mem.engRow + t + 32 * g) : 0.0f;
#pragma unroll
        for (int g = 0; g < kStepBlock / 32; g++) x += warp_sum_f(v[g]);
        if (lane == 0) atomicAdd(&sh.acc[c], to_fixed(x, ob));
    }
    if (ob) atomicOr(&s.sc->nonfinite, 2);
}

// Triangles by block: the energies 'e' of all the triangles, summed over the block's
// triangle tiles as coop_block_sums does.  Warps w0, w0 + 1, ... share
// the tiles, the last one first.
__device__ __forceinline__ void coop_tri_block_sums(const DevSys &s, CoopShared &sh, const float *e, int ttiles, int w0) {
    const int lane = threadIdx.x & 31, nw = (blockDim.x >> 5) - w0, w = nw - 1 - ((int)(threadIdx.x >> 5) - w0);
    bool ob = false;
    for (int j = w; j < ttiles; j += nw) {
        const int t = (blockIdx.x + j * gridDim.x) * kTriTile + lane;
        float v[kTriTile / 32], x = 0.0f;
#pragma unroll
        for (int g = 0; g < kTriTile / 32; g++) v[g] = t + 32 * g < s.ntri ? __ldcg(e + t + 32 * g) : 0.0f;
#pragma unroll
        for (int g = 0; g < kTriTile / 32; g++) x += warp_sum_f(v[g]);
        if (lane == 0) atomicAdd(&sh.accTri, to_fixed(x, ob));
    }
    if (ob) atomicOr(&s.sc->nonfinite, 2);
}

}  // namespace

// A run or part of one: with 'begin', the run start (forced rebuild, first
// force pass, half kick and drift) and the checkpoint of the start state;
// then 'units' middle steps, each followed by its rebuild when the half-skin
// rule calls for one; with 'end', the last step.  slots: when not null, the
// positions after drift u go to slots + (u + 1) N too.  The parameters are grid
// constants: one whose address a function takes would be copied to local memory
// (256 disks, run(100): 825 us with the copy, 780 without).
template <bool MT, bool SG, bool WX, bool WY, bool SIG1, bool FAST, bool SLOT>
__global__ void __launch_bounds__(kCoopThreads, 1) k_coop(const __grid_constant__ DevSys s, const __grid_constant__ CoopArgs a) {
    extern __shared__ int4 dyn[];
    __shared__ CoopShared sh;
    DevScalars *sc = s.sc;
    // a launch of this run before this one was cut short (block 0 sets the word only
    // after an exchange that every block took part in, or one that gave up)
    if (!a.begin && __ldcg(&sc->runStop)) return;
    const int nt = MT ? s.numTypes * s.numTypes : 1;
    for (int q = threadIdx.x; q < nt; q += blockDim.x) sh.tab[q] = s.pair[q];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    CoopRun r = {};
    r.made = sc->runTag;
    r.dispHi = a.begin ? 0.0f : sc->dispHi;
    r.row = a.begin ? 0 : sc->obsRow;
    r.stepNow = a.begin ? s.stepBase : sc->stepNow;
    r.updates = a.begin ? 0 : sc->totalUpdates;
    r.cnt = sc->runFill;
    int p = a.parity;
    bool withhold = a.withhold && blockIdx.x == 0;
    // tile j of block b is tile b + j grid: 128 particles, worked by the whole
    // block, four lanes each
    static_assert(kCoopThreads == 4 * kStepBlock, "a quad per particle of a tile");
    const int ntiles = (s.N + kStepBlock - 1) / kStepBlock, groups = blockDim.x / kStepBlock;
    const int grp = threadIdx.x / kStepBlock, gt = threadIdx.x % kStepBlock;
    const bool tris = s.feaForces && s.ntri > 0;
    const int ntt = tris ? (s.ntri + kTriTile - 1) / kTriTile : 0, tgroups = blockDim.x / kTriTile;
    const int tgrp = threadIdx.x / kTriTile, tgt = threadIdx.x % kTriTile;
    const int per = (ntiles + gridDim.x - 1) / gridDim.x, tper = (ntt + gridDim.x - 1) / gridDim.x;
    const int ttiles = (int)blockIdx.x < ntt ? (ntt - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    CoopMem mem;
    mem.rows = a.rows;
    mem.tiles = coop_tiles(ntiles, gridDim.x, blockIdx.x, a.triLocal, mem.first, mem.stride);
    const bool local = tris && a.triLocal;
    const int nown = local ? a.triOfs[blockIdx.x + 1] - a.triOfs[blockIdx.x] : 0;
    mem.tri = a.triStaged || local ? dyn : nullptr;
    mem.triF = local ? reinterpret_cast<float2 *>(dyn + a.triMost) : nullptr;
    mem.term = reinterpret_cast<float *>(dyn + (a.triStaged ? tper * kTriTile : (a.triLocal ? a.triMost : 0)));
    if (a.triLocal) mem.term += 6 * a.triMost;
    mem.part = mem.term + coop_terms(FAST) * kTermComp;
    mem.count = reinterpret_cast<int *>(mem.part + (size_t)per * 3 * kStepBlock);
    mem.inc = a.incStaged ? mem.count + per * kStepBlock : nullptr;
    mem.list = mem.count + per * kStepBlock + (a.incStaged ? per * kIncWords * kStepBlock : 0);
    if constexpr (SLOT) {
        mem.engRow = s.N;
        mem.eng = nullptr;
        mem.slot = mem.list;
        mem.list += per * kStepBlock;
        if (!a.begin)  // as the last rebuild left it
            for (int t = threadIdx.x; t < s.N; t += blockDim.x) {
                const int i = s.sortedIds[t], k = i / kStepBlock - mem.first;
                if (k >= 0 && k % mem.stride == 0 && k / mem.stride < mem.tiles)
                    mem.slot[k / mem.stride * kStepBlock + i % kStepBlock] = t;
            }
    }
    const bool late = local || SLOT;  // a step's last sums are added after the next step's exchange
    if (a.begin) {
        const float2 *x = p ? s.pos1 : s.pos0;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.N; i += gridDim.x * blockDim.x) {
            a.ckPos[i] = x[i];
            a.ckVel[i] = s.vel[i];
            a.ckAcc[i] = s.acc[i];
        }
    }
    if (local) {
        const int *own = a.triOwn + a.triOfs[blockIdx.x];
        for (int k = threadIdx.x; k < nown; k += blockDim.x) {
            int4 q = __ldg(s.triIdx + (own[k] & 0x7fffffff));
            q.w = own[k];
            dyn[k] = q;
        }
    } else if (mem.tri)
        for (int j = tgrp; blockIdx.x + j * gridDim.x < ntt; j += tgroups) {
            const int t = (blockIdx.x + j * gridDim.x) * kTriTile + tgt;
            if (t < s.ntri) mem.tri[j * kTriTile + tgt] = __ldg(s.triIdx + t);
        }
    for (int j = grp; j < mem.tiles; j += groups) {
        const int i = (mem.first + j * mem.stride) * kStepBlock + gt;
        if (mem.inc && i < min(s.nBonded, s.N)) {
            int *inc = mem.inc + (size_t)j * kIncWords * kStepBlock + gt;
            const int tb = s.tStart[i], nT = s.feaForces ? s.tStart[i + 1] - tb : 0;
            const int bb = s.bStart[i], nB = s.bondForces ? s.bStart[i + 1] - bb : 0;
            const bool fits = nT <= kIncTri && nB <= kIncBond;
            inc[0] = fits ? (nT | nB << 8) : -1;
            for (int k = 0; fits && k < nT; k++) {
                const int en = __ldg(s.tEnt + tb + k);
                inc[(1 + k) * kStepBlock] = local ? __ldg(a.triLoc + tb + k) : 3 * (en >> 2) + (en & 3);  // its force
            }
            for (int k = 0; fits && k < nB; k++) {
                const int2 en = __ldg(s.bEnt + bb + k);
                inc[(1 + kIncTri + 2 * k) * kStepBlock] = en.x;
                inc[(2 + kIncTri + 2 * k) * kStepBlock] = en.y;
            }
        }
        if (!a.begin && i < s.N) {
            // lists from the last rebuild before this launch
            const int cnt = min(s.nbrCount[i], s.nbrCap);
            mem.count[j * kStepBlock + gt] = cnt;
            for (int k = 0; k < min(cnt, mem.rows); k++)
                mem.list[((size_t)j * mem.rows + k) * kListRow + gt] = s.nbr[nbr_at(k, i, s.Ncap)];
        }
    }
    if (threadIdx.x < 3) sh.acc[threadIdx.x] = 0ull;
    if (threadIdx.x == 3) sh.accTri = 0ull;
    __syncthreads();
    bool ok = true;
    const int updates0 = r.updates;
    bool rebuild = a.begin || (a.check && __ldcg(&sc->rebuild));
    const int total = (a.begin ? 1 : 0) + a.units + (a.end ? 1 : 0);
    for (int u = 0;; u++) {
        if (rebuild) {
            // (neither lists nor their lengths are read before a rebuild that was
            // made, or the lists of the launch before, loaded above)
            ok = coop_rebuild<SLOT>(s, sh, mem, r, p, withhold) == kRebuildDone;
            withhold = false;
            if (!ok) break;
        }
        if (u >= total) break;
        const int mode = (a.begin && u == 0) ? MODE_FIRST : ((a.end && u == total - 1) ? MODE_LAST : MODE_MID);
        const float2 *pin = p ? s.pos1 : s.pos0;
        float2 *pout = p ? s.pos0 : s.pos1;
        if (local) {
            // every triangle of the block's particles: the forces stay here
            float *te = a.triTmp + (size_t)(r.dueIn % 3u) * s.ntri;
            for (int k = threadIdx.x; k < nown; k += blockDim.x) {
                const int4 q = dyn[k];
                const int t = q.w & 0x7fffffff;
                float2 f[3];
                const float e = tri_eval(s, pin, t, q, f);
#pragma unroll
                for (int c = 0; c < 3; c++) mem.triF[3 * k + c] = f[c];
                if (q.w >= 0) continue;
                te[t] = e;
                if (u == total - 1) {  // as the last force evaluation of the plain kernels leaves them
                    s.triE[t] = e;
#pragma unroll
                    for (int c = 0; c < 3; c++) s.triF[3 * t + c] = f[c];
                }
            }
            __syncthreads();
        } else if (tris) {
            for (int j = tgrp; blockIdx.x + j * gridDim.x < ntt; j += tgroups) {
                const int t = (blockIdx.x + j * gridDim.x) * kTriTile + tgt;
                float e = 0.0f;
                if (t < s.ntri) e = tri_force(s, pin, t, mem.tri ? mem.tri[j * kTriTile + tgt] : __ldg(s.triIdx + t));
                e = warp_sum_f(e);
                if (lane == 0) sh.tred[j][warp % (kTriTile / 32)] = e;
            }
            __syncthreads();
            if (!(ok = coop_exchange(s, sh, r, 0u, withhold))) break;
            withhold = false;
        }
        [[maybe_unused]] const float *lastEng = nullptr;
        if constexpr (SLOT) {
            lastEng = mem.eng;
            mem.eng = a.eng + (size_t)(r.dueIn % 3u) * 3 * mem.engRow;
        }
        float vvm = 0.0f;
        bool bad = false;
        for (int j = 0; j < mem.tiles; j++) {
            const int col = threadIdx.x >> 2, i = (mem.first + j * mem.stride) * kStepBlock + col;
            coop_particle<MT, SG, WX, WY, SIG1, FAST, SLOT>(s, mem, sh.tab, i, i < s.N, j, col, threadIdx.x & 3, mode, r.stepNow,
                                                pin, pout, a.slots ? a.slots + (size_t)(u + 1) * s.N : nullptr, vvm,
                                                bad);
        }
        vvm = warp_max(vvm);
        const unsigned anybad = __ballot_sync(0xffffffffu, bad);
        if (lane == 0) {
            sh.vmax[warp] = vvm;
            if (anybad) atomicOr(&sc->nonfinite, 1);
        }
        __syncthreads();
        float mm = 0.0f;
        if (warp == 0) mm = warp_max(lane < kCoopThreads / 32 ? sh.vmax[lane] : 0.0f);
        if (!(ok = coop_exchange(s, sh, r, __float_as_uint(mm), withhold, false,
                                 [&] {
                                     if constexpr (!SLOT) coop_block_sums(s, sh, mem, local ? 0 : ttiles, 3);
                                     else if (r.dueIn > 0) coop_slot_sums(s, sh, mem, lastEng, 3);
                                     if (local && r.dueIn > 0)
                                         coop_tri_block_sums(s, sh, a.triTmp + (size_t)((r.dueIn - 1) % 3u) * s.ntri,
                                                             ttiles, 3);
                                 })))
            break;
        withhold = false;
        if (threadIdx.x < 3) {
            // visible to the others with this block's next exchange (by slot: the
            // previous step's; none, zeros, after the first)
            atomicAdd(coop_sums(s, SLOT ? r.dueIn - 1 : r.dueIn) + threadIdx.x, sh.acc[threadIdx.x]);
            sh.acc[threadIdx.x] = 0ull;
        }
        if (late && r.dueIn > 0) {
            if (local && threadIdx.x == 3) {
                atomicAdd(coop_sums(s, r.dueIn - 1), sh.accTri);
                sh.accTri = 0ull;
            }
            if (blockIdx.x == 0 && threadIdx.x == 0) sh.due[(r.dueIn - 1) & 3u].x = (unsigned)r.made - 1u;
            r.dueOk = r.dueIn;
        }
        // the rebuild rule (md3dsystem.cpp:177, nn.cpp:118), the same on every block
        const float vm2 = __uint_as_float(sh.maxBits);
        int reb = 0;
        if (mode != MODE_FIRST) {
            const float d = r.dispHi + sqrtf(vm2) * s.dt;
            reb = d > s.halfSkinF;  // (double)d > halfSkin
            r.dispHi = d;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            CoopDue &d = sh.due[r.dueIn & 3u];
            d.x = (unsigned)r.made - 1u;
            d.set = r.dueIn;
            d.mode = mode;
            d.row = r.row;
            d.reb = reb;
            d.vm = vm2;
            d.d = r.dispHi;
            sc->rebuild = reb;
        }
        r.dueIn++;
        if (!late) r.dueOk = r.dueIn;
        if (mode != MODE_FIRST) r.row++;
        if (mode != MODE_LAST) {
            r.stepNow++;
            p ^= 1;
        }
        rebuild = mode == MODE_MID && reb;
    }
    if constexpr (SLOT) if (ok && r.dueIn > 0) {
        coop_slot_sums(s, sh, mem, mem.eng, 0);
        __syncthreads();
        if (threadIdx.x < 3) atomicAdd(coop_sums(s, r.dueIn - 1) + threadIdx.x, sh.acc[threadIdx.x]);
    }
    if (ok && local && r.dueIn > 0) {
        // the last step's triangle energies
        coop_tri_block_sums(s, sh, a.triTmp + (size_t)((r.dueIn - 1) % 3u) * s.ntri, ttiles, 0);
        __syncthreads();
        if (threadIdx.x == 3) atomicAdd(coop_sums(s, r.dueIn - 1), sh.accTri);
    }
    // the cell arrays of the last rebuild; then the last sums
    if (ok && r.updates != updates0) {
        coop_write_lists<FAST>(s, mem);
        ok = coop_cells<SLOT>(s, sh, r);
    }
    __syncthreads();
    if (ok) ok = coop_exchange(s, sh, r, 0u, false, true);
    if (ok && blockIdx.x == 0 && threadIdx.x == 64)
        for (; r.dueOut != r.dueIn; r.dueOut++) coop_totals(s, sh.due[r.dueOut & 3u]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->dispHi = r.dispHi;
        sc->obsRow = r.row;
        sc->stepNow = r.stepNow;
        sc->totalUpdates = r.updates;
        sc->runTag = r.made;
        sc->runFill = r.cnt;
        sc->runStop = !ok;
    }
}

// The kernel of a system with (MT) several types and (SG) a sigma per
// particle, in the fast mode or not.
template <bool MT, bool SG, bool WX, bool WY, bool FAST, bool SLOT>
const void *coop_sig(const DevSys &s) {
    if constexpr (!SG && !(FAST && MT)) {
        if (s.sigmaOne) return (const void *)k_coop<MT, SG, WX, WY, true, FAST, SLOT>;
    }
    return (const void *)k_coop<MT, SG, WX, WY, false, FAST, SLOT>;
}

template <bool MT, bool SG, bool FAST = false, bool SLOT = false>
const void *coop_image(const DevSys &s) {
    if (s.wrapx && s.wrapy) return coop_sig<MT, SG, true, true, FAST, SLOT>(s);
    if (s.wrapx) return coop_sig<MT, SG, true, false, FAST, SLOT>(s);
    return coop_sig<MT, SG, false, false, FAST, SLOT>(s);
}

// one translation unit each
const void *coop_kernel_one(const DevSys &s);    // k_coop.cu
const void *coop_kernel_types(const DevSys &s);  // k_coop_types.cu
const void *coop_kernel_sigma(const DevSys &s);  // k_coop_sigma.cu
const void *coop_kernel_fast(const DevSys &s);   // k_coop_fast.cu
const void *coop_kernel_slot(const DevSys &s);   // k_coop_slot.cu

}  // namespace femmd
