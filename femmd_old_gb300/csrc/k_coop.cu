// k_coop.cu -- launch of the whole-run kernel (k_coop.cuh), and its variant
// for one particle type.
#include <algorithm>
#include "k_coop.cuh"

namespace femmd {

const void *coop_kernel_one(const DevSys &s) { return coop_image<false, false>(s); }

namespace {

// Particles of the largest system that runs in one launch.  Measured on
// run(50) against the plain kernels' graph (us): LJ fluid 67,600 particles
// 1148 / 1539, 160,000 2095 / 1848 (equal near 125,000); disks in solvent
// 68,288 1512 / 1787, 150,800 2662 / 2111 (96,000); suspension 32,512
// 650 / 923, 130,048 1336 / 1254 (108,000).  Fast mode: LJ 97,969 1220 / 1419,
// disks in solvent 97,512 1717 / 2117, suspension 92,583 932 / 1262.
constexpr int kCoopMaxN = 98304;

const void *coop_kernel(const DevSys &s, bool bySlot) {
    if (s.fast) return bySlot ? coop_kernel_slot(s) : coop_kernel_fast(s);
    if (!s.sigmaByType) return coop_kernel_sigma(s);
    return s.numTypes > 1 ? coop_kernel_types(s) : coop_kernel_one(s);
}

constexpr size_t kCoopSmem = 180 * 1024;  // dynamic shared memory of a block at most

// Blocks of a system (one per tile, at most one per SM) and what their shared
// memory holds: terms, sums and counts always, then incidences and triangles
// where they fit, then as many list rows as do.
// False when the system does not fit.
bool coop_shape(const DevSys &s, int &grid, size_t &smem, CoopArgs &a) {
    const int ntiles = (s.N + kStepBlock - 1) / kStepBlock, ntt = (s.ntri + kTriTile - 1) / kTriTile;
    if (!(grid = coop_grid(s))) return false;
    const int per = (ntiles + grid - 1) / grid, tper = (ntt + grid - 1) / grid;
    if (per > kCoopMaxTiles || tper > kCoopMaxTiles) return false;
    const size_t own = (size_t)a.triMost * (sizeof(int4) + 3 * sizeof(float2));
    smem = coop_terms(s.fast) * (size_t)kTermComp * sizeof(float) + (size_t)per * 4 * kStepBlock * sizeof(int);  // terms, sums, counts
    const size_t inc = (size_t)per * kIncWords * kStepBlock * sizeof(int), tri = (size_t)tper * kTriTile * sizeof(int4);
    const size_t row = 4 * (size_t)per * kListRow * sizeof(int);  // four list rows
    if (a.eng) smem += (size_t)per * kStepBlock * sizeof(int);  // slots
    a.incStaged = s.nBonded > 0 && smem + inc + row <= kCoopSmem;
    if (a.incStaged) smem += inc;
    a.triLocal = a.triMost > 0 && a.incStaged && smem + own + row <= kCoopSmem;
    a.triStaged = ntt > 0 && !a.triLocal && smem + tri + row <= kCoopSmem;
    if (a.triStaged) smem += tri;
    if (a.triLocal) smem += own;
    a.rows = 4 * (int)std::min<size_t>(s.nbrCap / 4, (kCoopSmem - smem) / row);
    smem += a.rows / 4 * row;
    return a.rows > 0 || s.nbrCap == 0;
}

}  // namespace

// The blocks of a system: one per tile, at most one per SM (0: no device).  They
// depend on the topology alone: the exchanges count blocks over the life of the
// context, and the triangle forces can be turned on later.
int coop_grid(const DevSys &s) {
    int sms = 0, dev = 0;
    if (cudaGetDevice(&dev) || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) return 0;
    const int ntiles = (s.N + kStepBlock - 1) / kStepBlock, ntt = (s.ntri + kTriTile - 1) / kTriTile;
    return std::max(1, std::min(std::min(sms, kCoopMaxBlocks), std::max(ntiles, ntt)));
}

// Up to 128 tiles (a block has one then), cells whose starts fit the terms' place.
// The step kernels' per-step energies differ from sums in id order by float
// rounding; larger systems' sums are in id order (a slot of every particle after
// every rebuild would cost them a scan of all cells per block).
bool coop_by_slot(const DevSys &s) {
    return s.fast && s.numTypes <= 1 && s.nBonded == 0 && s.N <= 128 * kStepBlock &&
           s.ncells <= 2 * coop_terms(true) * kTermComp;
}

int coop_block(int ntiles, int grid, int tile) { return coop_pairs(ntiles, grid) ? tile / 2 : tile % grid; }

bool coop_run_fits(const DevSys &s, const CoopArgs &plan) {
    if ((s.fast && !s.sigmaByType) || s.areaUnits > 0 || s.trace || !s.cellCand || s.N <= 0) return false;
    int grid, resident = 0;
    size_t smem;
    CoopArgs a = plan;
    if (!coop_shape(s, grid, smem, a)) return false;
    // One type in the fast mode with long lists: from the fifth tile of a block on
    // shared memory does not hold them all, and the step kernel's packed loop is
    // faster.  LJ fluid, run(50), launch / plain kernels (us): capacity 56 (cutoff
    // 3.5), 70,000 particles 1149 / 1322, 80,000 1422 / 1380; 96 (cutoff 5), 1862 /
    // 1994 and 2293 / 2063; 48 (skin 1), 80,000 1063 / 1083, 98,000 1158 / 1140.
    const int ntiles = (s.N + kStepBlock - 1) / kStepBlock;
    if (s.fast && s.numTypes <= 1 && s.nBonded == 0 && ntiles > 4 * grid && s.nbrCap > 48) return false;
    if (kernel_setup(coop_kernel(s, a.eng), kCoopThreads, smem, &resident)) return false;
    return resident >= grid;
}

// The sizes a whole-run launch is made for: its cell table has kCellCap slots of 20
// bytes per cell (250 MB at most), so that a nearly empty box is left to the plain
// kernels.  Not a small fluid's in the fast mode: 2000 particles in 25,281 cells
// (density 0.01), run(100) 630 us against 1590 by the plain kernels; 64 in 8100,
// 411 against 1487.
bool coop_size_ok(const DevSys &s) {
    return s.N > 0 && s.N <= kCoopMaxN && (s.ncells <= 4 * s.N + 4096 || coop_by_slot(s));
}

cudaError_t launch_coop_run(cudaStream_t st, const DevSys &s, const CoopArgs &a) {
    int grid;
    size_t smem;
    DevSys sa = s;
    CoopArgs aa = a;
    if (!coop_shape(s, grid, smem, aa)) return cudaErrorInvalidConfiguration;
    void *args[] = {&sa, &aa};
    return cudaLaunchCooperativeKernel(coop_kernel(s, a.eng), dim3(grid), dim3(kCoopThreads), args, smem, st);
}

}  // namespace femmd
