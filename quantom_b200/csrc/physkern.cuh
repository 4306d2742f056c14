// Launchers of the physics-semantics kernels (kernels_physics.cu), called by
// the host side in physics_host.cu.
#pragma once
#include <algorithm>

#include "physdev.cuh"

namespace lima {

constexpr int kTB = 256;         // threads per block of the per-particle kernels and the step kernel
constexpr int kGroup = 8;        // columns of the list: the lanes of a particle come in groups of 8
constexpr int kBuildWarps = 4;   // warps per block of the list build
// The list build gives a warp one particle below this box size (more warps,
// shorter streams) and four from it on (fewer tests and one stream's fetches
// for four).  A host-issued rebuild with 1 / 4 particles a warp: 4,096
// particles 61 / 72 us, 8,192 76 / 78, 32,024 136 / 124, 258,192 748 / 571
// (14 us of each the call's synchronisation).  No size between 8,192, where the two
// are level, and 32,024 was measured.
constexpr int kBuildOneBelow = 16384;
constexpr int kMaxTypes = 32;    // LIMA_MAX_ATOM_TYPES
constexpr int kScanThreads = 1024;
// shared memory, static and dynamic together, that a block gets without the
// kernel's MaxDynamicSharedMemorySize being raised
constexpr size_t kSmemPlain = 48 * 1024;
// Before a launch with `dynamic` bytes of a kernel that has `fixed` static
// ones.  The limit belongs to the kernel and is shared by every context and
// host thread of the process, so it is only ever set to `most`, the largest
// size the kernel is launched with: set to each launch's own size, one thread
// could lower it between another's call here and its launch.  A failure is the
// error that cudaGetLastError gives next.
template <typename K>
inline void allow_smem(K kernel, size_t dynamic, size_t fixed, size_t most) {
    if (dynamic + fixed > kSmemPlain)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

// Lanes per particle in the step kernel: 8 (one list column each), more in
// boxes too small to fill the SMs' warps, where a lane's chain of chunk loads
// and gathers is the time.  Per step with 8 / 16 / 32 lanes: 880 particles
// 16.3 / 15.0 / 14.2 us, 1,948 17.5 / 16.3 / 15.8, 4,096 18.3 / 16.6 / 18.6,
// 8,192 20.1 / 21.4 / 23.1.  With energies (more sums to reduce, and the frame
// behind it) 200 steps: 880 4.60 / 4.52 / 3.97 ms, 1,948 4.72 / 5.11 / 5.09,
// 3,893 4.99 / 5.11 / 5.77.  The lines lie between these sizes (at a 1.2 nm cutoff,
// ~295 entries a list); none between them was measured, nor another cutoff.
constexpr int kStep32Below = 2048, kStep16Below = 6144, kStepEnergy32Below = 1024;
// the step kernel reads its list rows from shared memory, staged by bulk
// copies in groups of kStageRows rows (false: per-lane loads from the list).
// Built into liblima_b200_staged.so (LIMA_STAGED_LIST=1) beside the default
// library; it measured no faster on the 32k box.
#ifndef LIMA_STAGED_LIST
#define LIMA_STAGED_LIST 0
#endif
constexpr bool kStagedList = LIMA_STAGED_LIST != 0;
constexpr int kStageRows = 8;
// Verlet-list layout: entry k of particle slot i is column k % 8 of row k / 8,
// and a particle's rows come in chunks of kListChunk / 8 = 4: column g of
// chunk q holds rows 4q .. 4q + 3 in consecutive words, so the lane that owns
// column g reads its next four entries with one 8-byte (16-bit ids) or
// 16-byte (32-bit ids) load, and the 32 words of one chunk of consecutive
// particles follow each other.  The capacity per particle is a multiple of
// kListChunk.
constexpr int kListChunk = 32;
static_assert(kGroup == 8 && kListChunk == 4 * kGroup, "chunks of four 8-entry rows");
__host__ __device__ inline uint32_t nl_word(uint32_t n_pad, uint32_t i, uint32_t k) {
    return ((k >> 5) * n_pad + i) * 32u + (k & 7u) * 4u + ((k >> 3) & 3u);
}
// list capacity per particle: `want` entries rounded up to whole chunks
__host__ __device__ inline int nl_round_cap(int want) { return (want + kListChunk - 1) / kListChunk * kListChunk; }
// list entry `idx` (a word index of the layout above) in either id width
__device__ __forceinline__ uint32_t nl_load(const PhysDev& d, size_t idx) {
    return d.nl16 ? (uint32_t)reinterpret_cast<const uint16_t*>(d.nl)[idx] : d.nl[idx];
}
// whether the step kernels of this library take 16-bit list ids for n_pad
// slots: whenever they fit, except in the staged variant (32-bit rows)
constexpr int kIds16Slots = 65536;
bool list_ids_16bit(int n_pad);
// the step kernels of more than 8 lanes and the list build of one particle a
// warp exist for 16-bit ids alone (in the staged library the build's are 32-bit)
static_assert(kStep32Below <= kStep16Below && kStep16Below < kIds16Slots && kStepEnergy32Below < kIds16Slots &&
                  kBuildOneBelow < kIds16Slots,
              "small-box kernels take 16-bit ids");
// bytes of one list entry
__host__ __device__ inline size_t nl_entry_bytes(const PhysDev& d) { return d.nl16 ? 2 : 4; }

// lanes that walk one particle's list in the step kernel, and its blocks
int step_lanes(const PhysDev& d, bool energy);
int step_blocks(const PhysDev& d, bool energy);
// blocks of the bonded kernel (one thread per term; none without terms)
__host__ __device__ inline int bonded_blocks(const PhysDev& d) {
    const int nt = d.n_bonds + d.n_angles + d.n_dih;
    return (nt + kTB - 1) / kTB;
}

// the counting sort of the slots by the cell of `pos`: cell_key, cstart, order
void launch_sort(const PhysDev& d, const float4* pos, cudaStream_t s);
// the sort by the cell of pos[cur], and every per-slot array into cell order in the tmp arrays, reference positions
void launch_sort_permute(const PhysDev& d, int cur, bool mixed, cudaStream_t s);
// reference positions of an in-place build (particles not moved)
void launch_set_xref(const PhysDev& d, const float4* pos, cudaStream_t s);
// The Verlet list of positions pos (orig: orig ids by slot).  items
// (nullable): slots in cell order when the particles were not re-sorted.
// copy_cur >= 0: pos/orig are the permuted tmp arrays, and the build copies
// every tmp array back into the step arrays of that parity.
void launch_build_list(const PhysDev& d, const float4* pos, const uint32_t* orig, const uint32_t* items, int copy_cur,
                       bool mixed, cudaStream_t s);
// The bonded kernel of parity `cur` (term forces; ENERGY: block partials); returns the kernels launched
int launch_bonded(const PhysDev& d, int cur, bool energy, cudaStream_t s);
// The step kernel of parity `cur` (slot cur) or an energy evaluation (slot
// kSlotEval, integrate false), launched with a programmatic dependency on the
// bonded kernel before it.  tail: device-launchable rebuild graph the last
// block launches when a rebuild is due (nullptr: none).
void launch_step(const PhysDev& d, int cur, bool mixed, bool energy, bool integrate, int slot, cudaGraphExec_t tail,
                 cudaStream_t s);

}  // namespace lima
