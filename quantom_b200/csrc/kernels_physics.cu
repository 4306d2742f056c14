// Physics-semantics step kernels: Lorentz-Berthelot LJ with cutoff
// (+ potential switch), harmonic bonds/angles, periodic dihedrals, velocity
// Verlet with an optional Berendsen thermostat.  FP32 forces; in MIXED
// precision the force sums are compensated (every 8 pairs per lane and across
// lanes) and positions/velocities carry FP32 low parts; energy, virial and
// kinetic-energy reductions and the thermostat scalar are FP64, summed in a
// fixed order (run-to-run identical).
//
// Layout: particles sorted by cell (side >= r_list/2, x-major), so the
// kGroup = 8 lanes of the 4 particles a warp handles share a cell and read
// largely the same neighbours — the position gathers of a warp hit L1.
//
// Per step, one launch (captured in a CUDA graph):
//   k_step   8 or more lanes per particle walk its Verlet list (blocked so the
//            lanes of consecutive particles read one line), branch-free LJ +
//            switch; a compound particle's lanes also evaluate the bonded
//            terms it takes part in and keep its role's force; partial forces
//            reduced with warp shuffles; lane 0 kicks, drifts and gives the
//            kinetic energy.  Each block sums its FP64 values in a fixed
//            order into a partial; the block that finishes last adds the
//            partials in block order, sets the next step's Berendsen scalar
//            and, when a particle moved more than skin/2, tail-launches the
//            rebuild graph, which runs before the next step.
// Rebuild (a device-launchable graph, or host launches): k_sort_count (which
// also scans the counts), k_sort_fill, k_sort_order (a stable counting sort by
// cell; it also moves every per-slot array into the new order, through tmp
// arrays) and k_build_list — one warp per one or four particles over the
// columns of their 5x5x5 cell neighbourhood that their bounding box can
// reach, which also copies the permuted arrays back.
#include <type_traits>

#include "cellrange.cuh"
#include "physdev.cuh"
#include "physkern.cuh"
#include "physmath.cuh"
#include "refdev.cuh"

namespace lima {
namespace {

// error-free sum: s + e == a + b exactly
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float bp = s - a;
    e = (a - (s - bp)) + (b - bp);
}
// (hi, lo) += x
__device__ __forceinline__ void ds_add(float& hi, float& lo, float x) {
    float s, e;
    two_sum(hi, x + lo, s, e);
    hi = s;
    lo = e;
}

// lane 0 receives the warp's sum; the order of the additions is fixed
__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void cell_xyz(const PhysDev& d, float4 p, int& cx, int& cy, int& cz) {
    const float inv = (float)d.m / d.L;
    cx = cell_of(p.x, inv, d.m);
    cy = cell_of(p.y, inv, d.m);
    cz = cell_of(p.z, inv, d.m);
}

}  // namespace

// ----------------------------------------------------- counting sort by cell ---
// Cell of every slot and its arrival rank in the cell (atomic, so the ranks
// are put in slot order later).  The block that finishes last then scans the
// cell occupancies into cstart (cstart[n_cells] = n) and resets them to zero
// for the next sort, thread t owning a contiguous run of cells: a launch of its
// own for that one block cost about 3 us of a rebuild.
__global__ void __launch_bounds__(kScanThreads) k_sort_count(PhysDev d, const float4* __restrict__ pos) {
    __shared__ uint32_t s_warp[kScanThreads / 32];
    __shared__ int s_last;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.n) {
        int cx, cy, cz;
        cell_xyz(d, pos[i], cx, cy, cz);
        const uint32_t c = (uint32_t)((cx * d.m + cy) * d.m + cz);
        d.cell_key[i] = c;
        d.cell_rank[i] = atomicAdd(&d.ccount[c], 1u);
    }
    __threadfence();
    __syncthreads();
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (t == 0) s_last = atomicAdd(d.sort_done, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int per = (d.n_cells + kScanThreads - 1) / kScanThreads;
    const int b = min(d.n_cells, t * per), e = min(d.n_cells, b + per);
    uint32_t sum = 0u;
    for (int c = b; c < e; c++) sum += __ldcg(&d.ccount[c]);
    uint32_t x = sum;   // inclusive scan over the warp
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {   // kScanThreads / 32 == 32 warp totals
        uint32_t v = s_warp[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        s_warp[lane] = v;
    }
    __syncthreads();
    uint32_t run = (w ? s_warp[w - 1] : 0u) + x - sum;
    for (int c = b; c < e; c++) {
        const uint32_t k = __ldcg(&d.ccount[c]);
        d.cstart[c] = run;
        d.ccount[c] = 0u;
        run += k;
    }
    if (t == 0) {
        d.cstart[d.n_cells] = (uint32_t)d.n;
        *d.sort_done = 0u;   // for the next sort
    }
}

__global__ void k_sort_fill(PhysDev d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    d.order[d.cstart[d.cell_key[i]] + d.cell_rank[i]] = (uint32_t)i;
}

namespace {
// slot src of the step arrays becomes slot k of the tmp arrays; reference
// positions of the list; the orig <-> slot maps
__device__ __forceinline__ void permute_slot(const PhysDev& d, int cur, int mixed, uint32_t src, uint32_t k) {
    const float4 p = d.pos[cur][src];
    d.pos_tmp[0][k] = p;
    d.pos_tmp[1][k] = d.pos[cur ^ 1][src];
    d.vel_tmp[k] = d.vel[src];
    d.force_tmp[k] = d.force[src];
    if (mixed) {
        d.posc_tmp[k] = d.posc[src];
        d.velc_tmp[k] = d.velc[src];
    }
    const uint32_t o = d.orig_of_sorted[src];
    d.orig_tmp[k] = o;
    d.sorted_of_orig[o] = k;
    d.xref[k] = p;
}
}  // namespace

// One warp per cell: the cell's slots (in arrival order from k_sort_fill) put
// in ascending order, which makes the sort stable and the new order a
// function of the positions and the old order only.  Each lane ranks its slot
// by counting the smaller ones; cells of more than 32 particles are sorted by
// lane 0 (insertion sort).  PERMUTE: every per-slot array goes into the new
// order (tmp arrays) here too; else the order goes to d.order.
template <bool PERMUTE>
__global__ void k_sort_order(PhysDev d, int cur, int mixed) {
    const int lane = threadIdx.x & 31;
    const int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (c >= d.n_cells) return;
    const uint32_t b = d.cstart[c], n = d.cstart[c + 1] - b;
    if (n == 0u || (!PERMUTE && n == 1u)) return;
    if (n <= 32u) {
        const uint32_t v = (uint32_t)lane < n ? d.order[b + lane] : 0xffffffffu;
        uint32_t rank = 0u;
        for (uint32_t k = 0; k < n; k++) rank += __shfl_sync(0xffffffffu, v, (int)k) < v ? 1u : 0u;
        __syncwarp();
        if ((uint32_t)lane < n) {
            if (PERMUTE) permute_slot(d, cur, mixed, v, b + rank);
            else d.order[b + rank] = v;
        }
        return;
    }
    if (lane == 0)
        for (uint32_t k = b + 1; k < b + n; k++) {
            const uint32_t v = d.order[k];
            uint32_t j = k;
            while (j > b && d.order[j - 1] > v) {
                d.order[j] = d.order[j - 1];
                j--;
            }
            d.order[j] = v;
        }
    if (PERMUTE) {
        __threadfence_block();
        __syncwarp();
        for (uint32_t k = lane; k < n; k += 32u) permute_slot(d, cur, mixed, d.order[b + k], b + k);
    }
}

// every per-slot array into cell order, in large boxes
__global__ void k_permute(PhysDev d, int cur, int mixed) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < d.n) permute_slot(d, cur, mixed, d.order[k], (uint32_t)k);
}

__global__ void k_set_xref(PhysDev d, const float4* __restrict__ pos) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < d.n) d.xref[k] = pos[k];
}


// Verlet-list build: one warp per P consecutive particles of the cell order.
// The warp's particles are taken in groups that share a home column (cells
// (x, y, *)) and a z-window of at most m-4 cells.  For a group, each of the 25
// columns around it is culled when the xy gap between the group's bounding
// box and the column exceeds r_list, and otherwise contributes the cells that
// the group's z-range, widened by the reach sqrt(r_list^2 - gap^2), overlaps:
// one or two contiguous slot ranges of the cell order (at most m cells).  The
// ranges are walked as one stream of candidates, lane = candidate, 32 at a
// time (the next 32 in flight while these are tested), shifted into the home
// frame by whole box lengths.  Each particle's hits among them are a ballot:
// the hit of rank r is appended to the particle's row in shared memory, r
// entries past its count, by a predicated store.  At the end bonded exclusions
// are taken out of the rows of the particles that have any, and the rows go to
// the list in whole chunk columns, one vector store per lane.  Rows list their
// neighbours in stream order (deterministic).  Boxes with fewer than 5 cells
// per side stream all particles with the minimum image.
//
// Bound: issue slots (the candidate's range and address, the hits' ranks), and
// latency where there are few warps; the list is written once.  So the hits
// are ranked by ballots with predicated stores (8 particles a warp, 4 lanes a
// particle walking the candidates took ~50 instructions per 32 tests for hit
// masks, ranks and branches), loops run on values the compiler knows to be
// uniform, exclusions cost only the rows that have any, and small boxes put
// one particle on a warp (kBuildOneBelow).  A host-issued rebuild, sort,
// launches and synchronisation included, on one B200 (before -> now): 4,096
// particles 118 -> 45 us, 8,192 123 -> 58, 32,024 158 -> 112, 258,192 687 -> 575.
// pos/orig: positions and orig ids by slot.  items (nullable): the cell order
// as a list of slots when the particles were not moved into it (in-place
// rebuild).  copy_cur >= 0: the particles were permuted into the tmp arrays
// (pos = pos_tmp[0], orig = orig_tmp); the build also copies every slot back
// into the step arrays of parity copy_cur (the rebuild's last copy).
namespace {

constexpr int kMaxRanges = 50;   // 25 columns, one or two slot ranges each
constexpr int kBuildRow = 1024;  // entries of a row in shared memory at most (a multiple of 32); longer lists are written in parts

// a warp's shared memory: its ranges, then P rows of `cap` entries
struct BuildRange {
    float x, y, z;   // shift
    int delta;       // cell-order position of stream index f: f + delta
};
__host__ __device__ inline size_t build_warp_smem(int p, int cap, size_t id_bytes) {
    return sizeof(BuildRange) * kMaxRanges + sizeof(int) * kMaxRanges + 8 + p * cap * id_bytes;
}

// A value that is the same in every lane, in a form the compiler knows to be
// (a warp reduction): control flow on it needs no reconvergence code around
// the votes it holds.
__device__ __forceinline__ int uniform(int v) { return __reduce_max_sync(0xffffffffu, v); }

// One particle's hits among the warp's 32 candidates (r2 < rl2): the hit of
// rank r stores its id j r entries past `at`, the shared address of the row's
// next entry (nothing at or past `end`); `at` then moves past the hits.
template <typename ID>
__device__ __forceinline__ void append_hits(float r2, float rl2, uint32_t j, uint32_t lt, uint32_t end, uint32_t& at) {
    if (sizeof(ID) == 2)
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t.reg .b32 b, t;\n\t.reg .b16 h;\n\tcvt.u16.u32 h, %3;\n\tsetp.lt.f32 p, %1, %2;\n\t"
            "vote.sync.ballot.b32 b, p, 0xffffffff;\n\tand.b32 t, b, %4;\n\tpopc.b32 t, t;\n\tmad.lo.u32 t, t, 2, %0;\n\t"
            "setp.lt.and.u32 q, t, %5, p;\n\t@q st.shared.b16 [t], h;\n\tpopc.b32 t, b;\n\tmad.lo.u32 %0, t, 2, %0;\n\t}"
            : "+r"(at)
            : "f"(r2), "f"(rl2), "r"(j), "r"(lt), "r"(end)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t.reg .b32 b, t;\n\tsetp.lt.f32 p, %1, %2;\n\t"
            "vote.sync.ballot.b32 b, p, 0xffffffff;\n\tand.b32 t, b, %4;\n\tpopc.b32 t, t;\n\tmad.lo.u32 t, t, 4, %0;\n\t"
            "setp.lt.and.u32 q, t, %5, p;\n\t@q st.shared.b32 [t], %3;\n\tpopc.b32 t, b;\n\tmad.lo.u32 %0, t, 4, %0;\n\t}"
            : "+r"(at)
            : "f"(r2), "f"(rl2), "r"(j), "r"(lt), "r"(end)
            : "memory");
}

// The rows to the list: bonded exclusions out of them (in place and in order),
// then their whole chunks, and the last partial one too if `all`.  Otherwise
// what is left moves to the row's start.  cnt: entries in the row; done:
// entries of the particle already in the list (a multiple of 32).
template <typename ID, int P>
__device__ __forceinline__ void flush_rows(const PhysDev& d, const uint32_t* __restrict__ orig, ID* rows, int cap, int i,
                                           int base, bool all, uint32_t (&cnt)[P], uint32_t (&done)[P], int lane) {
    __syncwarp();
#pragma unroll 1
    for (int p = 0; p < P; p++) {
        if (base + p >= d.n) break;
        const int ip = __shfl_sync(0xffffffffu, i, p);
        uint32_t c = cnt[0], dn = done[0];
#pragma unroll
        for (int k = 1; k < P; k++) {
            c = p == k ? cnt[k] : c;
            dn = p == k ? done[k] : dn;
        }
        c = min(c, (uint32_t)cap);
        ID* r = rows + (size_t)p * cap;
        const uint32_t oi = d.n_cp > 0 ? orig[ip] : 0u;
        const bool bonded = oi < (uint32_t)d.n_cp;
        const uint32_t x0 = bonded ? d.excl_off[oi] : 0u, x1 = bonded ? d.excl_off[oi + 1] : 0u;
        if (x1 > x0) {
            const uint32_t n = c;
            c = 0u;
            for (uint32_t e0 = 0; e0 < n; e0 += 32) {
                const uint32_t e = e0 + lane;
                const uint32_t j = e < n ? (uint32_t)r[e] : 0u;
                const uint32_t oj = e < n ? orig[j] : 0xffffffffu;
                bool keep = e < n;
                if (oj < (uint32_t)d.n_cp)
                    for (uint32_t q = x0; q < x1; q++) keep = keep && d.excl_ids[q] != oj;
                const unsigned kb = __ballot_sync(0xffffffffu, keep);   // (also: every lane has read its entry)
                if (keep) r[c + __popc(kb & ((1u << lane) - 1u))] = (ID)j;
                c += __popc(kb);
                __syncwarp();
            }
        }
        // lane 8 s + g writes column g of the chunks s, s + 4, ... (words past the count are never read as ids)
        const int g = lane & 7;
        const uint32_t chunks = all ? (c + 31u) >> 5 : c >> 5;
        for (uint32_t q = lane >> 3; q < chunks; q += 4u) {
            const ID* e = r + q * 32u + g;
            const uint32_t e0 = e[0], e1 = e[8], e2 = e[16], e3 = e[24];
            const size_t qn = (dn >> 5) + q;
            if (qn < (size_t)(d.nl_cap >> 5)) {
                const size_t v = (qn * d.n_pad + ip) * kGroup + g;
                if (sizeof(ID) == 2)
                    reinterpret_cast<uint2*>(d.nl)[v] = make_uint2(e0 | (e1 << 16), e2 | (e3 << 16));
                else
                    reinterpret_cast<uint4*>(d.nl)[v] = make_uint4(e0, e1, e2, e3);
            }
        }
        const uint32_t whole = c & ~31u;
        if (!all) {
            const uint32_t e = whole + lane;
            const ID j = e < c ? r[e] : (ID)0;
            __syncwarp();
            if (e < c) r[lane] = j;
            __syncwarp();
            dn += whole;
            c -= whole;
        }
#pragma unroll
        for (int k = 0; k < P; k++)
            if (p == k) {
                cnt[k] = c;
                done[k] = dn;
            }
    }
}

// The group's candidate stream (`total` of them, the same in every lane;
// n_ranges ranges in rg, their first stream indices in rstart) against its
// particles: px.. (NaN: not in the group) at cell-order positions first,
// first + 1, ...  ITEMS: the cell order is a list of slots.
// A stream can be empty: a particle that is alone in its group and not finite,
// or more than the list radius outside the box, reaches none of the columns
// around its clamped cell.  It then has no range to fetch from.
template <bool MIN_IMAGE, bool ITEMS, typename ID, int P>
__device__ __forceinline__ void scan_stream(const PhysDev& d, const float4* __restrict__ pos,
                                            const uint32_t* __restrict__ items, const BuildRange* rg, const int* rstart,
                                            int n_ranges, int total, int first, const uint32_t* __restrict__ orig,
                                            ID* rows, int i, uint32_t (&done)[P], const float (&px)[P],
                                            const float (&py)[P], const float (&pz)[P], uint32_t row, uint32_t cap,
                                            uint32_t (&cnt)[P], int lane) {
    if (total <= 0) return;
    constexpr uint32_t kB = sizeof(ID);
    const uint32_t lt = (1u << lane) - 1u, le = lt | (1u << lane);
    const float rl2 = d.rlist2, nan = __int_as_float(0x7fc00000), L = d.L, invL = d.invL;
    uint32_t at[P], end[P];
#pragma unroll
    for (int p = 0; p < P; p++) {
        at[p] = row + (p * cap + cnt[p]) * kB;
        end[p] = row + (p + 1) * cap * kB;
    }
    // lane l knows where ranges l and l + 32 start; a round's ranges are found
    // from the mask of those that start inside it
    int s0 = lane < n_ranges ? rstart[lane] : 0x3fffffff;
    int s1 = lane + 32 < n_ranges ? rstart[lane + 32] : 0x3fffffff;
    int f = lane, before = -1;   // the lane's stream index, the range the round starts in
    float4 c;
    int q;   // the candidate's cell-order position
    auto fetch = [&]() {   // past the stream's end: its last candidate again, made to fail the test
        const unsigned m = __reduce_or_sync(
            0xffffffffu, ((unsigned)s0 < 32u ? 1u << s0 : 0u) | ((unsigned)s1 < 32u ? 1u << s1 : 0u));
        const int r = before + __popc(m & le);
        before += __popc(m);
        s0 -= 32;
        s1 -= 32;
        const BuildRange g = rg[r];
        q = min(f, total - 1) + g.delta;
        const int j = ITEMS ? (int)__ldg(items + q) : q;
        const float4 p = __ldg(pos + j);
        c = make_float4(f < total ? p.x + g.x : nan, p.y + g.y, p.z + g.z, __int_as_float(j));
        q -= first;
        f += 32;
    };
    fetch();
#pragma unroll 1
    for (int left = total; left > 0; left -= 32) {
        const float4 e = c;
        const int qe = q;
        fetch();   // in flight during the tests
#pragma unroll
        for (int p = 0; p < P; p++) {
            float dx = e.x - px[p], dy = e.y - py[p], dz = e.z - pz[p];
            if (MIN_IMAGE) {
                dx = mimg(dx, L, invL);
                dy = mimg(dy, L, invL);
                dz = mimg(dz, L, invL);
            }
            float r2 = dx * dx + dy * dy + dz * dz;
            r2 = qe == p ? nan : r2;   // not itself
            append_hits<ID>(r2, rl2, __float_as_uint(e.w), lt, end[p], at[p]);
        }
        // rows shorter than the list's and the exclusions still in them: to the list before one can run over
        if (cap < (uint32_t)d.nl_room) {
            uint32_t room = end[0] - at[0];
#pragma unroll
            for (int p = 1; p < P; p++) room = min(room, end[p] - at[p]);
            if (uniform(-(int)room) > -(int)(32u * kB)) {
#pragma unroll
                for (int p = 0; p < P; p++) cnt[p] = (at[p] - row) / kB - p * cap;
                flush_rows<ID, P>(d, orig, rows, (int)cap, i, first, false, cnt, done, lane);
#pragma unroll
                for (int p = 0; p < P; p++) at[p] = row + (p * cap + cnt[p]) * kB;
            }
        }
    }
#pragma unroll
    for (int p = 0; p < P; p++) cnt[p] = (at[p] - row) / kB - p * cap;
}

}  // namespace

template <typename ID, int P>
__global__ void __launch_bounds__(kBuildWarps * 32, P == 1 ? 8 : 0) k_build_list(const __grid_constant__ PhysDev d,
                                                                 const float4* __restrict__ pos,
                                                                 const uint32_t* __restrict__ orig,
                                                                 const uint32_t* __restrict__ items, int copy_cur,
                                                                 int mixed, int cap) {
    extern __shared__ float4 s_build[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gw = blockIdx.x * kBuildWarps + w;
    if (copy_cur >= 0) {   // the rebuild's copy of the permuted tmp arrays into the step arrays
        if (gw == 0 && lane == 0) *d.need_rebuild = 0;
        for (int k = gw * 32 + lane; k < d.n; k += gridDim.x * kBuildWarps * 32) {
            d.pos[copy_cur][k] = d.pos_tmp[0][k];
            d.pos[copy_cur ^ 1][k] = d.pos_tmp[1][k];
            d.vel[k] = d.vel_tmp[k];
            d.force[k] = d.force_tmp[k];
            if (mixed) {
                d.posc[k] = d.posc_tmp[k];
                d.velc[k] = d.velc_tmp[k];
            }
            d.orig_of_sorted[k] = d.orig_tmp[k];
        }
    }
    const int base = gw * P;
    if (base >= d.n) return;   // the whole warp
    char* smem = reinterpret_cast<char*>(s_build) + (size_t)w * build_warp_smem(P, cap, sizeof(ID));
    BuildRange* rg = reinterpret_cast<BuildRange*>(smem);
    int* rstart = reinterpret_cast<int*>(rg + kMaxRanges);
    ID* rows = reinterpret_cast<ID*>(rstart + kMaxRanges + 2);   // P rows of cap entries
    const uint32_t row = (uint32_t)__cvta_generic_to_shared(rows);
    // lane p < P owns particle p of the warp
    const int qi = base + lane;   // position in the cell order
    const bool have = lane < P && qi < d.n;
    const int i = have ? (items ? (int)items[qi] : qi) : 0;   // slot
    const float4 pi = have ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float nan = __int_as_float(0x7fc00000);
    uint32_t cnt[P], done[P];
#pragma unroll
    for (int p = 0; p < P; p++) cnt[p] = done[p] = 0u;
    float px[P], py[P], pz[P];
    auto members = [&](bool in) {
        const float x = in ? pi.x : nan;
#pragma unroll
        for (int p = 0; p < P; p++) {
            px[p] = __shfl_sync(0xffffffffu, x, p);
            py[p] = __shfl_sync(0xffffffffu, pi.y, p);
            pz[p] = __shfl_sync(0xffffffffu, pi.z, p);
        }
    };
    const int m = d.m;
    if (m < 5) {   // one range: every particle, minimum image
        if (lane == 0) {
            rg[0] = BuildRange{0.f, 0.f, 0.f, 0};
            rstart[0] = 0;
        }
        __syncwarp();
        members(have);
        if (items)
            scan_stream<true, true, ID, P>(d, pos, items, rg, rstart, 1, d.n, base, orig, rows, i, done, px, py, pz, row,
                                           (uint32_t)cap, cnt, lane);
        else
            scan_stream<true, false, ID, P>(d, pos, items, rg, rstart, 1, d.n, base, orig, rows, i, done, px, py, pz, row,
                                            (uint32_t)cap, cnt, lane);
    } else {
        const float cs = d.L / (float)m, ics = (float)m / d.L;   // cell side
        int cx = -1, cy = -1, cz = 0;
        if (have) cell_xyz(d, pi, cx, cy, cz);
        unsigned todo = __reduce_or_sync(0xffffffffu, have ? 1u << lane : 0u);   // one bit per particle
        while (todo) {   // warp-uniform
            const int lead = __ffs(todo) - 1;
            const int hx = __shfl_sync(0xffffffffu, cx, lead);
            const int hy = __shfl_sync(0xffffffffu, cy, lead);
            const int hz0 = __shfl_sync(0xffffffffu, cz, lead);
            const bool mine = ((todo >> lane) & 1u) && cx == hx && cy == hy && cz <= hz0 + (m - 5);
            todo &= ~__reduce_or_sync(0xffffffffu, mine ? 1u << lane : 0u);
            const int hz1 = __reduce_max_sync(0xffffffffu, mine ? cz : -1);   // the group's top cell
            members(mine);
            GroupBox b = {3.4e38f, -3.4e38f, 3.4e38f, -3.4e38f, 3.4e38f, -3.4e38f};
#pragma unroll
            for (int p = 0; p < P; p++) {   // a NaN x marks a particle outside the group
                const bool in = px[p] == px[p];
                b.xl = fminf(b.xl, px[p]);
                b.xh = fmaxf(b.xh, px[p]);
                b.yl = in ? fminf(b.yl, py[p]) : b.yl;
                b.yh = in ? fmaxf(b.yh, py[p]) : b.yh;
                b.zl = in ? fminf(b.zl, pz[p]) : b.zl;
                b.zh = in ? fmaxf(b.zh, pz[p]) : b.zh;
            }
            // lane c < 25: column (hx + c / 5 - 2, hy + c % 5 - 2), one or two ranges of slots
            int b0 = 0, l0 = 0, b1 = 0, l1 = 0;
            float sx = 0.f, sy = 0.f, sz0 = 0.f, sz1 = 0.f;
            if (lane < 25) {
                const ColumnCells o = column_cells(lane, m, d.L, cs, ics, d.rlist2, hx, hy, hz0, hz1, b);
                if (o.n0 > 0) {
                    b0 = (int)d.cstart[o.c0];
                    l0 = (int)d.cstart[o.c0 + o.n0] - b0;
                }
                if (o.n1 > 0) {
                    b1 = (int)d.cstart[o.c1];
                    l1 = (int)d.cstart[o.c1 + o.n1] - b1;
                }
                sx = o.sx;
                sy = o.sy;
                sz0 = o.sz0;
                sz1 = o.sz1;
            }
            // stream offsets: inclusive scan of the per-column lengths; the non-empty ranges in column order
            const int len = l0 + l1;
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int total = uniform(incl);   // the last lane's: no length is negative
            const unsigned has0 = __ballot_sync(0xffffffffu, l0 > 0), has1 = __ballot_sync(0xffffffffu, l1 > 0);
            const unsigned lt = (1u << lane) - 1u;
            int at = __popc(has0 & lt) + __popc(has1 & lt);
            __syncwarp();   // the previous group's readers are done
            const int st = incl - len;
            if (l0 > 0) {
                rg[at] = BuildRange{sx, sy, sz0, b0 - st};
                rstart[at++] = st;
            }
            if (l1 > 0) {
                rg[at] = BuildRange{sx, sy, sz1, b1 - st - l0};
                rstart[at] = st + l0;
            }
            __syncwarp();
            const int n_ranges = __popc(has0) + __popc(has1);
            if (items)
                scan_stream<false, true, ID, P>(d, pos, items, rg, rstart, n_ranges, total, base, orig, rows, i, done, px,
                                                py, pz, row, (uint32_t)cap, cnt, lane);
            else
                scan_stream<false, false, ID, P>(d, pos, items, rg, rstart, n_ranges, total, base, orig, rows, i, done,
                                                 px, py, pz, row, (uint32_t)cap, cnt, lane);
        }
    }
    uint32_t lost[P];   // hits past the end of a row: more than the list and the exclusions take
#pragma unroll
    for (int p = 0; p < P; p++) lost[p] = cnt[p] - min(cnt[p], (uint32_t)cap);
    flush_rows<ID, P>(d, orig, rows, cap, i, base, true, cnt, done, lane);
#pragma unroll
    for (int p = 0; p < P; p++)
        if (lane == p && have) {
            const uint32_t found = done[p] + cnt[p] + lost[p];
            d.nl_cnt[i] = min(found, (uint32_t)d.nl_cap);
            if (found > (uint32_t)d.nl_cap) {
                atomicOr(d.err, ERR_BIT_PHYS_LIST_OVERFLOW);
                atomicMax(d.nl_need, (int)found);
            }
        }
}

// ------------------------------------------------------------- bonded terms ---
// The bonded terms read the orig-ordered compound positions (pos_orig), none
// of the arrays a list rebuild re-sorts.  MIXED: every bond vector is
// (b_hi - a_hi) + (b_lo - a_lo), so the stiff bonded forces see the (hi, lo)
// positions, not their FP32 rounding.
namespace {

// programmatic dependent launch: let the next kernel of the stream start /
// wait until the kernels this one depends on have finished and their writes
// are visible (a no-op without a programmatic dependency)
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

#if LIMA_STAGED_LIST
// Bulk copies global -> shared memory completing on an mbarrier (the copy
// engine, not the threads, moves the bytes).  Sources are this GPU's own
// memory, and each copy lands in the issuing block's shared memory only.
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
// waits for the phase of `parity` to complete; false after the iteration limit
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    for (int it = 0; it < (1 << 20); it++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// orders this thread's earlier generic-proxy shared accesses (after a block
// barrier: the block's) before its following bulk-copy writes
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
#endif  // LIMA_STAGED_LIST

// lane 0 receives the warp's sum of v[0..K); then thread 0 adds the warps in
// order into out[0..K) (fixed order)
template <int K>
__device__ __forceinline__ void block_sums_fixed(double (&v)[K], double* out) {
    __shared__ double s_b[kTB / 32][K];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < K; q++) {
        const double x = warp_sum(v[q]);
        if (lane == 0) s_b[w][q] = x;
    }
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < K; q++) {
            double t = 0.0;
            for (int k = 0; k < (int)(blockDim.x / 32); k++) t += s_b[k][q];
            out[q] = t;
        }
}

}  // namespace

// One thread per bonded term: the forces on its atoms (w: each atom's share of
// the term's energy), each into its atom's run of term_force (bterm_pos).  The step kernel that
// follows is launched programmatically and starts right away; only the lanes
// that gather these slots wait for this kernel.  ENERGY: per-block FP64 sums
// of the bond, angle and dihedral energies and the virial into bpart.
template <bool ENERGY, bool MIXED>
__global__ void __launch_bounds__(kTB) k_bonded(PhysDev d, int cur) {
    pdl_launch_dependents();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double eb = 0.0, ea = 0.0, ed = 0.0, vir = 0.0;
    const float L = d.L, iL = d.invL;
    const float4* __restrict__ po = d.pos_orig[cur];
    const float4* __restrict__ pc = d.posc_orig[cur];
    // minimum-image vector from particle a to particle b (orig ids)
    auto V = [&](int a, int b, float& x, float& y, float& z) {
        const float4 pa = po[a], pb = po[b];
        x = mimg(pb.x - pa.x, L, iL);
        y = mimg(pb.y - pa.y, L, iL);
        z = mimg(pb.z - pa.z, L, iL);
        if (MIXED) {
            const float4 ca = pc[a], cb = pc[b];
            x += cb.x - ca.x;
            y += cb.y - ca.y;
            z += cb.z - ca.z;
        }
    };
    if (t < d.n_bonds) {
        const int4 ix = d.bond_idx[t];
        const float2 par = d.bond_par[t];
        float rx, ry, rz;
        V(ix.x, ix.y, rx, ry, rz);
        const float rr = sqrtf(rx * rx + ry * ry + rz * rz);
        const float dr = rr - par.x;
        const float f = -par.y * dr / rr;   // F_j = f * r
        if (ENERGY) {
            eb = 0.5 * (double)par.y * (double)dr * (double)dr;
            vir = (double)(f * rr * rr);
        }
        // w: each atom's share of the term's energy (per-particle potential energy)
        const float sh = ENERGY ? (float)(0.5 * eb) : 0.f;
        const uint32_t* at = d.bterm_pos + 2 * t;
        d.term_force[at[0]] = make_float4(-f * rx, -f * ry, -f * rz, sh);
        d.term_force[at[1]] = make_float4(f * rx, f * ry, f * rz, sh);
    } else if (t < d.n_bonds + d.n_angles) {
        const int a_ = t - d.n_bonds;
        const int4 ix = d.angle_idx[a_];
        const float2 par = d.angle_par[a_];
        float ux, uy, uz, vx, vy, vz;
        V(ix.y, ix.x, ux, uy, uz);
        V(ix.y, ix.z, vx, vy, vz);
        const float uu = ux * ux + uy * uy + uz * uz, vv = vx * vx + vy * vy + vz * vz;
        const float nu = sqrtf(uu), nv = sqrtf(vv);
        const float cx_ = uy * vz - uz * vy, cy_ = uz * vx - ux * vz, cz_ = ux * vy - uy * vx;
        const float sn = sqrtf(cx_ * cx_ + cy_ * cy_ + cz_ * cz_);
        const float cs = ux * vx + uy * vy + uz * vz;
        const float th = atan2f(sn, cs);
        const float dth = th - par.x;
        const float inuv = 1.f / (nu * nv);
        const float cosv = cs * inuv;
        const float s = fmaxf(sn * inuv, 1e-6f);
        const float gk = par.y * dth / s;   // (dV/dtheta) / sin(theta)
        const float fix = gk * (vx * inuv - cosv * ux / uu), fiy = gk * (vy * inuv - cosv * uy / uu),
                    fiz = gk * (vz * inuv - cosv * uz / uu);
        const float fkx = gk * (ux * inuv - cosv * vx / vv), fky = gk * (uy * inuv - cosv * vy / vv),
                    fkz = gk * (uz * inuv - cosv * vz / vv);
        if (ENERGY) {
            ea = 0.5 * (double)par.y * (double)dth * (double)dth;
            vir = (double)(ux * fix + uy * fiy + uz * fiz + vx * fkx + vy * fky + vz * fkz);
        }
        const float sh = ENERGY ? (float)(ea / 3.0) : 0.f;
        const uint32_t* at = d.bterm_pos + 2 * d.n_bonds + 3 * a_;
        d.term_force[at[0]] = make_float4(fix, fiy, fiz, sh);
        d.term_force[at[1]] = make_float4(-fix - fkx, -fiy - fky, -fiz - fkz, sh);
        d.term_force[at[2]] = make_float4(fkx, fky, fkz, sh);
    } else if (t < d.n_bonds + d.n_angles + d.n_dih) {
        const int q = t - d.n_bonds - d.n_angles;
        const int4 ix = d.dih_idx[q];
        const float4 par = d.dih_par[q];
        float b1x, b1y, b1z, b2x, b2y, b2z, b3x, b3y, b3z;
        V(ix.x, ix.y, b1x, b1y, b1z);
        V(ix.y, ix.z, b2x, b2y, b2z);
        V(ix.z, ix.w, b3x, b3y, b3z);
        const float m1x = b1y * b2z - b1z * b2y, m1y = b1z * b2x - b1x * b2z, m1z = b1x * b2y - b1y * b2x;
        const float m2x = b2y * b3z - b2z * b3y, m2y = b2z * b3x - b2x * b3z, m2z = b2x * b3y - b2y * b3x;
        const float m1m1 = m1x * m1x + m1y * m1y + m1z * m1z, m2m2 = m2x * m2x + m2y * m2y + m2z * m2z;
        const float b2b2 = b2x * b2x + b2y * b2y + b2z * b2z;
        const float nb2 = sqrtf(b2b2);
        const float m1m2 = m1x * m2x + m1y * m2y + m1z * m2z;
        const float xx = b1x * m2x + b1y * m2y + b1z * m2z;
        const float phi = atan2f(nb2 * xx, m1m2);   // IUPAC dihedral angle
        const float nn = par.z;
        float sv, cv;
        sincosf(nn * phi - par.x, &sv, &cv);
        const float dVdphi = -par.y * nn * sv;     // V = k (1 + cos(n phi - phi0))
        const float gi = dVdphi * nb2 / m1m1, gl = -dVdphi * nb2 / m2m2;
        const float fix = gi * m1x, fiy = gi * m1y, fiz = gi * m1z;
        const float flx = gl * m2x, fly = gl * m2y, flz = gl * m2z;
        const float p = (b1x * b2x + b1y * b2y + b1z * b2z) / b2b2;
        const float r = (b3x * b2x + b3y * b2y + b3z * b2z) / b2b2;
        const float fjx = -fix - p * fix + r * flx, fjy = -fiy - p * fiy + r * fly, fjz = -fiz - p * fiz + r * flz;
        const float fkx = -flx + p * fix - r * flx, fky = -fly + p * fiy - r * fly, fkz = -flz + p * fiz - r * flz;
        if (ENERGY) ed = (double)par.y * (1.0 + (double)cv);
        const float sh = ENERGY ? (float)(0.25 * ed) : 0.f;
        const uint32_t* at = d.bterm_pos + 2 * d.n_bonds + 3 * d.n_angles + 4 * q;
        d.term_force[at[0]] = make_float4(fix, fiy, fiz, sh);
        d.term_force[at[1]] = make_float4(fjx, fjy, fjz, sh);
        d.term_force[at[2]] = make_float4(fkx, fky, fkz, sh);
        d.term_force[at[3]] = make_float4(flx, fly, flz, sh);
        if (ENERGY) {
            vir = (double)(b1x * fjx + b1y * fjy + b1z * fjz + (b1x + b2x) * fkx + (b1y + b2y) * fky +
                           (b1z + b2z) * fkz + (b1x + b2x + b3x) * flx + (b1y + b2y + b3y) * fly +
                           (b1z + b2z + b3z) * flz);
        }
    }
    if (ENERGY) {
        double v[4] = {eb, ea, ed, vir};
        block_sums_fixed<4>(v, d.bpart + (size_t)blockIdx.x * 4);
    }
}

namespace {

// The FP64 sums of a step kernel (kinetic energy; with ENERGY also the LJ
// energy and virial), per block in a fixed order, then over the blocks by the
// block that finishes last (in block order).  That block adds the bonded
// kernel's block partials (ENERGY), folds the totals into e_last and the next
// Berendsen scalar and, when a rebuild is due and `tail` is set, launches it.
// TAIL: this kernel may launch the rebuild graph; a kernel that holds a
// device-side graph launch must itself run inside a graph, so the direct
// launches use the variant without it.
template <bool ENERGY, bool INTEGRATE, bool TAIL>
__device__ __forceinline__ void finish_sums(const PhysDev& d, int slot, cudaGraphExec_t tail, double (&v)[kRed]) {
    __shared__ double s_red[kTB / 32][kRed];
    __shared__ int s_last;
    constexpr int nq = ENERGY ? kRed : 1;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < nq; q++) {
        const double x = warp_sum(v[q]);
        if (lane == 0) s_red[w][q] = x;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < nq; q++) {
            double t = 0.0;
            for (int k = 0; k < kTB / 32; k++) t += s_red[k][q];
            d.part[(size_t)blockIdx.x * kRedStride + q] = t;
        }
        __threadfence();
        s_last = atomicAdd(d.done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // (read beside the partials; the block that finished last sees every block's request)
    const int due = TAIL && INTEGRATE && threadIdx.x == 0 ? *(volatile int*)d.need_rebuild : 0;
    double a[kRed];
#pragma unroll
    for (int q = 0; q < nq; q++) a[q] = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
        for (int q = 0; q < nq; q++) a[q] += __ldcg(&d.part[(size_t)b * kRedStride + q]);
#pragma unroll
    for (int q = 0; q < nq; q++) {
        const double x = warp_sum(a[q]);
        if (lane == 0) s_red[w][q] = x;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    double tot[kRed] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < nq; q++)
        for (int k = 0; k < kTB / 32; k++) tot[q] += s_red[k][q];
    const double kin = tot[0];
    const double temp = kin * d.temp_of_kin;
    d.e_last[LIMA_E_KINETIC] = kin;
    d.e_last[LIMA_E_TEMPERATURE] = temp;
    if (ENERGY) {
        // the bonded kernel's block partials (bond, angle, dihedral, virial), in block order
        pdl_wait();
        double bs[4] = {0.0, 0.0, 0.0, 0.0};
        const int nbb = bonded_blocks(d);
        for (int b = 0; b < nbb; b++)
#pragma unroll
            for (int q = 0; q < 4; q++) bs[q] += __ldcg(&d.bpart[(size_t)b * 4 + q]);
        d.e_last[LIMA_E_LJ] = tot[1];
        d.e_last[LIMA_E_BOND] = bs[0];
        d.e_last[LIMA_E_ANGLE] = bs[1];
        d.e_last[LIMA_E_DIHEDRAL] = bs[2];
        d.e_last[LIMA_E_VIRIAL] = tot[2] + bs[3];
        d.e_last[LIMA_E_TOTAL] = tot[1] + bs[0] + bs[1] + bs[2] + kin;
    }
    if (slot < 2) {
        float lam = 1.f;
        if (d.thermostat == LIMA_THERMOSTAT_BERENDSEN && temp > 0.0)
            lam = (float)sqrt(1.0 + d.dt_tau * (d.t_target / temp - 1.0));
        d.lambda[slot ^ 1] = lam;
    }
    *d.done = 0u;   // for the next launch
    if (TAIL && INTEGRATE && tail != nullptr && due) {
        if (cudaGraphLaunch(tail, cudaStreamGraphTailLaunch) == cudaSuccess)
            *d.rebuild_count += 1ull;
        else
            atomicOr(d.err, ERR_BIT_REBUILD_LAUNCH);
    }
}

}  // namespace

// ------------------------------------------------------------------ the step ---
// (lj_pair_step: physmath.cuh)
// The four ids of one chunk column (nl_word): one 8-byte load of 16-bit ids
// or one 16-byte load of 32-bit ids.
template <typename ID>
struct ChunkIds;
template <>
struct ChunkIds<uint16_t> {
    using V = uint2;
    static __device__ __forceinline__ void split(V v, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& e) {
        a = v.x & 0xffffu;
        b = v.x >> 16;
        c = v.y & 0xffffu;
        e = v.y >> 16;
    }
};
template <>
struct ChunkIds<uint32_t> {
    using V = uint4;
    static __device__ __forceinline__ void split(V v, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& e) {
        a = v.x;
        b = v.y;
        c = v.z;
        e = v.w;
    }
};

// One lane's entries of its particle's Verlet list: column g of every H-th
// 32-entry chunk, n_full whole chunks and, if tail, `tail` entries of the
// partial last one; four entries per chunk column (col: the lane's column of
// its first chunk; cstride: vectors between its chunks), each chunk one vector
// load and four position gathers in flight.
// In the last, partial chunk the words past the lane's count are not ids
// (the gathers for them re-read the first entry and are not evaluated).
// MIXED: compensated sums every two chunks (8 pairs).  WM: the axes that take
// the minimum image.  The plain FP32 walk loads each chunk's ids one chunk
// ahead (the mixed walk, and the energies of an unswitched cutoff, have no
// registers to spare for it).
template <bool MIXED, bool ENERGY, bool SWITCH, int WM, typename ID>
__device__ __forceinline__ void pair_rows(const PhysDev& d, const float2* row, float4 pi, const float4* __restrict__ pos,
                                          const typename ChunkIds<ID>::V* __restrict__ col, uint32_t cstride, int full,
                                          int tail, float& fx, float& fy, float& fz, float& cxx, float& cyy, float& czz,
                                          float& e_i, float& w_i) {
    constexpr bool kAhead = !MIXED && (SWITCH || !ENERGY);
    const int nch = full + (tail ? 1 : 0);
    uint32_t off = 0;
    int c = 0;
    typename ChunkIds<ID>::V nxt{};
    if (kAhead && nch > 0) nxt = __ldg(col);
    while (c < full) {
        const int cend = MIXED ? min(full, c + 2) : full;
        float px = 0.f, py = 0.f, pz = 0.f;
        for (; c < cend; c++, off += cstride) {
            uint32_t j0, j1, j2, j3;
            ChunkIds<ID>::split(kAhead ? nxt : __ldg(col + off), j0, j1, j2, j3);
            if (kAhead && c + 1 < nch) nxt = __ldg(col + off + cstride);
            const float4 p0 = __ldg(pos + j0), p1 = __ldg(pos + j1), p2 = __ldg(pos + j2), p3 = __ldg(pos + j3);
            lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p0, px, py, pz, e_i, w_i);
            lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p1, px, py, pz, e_i, w_i);
            lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p2, px, py, pz, e_i, w_i);
            lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p3, px, py, pz, e_i, w_i);
        }
        if (MIXED) {
            ds_add(fx, cxx, px);
            ds_add(fy, cyy, py);
            ds_add(fz, czz, pz);
        } else {
            fx += px;
            fy += py;
            fz += pz;
        }
    }
    if (tail) {
        uint32_t j0, j1, j2, j3;
        ChunkIds<ID>::split(kAhead ? nxt : __ldg(col + off), j0, j1, j2, j3);
        const float4 p0 = __ldg(pos + j0);
        const float4 p1 = __ldg(pos + (tail > 1 ? j1 : j0));
        const float4 p2 = __ldg(pos + (tail > 2 ? j2 : j0));
        float px = 0.f, py = 0.f, pz = 0.f;
        lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p0, px, py, pz, e_i, w_i);
        if (tail > 1) lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p1, px, py, pz, e_i, w_i);
        if (tail > 2) lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p2, px, py, pz, e_i, w_i);
        (void)j3;
        if (MIXED) {
            ds_add(fx, cxx, px);
            ds_add(fy, cyy, py);
            ds_add(fz, czz, pz);
        } else {
            fx += px;
            fy += py;
            fz += pz;
        }
    }
}

#if LIMA_STAGED_LIST
// One lane's entries of one staged group of list chunks: entry q of the lane
// at srow[(q / 4) * kChunkWords + q % 4] (shared memory; srow = the lane's
// column of the group's first chunk); MIXED: one compensated sum per group.
constexpr int kStageChunks = kStageRows / 4;   // list chunks per staged group
constexpr int kChunkWords = kTB * 4;           // words of one chunk of a block's 32 particles
__device__ __forceinline__ int staged_at(int q) { return (q >> 2) * kChunkWords + (q & 3); }
template <bool MIXED, bool ENERGY, bool SWITCH, int WM>
__device__ __forceinline__ void pair_staged(const PhysDev& d, const float2* row, float4 pi,
                                            const float4* __restrict__ pos, const uint32_t* srow, int nq, float& fx,
                                            float& fy, float& fz, float& cxx, float& cyy, float& czz, float& e_i,
                                            float& w_i) {
    float px = 0.f, py = 0.f, pz = 0.f;
    // staged ids are clamped into the position array (a wrong id stays a wrong force, not a stray read)
    const uint32_t lim = (uint32_t)d.n_pad - 1u;
    int q = 0;
    for (; q + 3 < nq; q += 4) {
        const uint32_t j0 = min(srow[staged_at(q)], lim), j1 = min(srow[staged_at(q + 1)], lim);
        const uint32_t j2 = min(srow[staged_at(q + 2)], lim), j3 = min(srow[staged_at(q + 3)], lim);
        const float4 p0 = __ldg(pos + j0), p1 = __ldg(pos + j1), p2 = __ldg(pos + j2), p3 = __ldg(pos + j3);
        lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p0, px, py, pz, e_i, w_i);
        lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p1, px, py, pz, e_i, w_i);
        lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p2, px, py, pz, e_i, w_i);
        lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, p3, px, py, pz, e_i, w_i);
    }
    for (; q < nq; q++)
        lj_pair_step<ENERGY, SWITCH, WM>(d, row, pi, __ldg(pos + min(srow[staged_at(q)], lim)), px, py, pz, e_i, w_i);
    if (MIXED) {
        ds_add(fx, cxx, px);
        ds_add(fy, cyy, py);
        ds_add(fz, czz, pz);
    } else {
        fx += px;
        fy += py;
        fz += pz;
    }
}

// The block's list chunks through shared memory: chunk q of the block's 32
// particles is four contiguous kilobytes of the list (nl_word: lane t of the
// block reads words 4t .. 4t + 3 of each chunk), so each chunk is one bulk
// copy.  Groups of kStageChunks chunks (kStageRows rows) alternate between
// two buffers: thread 0 issues group s + 1 while the block evaluates group
// s, and a block barrier after each group frees its buffer for group s + 2.  Waits are bounded; one that runs out sets
// ERR_BIT_TILE_TIMEOUT and ends the issuing, and thread 0 waits (bounded) for
// the copies already issued before the block moves on.
template <bool MIXED, bool ENERGY, bool SWITCH>
__device__ __forceinline__ void pair_walk_staged(const PhysDev& d, const float2* row, float4 pi,
                                                 const float4* __restrict__ pos, int rows, bool active, unsigned wm,
                                                 float& fx, float& fy, float& fz, float& cxx, float& cyy, float& czz,
                                                 float& e_i, float& w_i) {
    __shared__ __align__(128) uint32_t s_stage[2][kStageChunks][kChunkWords];
    __shared__ __align__(8) uint64_t s_bar[2];
    __shared__ int s_rows, s_fail;
    if (threadIdx.x == 0) {
        s_rows = 0;
        s_fail = 0;
        mbar_init(&s_bar[0], 1);
        mbar_init(&s_bar[1], 1);
        mbar_init_fence();
    }
    __syncthreads();
    if (active && threadIdx.x % kGroup == 0) atomicMax(&s_rows, rows);
    __syncthreads();
    const int bchunks = (s_rows + 3) / 4;
    const int nst = (bchunks + kStageChunks - 1) / kStageChunks;
    // chunk 0 of this block's particles: particle i0 = blockIdx.x * 32, word i0 * 32
    const uint32_t* src0 = d.nl + (size_t)blockIdx.x * kChunkWords;
    const size_t stride = (size_t)d.n_pad * kListChunk;   // words between chunks
    int issued = 0;   // thread 0: groups issued
    auto issue = [&](int st) {
        const int c0 = st * kStageChunks, nc = min(kStageChunks, bchunks - c0);
        uint64_t* bar = &s_bar[st & 1];
        fence_proxy_async_smem();
        mbar_expect_tx(bar, (uint32_t)(nc * kChunkWords * sizeof(uint32_t)));
        for (int q = 0; q < nc; q++)
            bulk_g2s(&s_stage[st & 1][q][0], src0 + (size_t)(c0 + q) * stride, kChunkWords * sizeof(uint32_t), bar);
        issued = st + 1;
    };
    if (threadIdx.x == 0 && nst > 0) issue(0);
    for (int st = 0; st < nst; st++) {
        if (threadIdx.x == 0 && st + 1 < nst && !*(volatile int*)&s_fail) issue(st + 1);
        const bool got = !*(volatile int*)&s_fail && mbar_wait_bounded(&s_bar[st & 1], (uint32_t)(st >> 1) & 1u);
        if (!got && !*(volatile int*)&s_fail) {
            s_fail = 1;
            atomicOr(d.err, ERR_BIT_TILE_TIMEOUT);
        }
        const int nq = got ? max(0, min(kStageRows, rows - st * kStageRows)) : 0;
        const uint32_t* srow = &s_stage[st & 1][0][threadIdx.x * 4];
#define LIMA_STAGED_CALL(WM) \
    pair_staged<MIXED, ENERGY, SWITCH, WM>(d, row, pi, pos, srow, nq, fx, fy, fz, cxx, cyy, czz, e_i, w_i)
        switch (wm) {
            case 0: LIMA_STAGED_CALL(0); break;
            case 1: LIMA_STAGED_CALL(1); break;
            case 2: LIMA_STAGED_CALL(2); break;
            case 4: LIMA_STAGED_CALL(4); break;
            default: LIMA_STAGED_CALL(7); break;
        }
#undef LIMA_STAGED_CALL
        __syncthreads();
    }
    // after a timeout: the groups issued and not yet seen complete
    if (threadIdx.x == 0 && s_fail)
        for (int st = max(0, issued - 2); st < issued; st++) mbar_wait_bounded(&s_bar[st & 1], (uint32_t)(st >> 1) & 1u);
    __syncthreads();
}
#endif  // LIMA_STAGED_LIST

// LPP lanes walk one particle's list: lane g + 8 h takes column g of the chunks
// h, h + LPP / 8, ...
template <int LPP, bool MIXED, bool ENERGY, bool INTEGRATE, bool SWITCH, bool TAIL, typename ID>
__device__ __forceinline__ void step_body(const PhysDev& d, int cur, int slot, cudaGraphExec_t tail) {
    // the LJ table as lj_pair_step reads it: (sigma^2, 24 eps)
    extern __shared__ float2 s_tab[];
    const int nt2 = d.n_types * d.n_types;
    for (int q = threadIdx.x; q < nt2; q += blockDim.x) {
        const float2 t = d.lj_table[q];
        s_tab[q] = make_float2(t.x, 6.f * t.y);
    }
    __syncthreads();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / LPP;
    const int lp = threadIdx.x % LPP, g = lp % kGroup, h = lp / kGroup;
    const bool active = i < d.n;
    // FP64 sums of this thread: kinetic energy, LJ energy, LJ virial
    double red[kRed] = {0.0, 0.0, 0.0};
    const float4* __restrict__ pos = d.pos[cur];
    const float4 pi = active ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2* row = &s_tab[__float_as_int(pi.w) * d.n_types];
    float fx = 0.f, fy = 0.f, fz = 0.f, cxx = 0.f, cyy = 0.f, czz = 0.f;
    float e_i = 0.f, w_i = 0.f;
    const int cnt = active ? (int)d.nl_cnt[i] : 0;
    // the axes that take the minimum image: those on which some particle of the
    // warp lies within r_c of a face (one axis alone, x and y, or all three)
    const unsigned wm = __reduce_or_sync(0xffffffffu, active ? face_axes(d, pi) : 0u);
#if LIMA_STAGED_LIST
    const int rows = cnt > g ? (cnt - g + kGroup - 1) / kGroup : 0;   // this lane's entries: g, g + 8, ... below cnt
    (void)h;
    pair_walk_staged<MIXED, ENERGY, SWITCH>(d, row, pi, pos, rows, active, wm, fx, fy, fz, cxx, cyy, czz, e_i, w_i);
#else
    // the lane's column of chunk 0 (nl_word with k = g), chunks n_pad * 8 vectors apart
    using V = typename ChunkIds<ID>::V;
    constexpr int H = LPP / kGroup;
    const uint32_t chunk = (uint32_t)d.n_pad * kGroup, cstride = H * chunk;
    const V* __restrict__ col = reinterpret_cast<const V*>(d.nl) + (uint32_t)i * kGroup + g + h * chunk;
    // this lane's chunks with four entries (whole ones, and the partial last one where it reaches
    // that far), then its 0 .. 3 entries of the last
    const int whole = cnt / kListChunk;
    const int last = whole % H == h ? max((cnt - whole * kListChunk - g + kGroup - 1) / kGroup, 0) : 0;
    const int full = (whole - h + H - 1) / H + (last >> 2), part = last & 3;
    {   // the warp's list chunks into L2 at once: chunk q of its 32 / LPP particles is
        // as many times 32 contiguous ids, one bulk prefetch per lane q (no completion to wait for)
        const int wch = ((int)__reduce_max_sync(0xffffffffu, (unsigned)cnt) + kListChunk - 1) / kListChunk;
        const int lane = threadIdx.x & 31;
        if (lane < wch) {
            const uint32_t i0 = (blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) / LPP;
            const char* a = reinterpret_cast<const char*>(d.nl) + ((size_t)lane * d.n_pad + i0) * kListChunk * sizeof(ID);
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(32 / LPP * kListChunk * sizeof(ID)))
                         : "memory");
        }
    }
#define LIMA_ROWS_CALL(WM) \
    pair_rows<MIXED, ENERGY, SWITCH, WM, ID>(d, row, pi, pos, col, cstride, full, part, fx, fy, fz, cxx, cyy, czz, e_i, \
                                             w_i)
    switch (wm) {
        case 0: LIMA_ROWS_CALL(0); break;
        case 1: LIMA_ROWS_CALL(1); break;
        case 2: LIMA_ROWS_CALL(2); break;
        case 3: LIMA_ROWS_CALL(3); break;
        case 4: LIMA_ROWS_CALL(4); break;
        default: LIMA_ROWS_CALL(7); break;
    }
#undef LIMA_ROWS_CALL
#endif
    // reduce the LPP lanes of this particle (warp shuffles)
#pragma unroll
    for (int o = LPP / 2; o > 0; o >>= 1) {
        if (MIXED) {
            const float ox = __shfl_xor_sync(0xffffffffu, fx, o), oy = __shfl_xor_sync(0xffffffffu, fy, o),
                        oz = __shfl_xor_sync(0xffffffffu, fz, o);
            const float ocx = __shfl_xor_sync(0xffffffffu, cxx, o), ocy = __shfl_xor_sync(0xffffffffu, cyy, o),
                        ocz = __shfl_xor_sync(0xffffffffu, czz, o);
            float s, e;
            two_sum(fx, ox, s, e); fx = s; cxx += ocx + e;
            two_sum(fy, oy, s, e); fy = s; cyy += ocy + e;
            two_sum(fz, oz, s, e); fz = s; czz += ocz + e;
        } else {
            fx += __shfl_xor_sync(0xffffffffu, fx, o);
            fy += __shfl_xor_sync(0xffffffffu, fy, o);
            fz += __shfl_xor_sync(0xffffffffu, fz, o);
        }
        if (ENERGY) {
            e_i += __shfl_xor_sync(0xffffffffu, e_i, o);
            w_i += __shfl_xor_sync(0xffffffffu, w_i, o);
        }
    }
    const uint32_t oi = active ? d.orig_of_sorted[i] : 0xffffffffu;
    if (active && lp == 0) {
        float e_b = 0.f;
        if (oi < (uint32_t)d.n_cp) {
            // the bonded kernel's forces on this particle (it runs beside this
            // kernel's list walk; wait for it only here)
            pdl_wait();
            float bx = 0.f, by = 0.f, bz = 0.f, bw = 0.f;
            const uint32_t q1 = d.bterm_off[oi + 1];
#pragma unroll 4
            for (uint32_t q = d.bterm_off[oi]; q < q1; q++) {
                const float4 tf = __ldcg(&d.term_force[q]);
                bx += tf.x;
                by += tf.y;
                bz += tf.z;
                bw += tf.w;
            }
            e_b = bw;
            if (MIXED) {
                ds_add(fx, cxx, bx);
                ds_add(fy, cyy, by);
                ds_add(fz, czz, bz);
            } else {
                fx += bx;
                fy += by;
                fz += bz;
            }
        }
        if (MIXED) {
            fx += cxx;
            fy += cyy;
            fz += czz;
        }
        // w: the particle's potential energy, its LJ pair halves plus its bonded-term shares
        d.force[i] = make_float4(fx, fy, fz, ENERGY ? e_i + e_b : 0.f);
        if (ENERGY) {
            red[1] = (double)e_i;
            red[2] = (double)w_i;
        }
        // velocity Verlet as kick-drift over half-step velocities
        const float4 v = d.vel[i];
        const float im = v.w;
        const float h = (float)(0.5 * d.dt);
        const float ax = fx * im, ay = fy * im, az = fz * im;
        const float L = d.L, iL = d.invL;
        if (MIXED) {
            float4 vc = d.velc[i];
            float vhx = v.x, vhy = v.y, vhz = v.z;
            ds_add(vhx, vc.x, ax * h);
            ds_add(vhy, vc.y, ay * h);
            ds_add(vhz, vc.z, az * h);
            const double vx = (double)vhx + vc.x, vy = (double)vhy + vc.y, vz = (double)vhz + vc.z;
            red[0] = 0.5 / (double)im * (vx * vx + vy * vy + vz * vz);
            if (INTEGRATE) {
                const float lam = d.lambda[slot];
                if (lam != 1.f) {   // scale (hi, lo): keep the product's rounding error in lo
                    float p = lam * vhx; vc.x = fmaf(lam, vhx, -p) + lam * vc.x; vhx = p;
                    p = lam * vhy; vc.y = fmaf(lam, vhy, -p) + lam * vc.y; vhy = p;
                    p = lam * vhz; vc.z = fmaf(lam, vhz, -p) + lam * vc.z; vhz = p;
                }
                ds_add(vhx, vc.x, ax * h);
                ds_add(vhy, vc.y, ay * h);
                ds_add(vhz, vc.z, az * h);
                float4 pc = d.posc[i];
                const float dtf = (float)d.dt;
                float x = pi.x, y = pi.y, z = pi.z;
                float tt = vhx * dtf; ds_add(x, pc.x, tt); pc.x += fmaf(vhx, dtf, -tt) + vc.x * dtf;
                tt = vhy * dtf; ds_add(y, pc.y, tt); pc.y += fmaf(vhy, dtf, -tt) + vc.y * dtf;
                tt = vhz * dtf; ds_add(z, pc.z, tt); pc.z += fmaf(vhz, dtf, -tt) + vc.z * dtf;
                if (x < 0.f) ds_add(x, pc.x, L); else if (x >= L) ds_add(x, pc.x, -L);
                if (y < 0.f) ds_add(y, pc.y, L); else if (y >= L) ds_add(y, pc.y, -L);
                if (z < 0.f) ds_add(z, pc.z, L); else if (z >= L) ds_add(z, pc.z, -L);
                if (x >= L) x -= L;
                if (y >= L) y -= L;
                if (z >= L) z -= L;
                d.pos[cur ^ 1][i] = make_float4(x, y, z, pi.w);
                if (oi < (uint32_t)d.n_cp) {
                    d.pos_orig[cur ^ 1][oi] = make_float4(x, y, z, pi.w);
                    d.posc_orig[cur ^ 1][oi] = pc;
                }
                d.posc[i] = pc;
                d.vel[i] = make_float4(vhx, vhy, vhz, im);
                d.velc[i] = vc;
                const float4 xr = d.xref[i];
                const float ddx = mimg(x - xr.x, L, iL), ddy = mimg(y - xr.y, L, iL), ddz = mimg(z - xr.z, L, iL);
                if (ddx * ddx + ddy * ddy + ddz * ddz > d.half_skin2) {
                    if (d.dynamic_list) atomicExch(d.need_rebuild, 1);
                    else atomicOr(d.err, ERR_BIT_LIST_STALE);
                }
                if (!(x == x) || !(y == y) || !(z == z)) atomicOr(d.err, ERR_BIT_NAN);
            }
        } else {
            float vx = v.x + ax * h, vy = v.y + ay * h, vz = v.z + az * h;
            red[0] = 0.5 / (double)im * ((double)vx * vx + (double)vy * vy + (double)vz * vz);
            if (INTEGRATE) {
                const float lam = d.lambda[slot];
                vx = lam * vx + ax * h;
                vy = lam * vy + ay * h;
                vz = lam * vz + az * h;
                const float dtf = (float)d.dt;
                float x = pi.x + vx * dtf, y = pi.y + vy * dtf, z = pi.z + vz * dtf;
                x += (x < 0.f) ? L : ((x >= L) ? -L : 0.f);
                y += (y < 0.f) ? L : ((y >= L) ? -L : 0.f);
                z += (z < 0.f) ? L : ((z >= L) ? -L : 0.f);
                if (x >= L) x -= L;
                if (y >= L) y -= L;
                if (z >= L) z -= L;
                d.pos[cur ^ 1][i] = make_float4(x, y, z, pi.w);
                if (oi < (uint32_t)d.n_cp) d.pos_orig[cur ^ 1][oi] = make_float4(x, y, z, pi.w);
                d.vel[i] = make_float4(vx, vy, vz, im);
                const float4 xr = d.xref[i];
                const float ddx = mimg(x - xr.x, L, iL), ddy = mimg(y - xr.y, L, iL), ddz = mimg(z - xr.z, L, iL);
                if (ddx * ddx + ddy * ddy + ddz * ddz > d.half_skin2) {
                    if (d.dynamic_list) atomicExch(d.need_rebuild, 1);
                    else atomicOr(d.err, ERR_BIT_LIST_STALE);
                }
                if (!(x == x) || !(y == y) || !(z == z)) atomicOr(d.err, ERR_BIT_NAN);
            }
        }
    }
    finish_sums<ENERGY, INTEGRATE, TAIL>(d, slot, tail, red);
}

// FP32: at most 48 registers, 5 blocks of 256 per SM.  Mixed keeps the
// compiler's own choice (a 5-block bound slowed it).
// ID: the list's slot-id type (uint16_t when the slots fit, else uint32_t).
template <int LPP, bool ENERGY, bool INTEGRATE, bool SWITCH, bool TAIL, typename ID>
__global__ void __launch_bounds__(kTB, 5) k_step(PhysDev d, int cur, int slot, cudaGraphExec_t tail) {
    step_body<LPP, false, ENERGY, INTEGRATE, SWITCH, TAIL, ID>(d, cur, slot, tail);
}
template <int LPP, bool ENERGY, bool INTEGRATE, bool SWITCH, bool TAIL, typename ID>
__global__ void __launch_bounds__(kTB) k_step_mixed(PhysDev d, int cur, int slot, cudaGraphExec_t tail) {
    step_body<LPP, true, ENERGY, INTEGRATE, SWITCH, TAIL, ID>(d, cur, slot, tail);
}

// ---------------------------------------------------------------- launchers --
int step_lanes(const PhysDev& d, bool energy) {
    if (kStagedList) return kGroup;
    if (energy) return d.n < kStepEnergy32Below ? 32 : kGroup;
    return d.n < kStep32Below ? 32 : (d.n < kStep16Below ? 16 : kGroup);
}

// the n_pad slots' lanes
int step_blocks(const PhysDev& d, bool energy) {
    return (int)(((size_t)d.n_pad * step_lanes(d, energy) + kTB - 1) / kTB);
}

namespace {

// The step kernel with a programmatic dependency on the kernel before it in
// the stream (the bonded kernel): it may start before that one has finished
// and waits for it only where it reads its results.
bool has_bonded(const PhysDev& d) { return d.n_bonds + d.n_angles + d.n_dih > 0; }

// (without bonded terms no bonded kernel comes before it: an ordinary launch)
template <typename K>
void launch_programmatic(K kernel, const PhysDev& d, int blocks, int cur, int slot, cudaGraphExec_t tail, size_t smem,
                         cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kTB);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = has_bonded(d) ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, d, cur, slot, tail);
}

template <int LPP, bool MIXED, bool ENERGY, bool INTEGRATE, bool TAIL, typename ID>
void step_variant_lanes(const PhysDev& d, int cur, int slot, cudaGraphExec_t tail, cudaStream_t s) {
    const size_t smem = sizeof(float2) * d.n_types * d.n_types;
    const int blocks = step_blocks(d, ENERGY);
    if (MIXED && d.use_switch)
        launch_programmatic(k_step_mixed<LPP, ENERGY, INTEGRATE, true, TAIL, ID>, d, blocks, cur, slot, tail, smem, s);
    else if (MIXED)
        launch_programmatic(k_step_mixed<LPP, ENERGY, INTEGRATE, false, TAIL, ID>, d, blocks, cur, slot, tail, smem, s);
    else if (d.use_switch)
        launch_programmatic(k_step<LPP, ENERGY, INTEGRATE, true, TAIL, ID>, d, blocks, cur, slot, tail, smem, s);
    else
        launch_programmatic(k_step<LPP, ENERGY, INTEGRATE, false, TAIL, ID>, d, blocks, cur, slot, tail, smem, s);
}

template <bool MIXED, bool ENERGY, bool INTEGRATE, bool TAIL, typename ID>
void step_variant_id(const PhysDev& d, int cur, int slot, cudaGraphExec_t tail, cudaStream_t s) {
    // more than 8 lanes: boxes whose ids are 16-bit; 16 lanes: without energies (step_lanes)
    if constexpr (sizeof(ID) == 2) {
        const int lanes = step_lanes(d, ENERGY);
        if (lanes == 32) return step_variant_lanes<32, MIXED, ENERGY, INTEGRATE, TAIL, ID>(d, cur, slot, tail, s);
        if constexpr (!ENERGY)
            if (lanes == 16) return step_variant_lanes<16, MIXED, ENERGY, INTEGRATE, TAIL, ID>(d, cur, slot, tail, s);
    }
    step_variant_lanes<8, MIXED, ENERGY, INTEGRATE, TAIL, ID>(d, cur, slot, tail, s);
}

template <bool MIXED, bool ENERGY, bool INTEGRATE, bool TAIL>
void step_variant(const PhysDev& d, int cur, int slot, cudaGraphExec_t tail, cudaStream_t s) {
    if constexpr (!kStagedList)   // (the staged library's ids are 32-bit)
        if (d.nl16) return step_variant_id<MIXED, ENERGY, INTEGRATE, TAIL, uint16_t>(d, cur, slot, tail, s);
    step_variant_id<MIXED, ENERGY, INTEGRATE, TAIL, uint32_t>(d, cur, slot, tail, s);
}

template <bool MIXED, bool ENERGY, bool INTEGRATE>
void step_tail(const PhysDev& d, int cur, int slot, cudaGraphExec_t tail, cudaStream_t s) {
    if (tail)
        step_variant<MIXED, ENERGY, INTEGRATE, true>(d, cur, slot, tail, s);
    else
        step_variant<MIXED, ENERGY, INTEGRATE, false>(d, cur, slot, nullptr, s);
}

}  // namespace

namespace {
void sort_cells(const PhysDev& d, const float4* pos, cudaStream_t s) {
    k_sort_count<<<(d.n + kScanThreads - 1) / kScanThreads, kScanThreads, 0, s>>>(d, pos);
    k_sort_fill<<<(d.n + kTB - 1) / kTB, kTB, 0, s>>>(d);
}
int order_blocks(const PhysDev& d) { return (int)(((size_t)d.n_cells * 32 + kTB - 1) / kTB); }
}  // namespace

void launch_sort(const PhysDev& d, const float4* pos, cudaStream_t s) {
    sort_cells(d, pos, s);
    k_sort_order<false><<<order_blocks(d), kTB, 0, s>>>(d, 0, 0);
}

void launch_sort_permute(const PhysDev& d, int cur, bool mixed, cudaStream_t s) {
    sort_cells(d, d.pos[cur], s);
    if (d.n < kPermuteAloneFrom) {
        k_sort_order<true><<<order_blocks(d), kTB, 0, s>>>(d, cur, mixed ? 1 : 0);
    } else {
        k_sort_order<false><<<order_blocks(d), kTB, 0, s>>>(d, cur, 0);
        k_permute<<<(d.n + kTB - 1) / kTB, kTB, 0, s>>>(d, cur, mixed ? 1 : 0);
    }
}

void launch_set_xref(const PhysDev& d, const float4* pos, cudaStream_t s) {
    k_set_xref<<<(d.n + kTB - 1) / kTB, kTB, 0, s>>>(d, pos);
}

bool list_ids_16bit(int n_pad) { return !kStagedList && n_pad <= kIds16Slots; }

namespace {
template <typename ID, int P>
void build_list(const PhysDev& d, const float4* pos, const uint32_t* orig, const uint32_t* items, int copy_cur,
                bool mixed, cudaStream_t s) {
    const int warps = (d.n + P - 1) / P;
    // room for the exclusions too: a row overflows by what is left without them
    const int cap = std::min(nl_round_cap(d.nl_room), kBuildRow);
    const size_t smem = kBuildWarps * build_warp_smem(P, cap, sizeof(ID));
    allow_smem(k_build_list<ID, P>, smem, 0, kBuildWarps * build_warp_smem(P, kBuildRow, sizeof(ID)));
    k_build_list<ID, P><<<(warps + kBuildWarps - 1) / kBuildWarps, kBuildWarps * 32, smem, s>>>(
        d, pos, orig, items, copy_cur, mixed ? 1 : 0, cap);
}
}  // namespace

void launch_build_list(const PhysDev& d, const float4* pos, const uint32_t* orig, const uint32_t* items, int copy_cur,
                       bool mixed, cudaStream_t s) {
    // (measured at kBuildOneBelow; boxes below it have this library's narrowest ids)
    using Narrow = typename std::conditional<kStagedList, uint32_t, uint16_t>::type;
    if (d.n < kBuildOneBelow) return build_list<Narrow, 1>(d, pos, orig, items, copy_cur, mixed, s);
    if constexpr (!kStagedList)
        if (d.nl16) return build_list<uint16_t, 4>(d, pos, orig, items, copy_cur, mixed, s);
    build_list<uint32_t, 4>(d, pos, orig, items, copy_cur, mixed, s);
}

namespace {
// position and half-step velocity of orig id o in FP64 (hi + lo)
__device__ __forceinline__ void state_of_orig(const PhysDev& d, int cur, uint32_t o, double* x, double* v) {
    const uint32_t k = d.sorted_of_orig[o];
    const float4 p = d.pos[cur][k], w = d.vel[k];
    x[0] = p.x; x[1] = p.y; x[2] = p.z;
    v[0] = w.x; v[1] = w.y; v[2] = w.z;
    if (d.precision == LIMA_PRECISION_MIXED) {
        const float4 pc = d.posc[k], wc = d.velc[k];
        x[0] += pc.x; x[1] += pc.y; x[2] += pc.z;
        v[0] += wc.x; v[1] += wc.y; v[2] += wc.z;
    }
}

// one thread per compound slot (c, t)
__global__ void k_read_compounds(PhysDev d, int cur, lima_compound_state* __restrict__ states,
                                 lima_float3* __restrict__ prev) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= d.n_c * LIMA_MAX_COMPOUND_PARTICLES) return;
    const int c = q / LIMA_MAX_COMPOUND_PARTICLES, t = q % LIMA_MAX_COMPOUND_PARTICLES;
    const uint32_t b = d.cp_base[c];
    const int n = (int)(d.cp_base[c + 1] - b);
    lima_float3 a = {0.f, 0.f, 0.f}, r = {0.f, 0.f, 0.f};
    if (t < n) {
        double x[3], v[3], x0[3], vv[3];
        state_of_orig(d, cur, b + t, x, v);
        state_of_orig(d, cur, b, x0, vv);
        const double L = d.L;
        double qq[3];
        for (int k = 0; k < 3; k++) {
            double dd = x[k] - x0[k];
            dd -= L * nearbyint(dd / L);
            qq[k] = t == 0 ? x[k] : x0[k] + dd;
        }
        a = lima_float3{(float)qq[0], (float)qq[1], (float)qq[2]};
        r = lima_float3{(float)(qq[0] - v[0] * d.dt), (float)(qq[1] - v[1] * d.dt), (float)(qq[2] - v[2] * d.dt)};
    }
    if (states) {
        states[c].positions[t] = a;
        if (t == 0) {
            // the count and the struct's padding bytes
            uint32_t* tail = reinterpret_cast<uint32_t*>(&states[c].n_particles);
            *tail = (uint32_t)n;
        }
    }
    if (prev) prev[q] = r;
}

// positions alone, as flat xyz: compound slots (the values k_read_compounds
// gives), then solvents
__global__ void k_read_positions(PhysDev d, int cur, lima_float3* __restrict__ cxyz, lima_float3* __restrict__ sxyz) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x, nc = d.n_c * LIMA_MAX_COMPOUND_PARTICLES;
    double x[3], v[3];
    if (q >= nc) {
        const int s = q - nc;
        if (s >= d.n_s || !sxyz) return;
        state_of_orig(d, cur, (uint32_t)(d.n_cp + s), x, v);
        sxyz[s] = lima_float3{(float)x[0], (float)x[1], (float)x[2]};
        return;
    }
    if (!cxyz) return;
    const int c = q / LIMA_MAX_COMPOUND_PARTICLES, t = q % LIMA_MAX_COMPOUND_PARTICLES;
    const uint32_t b = d.cp_base[c];
    lima_float3 a = {0.f, 0.f, 0.f};
    if (t < (int)(d.cp_base[c + 1] - b)) {
        state_of_orig(d, cur, b + t, x, v);
        if (t > 0) {
            double x0[3], v0[3];
            state_of_orig(d, cur, b, x0, v0);
            const double L = d.L;
            for (int k = 0; k < 3; k++) {
                const double dd = x[k] - x0[k];
                x[k] = x0[k] + (dd - L * nearbyint(dd / L));
            }
        }
        a = lima_float3{(float)x[0], (float)x[1], (float)x[2]};
    }
    cxyz[q] = a;
}

__global__ void k_read_solvents(PhysDev d, int cur, lima_solvent* __restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.n_s) return;
    double x[3], v[3];
    state_of_orig(d, cur, (uint32_t)(d.n_cp + s), x, v);
    out[s].pos = lima_float3{(float)x[0], (float)x[1], (float)x[2]};
    out[s].pos_tsub1 = lima_float3{(float)(x[0] - v[0] * d.dt), (float)(x[1] - v[1] * d.dt), (float)(x[2] - v[2] * d.dt)};
}
}  // namespace

void launch_read_compounds(const PhysDev& d, int cur, lima_compound_state* states, lima_float3* prev, cudaStream_t s) {
    const int n = d.n_c * LIMA_MAX_COMPOUND_PARTICLES;
    if (n > 0) k_read_compounds<<<(n + kTB - 1) / kTB, kTB, 0, s>>>(d, cur, states, prev);
}

void launch_read_positions(const PhysDev& d, int cur, lima_float3* cxyz, lima_float3* sxyz, cudaStream_t s) {
    const int n = d.n_c * LIMA_MAX_COMPOUND_PARTICLES + d.n_s;
    if (n > 0) k_read_positions<<<(n + kTB - 1) / kTB, kTB, 0, s>>>(d, cur, cxyz, sxyz);
}

void launch_read_solvents(const PhysDev& d, int cur, lima_solvent* out, cudaStream_t s) {
    if (d.n_s > 0) k_read_solvents<<<(d.n_s + kTB - 1) / kTB, kTB, 0, s>>>(d, cur, out);
}

int launch_bonded(const PhysDev& d, int cur, bool energy, cudaStream_t s) {
    const int nb = bonded_blocks(d);
    if (nb == 0) return 0;
    const bool mixed = d.precision == LIMA_PRECISION_MIXED;
    if (energy && mixed)
        k_bonded<true, true><<<nb, kTB, 0, s>>>(d, cur);
    else if (energy)
        k_bonded<true, false><<<nb, kTB, 0, s>>>(d, cur);
    else if (mixed)
        k_bonded<false, true><<<nb, kTB, 0, s>>>(d, cur);
    else
        k_bonded<false, false><<<nb, kTB, 0, s>>>(d, cur);
    return 1;
}

void launch_step(const PhysDev& d, int cur, bool mixed, bool energy, bool integrate, int slot, cudaGraphExec_t tail,
                 cudaStream_t s) {
    if (mixed) {
        if (!integrate) step_variant<true, true, false, false>(d, cur, slot, nullptr, s);
        else if (energy) step_tail<true, true, true>(d, cur, slot, tail, s);
        else step_tail<true, false, true>(d, cur, slot, tail, s);
    } else {
        if (!integrate) step_variant<false, true, false, false>(d, cur, slot, nullptr, s);
        else if (energy) step_tail<false, true, true>(d, cur, slot, tail, s);
        else step_tail<false, false, true>(d, cur, slot, tail, s);
    }
}

}  // namespace lima
