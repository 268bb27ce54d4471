// Uniform-grid binning for B200: cell hash -> histogram -> scan -> stable
// counting sort -> work list, and the permutation kernels.
//
// Replaces HashGrid::initialize / bin_particles / backward_bin_particles of the
// reference (sphops/sph_cuda.cu:32-206,1926-2056).  Differences by design:
//  * the slot order inside a cell is the original particle order (stable), so
//    the permutation is deterministic; the reference orders by atomic arrival;
//  * histograms use warp-aggregated atomics, held in shared memory when the
//    per-system cell table fits, so a cell-coherent input (every step after the
//    first of a rollout) does not serialise on one address;
//  * cell counts and work-item counts are scanned together, and the work list
//    is written by the scan's last phase.
// All kernels are HBM-bound integer work; nothing here is GEMM shaped.
#include <cooperative_groups.h>

#include <mutex>

#include "ops.cuh"
#include "mlp_grad_reduce.cuh"
#include "weight_image.cuh"

namespace npa {

constexpr int kBinThreads = 256;
// Particles per thread in the hash pass: as many as share a shared-memory histogram well, and one where the atomics go to global memory:
// each is a round trip that the next waits for, and eight after another were all of the pass (65,536 and 524,288 particles in 3D 14.5 and
// 15 us,
// now 4.2 and 6.6).
template <bool SMEM>
constexpr int kBinPerThread = SMEM ? 8 : 1;
constexpr int kSmemHistCells = 8192;                   // 32 KB of shared histogram at most
constexpr int kScanThreads = 256;
constexpr int kScanPerThread = 8;
constexpr int kScanTile = kScanThreads * kScanPerThread;
// Up to so many tiles every CTA of scan_apply_kernel adds up the tiles before its own by itself, tiles^2 x 8 bytes from L2 in all; beyond, a
// launch of one CTA makes prefixes of their sums.  The whole build by prefixes / by itself, us, on a stream: 256 tiles (2 x 64^3 cells) 26.9 / 25.4,
// 512 (1,024^2) 24.9 / 23.1, 1,024 (128^3) 36.4 / 37.1, 2,048 57.7 / 58.6, 4,096 95 / 100; in a graph 26.1 / 24.8, 22.8 / 22.1, 33.2 / 33.0, 52.4 / 52.1,
// 93 / 92.
constexpr int kScanPartials = 512;
// Cells with more particles than this are ranked by rank_crowded_kernel (linear in the population)
// instead of the per-particle scan of rank_kernel (quadratic in it).
constexpr int kCrowdedCell = 256;
constexpr int kRankWindow = 1 << 17;  // particle indices per bitmap window of rank_crowded_kernel (32 KB of shared memory)
constexpr int kRankCtas = 64;

struct BinScratch {
    uint32_t *counts;   // [B*cells + 1], then one word: number of crowded cells (zeroed with the counts)
    uint32_t *crowded;  // [B*N / kCrowdedCell + 1] global cell index of each crowded cell
    uint32_t *arrive;   // [B*N]  arrival number of the particle inside its cell (any order)
    uint32_t *cellid;   // [B*N]
    uint32_t *order;    // [B*N]  slot -> particle, unsorted inside a cell
    unsigned long long *partials;  // [tiles + 1] packed (blocks << 32 | particles)
    size_t zero_bytes;  // the counts are zeroed per call
    int tiles;
};

static size_t align_up(size_t v) { return (v + 255) & ~(size_t)255; }

static size_t layout_scratch(const Geom &g, void *base, BinScratch *s) {
    const size_t nc = (size_t)g.B * g.cells;
    const size_t np = (size_t)g.B * g.N;
    const int tiles = (int)((nc + kScanTile - 1) / kScanTile);
    size_t off = 0;
    char *p = (char *)base;
    size_t counts_off = off;
    off += align_up((nc + 2) * 4);
    size_t zero_end = off;
    size_t crowded_off = off;
    off += align_up((np / kCrowdedCell + 1) * 4);
    size_t arrive_off = off;
    off += align_up(np * 4);
    size_t cellid_off = off;
    off += align_up(np * 4);
    size_t order_off = off;
    off += align_up(np * 4);
    size_t part_off = off;
    off += align_up((size_t)(tiles + 1) * 8);
    if (s) {
        s->counts = (uint32_t *)(p + counts_off);
        s->crowded = (uint32_t *)(p + crowded_off);
        s->arrive = (uint32_t *)(p + arrive_off);
        s->cellid = (uint32_t *)(p + cellid_off);
        s->order = (uint32_t *)(p + order_off);
        s->partials = (unsigned long long *)(p + part_off);
        s->zero_bytes = zero_end;
        s->tiles = tiles;
    }
    return off;
}

// ---------------------------------------------------------------------------
// Pass 1: cell id per particle + per-cell histogram.
// ---------------------------------------------------------------------------
template <int D>
__device__ inline uint32_t particle_cell(const float *__restrict__ x, size_t idx, const Geom &g) {
    int cx, cy, cz = 0;
    if (D == 2) {
        float2 p = __ldg(reinterpret_cast<const float2 *>(x) + idx);
        cx = axis_cell(p.x, g, 0);
        cy = axis_cell(p.y, g, 1);
    } else {
        float4 p = __ldg(reinterpret_cast<const float4 *>(x) + idx);
        cx = axis_cell(p.x, g, 0);
        cy = axis_cell(p.y, g, 1);
        cz = axis_cell(p.z, g, 2);
    }
    return cell_hash<D>(g, cx, cy, cz);
}

// One atomic per distinct cell per warp: lanes holding the same key elect their lowest lane, which
// adds the group's population; every lane gets its arrival number in the cell (the counter's old
// value plus its rank in the group), which later serves as its unsorted slot inside the cell.
__device__ inline uint32_t warp_aggregated_take(uint32_t *hist, uint32_t key, bool valid) {
    const unsigned mask = __ballot_sync(kFull, valid);
    if (!valid) return 0;
    const unsigned peers = __match_any_sync(mask, key);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&hist[key], (uint32_t)__popc(peers));
    base = __shfl_sync(peers, base, leader);
    return base + (uint32_t)__popc(peers & ((1u << lane) - 1));
}

// The counts of a build start at zero.  A kernel and not a memset, so that its launch and that of the next overlap.
__global__ void __launch_bounds__(kBinThreads) zero_counts_kernel(uint4 *__restrict__ counts, size_t quads) {
    after_previous_kernel();
    for (size_t q = blockIdx.x * (size_t)kBinThreads + threadIdx.x; q < quads; q += (size_t)gridDim.x * kBinThreads)
        counts[q] = make_uint4(0u, 0u, 0u, 0u);
}

template <int D, bool SMEM>
__global__ void __launch_bounds__(kBinThreads)
hash_count_kernel(const float *__restrict__ x, uint32_t *__restrict__ cellid, uint32_t *__restrict__ arrive,
                  uint32_t *__restrict__ counts, Geom g) {
    after_previous_kernel();
    extern __shared__ uint32_t hist[];
    const int b = blockIdx.y;
    constexpr int PT = kBinPerThread<SMEM>;
    const int base = blockIdx.x * kBinThreads * PT;
    if (SMEM) {
        for (int c = threadIdx.x; c < g.cells; c += kBinThreads) hist[c] = 0;
        __syncthreads();
    }
    uint32_t *gl = counts + (size_t)b * g.cells;
    uint32_t keys[PT], arr[PT];
#pragma unroll
    for (int k = 0; k < PT; ++k) {
        const int i = base + k * kBinThreads + threadIdx.x;
        keys[k] = i < g.N ? particle_cell<D>(x, (size_t)b * g.N + i, g) : 0u;
    }
#pragma unroll
    for (int k = 0; k < PT; ++k) {
        const int i = base + k * kBinThreads + threadIdx.x;
        if (i < g.N) cellid[(size_t)b * g.N + i] = keys[k];
        arr[k] = warp_aggregated_take(SMEM ? hist : gl, keys[k], i < g.N);
    }
    if (SMEM) {
        // the CTA's populations go to the global counters in one atomic per cell; the old values
        // (where this CTA's particles start in the cell) replace the local counts
        __syncthreads();
        for (int c0 = threadIdx.x; c0 < g.cells; c0 += kBinThreads * 8) {  // eight round trips at a time
            uint32_t v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int c = c0 + u * kBinThreads;
                v[u] = c < g.cells ? hist[c] : 0u;
                if (v[u]) v[u] = atomicAdd(&gl[c], v[u]);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (c0 + u * kBinThreads < g.cells) hist[c0 + u * kBinThreads] = v[u];
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < PT; ++k) {
        const int i = base + k * kBinThreads + threadIdx.x;
        if (i < g.N) arrive[(size_t)b * g.N + i] = arr[k] + (SMEM ? hist[keys[k]] : 0u);
    }
}

// ---------------------------------------------------------------------------
// Exclusive scan of (particles per cell, work items per cell), packed as one 64-bit word so both prefix sums ride the same shuffles:
// the sums of tiles of cells, then in each tile the sum of the tiles before it and the cells' own prefixes (of more than
// kScanPartials tiles the sums are scanned in a launch between).
// ---------------------------------------------------------------------------
__device__ inline unsigned long long pack_cell(uint32_t count, int mpb) {
    uint32_t blocks = (count + (uint32_t)mpb - 1) / (uint32_t)mpb;
    return ((unsigned long long)blocks << 32) | count;
}

__device__ inline unsigned long long warp_inclusive(unsigned long long v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long t = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive scan of one value per thread across the CTA; returns the prefix of
// this thread and the CTA total through `total`.
template <int THREADS>
__device__ inline unsigned long long block_exclusive(unsigned long long v, unsigned long long &total) {
    __shared__ unsigned long long warp_tot[THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long inc = warp_inclusive(v);
    if (lane == 31) warp_tot[w] = inc;
    __syncthreads();
    if (w == 0) {
        unsigned long long t = lane < THREADS / 32 ? warp_tot[lane] : 0ull;
        unsigned long long ti = warp_inclusive(t);
        if (lane < THREADS / 32) warp_tot[lane] = ti - t;
        if (lane == THREADS / 32 - 1) total = ti;
    }
    __syncthreads();
    unsigned long long r = warp_tot[w] + inc - v;
    return r;
}

__global__ void __launch_bounds__(kScanThreads)
scan_tile_sums_kernel(const uint32_t *__restrict__ counts, unsigned long long *__restrict__ partials,
                      int n, int mpb) {
    after_previous_kernel();
    __shared__ unsigned long long tot;
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanPerThread;
    unsigned long long v = 0;
#pragma unroll
    for (int k = 0; k < kScanPerThread; ++k)
        if (base + k < n) v += pack_cell(counts[base + k], mpb);
    block_exclusive<kScanThreads>(v, tot);
    __syncthreads();
    if (threadIdx.x == 0) partials[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(1024)
scan_partials_kernel(unsigned long long *partials, int tiles) {
    after_previous_kernel();
    __shared__ unsigned long long tot;
    __shared__ unsigned long long carry_s;
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (int base = 0; base < tiles; base += 1024) {
        const int i = base + threadIdx.x;
        unsigned long long v = i < tiles ? partials[i] : 0ull;
        unsigned long long ex = block_exclusive<1024>(v, tot);
        unsigned long long carry = carry_s;
        if (i < tiles) partials[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry_s = carry + tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) partials[tiles] = carry_s;
}

// Writes bin_offsets, the work list rows of every non-empty cell, and zeroes
// the unused tail of the work list (rows [total_items, max_blocks)).  SCANNED: the partial sums are prefixes already, the grand total last.
template <bool SCANNED>
__global__ void __launch_bounds__(kScanThreads)
scan_apply_kernel(const uint32_t *__restrict__ counts, const unsigned long long *__restrict__ partials,
                  int32_t *__restrict__ bin_offsets, int4 *__restrict__ block_info, uint32_t *__restrict__ crowded,
                  uint32_t *__restrict__ crowded_count, int n, Geom g) {
    after_previous_kernel();
    __shared__ unsigned long long tot, sums[2][kScanThreads / 32];
    unsigned long long before = 0, grand = 0;  // the tiles before this one, all tiles
    if (SCANNED) {
        before = partials[blockIdx.x];
        grand = partials[gridDim.x];
    } else {
        for (int t = threadIdx.x; t < (int)gridDim.x; t += kScanThreads) {
            const unsigned long long v = partials[t];
            grand += v;
            if (t < (int)blockIdx.x) before += v;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            before += __shfl_xor_sync(kFull, before, o);
            grand += __shfl_xor_sync(kFull, grand, o);
        }
        if ((threadIdx.x & 31) == 0) {
            sums[0][threadIdx.x >> 5] = before;
            sums[1][threadIdx.x >> 5] = grand;
        }
        __syncthreads();
        before = grand = 0;
#pragma unroll
        for (int w = 0; w < kScanThreads / 32; ++w) {
            before += sums[0][w];
            grand += sums[1][w];
        }
    }
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanPerThread;
    uint32_t c[kScanPerThread];
    unsigned long long v = 0;
#pragma unroll
    for (int k = 0; k < kScanPerThread; ++k) {
        c[k] = base + k < n ? counts[base + k] : 0u;
        v += pack_cell(c[k], g.mpb);
    }
    unsigned long long run = before + block_exclusive<kScanThreads>(v, tot);
#pragma unroll
    for (int k = 0; k < kScanPerThread; ++k) {
        const int cell = base + k;
        if (cell < n) {
            const uint32_t start = (uint32_t)run;
            uint32_t row = (uint32_t)(run >> 32);
            bin_offsets[cell] = (int32_t)start;
            if (c[k] > (uint32_t)kCrowdedCell) crowded[atomicAdd(crowded_count, 1u)] = (uint32_t)cell;
            const int sys = cell / g.cells;
            for (uint32_t off = 0; off < c[k]; off += (uint32_t)g.mpb, ++row)
                block_info[row] = make_int4(cell, (int)off, (int)min((uint32_t)g.mpb, c[k] - off), sys);
        }
        run += pack_cell(c[k], g.mpb);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) bin_offsets[n] = (int32_t)(uint32_t)grand;
    const int total_items = (int)(grand >> 32);
    for (int r = total_items + blockIdx.x * kScanThreads + threadIdx.x; r < g.max_blocks;
         r += gridDim.x * kScanThreads)
        block_info[r] = make_int4(0, 0, 0, 0);
}

// ---------------------------------------------------------------------------
// Pass 2: scatter particle indices to their cell's slots (any order inside the
// cell), then rank each slot by original index -> stable permutation.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBinThreads)
scatter_kernel(const uint32_t *__restrict__ cellid, const uint32_t *__restrict__ arrive,
               const int32_t *__restrict__ bin_offsets, uint32_t *__restrict__ order, Geom g) {
    after_previous_kernel();
    const int b = blockIdx.y;
    const int i = blockIdx.x * kBinThreads + threadIdx.x;
    if (i >= g.N) return;
    const size_t idx = (size_t)b * g.N + i;
    const size_t cell = (size_t)b * g.cells + cellid[idx];
    order[(uint32_t)bin_offsets[cell] + arrive[idx]] = (uint32_t)i;  // no atomics: the slot was drawn in pass 1
}

// Stable ranks inside crowded cells (a collapsed system, or particles clamped into an edge cell): a
// CTA takes one crowded cell at a time, marks the original indices of its particles in a bitmap over
// the system's particle indices (in windows of kRankWindow indices), turns the bitmap into prefix
// popcounts, and a particle's rank is the number of marked indices below its own.  Linear in the
// population plus N / 32 words per window; no sort, no atomics in global memory.
__device__ inline void rank_crowded(const int32_t *__restrict__ bin_offsets, const uint32_t *__restrict__ order,
                                    int32_t *__restrict__ permutation, const uint32_t *__restrict__ crowded,
                                    const uint32_t *__restrict__ crowded_count, const Geom &g, uint32_t first, uint32_t stride) {
    extern __shared__ uint32_t rank_smem[];
    __shared__ uint32_t warp_tot[8];
    __shared__ uint32_t carry;
    const int win = g.N < kRankWindow ? g.N : kRankWindow;
    const int words = (win + 31) / 32;
    uint32_t *bits = rank_smem, *pre = rank_smem + words;
    const uint32_t n = *crowded_count;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (uint32_t entry = first; entry < n; entry += stride) {
        const uint32_t cell = crowded[entry];
        const uint32_t sys = (cell / (uint32_t)g.cells) * (uint32_t)g.N;
        const uint32_t s = (uint32_t)bin_offsets[cell], e = (uint32_t)bin_offsets[cell + 1];
        uint32_t below = 0;  // particles of the cell with an index below the current window
        for (uint32_t w0 = 0; w0 < (uint32_t)g.N; w0 += (uint32_t)win) {
            for (int k = threadIdx.x; k < words; k += 256) bits[k] = 0u;
            if (threadIdx.x == 0) carry = 0u;
            __syncthreads();
            for (uint32_t q = s + threadIdx.x; q < e; q += 256) {
                const uint32_t i = order[q] - w0;
                if (i < (uint32_t)win) atomicOr(&bits[i >> 5], 1u << (i & 31));
            }
            __syncthreads();
            // exclusive prefix of the word popcounts, 256 words per round
            for (int base = 0; base < words; base += 256) {
                const int k = base + threadIdx.x;
                const uint32_t v = k < words ? (uint32_t)__popc(bits[k]) : 0u;
                uint32_t inc = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(kFull, inc, o);
                    if (lane >= o) inc += t;
                }
                if (lane == 31) warp_tot[w] = inc;
                __syncthreads();
                uint32_t before = carry;
                for (int ww = 0; ww < w; ++ww) before += warp_tot[ww];
                if (k < words) pre[k] = before + inc - v;
                __syncthreads();
                if (threadIdx.x == 255) carry = before + inc;
                __syncthreads();
            }
            for (uint32_t q = s + threadIdx.x; q < e; q += 256) {
                const uint32_t idx = order[q];
                const uint32_t i = idx - w0;
                if (i < (uint32_t)win) {
                    const uint32_t rank = below + pre[i >> 5] + (uint32_t)__popc(bits[i >> 5] & ((1u << (i & 31)) - 1u));
                    permutation[sys + idx] = (int32_t)(s - sys + rank);
                }
            }
            below += carry;
            __syncthreads();
        }
    }
}

// The last kRankCtas columns of the grid take the crowded cells, the others a particle slot per thread.
__global__ void __launch_bounds__(kBinThreads)
rank_kernel(const uint32_t *__restrict__ cellid, const int32_t *__restrict__ bin_offsets, const uint32_t *__restrict__ order,
            int32_t *__restrict__ permutation, const uint32_t *__restrict__ crowded, const uint32_t *__restrict__ crowded_count, Geom g,
            int rank_columns) {
    after_previous_kernel();
    if ((int)blockIdx.x >= rank_columns) {
        if (blockIdx.y == 0)
            rank_crowded(bin_offsets, order, permutation, crowded, crowded_count, g, blockIdx.x - rank_columns, gridDim.x - rank_columns);
        return;
    }
    const int b = blockIdx.y;
    const int p = blockIdx.x * kBinThreads + threadIdx.x;
    if (p >= g.N) return;
    const size_t sys = (size_t)b * g.N;
    const uint32_t i = order[sys + p];
    const uint32_t key = cellid[sys + i];
    const size_t cell = (size_t)b * g.cells + key;
    const uint32_t s = (uint32_t)bin_offsets[cell], e = (uint32_t)bin_offsets[cell + 1];
    if (e - s > (uint32_t)kCrowdedCell) return;  // ranked by the crowded-cell blocks
    uint32_t rank = 0;
    for (uint32_t q = s; q < e; ++q) rank += order[q] < i ? 1u : 0u;
    permutation[sys + i] = (int32_t)(s - (uint32_t)sys + rank);
}

// ---------------------------------------------------------------------------
// Small systems: everything but the work list in one launch, a CTA per system with the cell table, the cell ids and the
// slots in shared memory.  The general path is six dependent launches of 1.5-8 us each for 8 x 4,096 particles
// (21 us): what bounds it there is launch latency, not memory.  With the work list's launch this takes 13 us (9.2 + 3.7), 6.5 for one system of 2,500.
// ---------------------------------------------------------------------------
constexpr int kSmallThreads = 1024;
constexpr int kSmallParticles = 16384;
constexpr size_t kSmallSmem = 200 * 1024, kClusterSmem = 220 * 1024;

// Place of a cell in the shared table: one word of padding per 32, so that threads that walk consecutive cells each do not
// meet on one bank.
__host__ __device__ inline int table_at(int c) { return c + (c >> 5); }

static size_t small_smem(const Geom &g) {
    return (size_t)(table_at(g.cells) + 1) * 4 + (size_t)((g.N + 1) & ~1) * 4 + (size_t)((g.N + 31) / 32) * 8;
}

// Which way to build a grid, from estimates of all in microseconds.
//  * Small, one CTA per system: a fixed part; the particles; ranking inside cells (pairs of a cell, or a bitmap beyond kCrowdedCell);
//    the cell table, which a thread walks in consecutive cells -- once in shared memory and, with several systems, again in
//    global memory, where long runs per thread scatter the loads.
//  * Cluster, eight CTAs per system: a fixed part; the share of a CTA; ranking among the share's particles of a cell; the systems, and
//    the cells where there are more CTAs than SMs; the rows as above.
//  * General: six launches (seven beyond kScanPartials tiles of cells); the shared histogram; the particles and cells of all systems; ranking, spread over the chip; crowded cells.
// Small was fitted to 560 sizes (2D and 3D, 256 to 16,384 particles, 1 to 64 systems, 16 to 32,768 cells), cluster and general, whose
// launches overlap on a stream, to 777 sizes (2,500 to 65,536 particles, 1 to 32 systems, 9 to 32,768 cells) on a stream and in a graph:
// 0.3 % behind the best way on average, 16 % at worst.  Some sizes, small / cluster / general, us, in a graph: 1 system of 2,500 in
// 10 x 10 7.7 / 8.1 / 20; 8 of 4,096 in 16 x 16 13 / 11 / 22; 8 of 16,384 in 40 x 40 27 / 14 / 25; 4 of 16,384 in 32^3 - / 86 / 17;
// 2 of 30,000 in 24^3 - / 33 / 17; 1 of 65,536 in 64 x 64 - / 20 / 25, in 16 x 16 - / 24 / 39.
enum class GridBuild { kSmall, kCluster, kGeneral };

static double rows_estimate(const Geom &g) {
    const double c = g.cells;
    return g.B > 1 ? 3.0 + c * c / 2.2e7 + c / 4000.0 : c / 2500.0;
}

constexpr int kClusterCtas = 8;
static size_t cluster_smem(const Geom &g, int ctas);

static GridBuild grid_build(const Geom &g) {
    const double n = g.N, c = g.cells, all = n * g.B, per_cell = n / c, ranking = per_cell > kCrowdedCell ? 0.0 : n * per_cell;
    const double none = 1e30;
    const bool fits = g.N <= kSmallParticles && g.cells < 65536 && small_smem(g) <= kSmallSmem;
    const double small = fits ? 4.0 + n / 900.0 + (per_cell > kCrowdedCell ? 10.0 : ranking / 54000.0) + rows_estimate(g) : none;
    const double crowded = per_cell > 0.9 * kCrowdedCell ? 1.6 + per_cell * 0.0078 + all * 8.3e-5 : 0.0;  // (half of the cells, at the mean)
    const double general = 14.5 + (g.cells <= kSmemHistCells ? 6.6 + c / 8400.0 : 0.0) + all / 35000.0 + c * g.B / 123000.0 +
                           ranking * g.B * 3.05e-7 + crowded;
    const bool shares = g.N > 2048 && g.N <= 65536 && g.cells < 65536 && cluster_smem(g, kClusterCtas) <= kClusterSmem;
    const double share_ranking = per_cell > kCrowdedCell * kClusterCtas ? 19.0 : n * per_cell / 2.6e6;
    const double beyond = kClusterCtas * g.B > 148 ? c * (kClusterCtas * g.B - 148) / 160000.0 : 0.0;  // CTAs beyond one per SM
    const double cluster = shares ? 7.5 + n / 4800.0 + share_ranking + g.B / 24.0 + beyond + rows_estimate(g) : none;
    if (cluster < small && cluster < general) return GridBuild::kCluster;
    return small <= general ? GridBuild::kSmall : GridBuild::kGeneral;
}

// Exclusive scan over the CTA's cell table: every thread takes `per` consecutive cells.  Calls emit(cell, count, prefix)
// in cell order; returns the grand total.  prefix and total count (work items << 32 | particles).
template <int THREADS = kSmallThreads, typename Count, typename Emit>
__device__ inline unsigned long long scan_cells(const Geom &g, Count &&count, Emit &&emit) {
    __shared__ unsigned long long tot;
    const int per = (g.cells + THREADS - 1) / THREADS, c0 = threadIdx.x * per, c1 = min(c0 + per, g.cells);
    unsigned long long v = 0;
    for (int c = c0; c < c1; ++c) v += pack_cell(count(c), g.mpb);
    unsigned long long run = block_exclusive<THREADS>(v, tot);
    for (int c = c0; c < c1; ++c) {
        const uint32_t n = count(c);
        emit(c, n, run);
        run += pack_cell(n, g.mpb);
    }
    __syncthreads();
    return tot;
}

// Rows of one system from its cell starts; row0 = rows of the systems before it.
__device__ inline void write_rows(int4 *__restrict__ block_info, const Geom &g, int b, int cell, uint32_t n, uint32_t row) {
    for (uint32_t off = 0; off < n; off += (uint32_t)g.mpb, ++row)
        block_info[row] = make_int4(b * g.cells + cell, (int)off, (int)min((uint32_t)g.mpb, n - off), b);
}

template <int D>
__global__ void __launch_bounds__(kSmallThreads)
bin_small_kernel(const float *__restrict__ x, int32_t *__restrict__ permutation, int32_t *__restrict__ bin_offsets,
                 int4 *__restrict__ block_info, uint32_t *__restrict__ rows_of_system, Geom g) {
    after_previous_kernel();
    extern __shared__ uint32_t small_mem[];
    __shared__ uint32_t crowded_n, s_crowded[kSmallParticles / kCrowdedCell];
    uint32_t *table = small_mem;                                     // per cell: count, then next free slot, then end
    uint16_t *key = reinterpret_cast<uint16_t *>(table + table_at(g.cells) + 1);  // [N] cell of the particle
    uint16_t *order = key + ((g.N + 1) & ~1);                        // [N] particle of the slot, any order in a cell
    const int words = (g.N + 31) / 32;
    uint32_t *bits = reinterpret_cast<uint32_t *>(order + ((g.N + 1) & ~1)), *pre = bits + words;  // crowded cells only
    const int b = blockIdx.x, tid = threadIdx.x;
    const size_t sys = (size_t)b * g.N;
    for (int c = tid; c <= table_at(g.cells); c += kSmallThreads) table[c] = 0u;
    if (tid == 0) crowded_n = 0u;
    __syncthreads();
    for (int i = tid; i < g.N; i += kSmallThreads) {
        const uint32_t k = particle_cell<D>(x, sys + i, g);
        key[i] = (uint16_t)k;
        atomicAdd(&table[table_at((int)k)], 1u);
    }
    __syncthreads();
    const unsigned long long total = scan_cells(
        g, [&](int c) { return table[table_at(c)]; },
        [&](int c, uint32_t n, unsigned long long run) {
            if (g.B == 1) write_rows(block_info, g, 0, c, n, (uint32_t)(run >> 32));
            if (n > (uint32_t)kCrowdedCell) s_crowded[atomicAdd(&crowded_n, 1u)] = (uint32_t)c;
            table[table_at(c)] = (uint32_t)run;
        });
    for (int c = tid; c < g.cells; c += kSmallThreads) bin_offsets[(size_t)b * g.cells + c] = (int32_t)((uint32_t)sys + table[table_at(c)]);
    if (tid == 0) {
        rows_of_system[b] = (uint32_t)(total >> 32);
        if (b == g.B - 1) bin_offsets[(size_t)g.B * g.cells] = (int32_t)((size_t)g.B * g.N);
    }
    if (g.B == 1)
        for (int r = (int)(total >> 32) + tid; r < g.max_blocks; r += kSmallThreads) block_info[r] = make_int4(0, 0, 0, 0);
    __syncthreads();
    for (int i = tid; i < g.N; i += kSmallThreads) order[atomicAdd(&table[table_at(key[i])], 1u)] = (uint16_t)i;
    __syncthreads();
    // every slot of a cell is taken: its entry is now its end, the entry before it its start
    auto cell_start = [&](uint32_t c) { return c ? table[table_at((int)c - 1)] : 0u; };
    for (int p = tid; p < g.N; p += kSmallThreads) {
        const uint32_t i = order[p], c = key[i], s = cell_start(c), e = table[table_at((int)c)];
        if (e - s > (uint32_t)kCrowdedCell) continue;
        uint32_t rank = 0;
        for (uint32_t q = s; q < e; ++q) rank += order[q] < i ? 1u : 0u;
        permutation[sys + i] = (int32_t)(s + rank);
    }
    // crowded cells: a bitmap over the particle indices and its prefix popcounts, as in rank_crowded
    for (uint32_t k = 0; k < crowded_n; ++k) {
        const uint32_t s = cell_start(s_crowded[k]), e = table[table_at((int)s_crowded[k])];
        __syncthreads();
        for (int w = tid; w < words; w += kSmallThreads) bits[w] = 0u;
        __syncthreads();
        for (uint32_t q = s + tid; q < e; q += kSmallThreads) atomicOr(&bits[order[q] >> 5], 1u << (order[q] & 31));
        __syncthreads();
        __shared__ unsigned long long marked;
        const unsigned long long mine = tid < words ? (unsigned long long)__popc(bits[tid]) : 0ull;  // words <= 512
        const unsigned long long before = block_exclusive<kSmallThreads>(mine, marked);
        if (tid < words) pre[tid] = (uint32_t)before;
        __syncthreads();
        for (uint32_t q = s + tid; q < e; q += kSmallThreads) {
            const uint32_t i = order[q];
            permutation[sys + i] = (int32_t)(s + pre[i >> 5] + (uint32_t)__popc(bits[i >> 5] & ((1u << (i & 31)) - 1u)));
        }
    }
}

// ---------------------------------------------------------------------------
// Systems of up to 65,536 particles by one cluster of CTAs each.  A CTA counts and orders its share of the particles (consecutive
// indices) in shared memory; the CTAs then share the cells: the owner of a slice of them reads the counts of all CTAs through
// distributed shared memory, scans them and leaves every CTA the slot of its first particle in each cell.  Stable: the particles of a
// cell lie CTA by CTA, and inside a CTA in index order.  Counts and slots are 16 bits, two to a word (shares of at most 8,192).
// Bound by latency: four passes over the share and three meetings of the cluster.  Back to back on a stream, work list included,
// us: 8 systems of 16,384 in 40 x 40 25 (one CTA per system) -> 13, 1 of 16,384 in 64 x 64 21 -> 11, 1 of 4,096 in 10 x 10 9.6 -> 7.4, 8 of
// 4,096 in 16 x 16 11.2 -> 10; 1 of 65,536 in 64 x 64 32 (general launches) -> 20, 2 of 32,768 in 20^3 37 -> 26.
// ---------------------------------------------------------------------------
constexpr int kClusterThreads = 512, kClusterMost = 8, kClusterShare = 8192;

static size_t cluster_smem(const Geom &g, int ctas) {
    const int words = (g.cells + 1) / 2, slice = (words + ctas - 1) / ctas, share = (g.N + ctas - 1) / ctas;
    return (size_t)(table_at(words) + 1) * 8 + (size_t)slice * 8 + (size_t)((share + 31) / 32) * 8 + (size_t)((share + 1) & ~1) * 4;
}

__device__ inline uint32_t half_of(const uint32_t *words, uint32_t c) { return (words[table_at((int)(c >> 1))] >> (16 * (c & 1))) & 0xffffu; }

template <int D>
__global__ void __launch_bounds__(kClusterThreads)
bin_cluster_kernel(const float *__restrict__ x, int32_t *__restrict__ permutation, int32_t *__restrict__ bin_offsets,
                   int4 *__restrict__ block_info, uint32_t *__restrict__ rows_of_system, Geom g) {
    after_previous_kernel();
    constexpr int T = kClusterThreads;
    extern __shared__ uint32_t cluster_mem[];
    __shared__ uint32_t s_bound[kClusterMost], s_items, crowded_n, s_crowded[kClusterShare / kCrowdedCell];
    __shared__ unsigned long long scan_total;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int K = (int)cluster.num_blocks(), r = (int)cluster.block_rank(), b = blockIdx.x / K, tid = threadIdx.x;
    const int words = (g.cells + 1) / 2, slice = (words + K - 1) / K, share = (g.N + K - 1) / K;
    const int i0 = min(r * share, g.N), mine = min(share, g.N - i0), marks = (share + 31) / 32;
    uint32_t *first = cluster_mem;                            // per cell: particles of this CTA, then the slot of the first of them
    uint32_t *next = first + table_at(words) + 1;             // per cell: next place in this CTA's order, then their end
    uint32_t *total = next + table_at(words) + 1;             // per cell of this CTA's slice: particles of the system
    uint32_t *bits = total + 2 * slice, *pre = bits + marks;  // crowded cells only
    uint16_t *key = reinterpret_cast<uint16_t *>(pre + marks), *order = key + ((share + 1) & ~1);
    const size_t sys = (size_t)b * g.N;
    for (int w = tid; w <= table_at(words); w += T) first[w] = 0u;
    if (tid < K) s_bound[tid] = (uint32_t)mine;
    if (tid == 0) crowded_n = 0u;
    __syncthreads();
    for (int i = tid; i < mine; i += T) {
        const uint32_t c = particle_cell<D>(x, sys + i0 + i, g);
        key[i] = (uint16_t)c;
        atomicAdd(&first[table_at((int)(c >> 1))], 1u << (16 * (c & 1)));
    }
    __syncthreads();
    {   // places in this CTA's order, and how many of its particles lie before each slice of the cells
        const int per = (words + T - 1) / T, w0 = tid * per, w1 = min(w0 + per, words);
        unsigned long long v = 0;
        for (int w = w0; w < w1; ++w) {
            const uint32_t n = first[table_at(w)];
            v += (n & 0xffffu) + (n >> 16);
        }
        uint32_t run = (uint32_t)block_exclusive<T>(v, scan_total);
        for (int w = w0; w < w1; ++w) {
            const uint32_t n = first[table_at(w)], lo = n & 0xffffu, hi = n >> 16;
            if (w % slice == 0) s_bound[w / slice] = run;
            if (lo > (uint32_t)kCrowdedCell) s_crowded[atomicAdd(&crowded_n, 1u)] = (uint32_t)(2 * w);
            if (hi > (uint32_t)kCrowdedCell) s_crowded[atomicAdd(&crowded_n, 1u)] = (uint32_t)(2 * w + 1);
            next[table_at(w)] = run | ((run + lo) << 16);
            run += lo + hi;
        }
    }
    cluster.sync();
    // this CTA's slice of the cells
    unsigned long long before = 0;  // work items of the slice << 32 | particles of the system, up to here
    for (int q = 0; q < K; ++q) before += cluster.map_shared_rank(s_bound, q)[r];
    for (int base = 0; base < slice; base += T) {
        const int w = r * slice + base + tid;
        const bool valid = base + tid < slice && w < words;
        uint32_t n[kClusterMost], lo = 0, hi = 0;
#pragma unroll
        for (int q = 0; q < kClusterMost; ++q) {
            n[q] = valid && q < K ? cluster.map_shared_rank(first, q)[table_at(w)] : 0u;
            lo += n[q] & 0xffffu;
            hi += n[q] >> 16;
        }
        const unsigned long long at = before + block_exclusive<T>(pack_cell(lo, g.mpb) + pack_cell(hi, g.mpb), scan_total);
        if (valid) {
            uint32_t slot_lo = (uint32_t)at, slot_hi = slot_lo + lo;
            int32_t *o = bin_offsets + (size_t)b * g.cells + 2 * w;
            o[0] = (int32_t)((uint32_t)sys + slot_lo);
            if (2 * w + 1 < g.cells) o[1] = (int32_t)((uint32_t)sys + slot_hi);
            if (g.B == 1) {
                total[2 * (base + tid)] = lo;
                total[2 * (base + tid) + 1] = hi;
            }
#pragma unroll
            for (int q = 0; q < kClusterMost; ++q) {
                if (q >= K) break;
                cluster.map_shared_rank(first, q)[table_at(w)] = (slot_lo & 0xffffu) | (slot_hi << 16);
                slot_lo += n[q] & 0xffffu;
                slot_hi += n[q] >> 16;
            }
        }
        before += scan_total;
        __syncthreads();
    }
    if (tid == 0) {
        s_items = (uint32_t)(before >> 32);
        if (b == g.B - 1 && r == 0) bin_offsets[(size_t)g.B * g.cells] = (int32_t)((size_t)g.B * g.N);
    }
    for (int i = tid; i < mine; i += T) {
        const uint32_t c = key[i], shift = 16 * (c & 1);
        order[(atomicAdd(&next[table_at((int)(c >> 1))], 1u << shift) >> shift) & 0xffffu] = (uint16_t)i;
    }
    cluster.sync();
    // every place of a cell is taken: its entry is now its end, the entry before it its start
    auto cell_start = [&](uint32_t c) { return c ? half_of(next, c - 1) : 0u; };
    for (int p = tid; p < mine; p += T) {
        const uint32_t i = order[p], c = key[i], s = cell_start(c), e = half_of(next, c);
        if (e - s > (uint32_t)kCrowdedCell) continue;
        uint32_t rank = 0;
        for (uint32_t q = s; q < e; ++q) rank += order[q] < i ? 1u : 0u;
        permutation[sys + i0 + i] = (int32_t)(half_of(first, c) + rank);
    }
    // crowded cells: a bitmap over the particle indices and its prefix popcounts, as above
    for (uint32_t k = 0; k < crowded_n; ++k) {
        const uint32_t c = s_crowded[k], s = cell_start(c), e = half_of(next, c);
        __syncthreads();
        for (int w = tid; w < marks; w += T) bits[w] = 0u;
        __syncthreads();
        for (uint32_t q = s + tid; q < e; q += T) atomicOr(&bits[order[q] >> 5], 1u << (order[q] & 31));
        __syncthreads();
        const unsigned long long here = tid < marks ? (unsigned long long)__popc(bits[tid]) : 0ull;  // marks <= 256
        const unsigned long long earlier = block_exclusive<T>(here, scan_total);
        if (tid < marks) pre[tid] = (uint32_t)earlier;
        __syncthreads();
        for (uint32_t q = s + tid; q < e; q += T) {
            const uint32_t i = order[q];
            permutation[sys + i0 + i] = (int32_t)(half_of(first, c) + pre[i >> 5] + (uint32_t)__popc(bits[i >> 5] & ((1u << (i & 31)) - 1u)));
        }
    }
    // rows: their number for rows_small_kernel, or with a single system the work list itself
    uint32_t row = 0, rows = 0;
    for (int q = 0; q < K; ++q) {
        const uint32_t n = *cluster.map_shared_rank(&s_items, q);
        if (q < r) row += n;
        rows += n;
    }
    if (g.B > 1) {
        if (r == 0 && tid == 0) rows_of_system[b] = rows;
    } else {
        for (int base = 0; base < slice; base += T) {
            const int w = r * slice + base + tid;
            const bool valid = base + tid < slice && w < words;
            const uint32_t lo = valid ? total[2 * (base + tid)] : 0u, hi = valid ? total[2 * (base + tid) + 1] : 0u;
            const unsigned long long n_lo = pack_cell(lo, g.mpb) >> 32, n_hi = pack_cell(hi, g.mpb) >> 32;
            __syncthreads();
            const uint32_t at = row + (uint32_t)block_exclusive<T>(n_lo + n_hi, scan_total);
            write_rows(block_info, g, 0, 2 * w, lo, at);
            write_rows(block_info, g, 0, 2 * w + 1, hi, at + (uint32_t)n_lo);
            row += (uint32_t)scan_total;
        }
        for (int k = (int)rows + r * T + tid; k < g.max_blocks; k += K * T) block_info[k] = make_int4(0, 0, 0, 0);
    }
    cluster.sync();  // a CTA's shared memory stays until all have read it
}

// Cells of a system up to which its work list is written beside the reorder, by a block of 256 threads, instead of by a launch of its own with 1,024.
// Grid build and reorder, launch / beside, us: 8 x 4,096 particles in 2D, 256 cells 12.9 / 9.9, 1,024 13.2 / 11.0, 4,096 16.2 / 16.1; 64 x 512, 64 cells
// 9.5 / 6.5, 4,096 12.3 / 12.0; 8 x 4,096 in 3D, 4,096 cells 16.5 / 16.6; 300 x 100, 36 cells 13.4 / 9.0.
constexpr int kRowsBesideCells = 2048;

// Work list of several small systems, a CTA each: the rows of a system start behind those of the systems before it.
template <int THREADS>
__device__ inline void write_system_rows(const int32_t *__restrict__ bin_offsets, int4 *__restrict__ block_info,
                                         const uint32_t *__restrict__ rows_of_system, const Geom &g, int b) {
    __shared__ unsigned long long before_s;
    const int tid = threadIdx.x;
    unsigned long long before = 0, all = 0;  // rows of the systems before this one, rows in all
    for (int k = tid; k < g.B; k += THREADS) {
        const uint32_t r = rows_of_system[k];
        all += r;
        if (k < b) before += r;
    }
    block_exclusive<THREADS>(before | (all << 32), before_s);  // both totals below 2^29
    __syncthreads();
    const uint32_t row0 = (uint32_t)before_s, grand = (uint32_t)(before_s >> 32);
    const int32_t *off = bin_offsets + (size_t)b * g.cells;
    scan_cells<THREADS>(g, [&](int c) { return (uint32_t)(off[c + 1] - off[c]); },
                        [&](int c, uint32_t n, unsigned long long run) { write_rows(block_info, g, b, c, n, row0 + (uint32_t)(run >> 32)); });
    for (long long r = (long long)grand + (long long)b * THREADS + tid; r < g.max_blocks; r += (long long)g.B * THREADS)
        block_info[r] = make_int4(0, 0, 0, 0);
}

__global__ void __launch_bounds__(kSmallThreads)
rows_small_kernel(const int32_t *__restrict__ bin_offsets, int4 *__restrict__ block_info, const uint32_t *__restrict__ rows_of_system, Geom g) {
    after_previous_kernel();
    write_system_rows<kSmallThreads>(bin_offsets, block_info, rows_of_system, g, blockIdx.x);
}

// ---------------------------------------------------------------------------
// Permutation kernels.  One thread moves one 16-byte piece of a feature row
// (or one float when C % 4 != 0); the thread that owns piece 0 also moves the
// position and the mass.  FORWARD: out[perm[i]] = in[i]; else out[i] = in[perm[i]].
// ---------------------------------------------------------------------------
template <int D, bool FORWARD, typename VEC>
__device__ inline void permute_piece(const float *__restrict__ x, const float *__restrict__ s, const float *__restrict__ m,
                                     const int32_t *__restrict__ perm, float *__restrict__ xo, float *__restrict__ so,
                                     float *__restrict__ mo, int pieces, long long total, int N, unsigned block) {
    const long long t = (long long)block * 256 + threadIdx.x;
    if (t >= total) return;
    const long long particle = t / pieces;
    const int piece = (int)(t - particle * pieces);
    const long long sys0 = (particle / N) * N;
    const long long other = sys0 + __ldg(perm + particle);
    const long long src = FORWARD ? particle : other;
    const long long dst = FORWARD ? other : particle;
    if (s) {
        const VEC *in = reinterpret_cast<const VEC *>(s);
        VEC *out = reinterpret_cast<VEC *>(so);
        out[dst * pieces + piece] = __ldg(in + src * pieces + piece);
    }
    if (piece == 0) {
        if (x) {
            if (D == 2)
                reinterpret_cast<float2 *>(xo)[dst] = __ldg(reinterpret_cast<const float2 *>(x) + src);
            else
                reinterpret_cast<float4 *>(xo)[dst] = __ldg(reinterpret_cast<const float4 *>(x) + src);
        }
        if (m) mo[dst] = __ldg(m + src);
    }
}

template <int D, bool FORWARD, typename VEC>
__global__ void __launch_bounds__(256)
permute_kernel(const float *__restrict__ x, const float *__restrict__ s, const float *__restrict__ m,
               const int32_t *__restrict__ perm, float *__restrict__ xo, float *__restrict__ so,
               float *__restrict__ mo, int pieces, long long total, int N) {
    after_previous_kernel();
    permute_piece<D, FORWARD, VEC>(x, s, m, perm, xo, so, mo, pieces, total, N, blockIdx.x);
}

// The inverse reorder of a step's gradients, with the sum of the weight gradients by blocks before those of the particles: sixteen runs of
// sixteen quads each instead of thirty-two, the same order of sums.  The sum is a round trip to L2 long and was a launch of its own behind the
// gradients, which nothing waits for: training step of 8 x 4,096 particles in 2D 171.9 -> 166.6 us, 64 x 512 167.9 -> 160.1, of 4 x 16,384 in 3D
// 294.4 -> 291.6, of 4 x 65,536 no difference (1,608 -> 1,416 and 1,611 -> 1,419 against the same earlier code).
template <int D, typename VEC>
__global__ void __launch_bounds__(256)
permute_reduce_kernel(const float *__restrict__ x, const float *__restrict__ s, const int32_t *__restrict__ perm, float *__restrict__ xo,
                      float *__restrict__ so, int pieces, long long total, int N, unsigned first, const __grid_constant__ GradReduce grads) {
    after_previous_kernel();
    if (blockIdx.x < first) reduce_weight_grads<256 / kReduceRuns>(grads, (int)blockIdx.x);
    else permute_piece<D, false, VEC>(x, s, nullptr, perm, xo, so, nullptr, pieces, total, N, blockIdx.x - first);
}

// The reorder of a step, with the images of the MLP's weights made by blocks behind those of the particles, and the work list of several
// small systems by blocks before them: they have no launch of their own then (2 us of a small step each, and 5 us of the host).
template <int D, typename VEC>
__global__ void __launch_bounds__(256)
permute_images_kernel(const float *__restrict__ x, const float *__restrict__ s, const int32_t *__restrict__ perm, float *__restrict__ xo,
                      float *__restrict__ so, int pieces, long long total, int N, unsigned blocks, const __grid_constant__ ImageJobs jobs,
                      const __grid_constant__ RowsJob rest) {
    after_previous_kernel();
    if (blockIdx.x < (unsigned)rest.systems) {
        write_system_rows<256>(rest.bin_offsets, rest.block_info, rest.rows_of_system, rest.g, (int)blockIdx.x);
        return;
    }
    const unsigned block = blockIdx.x - rest.systems;
    if (block < blocks) permute_piece<D, true, VEC>(x, s, nullptr, perm, xo, so, nullptr, pieces, total, N, block);
    else write_image_element(jobs, (int)(block - blocks) * 256 + threadIdx.x);
}

static unsigned blocks_beside(const ImageJobs &jobs, const RowsJob &rest) { return (unsigned)(jobs.total() + 255) / 256 + (unsigned)rest.systems; }

// `images`: with those blocks, which only the reorders of a step have: ImageJobs and RowsJob forward, GradReduce back.
template <bool FORWARD, typename... Images>
static int launch_permute(const Geom &g, int C, const float *x, const float *s, const float *m,
                          const int32_t *perm, float *xo, float *so, float *mo, cudaStream_t st, const Images &...images) {
    static_assert(sizeof...(Images) == (FORWARD ? 2 : 1) || sizeof...(Images) == 0, "images by the forward reorder, weight gradients by the inverse one");
    if (!perm) return fail(NPA_ERR_INVALID_ARGUMENT, "permutation is NULL");
    if ((x == nullptr) != (xo == nullptr) || (s == nullptr) != (so == nullptr) || (m == nullptr) != (mo == nullptr))
        return fail(NPA_ERR_INVALID_ARGUMENT, "each input of a permutation needs its output (and vice versa)");
    if (s && C <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "channels must be positive, got %d", C);
    if (((uintptr_t)x | (uintptr_t)xo) % (g.dim == 2 ? 8 : 16))
        return fail(NPA_ERR_INVALID_ARGUMENT, "positions to permute must be aligned to one position (%d bytes)", g.dim == 2 ? 8 : 16);
    const bool vec = s && (C % 4 == 0) && ((((uintptr_t)s) | ((uintptr_t)so)) % 16 == 0);
    const int pieces = s ? (vec ? C / 4 : C) : 1;
    const long long total = (long long)g.B * g.N * pieces;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if constexpr (sizeof...(Images) == 2) {
        const unsigned all = blocks + blocks_beside(images...);
#define NPA_PERMUTE(DD, VEC) \
    launch_early(permute_images_kernel<DD, VEC>, all, 256, 0, st, x, s, perm, xo, so, pieces, total, g.N, blocks, images...)
        if (g.dim == 2) {
            if (vec) NPA_PERMUTE(2, float4); else NPA_PERMUTE(2, float);
        } else {
            if (vec) NPA_PERMUTE(3, float4); else NPA_PERMUTE(3, float);
        }
#undef NPA_PERMUTE
        return check_launch("permute_images_kernel");
    }
    if constexpr (sizeof...(Images) == 1) {
        const unsigned first = (images.blocks(256 / kReduceRuns) + ...);
#define NPA_PERMUTE(DD, VEC) \
    launch_early(permute_reduce_kernel<DD, VEC>, first + blocks, 256, 0, st, x, s, perm, xo, so, pieces, total, g.N, first, images...)
        if (g.dim == 2) {
            if (vec) NPA_PERMUTE(2, float4); else NPA_PERMUTE(2, float);
        } else {
            if (vec) NPA_PERMUTE(3, float4); else NPA_PERMUTE(3, float);
        }
#undef NPA_PERMUTE
        return check_launch("permute_reduce_kernel");
    }
#define NPA_PERMUTE(DD, VEC) \
    launch_early(permute_kernel<DD, FORWARD, VEC>, blocks, 256, 0, st, x, s, m, perm, xo, so, mo, pieces, total, g.N)
    if (g.dim == 2) {
        if (vec) NPA_PERMUTE(2, float4); else NPA_PERMUTE(2, float);
    } else {
        if (vec) NPA_PERMUTE(3, float4); else NPA_PERMUTE(3, float);
    }
#undef NPA_PERMUTE
    return check_launch(FORWARD ? "permute_kernel(forward)" : "permute_kernel(inverse)");
}

int bin_particles_and_images(const npa_grid *grid, int channels, const float *x, const float *s, const int32_t *permutation, float *x_out,
                             float *s_out, const ImageJobs &jobs, cudaStream_t stream, const RowsJob &rest) {
    Geom g;
    const int rc = make_geom(grid, &g);
    return rc != NPA_OK ? rc : launch_permute<true>(g, channels, x, s, nullptr, permutation, x_out, s_out, nullptr, stream, jobs, rest);
}

// ---------------------------------------------------------------------------
// safe inverse of symmetric 2x2 / 3x3 matrices (sphops/sph_cuda.cu:3095-3179):
// only the upper triangle is read; |det| < tol gives the identity.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
safe_inv2_kernel(const float4 *__restrict__ in, float4 *__restrict__ out, long long n, float tol) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const float4 a = __ldg(in + i);
    const float det = a.x * a.w - a.y * a.y;
    if (fabsf(det) < tol) {
        out[i] = make_float4(1.f, 0.f, 0.f, 1.f);
    } else {
        const float r = 1.0f / det;
        out[i] = make_float4(a.w * r, -a.y * r, -a.y * r, a.x * r);
    }
}

__global__ void __launch_bounds__(256)
safe_inv3_kernel(const float *__restrict__ in, float *__restrict__ out, long long n, float tol) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const float *p = in + i * 9;
    const float a = p[0], b = p[1], c = p[2], d = p[4], e = p[5], f = p[8];
    const float t1 = d * f - e * e, t2 = c * e - b * f, t3 = b * e - c * d;
    const float det = a * t1 + b * t2 + c * t3;
    float *o = out + i * 9;
    if (fabsf(det) < tol) {
        o[0] = 1.f; o[1] = 0.f; o[2] = 0.f;
        o[3] = 0.f; o[4] = 1.f; o[5] = 0.f;
        o[6] = 0.f; o[7] = 0.f; o[8] = 1.f;
    } else {
        const float r = 1.0f / det;
        const float m01 = t2 * r, m02 = t3 * r, m12 = (b * c - a * e) * r;
        o[0] = t1 * r;  o[1] = m01;                o[2] = m02;
        o[3] = m01;     o[4] = (a * f - c * c) * r; o[5] = m12;
        o[6] = m02;     o[7] = m12;                o[8] = (a * d - b * b) * r;
    }
}

// out = raw . inv(M) per particle, one thread per (particle, feature): HBM bound (8 D floats per thread and the D x D
// matrix of the particle from L1).  The product has inner dimension D: as a batched library GEMM it took 227 us for 32,768
// 2 x 2 matrices and 16 features (and 40 us for 15,003 and 13), most of it launch shape.
template <int D>
__global__ void __launch_bounds__(256)
corrected_gradient_kernel(const float *__restrict__ raw, const float *__restrict__ moment, float *__restrict__ out, long long total, int C,
                          float tol) {
    after_previous_kernel();
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    if (t >= total) return;
    const float *mp = moment + (t / C) * (D * D);
    float m[D * (D + 1) / 2], L[D * D], v[D];
    int k = 0;
#pragma unroll
    for (int p = 0; p < D; ++p)
#pragma unroll
        for (int q = p; q < D; ++q) m[k++] = __ldg(mp + p * D + q);
    safe_inverse_sym<D>(m, tol, L);
#pragma unroll
    for (int d = 0; d < D; ++d) v[d] = raw[t * D + d];
#pragma unroll
    for (int d = 0; d < D; ++d) {
        float acc = 0.f;
#pragma unroll
        for (int p = 0; p < D; ++p) acc = fmaf(v[p], L[p * D + d], acc);
        out[t * D + d] = acc;
    }
}

}  // namespace npa

using namespace npa;

extern "C" {

int64_t npa_grid_scratch_bytes(const npa_grid *gd) {
    Geom g;
    int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    return (int64_t)layout_scratch(g, nullptr, nullptr);
}

int npa_grid_build_kernels(const npa_grid *gd) {
    Geom g;
    const int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    if (grid_build(g) != GridBuild::kGeneral) return g.B == 1 ? 1 : 2;
    return ((long long)g.B * g.cells + kScanTile - 1) / kScanTile > kScanPartials ? 7 : 6;
}

int npa_grid_build(const npa_grid *gd, const float *x, int32_t *permutation, int32_t *bin_offsets,
                   int32_t *block_info, void *scratch, int64_t scratch_bytes, void *stream) {
    return grid_build_leaving(gd, x, permutation, bin_offsets, block_info, scratch, scratch_bytes, (cudaStream_t)stream, nullptr);
}

}  // extern "C"

namespace npa {

static int build_rows(const Geom &g, const int32_t *bin_offsets, int32_t *block_info, const uint32_t *rows_of_system, cudaStream_t st, RowsJob *rest) {
    const RowsJob job = {bin_offsets, reinterpret_cast<int4 *>(block_info), rows_of_system, g, g.B};
    if (rest && g.cells <= kRowsBesideCells) {
        *rest = job;
        return NPA_OK;
    }
    launch_early(rows_small_kernel, g.B, kSmallThreads, 0, st, bin_offsets, job.block_info, rows_of_system, g);
    return check_launch("rows_small_kernel");
}

int grid_build_leaving(const npa_grid *gd, const float *x, int32_t *permutation, int32_t *bin_offsets, int32_t *block_info, void *scratch,
                       int64_t scratch_bytes, cudaStream_t st, RowsJob *rest) {
    Geom g;
    int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    if (!x || !permutation || !bin_offsets || !block_info || !scratch)
        return fail(NPA_ERR_INVALID_ARGUMENT, "npa_grid_build: x, permutation, bin_offsets, block_info and scratch must be non-NULL");
    if (((uintptr_t)x % (g.dim == 2 ? 8 : 16)) || ((uintptr_t)block_info % 16) || ((uintptr_t)scratch % 16))
        return fail(NPA_ERR_INVALID_ARGUMENT, "npa_grid_build: x / block_info / scratch are not aligned to their vector width");
    BinScratch s;
    const size_t need = layout_scratch(g, scratch, &s);
    if (scratch_bytes < (int64_t)need)
        return fail(NPA_ERR_SCRATCH_TOO_SMALL, "npa_grid_build: scratch has %lld bytes, %zu needed", (long long)scratch_bytes, need);
    const GridBuild way = grid_build(g);
    if (way == GridBuild::kCluster) {
        const int ctas = kClusterCtas;
        const auto kernel = g.dim == 2 ? bin_cluster_kernel<2> : bin_cluster_kernel<3>;
        const size_t bytes = cluster_smem(g, ctas);
        int unused = 0;
        if ((rc = persistent_ctas(kernel, kClusterThreads, bytes, &unused)) != NPA_OK) return rc;  // shared-memory limit
        launch_cluster(ctas, kernel, g.B * ctas, kClusterThreads, bytes, st, x, permutation, bin_offsets, reinterpret_cast<int4 *>(block_info), s.counts, g);
        if ((rc = check_launch("bin_cluster_kernel")) != NPA_OK || g.B == 1) return rc;
        return build_rows(g, bin_offsets, block_info, s.counts, st, rest);
    }
    if (way == GridBuild::kSmall) {
        const size_t bytes = small_smem(g);
        int unused = 0;
        if (g.dim == 2) {
            if ((rc = persistent_ctas(bin_small_kernel<2>, kSmallThreads, bytes, &unused)) != NPA_OK) return rc;  // shared-memory limit
            launch_early(bin_small_kernel<2>, g.B, kSmallThreads, bytes, st, x, permutation, bin_offsets, reinterpret_cast<int4 *>(block_info), s.counts, g);
        } else {
            if ((rc = persistent_ctas(bin_small_kernel<3>, kSmallThreads, bytes, &unused)) != NPA_OK) return rc;
            launch_early(bin_small_kernel<3>, g.B, kSmallThreads, bytes, st, x, permutation, bin_offsets, reinterpret_cast<int4 *>(block_info), s.counts, g);
        }
        if ((rc = check_launch("bin_small_kernel")) != NPA_OK || g.B == 1) return rc;
        return build_rows(g, bin_offsets, block_info, s.counts, st, rest);
    }
    const size_t quads = s.zero_bytes / 16;  // (a multiple of 256 bytes)
    const size_t zero_ctas = (quads + kBinThreads - 1) / kBinThreads;
    launch_early(zero_counts_kernel, (unsigned)(zero_ctas < 148 * 8 ? zero_ctas : 148 * 8), kBinThreads, 0, st, reinterpret_cast<uint4 *>(s.counts), quads);
    if ((rc = check_launch("zero_counts_kernel")) != NPA_OK) return rc;

    const bool smem = g.cells <= kSmemHistCells;
    const int per_cta = kBinThreads * (smem ? kBinPerThread<true> : kBinPerThread<false>);
    const dim3 pgrid((g.N + per_cta - 1) / per_cta, g.B);
    const size_t smem_bytes = smem ? (size_t)g.cells * 4 : 0;
    if (g.dim == 2) {
        if (smem) launch_early(hash_count_kernel<2, true>, pgrid, kBinThreads, smem_bytes, st, x, s.cellid, s.arrive, s.counts, g);
        else launch_early(hash_count_kernel<2, false>, pgrid, kBinThreads, 0, st, x, s.cellid, s.arrive, s.counts, g);
    } else {
        if (smem) launch_early(hash_count_kernel<3, true>, pgrid, kBinThreads, smem_bytes, st, x, s.cellid, s.arrive, s.counts, g);
        else launch_early(hash_count_kernel<3, false>, pgrid, kBinThreads, 0, st, x, s.cellid, s.arrive, s.counts, g);
    }
    if ((rc = check_launch("hash_count_kernel")) != NPA_OK) return rc;

    const int n = g.B * g.cells;
    launch_early(scan_tile_sums_kernel, s.tiles, kScanThreads, 0, st, s.counts, s.partials, n, g.mpb);
    if ((rc = check_launch("scan_tile_sums_kernel")) != NPA_OK) return rc;
    const bool scanned = s.tiles > kScanPartials;
    if (scanned) {
        launch_early(scan_partials_kernel, 1, 1024, 0, st, s.partials, s.tiles);
        if ((rc = check_launch("scan_partials_kernel")) != NPA_OK) return rc;
    }
    uint32_t *crowded_count = s.counts + (size_t)n + 1;
    launch_early(scanned ? scan_apply_kernel<true> : scan_apply_kernel<false>, s.tiles, kScanThreads, 0, st, s.counts, s.partials, bin_offsets,
                 reinterpret_cast<int4 *>(block_info), s.crowded, crowded_count, n, g);
    if ((rc = check_launch("scan_apply_kernel")) != NPA_OK) return rc;

    const dim3 tgrid((g.N + kBinThreads - 1) / kBinThreads, g.B);
    launch_early(scatter_kernel, tgrid, kBinThreads, 0, st, s.cellid, s.arrive, bin_offsets, s.order, g);
    if ((rc = check_launch("scatter_kernel")) != NPA_OK) return rc;
    const int win = g.N < kRankWindow ? g.N : kRankWindow;
    const dim3 rgrid(tgrid.x + kRankCtas, g.B);
    launch_early(rank_kernel, rgrid, kBinThreads, (size_t)((win + 31) / 32) * 8, st, s.cellid, bin_offsets, s.order, permutation, s.crowded, crowded_count, g,
                                                                         (int)tgrid.x);
    return check_launch("rank_kernel");
}

}  // namespace npa

// Work arrays of npa_grid_build_static(): a fixed device array owned by the library, so that the
// call needs no scratch from the caller and allocates nothing.  In host code the symbol is only a
// handle; its device address is looked up once per device and cached below.
static __device__ __align__(256) unsigned char g_static_scratch[NPA_STATIC_SCRATCH_BYTES];

namespace npa {
constexpr int kMaxDevices = 64;
static std::mutex g_static_mutex;
static void *g_static_ptr[kMaxDevices] = {nullptr};

// Device address of g_static_scratch on the current device (queried once per device).
static int static_scratch_address(void **out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(NPA_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return fail(NPA_ERR_UNSUPPORTED, "device ordinal %d is out of range", dev);
    std::lock_guard<std::mutex> lock(g_static_mutex);
    if (!g_static_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess || !p)
            return fail(NPA_ERR_CUDA, "cudaGetSymbolAddress(static scratch) on device %d: %s", dev, cudaGetErrorString(e));
        g_static_ptr[dev] = p;
    }
    *out = g_static_ptr[dev];
    return NPA_OK;
}
}  // namespace npa

extern "C" {

int npa_grid_build_static(const npa_grid *gd, const float *x, int32_t *permutation, int32_t *bin_offsets,
                          int32_t *block_info, void *stream) {
    const int64_t need = npa_grid_scratch_bytes(gd);
    if (need < 0) return (int)need;
    if (need > (int64_t)NPA_STATIC_SCRATCH_BYTES)
        return fail(NPA_ERR_SCRATCH_TOO_SMALL,
                    "npa_grid_build_static: this grid needs %lld bytes of work arrays, the built-in array holds %u; "
                    "use npa_grid_build with caller scratch", (long long)need, (unsigned)NPA_STATIC_SCRATCH_BYTES);
    void *scratch = nullptr;
    int rc = static_scratch_address(&scratch);
    if (rc != NPA_OK) return rc;
    return npa_grid_build(gd, x, permutation, bin_offsets, block_info, scratch, (int64_t)NPA_STATIC_SCRATCH_BYTES, stream);
}

int npa_bin_particles(const npa_grid *gd, int32_t channels, const float *x, const float *s,
                      const float *mass, const int32_t *permutation, float *x_out, float *s_out,
                      float *mass_out, void *stream) {
    Geom g;
    int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    return launch_permute<true>(g, channels, x, s, mass, permutation, x_out, s_out, mass_out, (cudaStream_t)stream);
}

int npa_unbin_particles(const npa_grid *gd, int32_t channels, const float *x_bin, const float *s_bin,
                        const float *mass_bin, const int32_t *permutation, float *x_out, float *s_out,
                        float *mass_out, void *stream) {
    Geom g;
    int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    return launch_permute<false>(g, channels, x_bin, s_bin, mass_bin, permutation, x_out, s_out, mass_out, (cudaStream_t)stream);
}

int npa_step_unbin(const npa_grid *gd, int32_t channels, const float *x_bin, const float *s_bin, const int32_t *permutation, float *x_out,
                   float *s_out, int32_t in_dim, int32_t out_dim, const float *partial, int64_t partial_floats, float *dW1, float *dW2, float *db1,
                   void *stream) {
    const char *me = "npa_step_unbin";
    Geom g;
    const int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    if (!x_bin && !s_bin) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: positions or features must be given", me);
    if (!partial || !dW1 || !dW2 || !db1 || (uintptr_t)partial % 16)
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: partial, dW1, dW2 and db1 must be non-NULL, partial 16-byte aligned", me);
    const int64_t rows = (int64_t)g.B * g.N, need = npa_mlp_weight_grad_tcgen05_scratch_floats(rows, in_dim, out_dim);
    if (need <= 0 || partial_floats < need)
        return fail(need <= 0 ? NPA_ERR_INVALID_ARGUMENT : NPA_ERR_SCRATCH_TOO_SMALL, "%s: partial has %lld floats, %lld needed", me, (long long)partial_floats,
                    (long long)need);
    GradReduce a = grad_plan(rows, in_dim, out_dim);
    a.partial = partial; a.dW1 = dW1; a.dW2 = dW2; a.db1 = db1;
    return launch_permute<false>(g, channels, x_bin, s_bin, nullptr, permutation, x_out, s_out, nullptr, (cudaStream_t)stream, a);
}

int npa_safe_inv_sym_mat(int32_t dim, int64_t n, const float *m, float *m_inv, float tol, void *stream) {
    if (dim != 2 && dim != 3) return fail(NPA_ERR_INVALID_ARGUMENT, "safe_inverse only supports 2x2 or 3x3 matrices.");
    if (n < 0 || !m || !m_inv) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_safe_inv_sym_mat: bad arguments");
    if (n == 0) return NPA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (dim == 2) {
        if (((uintptr_t)m | (uintptr_t)m_inv) % 16)
            return fail(NPA_ERR_INVALID_ARGUMENT, "npa_safe_inv_sym_mat: 2x2 matrices must be 16-byte aligned");
        safe_inv2_kernel<<<blocks, 256, 0, st>>>(reinterpret_cast<const float4 *>(m), reinterpret_cast<float4 *>(m_inv), n, tol);
    } else {
        safe_inv3_kernel<<<blocks, 256, 0, st>>>(m, m_inv, n, tol);
    }
    return check_launch("safe_inv_kernel");
}

int npa_corrected_gradient(int32_t dim, int64_t n, int32_t channels, const float *raw, const float *moment, float tol, float *out,
                           void *stream) {
    if (dim != 2 && dim != 3) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_corrected_gradient: dim must be 2 or 3, got %d", dim);
    if (n < 0 || channels <= 0 || !raw || !moment || !out) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_corrected_gradient: bad arguments");
    if (n == 0) return NPA_OK;
    const long long total = (long long)n * channels;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if (dim == 2) launch_early(corrected_gradient_kernel<2>, blocks, 256, 0, (cudaStream_t)stream, raw, moment, out, total, channels, tol);
    else launch_early(corrected_gradient_kernel<3>, blocks, 256, 0, (cudaStream_t)stream, raw, moment, out, total, channels, tol);
    return check_launch("corrected_gradient_kernel");
}

}  // extern "C"
