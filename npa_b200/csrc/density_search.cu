// Density and neighbour count by the cell search, and the recording of the neighbour lists: the one
// search of a snapshot, whose lists every later sweep reads.
//
// Linear hash (density_tile_kernel): particles of an x-row of cells are consecutive, so a warp takes 16
// consecutive particles, two lanes each, and tests them against the candidates of the 3 (9) rows of cells
// around the ones they span.  The candidates are staged end to end in shared memory and read as
// broadcasts, two at a time in packed fp32x2; a lane shifts the sign of every r^2 - h^2 into a word, walks
// the set bits of each 32 and collects slot numbers (bytes) in shared memory; the lists leave in runs,
// four lanes to a list.  No work items, no tickets, no reductions but the one between a particle's lanes.
// Morton hash, and fewer than 16,384 particles (density_item_kernel): the neighbours of 32 consecutive particles are scattered over many
// short ranges; a warp takes the particles of one cell, lays the candidates of its 3^D cells end to end,
// one gather per item, and tests 32 candidates, a lane each, against four particles at once; a scan of the
// accepted bits places the entries.
// Both are bound by instruction issue: about 8 warp instructions per 32 tests in the first, 11 in the second, which
// also spends as much again on its lists and on setting up an item.
// Measured, B200, density + lists, us (before: a lane per particle with every list entry written as a word of its own,
// and a walk per particle on Morton and 3D periodic grids): 262,144 particles 3D, ~240 candidates 140 -> 93;
// 524,288 particles 3D periodic 542 -> 213 (265 while its candidates were staged range by range); 65,536 particles 3D Morton, thin cells 61 -> 45; 4,096 particles 2D
// periodic, 370 candidates 45 -> 17; 32,768 particles in 2D 20 -> 13.  Of the 93 us staging takes 25, the tests 30, the collecting of
// the entries 25 and their way out a dozen (kernels without one part).
#include "neighbors.cuh"
#include "ops.cuh"

namespace npa {

constexpr int kSearchWarps = 4;
constexpr int kSearchSlots = 320;  // candidates staged at a time per warp
constexpr int kSearchRun = 128;    // accepted neighbours of a particle collected before they go to its list
constexpr float kFarAway = 1.0e18f;

// v + k * L as an unevaluated sum hi + lo (error-free two-sum; L itself is split in g.L + g.Llo).  With the image
// shift on the candidate's side, (hi - x_i) + lo is as accurate as an unshifted difference.
__device__ inline void shifted(const Geom &g, int d, float v, int k, float &hi, float &lo) {
    const float b = (float)k * g.L[d];
    const float sum = __fadd_rn(v, b);
    const float bb = __fsub_rn(sum, v);
    const float err = __fadd_rn(__fsub_rn(v, __fsub_rn(sum, bb)), __fsub_rn(b, bb));
    hi = sum;
    lo = __fadd_rn((float)k * g.Llo[d], err);
}

// hash_to_cell with the divisions of the linear hash in floating point: (n + 1/2) / d is farther from an integer than
// the rounding error reaches while there are fewer than 2^21 cells.
template <int D>
__device__ inline void item_cell(const Geom &g, uint32_t hsh, int &cx, int &cy, int &cz) {
    if (g.morton || g.cells >= (1 << 21)) {
        hash_to_cell<D>(g, hsh, cx, cy, cz);
        return;
    }
    const int rows = (int)__fdividef((float)hsh + 0.5f, (float)g.g[0]);
    cx = (int)hsh - rows * g.g[0];
    cz = D == 3 ? (int)__fdividef((float)rows + 0.5f, (float)g.g[1]) : 0;
    cy = rows - cz * g.g[1];
}

// ---------------------------------------------------------------------------------------------------------
// Linear hash: two lanes per particle.
// ---------------------------------------------------------------------------------------------------------
constexpr int kTileWarps = 2;
constexpr int kTileSlots = 256;  // candidates staged at a time per warp; a slot number is a byte
constexpr int kShare = 2;        // lanes per particle, below
constexpr int kTileRun = 132;    // bytes per lane for the slots accepted since the last flush (33 words: spread over the banks)

// Signs of two differences r^2 - h^2 shifted into a word, the first candidate's bit ending up highest: the bit is set
// where r^2 < h^2.
__device__ __forceinline__ unsigned shift_sign(unsigned m, float d) { return __funnelshift_l(__float_as_uint(d), m, 1); }

template <int V> struct Mode {
    static constexpr int value = V;
};

template <bool MASS> struct TileStage {
    float x[kTileSlots], y[kTileSlots], z[kTileSlots];
    int j[kTileSlots];  // particle; COUNT: image shift code
    float m[MASS ? kTileSlots : 4];
    unsigned char run[32 * kTileRun];
};

// kShare lanes share a particle (each takes every kShare-th batch of 32 candidates): 32 / kShare particles per warp.  Fewer
// particles span fewer cells and meet fewer candidates that none of them accepts, but set up more often: 262,144
// particles in 3D took 105 / 98 / 126 us with 1 / 2 / 4 lanes, 524,288 periodic 340 / 321 / 403, 32,768 in 2D 15.1 / 13.6 / 16.2.
template <int D, bool PER, bool COUNT, bool MASS>
__global__ void __launch_bounds__(kTileWarps * 32, 12)
density_tile_kernel(const __grid_constant__ ScalarFwdArgs a, const __grid_constant__ Geom g) {
    after_previous_kernel();
    constexpr int PT = 32 / kShare;
    extern __shared__ __align__(16) unsigned char s_tile[];
    __shared__ int4 s_rng[kTileWarps][kMaxRanges];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = lane / PT;
    TileStage<MASS> &S = reinterpret_cast<TileStage<MASS> *>(s_tile)[warp];
    int4 *rng = s_rng[warp];
    const int total_particles = g.B * g.N, K = a.pair_stride;
    const unsigned first = (blockIdx.x * kTileWarps + warp) * PT;
    if (first >= (unsigned)total_particles) return;
    const int i = (int)min(first + lane % PT, (unsigned)total_particles - 1u);
    const bool ivalid = first + lane % PT < (unsigned)total_particles;
    const Pos<D> pi = load_pos<D>(a.x, i);
    const int sys = i / g.N;
    int cx, cy, cz;  // in cell order, so the particles of a row of cells stand together with cx ascending
    snapshot_cell_of<D>(g, a.bin_offsets + (size_t)sys * g.cells, i, pi.x, pi.y, pi.z, cx, cy, cz);
    const int key = (sys * g.g[2] + cz) * g.g[1] + cy;
    const bool stray = PER && outside_cells<D>(g, pi, cx, cx, cy, cy, cz, cz);
    unsigned left = __ballot_sync(kFull, ivalid) & ((1u << PT) - 1u);  // particles to do
    while (left) {
        // ---- the particles of one x-row of cells, and the candidates of the rows around the cells they span
        const int lead = __ffs(left) - 1;
        const int lead_key = __shfl_sync(kFull, key, lead);
        const bool mine = ivalid && key == lead_key;
        const unsigned seg = (__ballot_sync(kFull, mine) & left) | (1u << lead);
        left &= ~seg;
        const int last = 31 - __clz(seg);
        const int cx0 = __shfl_sync(kFull, cx, lead), cx1 = __shfl_sync(kFull, cx, last);
        const int row_y = __shfl_sync(kFull, cy, lead), row_z = __shfl_sync(kFull, cz, lead);
        __syncwarp();
        const int nr = build_ranges_span<D>(g, a.bin_offsets, __shfl_sync(kFull, sys, lead), cx0, cx1, row_y, row_z, rng);
        const int4 own = lane < nr ? rng[lane] : make_int4(0, 0, shift_code(0, 0, 0), 0);
        int incl = own.y - own.x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(kFull, incl, 31);
        const int ordinal = incl - (own.y - own.x);
        if (lane < nr) rng[lane] = make_int4(own.x - ordinal, ordinal, own.z, own.y - own.x);
        const bool wrapped = PER && __any_sync(kFull, own.z != shift_code(0, 0, 0));
        // an axis too short to know the image of a cell, or a position outside its cell: the half-box test decides pair by pair
        bool check = PER && (g.g[0] <= 3 || g.g[1] <= 2 || (D == 3 && g.g[2] <= 2) || cx1 - cx0 + 3 >= g.g[0]);
        if (PER) check = check || __any_sync(kFull, mine && stray);
        const int cap = wrapped && !COUNT ? kTileSlots / 2 : kTileSlots;  // the low parts take the other half
        const bool lists = !COUNT && a.pair_cache != nullptr;

        float rho = 0.f;
        int found = 0;  // of the particle, the same in its lanes
        unsigned long long sum2 = 0ull;
        for (int c0 = 0; c0 < total; c0 += cap) {
            const int count = min(cap, total - c0), padded = (count + 32 * kShare - 1) / (32 * kShare) * (32 * kShare);
            __syncwarp();
            bool outside = false;
            if (!PER) {
                // every lane stages its slots of the chunk: the range of a slot is the last one that starts at or before it;
                // all loads are in flight together (range by range the gather was a chain of round trips, a third of the time)
                constexpr int kPer = kTileSlots / 32;
                int from[kPer];
#pragma unroll
                for (int u = 0; u < kPer; ++u) from[u] = 0;
                for (int r = 0; r < nr; ++r) {
                    const int4 R = rng[r];  // particle of ordinal 0 as if the range began there, ordinal of the first candidate
#pragma unroll
                    for (int u = 0; u < kPer; ++u) {
                        from[u] = c0 + u * 32 + lane >= R.y ? R.x : from[u];
                    }
                }
                Pos<D> p[kPer];
                float mass[kPer];
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    const int k = u * 32 + lane, j = from[u] + c0 + k;
                    const bool real = k < count;
                    p[u] = Pos<D>{kFarAway, kFarAway, kFarAway};
                    mass[u] = 0.f;
                    from[u] = real ? j : 0;
                    if (real) p[u] = load_pos<D>(a.x, j);
                    if (MASS && real) mass[u] = __ldg(a.mass + j);
                }
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    const int k = u * 32 + lane;
                    if (k >= padded) break;
                    S.x[k] = p[u].x; S.y[k] = p[u].y;
                    if (D == 3) S.z[k] = p[u].z;
                    S.j[k] = COUNT ? shift_code(0, 0, 0) : from[u];
                    if (MASS) S.m[k] = mass[u];
                }
            } else {  // up to 27 ranges, with image shifts: the same, four slots a lane at a time
                const bool low = wrapped && !COUNT;
                for (int base = 0; base < padded; base += 4 * 32) {
                    int which[4];  // range of the slot
#pragma unroll
                    for (int u = 0; u < 4; ++u) which[u] = 0;
                    for (int r = 1; r < nr; ++r) {
                        const int at = rng[r].y - c0 - base - lane;
#pragma unroll
                        for (int u = 0; u < 4; ++u) which[u] += u * 32 >= at ? 1 : 0;
                    }
                    Pos<D> p[4];
                    int code[4], from[4];
                    float mass[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int k = base + u * 32 + lane;
                        const int4 R = rng[which[u]];
                        const bool real = k < count;
                        p[u] = Pos<D>{kFarAway, kFarAway, kFarAway};
                        from[u] = real ? R.x + c0 + k : 0;
                        code[u] = real ? R.z : shift_code(0, 0, 0);
                        if (real) p[u] = load_pos<D>(a.x, from[u]);
                        mass[u] = MASS && real ? __ldg(a.mass + from[u]) : 0.f;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int k = base + u * 32 + lane;
                        if (k >= padded) break;
                        if (low) {
                            float lx = 0.f, ly = 0.f, lz = 0.f, hx = p[u].x, hy = p[u].y, hz = p[u].z;
                            if (k < count) {
                                shifted(g, 0, p[u].x, (code[u] & 3) - 1, hx, lx);
                                shifted(g, 1, p[u].y, ((code[u] >> 2) & 3) - 1, hy, ly);
                                if (D == 3) shifted(g, 2, p[u].z, ((code[u] >> 4) & 3) - 1, hz, lz);
                            }
                            p[u] = Pos<D>{hx, hy, hz};
                            S.x[kTileSlots / 2 + k] = lx; S.y[kTileSlots / 2 + k] = ly;
                            if (D == 3) S.z[kTileSlots / 2 + k] = lz;
                        }
                        if (k < count && (!COUNT || !wrapped)) outside |= outside_cells<D>(g, p[u], cx0 - 1, cx1 + 1, row_y - 1, row_y + 1, row_z - 1, row_z + 1);
                        S.x[k] = p[u].x; S.y[k] = p[u].y;
                        if (D == 3) S.z[k] = p[u].z;
                        S.j[k] = COUNT ? code[u] : from[u];
                        if (MASS) S.m[k] = mass[u];
                    }
                }
            }
            if (PER) check = check || __any_sync(kFull, outside);
            __syncwarp();

            int held = 0;  // slots in this lane's run
            unsigned char *run = S.run + lane * kTileRun;
            auto flush = [&]() {
                int before = 0, sum = held;  // entries of the particle's other lanes ahead of this one's, and all of them
#pragma unroll
                for (int q = 1; q < kShare; ++q) {
                    const int v = __shfl_sync(kFull, held, (lane + q * PT) & 31);
                    sum += v;
                    if (((lane + q * PT) & 31) / PT < part) before += v;
                }
                const int at = found + before, take = min(held, K - 1 - at);  // entries that still fit
                __syncwarp();
                // four lanes write a list, two entries each at a time, eight lists at once (eight lanes and one entry: 262,144 particles in
                // 3D 100 us instead of 93, 524,288 periodic 231 instead of 213; two lanes 94 and 214, but 40 instead of 37 in 2D)
#pragma unroll 1
                for (int l0 = 0; l0 < 32; l0 += 8) {
                    const int l = l0 + (lane >> 2);
                    const int n = __shfl_sync(kFull, take, l);
                    int32_t *list = a.pair_cache + (long long)__shfl_sync(kFull, i, l) * K + 1 + __shfl_sync(kFull, at, l);
                    const unsigned char *from = S.run + l * kTileRun;
                    int e = lane & 3;
                    for (; e + 4 < n; e += 8) {
                        const int j0 = S.j[from[e]], j1 = S.j[from[e + 4]];
                        list[e] = j0;
                        list[e + 4] = j1;
                    }
                    if (e < n) list[e] = S.j[from[e]];
                }
                found += sum;
                held = 0;
                __syncwarp();
            };
            // the 32 candidates from slot s0, the first one's bit highest
            auto test = [&](auto mode, int s0) {
                constexpr int kMode = decltype(mode)::value;  // 0: plain, 1: with low parts, 2: pair by pair
                const unsigned long long nx = pack2(-pi.x, -pi.x), ny = pack2(-pi.y, -pi.y), nz = pack2(-pi.z, -pi.z);
                const unsigned long long nh = pack2(-g.h2, -g.h2);
                unsigned m = 0u;
                if (kMode == 2) {
#pragma unroll 4
                    for (int k = 0; k < 32; ++k) {
                        const int c = s0 + k;
                        float rx, ry, rz;
                        Origin<D, PER> org;
                        if (COUNT) {
                            org = make_origin<D, PER>(g, pi.x, pi.y, pi.z, S.j[c]);
                        } else {
                            org.x[0] = pi.x; org.x[1] = pi.y; org.x[2] = pi.z;
                            org.c[0] = wrapped ? S.x[kTileSlots / 2 + c] : 0.f;
                            org.c[1] = wrapped ? S.y[kTileSlots / 2 + c] : 0.f;
                            org.c[2] = wrapped && D == 3 ? S.z[kTileSlots / 2 + c] : 0.f;
                        }
                        const float q = displacement<D, PER, COUNT>(g, org, S.x[c], S.y[c], D == 3 ? S.z[c] : 0.f, rx, ry, rz);
                        const bool acc = q < g.h2 && c < count;
                        m = (m << 1) | (acc ? 1u : 0u);
                        if (!COUNT) {
                            const float t = acc ? g.h2 - q : 0.f;
                            rho = fmaf(MASS ? S.m[c] : 1.0f, t * t * t, rho);
                        }
                    }
                } else {
#pragma unroll 4
                    for (int k = 0; k < 32; k += 4) {
                        const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(S.x + s0 + k), Y = *reinterpret_cast<const ulonglong2 *>(S.y + s0 + k);
                        ulonglong2 Z = make_ulonglong2(0ull, 0ull), LX = Z, LY = Z, LZ = Z, M = Z;
                        if (D == 3) Z = *reinterpret_cast<const ulonglong2 *>(S.z + s0 + k);
                        if (kMode == 1) {
                            LX = *reinterpret_cast<const ulonglong2 *>(S.x + kTileSlots / 2 + s0 + k);
                            LY = *reinterpret_cast<const ulonglong2 *>(S.y + kTileSlots / 2 + s0 + k);
                            if (D == 3) LZ = *reinterpret_cast<const ulonglong2 *>(S.z + kTileSlots / 2 + s0 + k);
                        }
                        if (MASS) M = *reinterpret_cast<const ulonglong2 *>(S.m + s0 + k);
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            unsigned long long rx = add2(v ? X.y : X.x, nx), ry = add2(v ? Y.y : Y.x, ny), rz = 0ull;
                            if (D == 3) rz = add2(v ? Z.y : Z.x, nz);
                            if (kMode == 1) {
                                rx = add2(rx, v ? LX.y : LX.x);
                                ry = add2(ry, v ? LY.y : LY.x);
                                if (D == 3) rz = add2(rz, v ? LZ.y : LZ.x);
                            }
                            unsigned long long q;
                            if (COUNT) {  // no fused multiply-adds: borderline pairs as in the fp32 oracle
                                q = add2(mul2(rx, rx), mul2(ry, ry));
                                if (D == 3) q = add2(q, mul2(rz, rz));
                            } else {
                                q = fma2(ry, ry, mul2(rx, rx));
                                if (D == 3) q = fma2(rz, rz, q);
                            }
                            float d0, d1;
                            unpack2(add2(q, nh), d0, d1);  // r^2 - h^2, negative inside the cut-off
                            m = shift_sign(shift_sign(m, d0), d1);
                            if (!COUNT) {
                                const unsigned long long w = pack2(fmaxf(-d0, 0.f), fmaxf(-d1, 0.f));
                                const unsigned long long c3 = mul2(mul2(w, w), w);
                                sum2 = MASS ? fma2(v ? M.y : M.x, c3, sum2) : add2(sum2, c3);
                            }
                        }
                    }
                }
                return mine ? m : 0u;
            };
            // One copy of the rest for all ways of testing: with a copy for each, a sixth of the periodic kernel's stalls were
            // waits for instructions (524,288 particles 311 us, so 281, when that was tried).
            for (int s0 = part * 32; s0 < padded; s0 += 32 * kShare) {
                unsigned m;
                if (PER && (check || (COUNT && wrapped))) m = test(Mode<2>(), s0);
                else if (PER && wrapped) m = test(Mode<1>(), s0);
                else m = test(Mode<0>(), s0);
                if (COUNT) {
                    found += __popc(m);
                } else if (lists) {
                    // as many rounds as the fullest lane has neighbours here: no divergence
                    for (int left_over = __reduce_max_sync(kFull, __popc(m)); left_over > 0; --left_over) {
                        const int b = __clz(m);
                        if (m) run[held] = (unsigned char)(s0 + b);
                        held += m != 0u;
                        m &= ~(0x80000000u >> (b & 31));
                    }
                    // (the lanes of a warp go round equally often: padded is a multiple of 32 kShare)
                    if (s0 + 32 * kShare >= padded || __any_sync(kFull, held > kTileRun - 4 - 32)) flush();
                }
            }
        }
        float lo, hi;
        unpack2(sum2, lo, hi);
        rho += lo + hi;
#pragma unroll
        for (int o = PT; o < 32; o <<= 1) {
            rho += __shfl_xor_sync(kFull, rho, o);
            if (COUNT) found += __shfl_xor_sync(kFull, found, o);
        }
        if (mine && part == 0) {
            if (COUNT) {
                a.count[i] = (float)found;
            } else {
                if (lists) a.pair_cache[(long long)i * K] = found <= K - 1 ? found : -1;
                const float r = g.c_s * rho;
                a.rho_out[i] = r;
                if (a.pv) a.pv[i] = make_float4(pi.x, pi.y, pi.z, (MASS ? __ldg(a.mass + i) : 1.0f) / r);
            }
        }
    }
}

template <int D, bool PER, bool COUNT, bool MASS>
static int launch_tile(const Geom &g, const ScalarFwdArgs &a, cudaStream_t st) {
    const auto kernel = density_tile_kernel<D, PER, COUNT, MASS>;
    const size_t dyn = sizeof(TileStage<MASS>) * kTileWarps;
    int unused = 0;
    const int rc = persistent_ctas(kernel, kTileWarps * 32, dyn, &unused);  // raises the shared-memory limit once
    if (rc != NPA_OK) return rc;
    const long long per_cta = (long long)kTileWarps * (32 / kShare), particles = (long long)g.B * g.N;
    launch_early(kernel, (unsigned)((particles + per_cta - 1) / per_cta), kTileWarps * 32, dyn, st, a, g);
    return check_launch("density_tile_kernel");
}

// ---------------------------------------------------------------------------------------------------------
// Morton hash: a lane per candidate.
// ---------------------------------------------------------------------------------------------------------
template <int D, bool PER>
__global__ void __launch_bounds__(kSearchWarps * 32, 8)
density_item_kernel(const __grid_constant__ ScalarFwdArgs a, const __grid_constant__ Geom g, int split) {
    after_previous_kernel();
    extern __shared__ float4 s_mem[];  // per warp: candidates (x, y, z, index), then their masses when there are any
    __shared__ int4 s_rng[kSearchWarps][32];
    __shared__ int s_run[kSearchWarps][4][kSearchRun];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool masses = a.mass != nullptr;
    float4 *cand = s_mem + warp * (masses ? kSearchSlots + kSearchSlots / 4 : kSearchSlots);
    float *cmass = reinterpret_cast<float *>(cand + kSearchSlots);
    int4 *rng = s_rng[warp];
    const unsigned below = (1u << lane) - 1u;
    const int K = a.pair_stride;
    const unsigned long long hh = pack2(g.h2, g.h2), minus = pack2(-1.f, -1.f);

    const int vrows = g.max_blocks * split;
    for (int vrow = blockIdx.x * kSearchWarps + warp; vrow < vrows; vrow += gridDim.x * kSearchWarps) {
        const int row = split == 1 ? vrow : vrow / split, part = vrow - row * split;
        const WorkItem it = load_item(a.block_info, a.bin_offsets, row);
        if (it.count <= 0) break;  // rows after the last work item are zero
        const int share = split == 1 ? it.count : ((it.count + split - 1) / split + 3) & ~3;
        const int k0 = part * share, k1 = min(k0 + share, it.count);
        if (k0 >= k1) continue;

        // the non-empty candidate ranges: start, length, image shift, ordinal of the first candidate
        int cx, cy, cz, start, end, code;
        item_cell<D>(g, (uint32_t)(it.cell - it.sys * g.cells), cx, cy, cz);
        range_piece<D>(g, a.bin_offsets + (size_t)it.sys * g.cells, cx, cy, cz, lane, start, end, code);
        const int len = max(end - start, 0);
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(kFull, incl, 31);
        const unsigned some = __ballot_sync(kFull, len > 0);
        const int nr = __popc(some);
        __syncwarp();
        if (len > 0) rng[__popc(some & below)] = make_int4(start, len, code, incl - len);
        __syncwarp();
        const bool wrapped = PER && __any_sync(kFull, len > 0 && code != shift_code(0, 0, 0));
        // an axis too short to know the image of a cell, or a position outside its cell: the half-box test decides pair by pair
        bool general = PER && (wrapped || g.g[0] <= 3 || g.g[1] <= 2 || (D == 3 && g.g[2] <= 2));
        const int cap = wrapped ? kSearchSlots / 2 : kSearchSlots;  // the low parts take the other half

        for (int kb = k0; kb < k1; kb += 32) {
            const int nb = min(32, k1 - kb);
            // (a particle is one of its own candidates, and within their window on four cells an axis its images stay clear: a
            // test of its own is needed where it may be staged in a later chunk, or an axis has three)
            if (PER && !general && (total > cap || g.g[1] == 3 || (D == 3 && g.g[2] == 3)))
                general = __any_sync(kFull, lane < nb && outside_cells<D>(g, load_pos<D>(a.x, it.first + kb + min(lane, nb - 1)), cx, cx, cy, cy, cz, cz));
            float rho = 0.f;  // of particle kb + lane
            int found = 0;
            for (int c0 = 0; c0 < total; c0 += cap) {
                const int count = min(cap, total - c0), padded = (count + 31) & ~31;
                if (total > cap || kb == k0) {  // otherwise the candidates are there already
                    bool outside = false;
                    __syncwarp();
                    auto stage = [&](int group) {  // `group` lanes per range
                        for (int r = lane / group; r < nr; r += 32 / group) {
                            const int4 R = rng[r];
                            const int e = min(R.y, c0 + count - R.w);
                            for (int k = max(0, c0 - R.w) + lane % group; k < e; k += group) {
                                const int j = R.x + k, slot = R.w + k - c0;
                                Pos<D> p = load_pos<D>(a.x, j);
                                if (PER && !wrapped) outside |= outside_cells<D>(g, p, cx - 1, cx + 1, cy - 1, cy + 1, cz - 1, cz + 1);
                                if (PER && wrapped) {  // (these are tested pair by pair in any case)
                                    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f);
                                    float hx, hy, hz = 0.f;
                                    shifted(g, 0, p.x, (R.z & 3) - 1, hx, lo.x);
                                    shifted(g, 1, p.y, ((R.z >> 2) & 3) - 1, hy, lo.y);
                                    if (D == 3) shifted(g, 2, p.z, ((R.z >> 4) & 3) - 1, hz, lo.z);
                                    p = Pos<D>{hx, hy, hz};
                                    cand[kSearchSlots / 2 + slot] = lo;
                                }
                                cand[slot] = make_float4(p.x, p.y, p.z, __int_as_float(j));
                                if (masses) cmass[slot] = __ldg(a.mass + j);
                            }
                        }
                    };
                    if (total > 20 * nr) stage(32);  // lanes per range by the mean length of the ranges
                    else if (total > 8 * nr) stage(16);
                    else stage(8);
                    if (count + lane < padded) {
                        cand[count + lane] = make_float4(kFarAway, kFarAway, kFarAway, __int_as_float(0));
                        if (PER && wrapped) cand[kSearchSlots / 2 + count + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (masses) cmass[count + lane] = 0.f;
                    }
                    if (PER) general |= __any_sync(kFull, outside) != 0;
                    __syncwarp();
                }
                for (int p0 = 0; p0 < nb; p0 += 4) {
                    Pos<D> pi[4];
                    unsigned hits[4] = {0u, 0u, 0u, 0u};  // bit s: this lane's candidate of step s is a neighbour
#pragma unroll
                    for (int u = 0; u < 4; ++u) pi[u] = load_pos<D>(a.x, it.first + kb + min(p0 + u, nb - 1));
                    float sum[4];
                    if (PER && general) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) sum[u] = 0.f;
                        unsigned bit = 1u;
                        for (int c = lane; c < padded; c += 32, bit <<= 1) {
                            const float4 cc = cand[c];
                            float4 lo = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (PER && wrapped) lo = cand[kSearchSlots / 2 + c];
                            const float m = masses ? cmass[c] : 1.0f;
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                float rx, ry, rz, q;
                                Origin<D, PER> org;
                                org.x[0] = pi[u].x; org.x[1] = pi[u].y; org.x[2] = pi[u].z;
                                org.c[0] = lo.x; org.c[1] = lo.y; org.c[2] = lo.z;
                                q = displacement<D, PER, false>(g, org, cc.x, cc.y, cc.z, rx, ry, rz);
                                const bool acc = q < g.h2 && c < count;
                                hits[u] |= acc ? bit : 0u;
                                const float t = acc ? g.h2 - q : 0.f;
                                sum[u] = fmaf(m, t * t * t, sum[u]);
                            }
                        }
                    } else {
                        unsigned long long nx[2], ny[2], nz[2], acc2[2] = {0ull, 0ull};
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            nx[v] = pack2(-pi[2 * v].x, -pi[2 * v + 1].x);
                            ny[v] = pack2(-pi[2 * v].y, -pi[2 * v + 1].y);
                            nz[v] = pack2(-pi[2 * v].z, -pi[2 * v + 1].z);
                        }
                        unsigned bit = 1u;
                        for (int c = lane; c < padded; c += 32, bit <<= 1) {
                            const float4 cc = cand[c];
                            const unsigned long long xx = pack2(cc.x, cc.x), yy = pack2(cc.y, cc.y), zz = pack2(cc.z, cc.z);
                            const float m = masses ? cmass[c] : 1.0f;
#pragma unroll
                            for (int v = 0; v < 2; ++v) {
                                const unsigned long long rx = add2(xx, nx[v]), ry = add2(yy, ny[v]);
                                unsigned long long q = fma2(ry, ry, mul2(rx, rx));
                                if (D == 3) {
                                    const unsigned long long rz = add2(zz, nz[v]);
                                    q = fma2(rz, rz, q);
                                }
                                float t0, t1;
                                unpack2(fma2(q, minus, hh), t0, t1);  // h^2 - r^2, positive inside the cut-off
                                hits[2 * v] |= t0 > 0.f ? bit : 0u;
                                hits[2 * v + 1] |= t1 > 0.f ? bit : 0u;
                                const unsigned long long t = pack2(fmaxf(t0, 0.f), fmaxf(t1, 0.f));
                                const unsigned long long w = mul2(mul2(t, t), t);
                                acc2[v] = masses ? fma2(pack2(m, m), w, acc2[v]) : add2(acc2[v], w);
                            }
                        }
                        unpack2(acc2[0], sum[0], sum[1]);
                        unpack2(acc2[1], sum[2], sum[3]);
                    }
                    {
                        // the four sums over the warp: pairs of lanes exchange values first
                        const bool odd = lane & 1, two = lane & 2;
                        float v0 = (odd ? sum[1] : sum[0]) + __shfl_xor_sync(kFull, odd ? sum[0] : sum[1], 1);
                        float v1 = (odd ? sum[3] : sum[2]) + __shfl_xor_sync(kFull, odd ? sum[2] : sum[3], 1);
                        float v = (two ? v1 : v0) + __shfl_xor_sync(kFull, two ? v0 : v1, 2);
                        v += __shfl_xor_sync(kFull, v, 4);
                        v += __shfl_xor_sync(kFull, v, 8);
                        v += __shfl_xor_sync(kFull, v, 16);  // lane l holds the sum of particle l & 3
                        if ((lane & ~3) == p0) rho += v;
                    }
                    if (a.pair_cache) {
                        // counts of two particles per word: totals, and where this lane's entries start
                        unsigned own[2], at[2], all[2];
#pragma unroll
                        for (int v = 0; v < 2; ++v) {
                            own[v] = (unsigned)__popc(hits[2 * v]) | ((unsigned)__popc(hits[2 * v + 1]) << 16);
                            at[v] = own[v];
#pragma unroll
                            for (int o = 1; o < 32; o <<= 1) {
                                const unsigned w = __shfl_up_sync(kFull, at[v], o);
                                if (lane >= o) at[v] += w;
                            }
                            all[v] = __shfl_sync(kFull, at[v], 31);
                            at[v] -= own[v];
                        }
                        {
                            const int *index = reinterpret_cast<const int *>(cand + lane) + 3;
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                if (p0 + u >= nb) break;
                                const int n = (int)((all[u >> 1] >> (16 * (u & 1))) & 0xffffu);
                                int pos = (int)((at[u >> 1] >> (16 * (u & 1))) & 0xffffu);
                                const int before = __shfl_sync(kFull, found, p0 + u), m = min(n, K - 1 - before);
                                int32_t *list = a.pair_cache + (it.first + kb + p0 + u) * (long long)K + 1 + before;
                                unsigned h = hits[u];
                                if (n <= kSearchRun) {
                                    int *run = s_run[warp][u] + pos;
                                    while (h) {
                                        const int s = __ffs(h) - 1;
                                        h &= h - 1u;
                                        *run++ = index[s * 128];
                                    }
                                    __syncwarp();
                                    for (int e = lane; e < m; e += 32) list[e] = s_run[warp][u][e];
                                } else {  // more than the run holds
                                    for (; h; h &= h - 1u, ++pos)
                                        if (pos < m) list[pos] = index[(__ffs(h) - 1) * 128];
                                }
                            }
                            __syncwarp();
                        }
                        if ((lane & ~3) == p0) found += (int)((((lane & 2) ? all[1] : all[0]) >> (16 * (lane & 1))) & 0xffffu);
                    }
                }
            }
            if (lane < nb) {
                const long long i = it.first + kb + lane;
                if (a.pair_cache) a.pair_cache[i * K] = found <= K - 1 ? found : -1;
                const float r = g.c_s * rho;
                a.rho_out[i] = r;
                if (a.pv) {
                    const Pos<D> p = load_pos<D>(a.x, i);
                    a.pv[i] = make_float4(p.x, p.y, p.z, (a.mass ? __ldg(a.mass + i) : 1.0f) / r);
                }
            }
        }
    }
}

template <int D, bool PER>
static int launch_item(const Geom &g, const ScalarFwdArgs &a, cudaStream_t st) {
    const auto kernel = density_item_kernel<D, PER>;
    const size_t dyn = (size_t)kSearchWarps * kSearchSlots * (a.mass ? 20 : 16);
    int ctas = 0;
    const int rc = persistent_ctas(kernel, kSearchWarps * 32, dyn, &ctas);
    if (rc != NPA_OK) return rc;
    // warps sharing an item, four particles of it at least each: enough for two items per resident warp
    const long long items = (long long)g.B * (g.cells < g.N ? g.cells : g.N);
    long long split = 2ll * ctas * kSearchWarps / items;
    const int most = (g.mpb < g.N ? g.mpb : g.N) / 4;
    if (split > most) split = most;
    if (split > 16) split = 16;
    if (split < 1) split = 1;
    const long long needed = ((long long)g.max_blocks * split + kSearchWarps - 1) / kSearchWarps;
    launch_early(kernel, (unsigned)(needed < ctas ? needed : ctas), kSearchWarps * 32, dyn, st, a, g, (int)split);
    return check_launch("density_item_kernel");
}

template <int D, bool PER>
static int launch_search(const Geom &g, bool count, const ScalarFwdArgs &a, cudaStream_t st) {
    // few particles: the item kernel's warps are shorter (2,500 particles in 2D 5.3 us against 8.4, 4,096 with 128
    // neighbours 17.5 against 27; 15,003 about equal, 32,768 18 against 15)
    if (g.morton || (!count && (long long)g.B * g.N < 16384)) return launch_item<D, PER>(g, a, st);
    if (count) return launch_tile<D, PER, true, false>(g, a, st);
    return a.mass ? launch_tile<D, PER, false, true>(g, a, st) : launch_tile<D, PER, false, false>(g, a, st);
}

int launch_density_search(const Geom &g, bool count, const ScalarFwdArgs &a, cudaStream_t st) {
    if (g.dim == 2) return g.periodic ? launch_search<2, true>(g, count, a, st) : launch_search<2, false>(g, count, a, st);
    return g.periodic ? launch_search<3, true>(g, count, a, st) : launch_search<3, false>(g, count, a, st);
}

}  // namespace npa
