// Density and neighbour lists of the packed perception, recorded for a backward or not: the order of its sums.
//
// A hidden unit of the MLP whose preactivation is within rounding of zero switches with the last bit of the
// perception vector, and with it a row of the weight gradient.  The packed perception therefore keeps one fixed
// association of its sums, whatever is done to make it faster: here the candidates in the
// order of the cell walk, two partial sums (even and odd positions of a row of cells) on a clamped grid; in
// packed_ordered.cuh the accepted pairs by their position in the list.  Everything else searches in density_search.cu.
//
// Linear hash: a warp takes a tile of up to 32 particles -- consecutive work-list rows of one x-row of cells, at most
// kTileSpan cells apart -- gives every particle a lane, loads 32 candidates at a time into shared memory and lets every lane test
// each of them.  Bound by instruction issue (about a dozen instructions per candidate and tile) and by the list entries,
// written a word at a time.  Measured, B200, us: 262,144 particles 3D, ~240 candidates 140; 32,768 particles 2D 20.
// Few particles, Morton and 3D periodic grids: a lane per candidate, below.
#include "neighbors.cuh"
#include "ops.cuh"

namespace npa {

constexpr int kTileSpan = 3;   // cells per tile
constexpr int kTicketRows = 8; // most work-list rows a warp draws per ticket

template <int D, bool PER>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
density_ordered_kernel(const __grid_constant__ ScalarFwdArgs a, const __grid_constant__ Geom g, int batch) {
    after_previous_kernel();
    __shared__ int4 s_ranges[kWarpsPerCta][kMaxRanges];
    __shared__ float4 s_cand[kWarpsPerCta][2][32];  // x, y, z, mass of the staged candidates (two batches)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int4 *rng = s_ranges[warp];
    const int K = a.pair_stride;

    bool finished = false;
    while (!finished) {
        int row = 0;
        if (lane == 0) row = (int)atomicAdd(a.tickets, (unsigned)batch);
        row = __shfl_sync(kFull, row, 0) + lane;
        WorkItem mine = {0, 0, 0, 0};
        int mcx = 0, mcy = 0, mcz = 0;
        if (lane < batch && row < g.max_blocks) mine = load_item(a.block_info, a.bin_offsets, row);
        if (mine.count > 0) hash_to_cell<D>(g, (uint32_t)(mine.cell - mine.sys * g.cells), mcx, mcy, mcz);
        int next = 0;
        while (next < batch) {
            const int h = next;
            const int hcount = __shfl_sync(kFull, mine.count, h);
            if (hcount <= 0) {  // rows after the last work item are zero
                finished = true;
                break;
            }
            const int hfirst = __shfl_sync(kFull, mine.first, h);
            const int hsys = __shfl_sync(kFull, mine.sys, h);
            const int hcx = __shfl_sync(kFull, mcx, h), hcy = __shfl_sync(kFull, mcy, h), hcz = __shfl_sync(kFull, mcz, h);
            // rows h, h+1, ... join the tile while they lie in the same x-row, within kTileSpan cells, and the
            // tile holds at most 32 particles (rows of one x-row are contiguous in memory)
            const bool in_batch = lane >= h && lane < batch && mine.count > 0;
            const int upto = in_batch ? mine.first + mine.count - hfirst : 0;
            const bool wide = g.periodic && (mcx - hcx + 3 >= g.g[0]);
            const bool okrow = in_batch && mine.sys == hsys && mcy == hcy && mcz == hcz && mcx >= hcx &&
                               mcx - hcx < kTileSpan && upto <= 32 && upto > 0 && (lane == h || !wide);
            const unsigned okm = __ballot_sync(kFull, okrow || lane == h);
            const unsigned run = ~okm & ~((1u << h) - 1u);
            const int stop = run ? __ffs(run) - 1 : 32;
            const int last = stop - 1;
            const int lcx = __shfl_sync(kFull, mcx, last);
            const int tile_count = __shfl_sync(kFull, mine.first + mine.count, last) - hfirst;
            next = stop;
            __syncwarp();
            const int nr = build_ranges_span<D>(g, a.bin_offsets, hsys, hcx, lcx, hcy, hcz, rng);

            for (int p0 = 0; p0 < tile_count; p0 += 32) {  // a lone row of more than 32 particles: passes of 32
                const bool ivalid = p0 + lane < tile_count;
                const long long i = hfirst + p0 + (ivalid ? lane : 0);
                const Pos<D> pi = load_pos<D>(a.x, i);
                int32_t *list = a.pair_cache + i * K + 1;
                float rho = 0.f;
                unsigned long long rho2 = 0ull;  // clamped: sums over the even and the odd candidates of the batches
                int listed = 0;

                // candidates are staged 32 at a time; the next batch is fetched from global memory while the
                // current one is tested.  A batch is (range r, first candidate j0); this walks them in order.
                auto fetch = [&](int r, int j0) {
                    if (r < nr) {
                        const int j = j0 + lane;
                        if (j < rng[r].y) {
                            const Pos<D> pj = load_pos<D>(a.x, j);
                            return make_float4(pj.x, pj.y, pj.z, a.mass ? __ldg(a.mass + j) : 1.0f);
                        }
                    }
                    return make_float4(0.f, 0.f, 0.f, 0.f);
                };
                int r = 0, j0 = nr > 0 ? rng[0].x : 0, buf = 0;
                float4 c_next = fetch(r, j0);
                while (r < nr) {
                    const int4 rg = rng[r];
                    float4 *cand = s_cand[warp][buf];
                    if (!PER) {  // four arrays x[32] y[32] z[32] m[32]: a pair of candidates is one 8-byte broadcast
                        float *cs = reinterpret_cast<float *>(cand);
                        cs[lane] = c_next.x; cs[32 + lane] = c_next.y; cs[64 + lane] = c_next.z; cs[96 + lane] = c_next.w;
                    } else {
                        cand[lane] = c_next;
                    }
                    __syncwarp();
                    // the batch after this one
                    int rn = r, jn0 = j0 + 32;
                    if (jn0 >= rg.y) {
                        rn = r + 1;
                        jn0 = rn < nr ? rng[rn].x : 0;
                    }
                    c_next = fetch(rn, jn0);
                    const int jn = min(32, rg.y - j0);
                    if (!PER && ivalid) {
                        const unsigned long long *cs = reinterpret_cast<const unsigned long long *>(cand);
                        const unsigned long long nox = pack2(-pi.x, -pi.x), noy = pack2(-pi.y, -pi.y), noz = pack2(-pi.z, -pi.z);
#pragma unroll 2
                        for (int k = 0; k < jn; k += 2) {
                            // candidates k and k + 1 (a batch that ends on an odd count is followed by a zero-mass entry)
                            const unsigned long long rx = add2(cs[k >> 1], nox), ry = add2(cs[16 + (k >> 1)], noy);
                            unsigned long long q = fma2(ry, ry, mul2(rx, rx));
                            if (D == 3) {
                                const unsigned long long rz = add2(cs[32 + (k >> 1)], noz);
                                q = fma2(rz, rz, q);
                            }
                            float q0, q1;
                            unpack2(q, q0, q1);
                            const bool acc0 = q0 < g.h2, acc1 = q1 < g.h2 && k + 1 < jn;
                            if (acc0 && listed < K - 1) list[listed] = j0 + k;
                            listed += acc0 ? 1 : 0;
                            if (acc1 && listed < K - 1) list[listed] = j0 + k + 1;
                            listed += acc1 ? 1 : 0;
                            const unsigned long long t = pack2(fmaxf(g.h2 - q0, 0.f), fmaxf(g.h2 - q1, 0.f));
                            rho2 = fma2(cs[48 + (k >> 1)], mul2(mul2(t, t), t), rho2);
                        }
                    } else if (ivalid) {
                        const Origin<D, PER> org = make_origin<D, PER>(g, pi.x, pi.y, pi.z, rg.z);
#pragma unroll 4
                        for (int k = 0; k < jn; ++k) {
                            const float4 c = cand[k];  // same address in every lane: one broadcast
                            float rx, ry, rz;
                            const float q = displacement<D, PER, false>(g, org, c.x, c.y, c.z, rx, ry, rz);
                            const bool acc = q < g.h2;
                            if (acc && listed < K - 1) list[listed] = j0 + k;
                            listed += acc ? 1 : 0;
                            // the kernel vanishes at the cut-off: no branch on `acc` is needed
                            const float t = fmaxf(g.h2 - q, 0.f);
                            rho = fmaf(c.w, t * t * t, rho);
                        }
                    }
                    r = rn;
                    j0 = jn0;
                    buf ^= 1;
                }
                __syncwarp();
                if (!PER) {
                    float lo, hi;
                    unpack2(rho2, lo, hi);
                    rho = lo + hi;
                }
                if (ivalid) {
                    list[-1] = listed <= K - 1 ? listed : -1;
                    const float d = g.c_s * rho;
                    a.rho_out[i] = d;
                    if (a.pv) a.pv[i] = make_float4(pi.x, pi.y, pi.z, (a.mass ? __ldg(a.mass + i) : 1.0f) / d);
                }
            }
        }
    }
    release_rows(a.tickets);
}

// Rows a warp draws per ticket: two tickets for each of 32 warps on 148 SMs, at most kTicketRows rows (consecutive rows
// of one ticket can merge into a tile; a single row cannot).  The tiles decide which candidates are even, so the rule
// depends on nothing but the size of the work list.
static int ticket_rows(const Geom &g) {
    const int batch = g.max_blocks / (2 * 32 * 148);
    return batch < 1 ? 1 : (batch > kTicketRows ? kTicketRows : batch);
}

template <int D, bool PER>
static int launch_ordered(const Geom &g, const ScalarFwdArgs &a, cudaStream_t st) {
    int ctas = 0;
    int rc = persistent_ctas(density_ordered_kernel<D, PER>, kWarpsPerCta * 32, 0, &ctas);
    if (rc != NPA_OK) return rc;
    const int batch = ticket_rows(g);
    const int needed = (g.max_blocks + batch * kWarpsPerCta - 1) / (batch * kWarpsPerCta);
    ScalarFwdArgs b = a;
    if ((rc = acquire_row_tickets(st, &b.tickets)) != NPA_OK) return rc;
    launch_early(density_ordered_kernel<D, PER>, needed < ctas ? needed : ctas, kWarpsPerCta * 32, 0, st, b, g, batch);
    return check_launch("density_ordered_kernel");
}

// ---------------------------------------------------------------------------------------------------------
// The same sums with a lane per candidate: a warp takes up to eight particles of an item, tests 32 candidates at a time
// against four of them and appends the accepted ones (kernel value, index and class) to the particle's run in shared
// memory by their rank in the ballot, that is in candidate order.  Afterwards a lane per particle and class walks
// the run.  CLS classes by the position in the range: 1 on the 2D periodic grid, 2 on the clamped one, 4 (the lanes of the
// walk per particle) with Morton order and on the 3D periodic grid.  Bound by instruction issue (~56 % of the slots, at 10 warps
// per SM; 4,096 particles in 2D with 370 candidates took the tile 43 us, this 18).
// ---------------------------------------------------------------------------------------------------------
constexpr int kItemWarps = 4;
constexpr int kItemSlots = 320;  // candidates staged at a time per warp
constexpr int kItemRun = 96;     // accepted neighbours of a particle between two flushes

template <bool V> struct Flag {
    static constexpr bool value = V;
};

struct ItemMem {
    float4 cand[kItemSlots];            // x, y, z, (index << 2) | class
    unsigned char code[kItemSlots];     // image shift
    float value[8][kItemRun + 1];       // (one more: the rows start on different banks)
    unsigned index[8][kItemRun + 1];
    int4 rng[32];
};

template <int D, bool PER, int CLS>
__global__ void __launch_bounds__(kItemWarps * 32, 4)
density_ordered_item_kernel(const __grid_constant__ ScalarFwdArgs a, const __grid_constant__ Geom g, int split) {
    after_previous_kernel();
    extern __shared__ __align__(16) unsigned char s_item[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, K = a.pair_stride;
    ItemMem &S = reinterpret_cast<ItemMem *>(s_item)[warp];
    const unsigned below = (1u << lane) - 1u;
    const int pl = lane >> 2, cls = lane & 3;  // the particle and the class this lane sums

    const int vrows = g.max_blocks * split;
    for (int vrow = blockIdx.x * kItemWarps + warp; vrow < vrows; vrow += gridDim.x * kItemWarps) {
        const int row = split == 1 ? vrow : vrow / split, part = vrow - row * split;
        const WorkItem it = load_item(a.block_info, a.bin_offsets, row);
        if (it.count <= 0) break;  // rows after the last work item are zero
        const int share = split == 1 ? it.count : ((it.count + split - 1) / split + 3) & ~3;
        const int k0 = part * share, k1 = min(k0 + share, it.count);
        if (k0 >= k1) continue;

        // the non-empty candidate ranges: start, length, image shift, ordinal of the first candidate
        int cx, cy, cz, start, end, code;
        hash_to_cell<D>(g, (uint32_t)(it.cell - it.sys * g.cells), cx, cy, cz);
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
        if (len > 0) S.rng[__popc(some & below)] = make_int4(start, len, code, incl - len);
        __syncwarp();
        const bool wrapped = PER && __any_sync(kFull, len > 0 && code != shift_code(0, 0, 0));
        // an axis too short to know the image of a cell, or a position outside its cell: the half-box test decides pair by pair
        bool check = PER && (g.g[0] <= 4 || g.g[1] <= 4 || (D == 3 && g.g[2] <= 4));

        float centre[3];
#pragma unroll
        for (int d = 0; d < D; ++d) centre[d] = ((float)((d == 0 ? cx : d == 1 ? cy : cz) - g.half[d]) + 0.5f) * g.h;

        for (int kb = k0; kb < k1; kb += 8) {
            const int nb = min(8, k1 - kb);
            float rho = 0.f;       // of particle kb + pl, the pairs of class cls
            int found = 0, held = 0;  // of particle kb + lane: entries in its list, and in its run
            auto flush = [&]() {
                __syncwarp();
                for (int p = 0; p < nb; ++p) {
                    const int n = __shfl_sync(kFull, held, p), at = __shfl_sync(kFull, found, p);
                    int32_t *list = a.pair_cache + (it.first + kb + p) * (long long)K + 1 + at;
                    for (int e = lane; e < min(n, K - 1 - at); e += 32) list[e] = (int)(S.index[p][e] >> 2);
                }
                const int n = __shfl_sync(kFull, held, pl), most = __reduce_max_sync(kFull, held);
                if (cls < CLS) {
                    if (a.mass) {
#pragma unroll 4
                        for (int e = 0; e < most; ++e) {
                            const unsigned id = S.index[pl][e];
                            if (e < n && (CLS == 1 || (int)(id & 3u) == cls)) rho = fmaf(__ldg(a.mass + (id >> 2)), S.value[pl][e], rho);
                        }
                    } else {  // (adding zero changes no sum: they start at zero and the terms are not negative)
#pragma unroll 8
                        for (int e = 0; e < most; ++e) {
                            const float v = S.value[pl][e];
                            rho += e < n && (CLS == 1 || (int)(S.index[pl][e] & 3u) == cls) ? v : 0.f;
                        }
                    }
                }
                found += held;
                held = 0;
                __syncwarp();
            };
            for (int c0 = 0; c0 < total; c0 += kItemSlots) {
                const int count = min(kItemSlots, total - c0);
                if (total > kItemSlots || kb == k0) {  // otherwise the candidates are there already
                    __syncwarp();
                    const int group = total > 20 * nr ? 32 : (total > 8 * nr ? 16 : 8);  // lanes per range by the mean length
                    for (int r = lane / group; r < nr; r += 32 / group) {
                        const int4 R = S.rng[r];
                        const int e = min(R.y, c0 + count - R.w);
                        for (int k = max(0, c0 - R.w) + lane % group; k < e; k += group) {
                            const int slot = R.w + k - c0;
                            S.cand[slot].w = __uint_as_float(((unsigned)(R.x + k) << 2) | (unsigned)(k & (CLS - 1)));
                            if (PER) S.code[slot] = (unsigned char)R.z;
                        }
                    }
                    __syncwarp();
                    // the positions: the loads of five steps in flight together.  Periodic: seen from here a candidate's cell may lie
                    // beyond an edge of the box; three cells around the centre hold it, or its position is not that of its cell
                    bool outside = false;
                    auto positions = [&](auto shifted_cells) {
                        for (int c0 = lane; c0 < count; c0 += 5 * 32) {
                            Pos<D> p[5];
                            int code[5];
#pragma unroll
                            for (int u = 0; u < 5; ++u) {
                                const int c = c0 + 32 * u;
                                if (c < count) p[u] = load_pos<D>(a.x, __float_as_uint(S.cand[c].w) >> 2);
                                code[u] = PER && decltype(shifted_cells)::value && c < count ? S.code[c] : shift_code(0, 0, 0);
                            }
#pragma unroll
                            for (int u = 0; u < 5; ++u) {
                                const int c = c0 + 32 * u;
                                if (c >= count) break;
                                S.cand[c].x = p[u].x; S.cand[c].y = p[u].y; S.cand[c].z = p[u].z;
                                if (PER) {
                                    const float v[3] = {p[u].x, p[u].y, p[u].z};
#pragma unroll
                                    for (int d = 0; d < D; ++d) {
                                        float t = v[d] - centre[d];
                                        if (decltype(shifted_cells)::value) {
                                            const int k = (code[u] >> (2 * d)) & 3;
                                            t += k == 1 ? 0.f : (k ? g.L[d] : -g.L[d]);
                                        }
                                        outside |= !(fabsf(t) <= 1.5f * g.h + 1e-5f * g.L[d]);
                                    }
                                }
                            }
                        }
                    };
                    if (PER && wrapped) positions(Flag<true>());
                    else positions(Flag<false>());
                    if (PER) check |= __any_sync(kFull, outside) != 0;
                    __syncwarp();
                }
                for (int p0 = 0; p0 < nb; p0 += 4) {
                    Pos<D> pi[4];
                    int n[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        pi[u] = load_pos<D>(a.x, it.first + kb + min(p0 + u, nb - 1));
                        n[u] = __shfl_sync(kFull, held, p0 + u);
                    }
                    if (PER && total > kItemSlots && c0 == 0) {  // (a single chunk holds, and tests, the particles themselves as well)
                        const Pos<D> own = lane & 2 ? (lane & 1 ? pi[3] : pi[2]) : (lane & 1 ? pi[1] : pi[0]);
                        check |= __any_sync(kFull, outside_cells<D>(g, own, cx, cx, cy, cy, cz, cz)) != 0;
                    }
                    for (int c = 0; c < count; c += 32) {
                        const bool real = c + lane < count;
                        const float4 cc = S.cand[real ? c + lane : 0];
                        const int image = PER && wrapped ? S.code[real ? c + lane : 0] : shift_code(0, 0, 0);
                        bool full = false;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            Origin<D, PER> org;
                            if (PER && wrapped) {
                                org = make_origin<D, PER>(g, pi[u].x, pi[u].y, pi[u].z, image);
                            } else {
                                org.x[0] = pi[u].x; org.x[1] = pi[u].y; org.x[2] = pi[u].z;
                                org.c[0] = org.c[1] = org.c[2] = 0.f;
                            }
                            float rx = (cc.x - org.x[0]) + org.c[0], ry = (cc.y - org.x[1]) + org.c[1], rz = D == 3 ? (cc.z - org.x[2]) + org.c[2] : 0.f;
                            if (PER && check) displacement<D, PER, CLS == 4>(g, org, cc.x, cc.y, cc.z, rx, ry, rz);
                            const float q = CLS == 4 ? sq_norm<D>(rx, ry, rz) : sq_norm_fast<D>(rx, ry, rz);
                            const bool acc = real && q < g.h2;
                            const unsigned hits = __ballot_sync(kFull, acc);
                            if (acc) {
                                const int e = n[u] + __popc(hits & below);
                                const float t = fmaxf(g.h2 - q, 0.f);
                                S.value[p0 + u][e] = t * t * t;
                                S.index[p0 + u][e] = __float_as_uint(cc.w);
                            }
                            n[u] += __popc(hits);
                            full |= n[u] > kItemRun - 32;
                        }
                        if (full) {  // a run may not hold another 32: empty them all
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                if (lane == p0 + u && p0 + u < nb) held = n[u];
                                n[u] = 0;
                            }
                            flush();
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (lane == p0 + u && p0 + u < nb) held = n[u];
                }
            }
            flush();
            // the classes meet as the lanes of the walk (distance 2 first) and the even and odd candidates do
            if (CLS == 4) rho += __shfl_xor_sync(kFull, rho, 2);
            if (CLS >= 2) rho += __shfl_xor_sync(kFull, rho, 1);
            const int listed = __shfl_sync(kFull, found, pl);
            if (cls == 0 && pl < nb) {
                const long long i = it.first + kb + pl;
                a.pair_cache[i * K] = listed <= K - 1 ? listed : -1;
                const float d = g.c_s * rho;
                a.rho_out[i] = d;
                if (a.pv) {
                    const Pos<D> p = load_pos<D>(a.x, i);
                    a.pv[i] = make_float4(p.x, p.y, p.z, (a.mass ? __ldg(a.mass + i) : 1.0f) / d);
                }
            }
        }
    }
}

template <int D, bool PER, int CLS>
static int launch_item(const Geom &g, const ScalarFwdArgs &a, cudaStream_t st) {
    const auto kernel = density_ordered_item_kernel<D, PER, CLS>;
    const size_t dyn = sizeof(ItemMem) * kItemWarps;
    int ctas = 0;
    const int rc = persistent_ctas(kernel, kItemWarps * 32, dyn, &ctas);
    if (rc != NPA_OK) return rc;
    // warps sharing an item, four particles of it at least each: enough for two items per resident warp
    const long long items = (long long)g.B * (g.cells < g.N ? g.cells : g.N);
    long long split = 2ll * ctas * kItemWarps / items;
    const int most = (g.mpb < g.N ? g.mpb : g.N) / 4;
    if (split > most) split = most;
    if (split > 16) split = 16;
    if (split < 1) split = 1;
    const long long needed = ((long long)g.max_blocks * split + kItemWarps - 1) / kItemWarps;
    launch_early(kernel, (unsigned)(needed < ctas ? needed : ctas), kItemWarps * 32, dyn, st, a, g, (int)split);
    return check_launch("density_ordered_item_kernel");
}

int launch_density_ordered(const Geom &g, const ScalarFwdArgs &a, cudaStream_t st) {
    if ((long long)g.B * g.N >= (1ll << 30)) return launch_density_search(g, false, a, st);  // a staged index has 30 bits here
    if (g.morton || (g.periodic && g.dim == 3)) {
        if (g.dim == 2) return g.periodic ? launch_item<2, true, 4>(g, a, st) : launch_item<2, false, 4>(g, a, st);
        return g.periodic ? launch_item<3, true, 4>(g, a, st) : launch_item<3, false, 4>(g, a, st);
    }
    // A tile takes as long as the candidates of a lane, whatever the number of particles; the item kernel's time grows with the
    // particles, and with the candidates of crowded cells, which make long items.  Item / tile (density and packed sweep
    // together, us): 2D clamped, 16 particles a cell: 2,048 15.6 / 17.3, 4,096 17.6 / 17.8, 8,192 28 / 23; 4 a cell: 1,024 10.0 / 10.6, 4,096 13.4 / 11.7;
    // 2D periodic (whose tiles test pair by pair), 16 a cell: 1,024 11 / 19, 4,096 18 / 28, 8,192 31 / 33, 16,384 44 / 43; 3D clamped,
    // 2 a cell: 4,096 15 / 16, 16,384 30 / 35, 32,768 51 / 61; 8 a cell: 16,384 44 / 45, 24,000 60 / 57; 16 a cell: 4,096 28 / 35,
    // 8,192 43 / 38.  Over 289 sizes up to 32,768 particles and 32 a cell these lines are at worst 12 % (3 us) behind the
    // better kernel and 0.3 % on average.  (Same sums: a row drawn alone is a tile of its own.)
    const long long particles = (long long)g.B * g.N, cells = g.cells;
    bool few;
    if (g.dim == 3) few = particles <= 6000 || (particles <= 20000 && g.N < 12 * cells) || (particles <= 33000 && g.N < 6 * cells);
    else if (g.periodic) few = particles <= 12000;
    else few = particles <= 4608 && 320ll * g.N >= particles * cells;
    if (few && ticket_rows(g) == 1) {
        if (g.dim == 3) return launch_item<3, false, 2>(g, a, st);
        return g.periodic ? launch_item<2, true, 1>(g, a, st) : launch_item<2, false, 2>(g, a, st);
    }
    if (g.dim == 3) return launch_ordered<3, false>(g, a, st);
    return g.periodic ? launch_ordered<2, true>(g, a, st) : launch_ordered<2, false>(g, a, st);
}

}  // namespace npa
