// Density and neighbour lists of a recorded step: the order of the sums of the packed perception.
//
// A hidden unit of the MLP whose preactivation is within rounding of zero switches with the last bit of the
// perception vector, and with it a row of the weight gradient.  The forward of a step that will be differentiated
// therefore keeps one fixed association of its sums, whatever is done to make it faster: here the candidates in the
// order of the cell walk, two partial sums (even and odd positions of a row of cells) on a clamped grid; in
// packed_ordered.cuh the accepted pairs by their position in the list.  Everything else searches in density_search.cu.
//
// Linear hash: a warp takes a tile of up to 32 particles -- consecutive work-list rows of one x-row of cells, at most
// kTileSpan cells apart -- gives every particle a lane, loads 32 candidates at a time into shared memory and lets every lane test
// each of them.  Bound by instruction issue (about a dozen instructions per candidate and tile) and by the list entries,
// written a word at a time.  Measured, B200, us: 262,144 particles 3D, ~240 candidates 140; 32,768 particles 2D 20.
// Morton and 3D periodic grids: the walk per particle of scalar_ops.cu.
#include "neighbors.cuh"
#include "ops.cuh"

namespace npa {

constexpr int kTileSpan = 3;   // cells per tile
constexpr int kTicketRows = 8; // most work-list rows a warp draws per ticket

template <int D, bool PER>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
density_ordered_kernel(const __grid_constant__ ScalarFwdArgs a, const __grid_constant__ Geom g, int batch) {
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

template <int D, bool PER>
static int launch_ordered(const Geom &g, const ScalarFwdArgs &a, cudaStream_t st) {
    int ctas = 0;
    int rc = persistent_ctas(density_ordered_kernel<D, PER>, kWarpsPerCta * 32, 0, &ctas);
    if (rc != NPA_OK) return rc;
    // rows a warp draws per ticket: two tickets for each of 32 warps on 148 SMs, at most kTicketRows rows (consecutive rows
    // of one ticket can merge into a tile; a single row cannot).  The tiles decide which candidates are even, so the rule
    // depends on nothing but the size of the work list.
    int batch = g.max_blocks / (2 * 32 * 148);
    batch = batch < 1 ? 1 : (batch > kTicketRows ? kTicketRows : batch);
    const int needed = (g.max_blocks + batch * kWarpsPerCta - 1) / (batch * kWarpsPerCta);
    ScalarFwdArgs b = a;
    if ((rc = acquire_row_tickets(st, &b.tickets)) != NPA_OK) return rc;
    density_ordered_kernel<D, PER><<<needed < ctas ? needed : ctas, kWarpsPerCta * 32, 0, st>>>(b, g, batch);
    return check_launch("density_ordered_kernel");
}

int launch_density_ordered(const Geom &g, const ScalarFwdArgs &a, cudaStream_t st) {
    if (g.morton || (g.periodic && g.dim == 3)) return launch_density_walk(g, a, st);
    if (g.dim == 3) return launch_ordered<3, false>(g, a, st);
    return g.periodic ? launch_ordered<2, true>(g, a, st) : launch_ordered<2, false>(g, a, st);
}

}  // namespace npa
