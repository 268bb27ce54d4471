// Blur and feature gradient, forward and backward, over recorded neighbour lists.
//
// The kernels of feature_kernels.cuh give a particle the whole warp: its pairs are dealt to 32 / LPP
// sub-groups and the sub-groups' partial sums are combined by shuffles once per particle.  At ~41 pairs
// per particle that combination, the half-empty last round of pair scalars and the walk over work-list
// rows are two thirds of the instructions (25 warp instructions per pair measured where the arithmetic
// needs 4).  With a list nothing ties a particle to a work item, so here a sub-group of LPP lanes owns a
// whole particle: lanes cover the features (4 each), every lane ends with the complete sum of its
// features and nothing is combined.  32 / LPP particles advance together through chunks of CH list
// entries:
//   stage B  every lane turns one (LPP = 4: two) list entries of its particle into pair scalars and leaves
//            them in the warp's shared memory; list entries are loaded two chunks ahead, particles one;
//   stage C  the lanes of a sub-group walk the chunk's entries: neighbour rows are fetched a few at a time
//            (128-bit loads, one line per sub-group) and multiplied in with fma.rn.f32x2.
// The price is imbalance: a warp runs as long as the longest of its lists (neighbouring particles, ~16 %
// over the mean for four lists of ~41).  Work items, tickets and cell ranges are not needed; blocks are
// plain blocks over consecutive particles, which lie in consecutive cells.
// A particle whose list overflowed (count -1) is searched by its sub-group's lanes over the cells around
// its position, LPP candidates a round, out of line so that the walk over lists keeps its registers.
//
// What bounds them: the L1 data path.  A 128-byte row of a neighbour is one wavefront, but so are every four
// bytes per lane of shared memory, broadcast or not: with the scalars stored twice for the packed arithmetic
// (32 bytes per pair) the forward took 231 us instead of 194.  Then latency: 16-24 warps per SM are resident, a third
// of the row sectors come from L2 (prefetching rows into L1 a chunk ahead was slower, 330 -> 340 us; one register
// set per row refilled early cost spills, 194 -> 234 us; five CTAs of the full backward instead of four 664 -> 758 us).
// Measured, B200, 262,144 particles in 3D, C = 32, ~41 neighbours, us, kernel with the whole warp per particle
// -> this one: blur + gradient 328 -> 164 (with the density gradient), features-only backward 499 -> 383, full
// backward 902 -> 560 (575 before rows were filled, 644 before that with one sum per term and 14 warps per SM; 524,288 periodic, C = 16: 700 -> 632 -> 596, with two list entries per
// lane and chunk and the registers of these 790).  In 2D the one sum gains little or loses
// little (blur and gradient together, 8 x 16,384, C = 32: 446 -> 441; 4 x 65,536, C = 64 723 -> 711; 8 x 4,096, C = 16 56.3 -> 56.4, C = 13 58.4
// -> 59.2; one operator alone, C = 16: gradient 43.5 -> 44.6, blur 30.7 -> 31.2, where the preparation of a particle shows).
#pragma once
#include "neighbors.cuh"
#include "ops.cuh"

namespace npa {

constexpr int kListWarps = 8;      // warps per CTA

// How a kernel addresses rows of C floats: float by float; four at a time (C a multiple of four, 16-byte aligned); or the same with
// C = 4 LPP known to the compiler: the rows fill the lanes, no lane lies beyond the last feature, there is one slice, and the rows of a
// neighbour lie at constant distances from one address.  Same sums.  Measured, B200, us, four at a time -> filled: 262,144 particles
// in 3D, C = 32, forward 176 -> 164, full backward 574 -> 560, features only 402 -> 383, packed sweep (packed_ordered.cuh) 418 -> 371;
// 2 x 262,144 periodic, C = 16, forward 236 -> 223, full backward 633 -> 596; 8 x 16,384 clustered in 2D, C = 32, 112 -> 107 and
// 339 -> 321; 8 x 4,096 in 2D, C = 16, packed sweep 35 -> 33, full backward 44.5 -> 43.5.
enum ListRows : int { kRowsAny = 0, kRowsVec = 1, kRowsFilled = 2 };
// Same, backward; with position gradients sixteen warps per SM either way (128 registers), in 3D as eight CTAs of two.
template <int D, bool FULL>
constexpr int kListBackwardWarps = FULL ? (D == 3 ? 2 : 4) : kListWarps;

// (x, y, z, m_j / rho_j) of particle j: one 16-byte gather when the density sweep left it packed.
template <int D>
__device__ inline float4 fetch_particle(const float *__restrict__ x, const float4 *__restrict__ pv, const float *__restrict__ rho,
                                        const float *__restrict__ mass, int j) {
    if (pv) return __ldg(pv + j);
    const Pos<D> p = load_pos<D>(x, j);
    const float m = mass ? __ldg(mass + j) : 1.0f;
    return make_float4(p.x, p.y, p.z, m / __ldg(rho + j));
}

// Four features f0..f0+3 of a row; lanes beyond the last feature read valid neighbours of it (unused).
template <int ROWS>
__device__ inline void load_row4(const float *__restrict__ row, int f0, int C, float (&v)[4]) {
    if (ROWS != kRowsAny) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(row + (ROWS == kRowsFilled ? f0 : min(f0, C - 4))));
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = __ldg(row + min(f0 + q, C - 1));
    }
}

template <int ROWS>
__device__ inline void store_row4(float *__restrict__ row, int f0, int C, const float (&v)[4]) {
    if (ROWS != kRowsAny) {
        if (ROWS == kRowsFilled || f0 < C) *reinterpret_cast<float4 *>(row + f0) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (f0 + q < C) row[f0 + q] = v[q];
    }
}

// Search of the cells around one particle (around the cell it was binned into) by the LPP lanes of its sub-group: candidate
// ranges in the order of the cell walk, LPP candidates per round.
template <int D, bool PER, int LPP>
struct SubgroupSearch {
    int cx, cy, cz, piece, j, end;
    const int32_t *off;
    Origin<D, PER> org;

    __device__ inline void begin(const Geom &g, const int32_t *bin_offsets, long long i, const Pos<D> &pi) {
        off = bin_offsets + (i / g.N) * (long long)g.cells;
        snapshot_cell_of<D>(g, off, (int)i, pi.x, pi.y, pi.z, cx, cy, cz);
        piece = -1;
        j = end = 0;
    }
    // Moves on to the next non-empty range when the current one is used up; false at the end.
    __device__ inline bool more(const Geom &g, const Pos<D> &pi) {
        while (j >= end) {
            if (++piece >= range_pieces<D>(g)) return false;
            int code;
            range_piece<D>(g, off, cx, cy, cz, piece, j, end, code);
            if (j < end) org = make_origin<D, PER>(g, pi.x, pi.y, pi.z, code);
        }
        return true;
    }
};

// Slot of this lane's entry when the accepted entries of its sub-group come first, in lane order, and the
// others fill the slots behind them; m = number of accepted entries of the sub-group.
template <int LPP>
__device__ inline int compact_slot(bool acc, int sg, int sl, int &m) {
    const unsigned all = LPP == 32 ? 0xffffffffu : ((1u << (LPP & 31)) - 1u);
    const unsigned bits = (__ballot_sync(kFull, acc) >> (sg * LPP)) & all;
    const unsigned below = (1u << sl) - 1u;
    m = __popc(bits);
    return acc ? __popc(bits & below) : m + __popc(~bits & below);
}

// Shared memory of one warp: the entries of two chunks per sub-group (one entry of padding keeps the sub-groups'
// broadcasts on different banks).
template <int LPP, bool ONE = false>  // ONE: an entry per lane in any case (registers)
struct ListShape {
    static constexpr int EPL = LPP == 4 && !ONE ? 2 : 1;  // list entries per lane and chunk
    static constexpr int CH = LPP * EPL, PP = 32 / LPP;
    static constexpr int kSlots = PP * (CH + 1), kIndexQuads = PP * (CH / 4 + 1);
};

// Starts the head of a particle's list (256 bytes) on its way into L1 while its count is still awaited.
template <int LPP>
__device__ inline int list_count(const int32_t *list, int stride, bool valid, int sl) {
    for (int q = sl; q < 8; q += LPP)
        if (q * 8 < stride) asm volatile("prefetch.global.L1 [%0];" ::"l"(list + q * 8));
    return valid ? __ldg(list) : 0;
}

// The particles first .. first + PP - 1 of a warp: those with a list (SEARCH false) or those whose list overflowed.
template <int D, bool PER, int LPP, int ROWS, int MASK, bool SEARCH>
__device__ __forceinline__ void list_forward(const FeatureFwdArgs &a, const Geom &g, float4 (*s_k)[ListShape<LPP>::kSlots],
                                             int4 (*s_j)[ListShape<LPP>::kIndexQuads], float *stage) {
    constexpr int EPL = ListShape<LPP>::EPL, CH = ListShape<LPP>::CH, PP = ListShape<LPP>::PP;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sg = lane / LPP, sl = lane % LPP;
    constexpr bool kFilled = ROWS == kRowsFilled, kVec = ROWS != kRowsAny;
    const int total = g.B * g.N, C = kFilled ? LPP * 4 : a.C;
    const int first = (blockIdx.x * kListWarps + warp) * PP;  // (less than total: the kernel has checked)
    bool ivalid = (unsigned)(first + sg) < (unsigned)total;
    const int i = ivalid ? first + sg : total - 1;
    const int32_t *list = a.pair_cache + (long long)i * a.pair_stride;
    const int count = list_count<LPP>(list, a.pair_stride, ivalid, sl);
    const Pos<D> pi = load_pos<D>(a.x, i);
    ++list;
    const int n = SEARCH ? 0 : max(count, 0);
    const int nmax = SEARCH ? 0 : __reduce_max_sync(kFull, n);
    ivalid = ivalid && (count < 0) == SEARCH;
    const unsigned pitch = (unsigned)C * 4u;
    constexpr bool kGrad = (MASK & F_GRAD) != 0, kBlur = (MASK & F_BLUR) != 0;
    constexpr bool kMoment = (MASK & F_MOMENT) != 0;
    constexpr bool kDg = (MASK & F_DGRAD) != 0;

    for (int fbase = 0; fbase < C; fbase += LPP * 4) {
        __syncwarp();  // the slice before has drained its buffers
        const int f0 = fbase + sl * 4;
        float si[4];
        load_row4<ROWS>(a.s + (long long)i * C, f0, C, si);
        const unsigned long long nsi01 = pack2(-si[0], -si[1]), nsi23 = pack2(-si[2], -si[3]);
        // packed sums of the features (0, 1) and (2, 3): blur, then the gradient axis by axis
        unsigned long long acc[2 + 2 * D];
#pragma unroll
        for (int q = 0; q < 2 + 2 * D; ++q) acc[q] = 0ull;
        float mom[D * (D + 1) / 2], dgs[EPL][3];  // lane-partial over the pairs
#pragma unroll
        for (int q = 0; q < D * (D + 1) / 2; ++q) mom[q] = 0.f;
#pragma unroll
        for (int k = 0; k < EPL; ++k) dgs[k][0] = dgs[k][1] = dgs[k][2] = 0.f;

        // pair scalars of one entry (zero volume: no pair) into slot `slot` of buffer `buf`
        auto put = [&](int buf, int slot, int k, float rx, float ry, float rz, float vj, float mj, int j) {
            const float q = sq_norm_fast<D>(rx, ry, rz);
            float w = 0.f, kv = 0.f;
            if (kBlur) {
                const float t = fmaxf(g.h2 - q, 0.f);
                w = vj * (t * t * t);
            }
            if ((kGrad || kMoment || kDg) && q > 0.f) {
                const Spiky sp = spiky_distance(q);
                const float phi = spiky_phi(sp, g.h);
                kv = vj * phi;
                if (kDg) {
                    const float md = mj * phi;
                    dgs[k][0] = fmaf(md, rx, dgs[k][0]);
                    dgs[k][1] = fmaf(md, ry, dgs[k][1]);
                    if (D == 3) dgs[k][2] = fmaf(md, rz, dgs[k][2]);
                }
            }
            if (kMoment) {
                mom[0] = fmaf(kv * rx, rx, mom[0]);
                mom[1] = fmaf(kv * rx, ry, mom[1]);
                if (D == 2) {
                    mom[2] = fmaf(kv * ry, ry, mom[2]);
                } else {
                    mom[2] = fmaf(kv * rx, rz, mom[2]);
                    mom[3] = fmaf(kv * ry, ry, mom[3]);
                    mom[D == 3 ? 4 : 0] = fmaf(kv * ry, rz, mom[D == 3 ? 4 : 0]);
                    mom[D == 3 ? 5 : 0] = fmaf(kv * rz, rz, mom[D == 3 ? 5 : 0]);
                }
            }
            const float kx = kv * rx, ky = kv * ry, kz = kv * rz;
            s_k[buf][sg * (CH + 1) + slot] = make_float4(kx, ky, kz, w);
            reinterpret_cast<int *>(&s_j[buf][sg * (CH / 4 + 1)])[slot] = j;
        };
        // the first m entries of a buffer (m uniform; slots up to the next multiple of four are filled)
        auto drain = [&](int buf, int m) {
            const float4 *ks = &s_k[buf][sg * (CH + 1)];
            const int4 *jj = &s_j[buf][sg * (CH / 4 + 1)];
#pragma unroll
            for (int e0 = 0; e0 < CH; e0 += 4) {
                if (e0 >= m) break;
                const int4 j4 = jj[e0 / 4];
                const int js[4] = {j4.x, j4.y, j4.z, j4.w};
                float r[4][4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    load_row4<ROWS>(reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.s) + (unsigned long long)(unsigned)js[u] * pitch),
                                   f0, C, r[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const unsigned long long s01 = pack2(r[u][0], r[u][1]), s23 = pack2(r[u][2], r[u][3]);
                    const float4 k4 = ks[e0 + u];
                    if (kBlur) {
                        const unsigned long long ww = pack2(k4.w, k4.w);
                        acc[0] = fma2(ww, s01, acc[0]);
                        acc[1] = fma2(ww, s23, acc[1]);
                    }
                    if (kGrad) {
                        const unsigned long long d01 = add2(s01, nsi01), d23 = add2(s23, nsi23);  // s_j - s_i
                        const float kd[3] = {k4.x, k4.y, k4.z};
#pragma unroll
                        for (int d = 0; d < D; ++d) {
                            const unsigned long long kk = pack2(kd[d], kd[d]);
                            acc[2 + 2 * d] = fma2(d01, kk, acc[2 + 2 * d]);
                            acc[3 + 2 * d] = fma2(d23, kk, acc[3 + 2 * d]);
                        }
                    }
                }
            }
        };

        int buf = 0;
        if constexpr (!SEARCH) {
            // indices are loaded two chunks ahead and particles one, so that neither waits for the other's latency
            int jn[EPL], ja[EPL];
            float4 pj[EPL];
            float mj[EPL];
            auto indices = [&](int c) {
#pragma unroll
                for (int k = 0; k < EPL; ++k) {
                    const int e = c + k * LPP + sl;
                    ja[k] = e < n ? __ldg(list + e) : -1;
                }
            };
            auto particles = [&]() {
#pragma unroll
                for (int k = 0; k < EPL; ++k) {
                    const int j = jn[k] >= 0 ? jn[k] : i;
                    pj[k] = fetch_particle<D>(a.x, a.pv, a.rho, a.mass, j);
                    mj[k] = kDg ? (a.mass ? __ldg(a.mass + j) : 1.0f) : 0.f;
                    if (jn[k] < 0) { pj[k].w = 0.f; mj[k] = 0.f; }
                }
            };
            auto advance = [&](int c) {
#pragma unroll
                for (int k = 0; k < EPL; ++k) jn[k] = ja[k];
                indices(c);
                particles();
            };
            indices(0);
            advance(CH);
            for (int c = 0; c < nmax; c += CH, buf ^= 1) {
#pragma unroll
                for (int k = 0; k < EPL; ++k) {
                    float rx, ry, rz;
                    listed_displacement<D, PER>(g, pi, Pos<D>{pj[k].x, pj[k].y, pj[k].z}, rx, ry, rz);
                    put(buf, k * LPP + sl, k, rx, ry, rz, pj[k].w, mj[k], jn[k] >= 0 ? jn[k] : i);
                }
                __syncwarp();
                advance(c + 2 * CH);
                drain(buf, nmax - c);
            }
        }
        if constexpr (SEARCH) {
            bool over = ivalid;
            SubgroupSearch<D, PER, LPP> search;
            if (over) search.begin(g, a.bin_offsets, i, pi);
            while (true) {
                over = over && search.more(g, pi);
                if (!__any_sync(kFull, over)) break;
                float rx = 0.f, ry = 0.f, rz = 0.f;
                bool hit = false;
                const int j = over ? search.j + sl : i;
                if (over) {
                    if (j < search.end) {
                        const Pos<D> p = load_pos<D>(a.x, j);
                        hit = displacement<D, PER, false>(g, search.org, p.x, p.y, p.z, rx, ry, rz) < g.h2;
                    }
                    search.j += LPP;
                }
                int m;
                const int slot = compact_slot<LPP>(hit, sg, sl, m);
                const int most = __reduce_max_sync(kFull, m);
                if (most == 0) continue;
                const float m_j = hit && a.mass ? __ldg(a.mass + j) : 1.0f;
                put(buf, slot, 0, rx, ry, rz, hit ? m_j / __ldg(a.rho + j) : 0.f, hit ? m_j : 0.f, hit ? j : i);
                __syncwarp();
                drain(buf, most);
                buf ^= 1;
            }
        }

        float blur[4], gr[4][D];
        unpack2(acc[0], blur[0], blur[1]);
        unpack2(acc[1], blur[2], blur[3]);
#pragma unroll
        for (int d = 0; d < D; ++d) {
            unpack2(acc[2 + 2 * d], gr[0][d], gr[1][d]);
            unpack2(acc[3 + 2 * d], gr[2][d], gr[3][d]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            blur[q] *= g.c_s;
#pragma unroll
            for (int d = 0; d < D; ++d) gr[q][d] *= g.c_g;
        }
        float dg[3] = {0.f, 0.f, 0.f};
        if (kDg && fbase == 0) {
            // partial sums over the entries with equal (entry mod 8) meet in the same order for LPP = 4 and 8
#pragma unroll
            for (int d = 0; d < D; ++d) dg[d] = g.c_g * subgroup_sum<LPP>(EPL == 2 ? dgs[0][d] + dgs[EPL - 1][d] : dgs[0][d]);
        }
        if (kMoment) {
#pragma unroll
            for (int q = 0; q < D * (D + 1) / 2; ++q) mom[q] = g.c_g * subgroup_sum<LPP>(mom[q]);
        }
        if (kBlur && a.blur && ivalid) store_row4<ROWS>(a.blur + (long long)i * C, f0, C, blur);
        float L[D * D];
        if (MASK & (F_PACK | F_CORRECTED)) {
            safe_inverse_sym<D>(mom, a.inv_tol, L);
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // gradient . inv(M)
                float v[D];
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    float s = 0.f;
#pragma unroll
                    for (int k = 0; k < D; ++k) s = fmaf(gr[q][k], L[k * D + d], s);
                    v[d] = s;
                }
#pragma unroll
                for (int d = 0; d < D; ++d) gr[q][d] = v[d];
            }
        }
        float *gout = (MASK & F_PACK) ? a.vgrad : a.grad;
        if (kGrad && gout && ivalid) {
            float *o = gout + ((long long)i * C + f0) * D;
            if (kVec) {
                if (kFilled || f0 < C) {
                    const float *v = &gr[0][0];
#pragma unroll
                    for (int k = 0; k < D; ++k) reinterpret_cast<float4 *>(o)[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (f0 + q < C) {
#pragma unroll
                        for (int d = 0; d < D; ++d) o[q * D + d] = gr[q][d];
                    }
            }
        }
        if (kDg && fbase == 0 && a.rho_grad_out && ivalid && sl == 0) {
#pragma unroll
            for (int d = 0; d < D; ++d) a.rho_grad_out[(long long)i * D + d] = dg[d];
        }
        if (kMoment && fbase == 0 && a.moment && ivalid && sl == 0) {
            float *o = a.moment + (long long)i * (D * D);
            int k = 0;
#pragma unroll
            for (int p = 0; p < D; ++p)
#pragma unroll
                for (int q = p; q < D; ++q, ++k) {
                    o[p * D + q] = mom[k];
                    o[q * D + p] = mom[k];
                }
        }
        if (MASK & F_PACK) {
            // the rows of z of the warp's particles are contiguous: assembled in shared memory, written as one run
            const int Z = a.zstride;
            float *zs = stage + sg * Z;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int f = f0 + q;
                float v[D];
#pragma unroll
                for (int d = 0; d < D; ++d) v[d] = a.coef * gr[q][d];
                if (a.log_norm_grad) log_normalize<D>(v);
                if (f < C) {
                    zs[f] = si[q];
                    zs[C + f] = blur[q];
#pragma unroll
                    for (int d = 0; d < D; ++d) zs[2 * C + f * D + d] = v[d];
                }
            }
            if (sl == 0) {
                float w[D];
#pragma unroll
                for (int d = 0; d < D; ++d) w[d] = a.dg_scale * dg[d];
                if (a.log_norm_dg) log_normalize<D>(w);
#pragma unroll
                for (int d = 0; d < D; ++d) zs[2 * C + C * D + d] = w[d];
            }
            __syncwarp();
            if (SEARCH) {
                if (ivalid)
                    for (int q = sl; q < Z; q += LPP) a.z[(long long)i * Z + q] = zs[q];
                return;
            }
            // (rows of particles without a list are written again by the search that follows)
            const int floats = min(PP, total - first) * Z;
            float *out = a.z + (long long)first * Z;
            if (PP % 4 == 0 && a.out_vec) {  // first is a multiple of four rows: 16-byte aligned when z is
                const int quads = floats / 4;
                for (int q = lane; q < quads; q += 32) reinterpret_cast<float4 *>(out)[q] = reinterpret_cast<const float4 *>(stage)[q];
                for (int q = quads * 4 + lane; q < floats; q += 32) out[q] = stage[q];
            } else {
                for (int q = lane; q < floats; q += 32) out[q] = stage[q];
            }
        }
    }
}

// Out of line, so that the search does not cost the walk over lists registers.
template <int D, bool PER, int LPP, int ROWS, int MASK>
__device__ __noinline__ void list_forward_search(const FeatureFwdArgs &a, const Geom &g, float4 (*s_k)[ListShape<LPP>::kSlots],
                                                 int4 (*s_j)[ListShape<LPP>::kIndexQuads], float *stage) {
    list_forward<D, PER, LPP, ROWS, MASK, true>(a, g, s_k, s_j, stage);
}

template <int D, bool PER, int LPP, int ROWS, int MASK>
__global__ void __launch_bounds__(kListWarps * 32, (MASK & F_MOMENT) ? 2 : 4)
feature_list_forward_kernel(const __grid_constant__ FeatureFwdArgs a, const __grid_constant__ Geom g) {
    after_previous_kernel();
    using S = ListShape<LPP>;
    __shared__ float4 s_k[kListWarps][2][S::kSlots];  // v_j (K.x, K.y, K.z, W)
    __shared__ int4 s_j[kListWarps][2][S::kIndexQuads];
    extern __shared__ float4 s_rows[];                 // F_PACK: the rows of z of a warp's particles
    const int warp = threadIdx.x >> 5, total = g.B * g.N;
    const unsigned first = (blockIdx.x * kListWarps + warp) * S::PP;
    if (first >= (unsigned)total) return;
    float *stage = reinterpret_cast<float *>(s_rows) + ((MASK & F_PACK) ? (size_t)warp * ((S::PP * a.zstride + 3) & ~3) : 0);
    list_forward<D, PER, LPP, ROWS, MASK, false>(a, g, s_k[warp], s_j[warp], stage);
    __syncwarp();
    const int i = (int)min(first + (threadIdx.x & 31u) / LPP, (unsigned)total - 1u);
    if (__any_sync(kFull, __ldg(a.pair_cache + (long long)i * a.pair_stride) < 0))
        list_forward_search<D, PER, LPP, ROWS, MASK>(a, g, s_k[warp], s_j[warp], stage);
}

// ---------------------------------------------------------------------------------------------------------
// Backward.  The upstream of the gradient comes with the axis in front of the features ([N, D, C], rows
// padded to a multiple of four; upstream_rows_kernel or the packed perception's own epilogue write it so),
// so that the lanes of a sub-group read one line per axis instead of runs 48 bytes apart.
//   ds_i   = v_i sum_j [ c_s W gB_j - sum_d K_d gG_j[d] ] - gG_i . T,        K = c_g phi r, T = sum_j v_j K
//   u_d    = v_j (s_i - s_j).gG_i[d] + v_i (s_i - s_j).gG_j[d],   t = v_j gB_i.s_j + v_i gB_j.s_i
//   dx_i   = sum_j (E t - psi r.u) r + phi u      (E, phi, psi with their constants)
//   drho_i = (v_i / m_i) v_i sum_j [ phi r.((s_i - s_j) gG_j) - c_s W gB_j.s_i ]
// With position gradients the scalars of a pair carry v_i, and v_j / v_i stands in for v_j: u_d / v_i = (s_i - s_j).(v_j / v_i gG_i[d] +
// gG_j[d]) is one sum over the features instead of two, and sum_d K_d gG_j[d] serves ds and, times s_i - s_j, drho.
// Sums over features stay lane-partial (packed pairs) until the particle is done.  The density gradient's own
// backward, dx_i += sum_j J (m_i g_j - m_j g_i), uses the same pair scalars and rides stage B.
// ---------------------------------------------------------------------------------------------------------
template <int D, bool PER, int LPP, int ROWS, int MASK, bool FULL, bool SEARCH>
__device__ __forceinline__ void list_backward(const FeatureListBwdArgs &a, const Geom &g, float4 (*s_k)[ListShape<LPP, FULL && D == 3>::kSlots],
                                              float4 (*s_e)[ListShape<LPP, FULL && D == 3>::kSlots], int4 (*s_j)[ListShape<LPP, FULL && D == 3>::kIndexQuads]) {
    constexpr int EPL = ListShape<LPP, FULL && D == 3>::EPL, CH = ListShape<LPP, FULL && D == 3>::CH, PP = ListShape<LPP, FULL && D == 3>::PP, WARPS = kListBackwardWarps<D, FULL>;
    constexpr bool kGrad = (MASK & F_GRAD) != 0, kBlur = (MASK & F_BLUR) != 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sg = lane / LPP, sl = lane % LPP;
    constexpr bool kFilled = ROWS == kRowsFilled, kVec = ROWS != kRowsAny;
    const int total = g.B * g.N, C = kFilled ? LPP * 4 : a.C;
    const int first = (blockIdx.x * WARPS + warp) * PP;
    bool ivalid = (unsigned)(first + sg) < (unsigned)total;
    const int i = ivalid ? first + sg : total - 1;
    const int32_t *list = a.pair_cache + (long long)i * a.pair_stride;
    const int count = list_count<LPP>(list, a.pair_stride, ivalid, sl);
    const Pos<D> pi = load_pos<D>(a.x, i);
    ++list;
    const int n = SEARCH ? 0 : max(count, 0);
    const int nmax = SEARCH ? 0 : __reduce_max_sync(kFull, n);
    ivalid = ivalid && (count < 0) == SEARCH;
    const float mi = a.mass ? __ldg(a.mass + i) : 1.0f;
    const float rhoi = __ldg(a.rho + i);
    const float vi = mi / rhoi;
    // v_i as the pair scalars carry it: a particle without volume has only its neighbours' terms, which v_j / v_i must be able to hold
    const float vs = fabsf(vi) < 1e-25f ? 1e-25f : vi, inv_vs = 1.0f / vs;
    const unsigned spitch = (unsigned)C * 4u, bpitch = (unsigned)a.gb_pitch * 4u, gpitch = (unsigned)a.gg_pitch * 4u;
    const int Cp = kFilled ? C : a.cp;
    float dx[3] = {0.f, 0.f, 0.f};           // lane-partial over features and pairs
    unsigned long long drp = 0ull;           // minus the sum in drho, lane-partial

    for (int fbase = 0; fbase < C; fbase += LPP * 4) {
        __syncwarp();
        const int f0 = fbase + sl * 4, fv = kFilled ? f0 : min(f0, Cp - 4);
        // the i side: s_i, gB_i, gG_i in packed pairs; a lane beyond the last feature contributes zeros (minus1: -1 where it has features)
        unsigned long long si[2] = {0ull, 0ull}, gbi[2] = {0ull, 0ull}, minus1[2] = {0ull, 0ull}, ggi[2 * D];
#pragma unroll
        for (int q = 0; q < 2 * D; ++q) ggi[q] = 0ull;
        if (FULL) {
            float t[4];
            load_row4<ROWS>(a.s + (long long)i * C, f0, C, t);
            const bool in = kFilled || f0 < C, live[4] = {in, kVec ? in : f0 + 1 < C, kVec ? in : f0 + 2 < C, kVec ? in : f0 + 3 < C};
#pragma unroll
            for (int q = 0; q < 4; ++q) t[q] = live[q] ? t[q] : 0.f;
            si[0] = pack2(t[0], t[1]); si[1] = pack2(t[2], t[3]);
            minus1[0] = pack2(live[0] ? -1.f : 0.f, live[1] ? -1.f : 0.f);
            minus1[1] = kVec ? minus1[0] : pack2(live[2] ? -1.f : 0.f, live[3] ? -1.f : 0.f);
            if (kBlur && in) {
                const float4 b = __ldg(reinterpret_cast<const float4 *>(a.gb + (long long)i * a.gb_pitch + f0));
                gbi[0] = pack2(b.x, live[1] ? b.y : 0.f);
                gbi[1] = pack2(live[2] ? b.z : 0.f, live[3] ? b.w : 0.f);
            }
            if (kGrad && in) {
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    const float4 b = __ldg(reinterpret_cast<const float4 *>(a.gg + (long long)i * a.gg_pitch + d * Cp + f0));
                    ggi[2 * d] = pack2(b.x, live[1] ? b.y : 0.f);
                    ggi[2 * d + 1] = pack2(live[2] ? b.z : 0.f, live[3] ? b.w : 0.f);
                }
            }
        }
        unsigned long long ds[2] = {0ull, 0ull};
        float tsum[3] = {0.f, 0.f, 0.f};  // T, lane-partial over the pairs

        auto put = [&](int buf, int slot, float rx, float ry, float rz, float vj, int j) {
            const float q = sq_norm_fast<D>(rx, ry, rz);
            const float t = fmaxf(g.h2 - q, 0.f);
            const bool pair = vj != 0.f || j != i;  // a filled-up slot is (self, zero volume)
            const float w = pair ? g.c_s * (t * t * t) : 0.f;
            float phi = 0.f, psi = 0.f;
            if ((kGrad || (FULL && a.g_dg)) && q > 0.f) {
                const Spiky sp = spiky_distance(q);
                phi = g.c_g * spiky_phi(sp, g.h);
                if (FULL) psi = g.c_g * spiky_psi(sp, g.h);
            }
            const float kx = phi * rx, ky = phi * ry, kz = phi * rz;
            tsum[0] = fmaf(vj, kx, tsum[0]);
            tsum[1] = fmaf(vj, ky, tsum[1]);
            if (D == 3) tsum[2] = fmaf(vj, kz, tsum[2]);
            const int at = sg * (CH + 1) + slot;
            s_k[buf][at] = FULL ? make_float4(rx, ry, rz, vs * w) : make_float4(-kx, -ky, -kz, w);
            if (FULL) {
                s_e[buf][at] = make_float4(vs * phi, vs * psi, vj * inv_vs, pair ? vs * (g.c_s * 6.0f * t * t) : 0.f);
                if (a.g_dg && fbase == 0 && q > 0.f) {
                    const float mj = a.mass ? __ldg(a.mass + j) : 1.0f;
                    const float rv[3] = {rx, ry, rz};
                    float u[3] = {0.f, 0.f, 0.f}, ru = 0.f;
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        u[d] = mi * __ldg(a.g_dg + (long long)j * D + d) - mj * __ldg(a.g_dg + (long long)i * D + d);
                        ru = fmaf(rv[d], u[d], ru);
                    }
                    const float sc = psi * ru;
#pragma unroll
                    for (int d = 0; d < D; ++d) dx[d] += phi * u[d] - sc * rv[d];
                }
            }
            reinterpret_cast<int *>(&s_j[buf][sg * (CH / 4 + 1)])[slot] = j;
        };

        struct Rows { float s[4], b[4], g[D][4]; };
        auto load = [&](int j, Rows &r) {
            const unsigned long long u = (unsigned)j;
            if (FULL) load_row4<ROWS>(reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.s) + u * spitch), f0, C, r.s);
            if (kBlur) {
                const float4 t = __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(a.gb + fv) + u * bpitch));
                r.b[0] = t.x; r.b[1] = t.y; r.b[2] = t.z; r.b[3] = t.w;
            }
            if (kGrad) {
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    const float4 t = __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(a.gg + fv + d * Cp) + u * gpitch));
                    r.g[d][0] = t.x; r.g[d][1] = t.y; r.g[d][2] = t.z; r.g[d][3] = t.w;
                }
            }
        };
        auto add = [&](int buf, int e, const Rows &r) {
            const int at = sg * (CH + 1) + e;
            const float4 ke = s_k[buf][at];
            const float4 ex = FULL ? s_e[buf][at] : make_float4(-1.f, 0.f, 0.f, 0.f);
            const unsigned long long w = pack2(ke.w, ke.w);
            unsigned long long b01, b23, k01 = 0ull, k23 = 0ull;  // k: minus sum_d K_d gG_j[d]
            if (kBlur) {
                b01 = pack2(r.b[0], r.b[1]); b23 = pack2(r.b[2], r.b[3]);
                ds[0] = fma2(w, b01, ds[0]);
                ds[1] = fma2(w, b23, ds[1]);
            }
            if (kGrad) {
                const float kv[3] = {ke.x, ke.y, ke.z};
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    const float m = FULL ? -(ex.x * kv[d]) : kv[d];  // -K
                    const unsigned long long kd = pack2(m, m);
                    if (!FULL) {
                        ds[0] = fma2(kd, pack2(r.g[d][0], r.g[d][1]), ds[0]);
                        ds[1] = fma2(kd, pack2(r.g[d][2], r.g[d][3]), ds[1]);
                    } else if (d == 0) {
                        k01 = mul2(kd, pack2(r.g[d][0], r.g[d][1]));
                        k23 = mul2(kd, pack2(r.g[d][2], r.g[d][3]));
                    } else {
                        k01 = fma2(kd, pack2(r.g[d][0], r.g[d][1]), k01);
                        k23 = fma2(kd, pack2(r.g[d][2], r.g[d][3]), k23);
                    }
                }
                if (FULL) {
                    ds[0] = add2(ds[0], k01);
                    ds[1] = add2(ds[1], k23);
                }
            }
            if (FULL) {
                const unsigned long long s01 = pack2(r.s[0], r.s[1]), s23 = pack2(r.s[2], r.s[3]), vj = pack2(ex.z, ex.z);
                const float rv[3] = {ke.x, ke.y, ke.z};
                float coef = 0.f;
                if (kBlur) {
                    const unsigned long long A = fma2(gbi[1], s23, mul2(gbi[0], s01));
                    const unsigned long long Bp = fma2(si[1], b23, mul2(si[0], b01));
                    float lo, hi;
                    unpack2(fma2(vj, A, Bp), lo, hi);
                    coef = ex.w * (lo + hi);
                    drp = fma2(w, Bp, drp);
                }
                if (kGrad) {
                    const unsigned long long e01 = fma2(s01, minus1[0], si[0]), e23 = fma2(s23, minus1[1], si[1]);  // s_i - s_j
                    drp = fma2(e01, k01, drp);
                    drp = fma2(e23, k23, drp);
                    float u[3] = {0.f, 0.f, 0.f};
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        const unsigned long long h01 = fma2(vj, ggi[2 * d], pack2(r.g[d][0], r.g[d][1]));
                        const unsigned long long h23 = fma2(vj, ggi[2 * d + 1], pack2(r.g[d][2], r.g[d][3]));
                        float lo, hi;
                        unpack2(fma2(h23, e23, mul2(h01, e01)), lo, hi);
                        u[d] = lo + hi;
                    }
                    float ru = rv[0] * u[0] + rv[1] * u[1];
                    if (D == 3) ru = fmaf(rv[2], u[2], ru);
                    coef = fmaf(-ex.y, ru, coef);
#pragma unroll
                    for (int d = 0; d < D; ++d) dx[d] = fmaf(ex.x, u[d], dx[d]);
                }
#pragma unroll
                for (int d = 0; d < D; ++d) dx[d] = fmaf(coef, rv[d], dx[d]);
            }
        };
        auto drain = [&](int buf, int m) {
            const int4 *jj = &s_j[buf][sg * (CH / 4 + 1)];
#pragma unroll
            for (int e0 = 0; e0 < CH; e0 += 4) {
                if (e0 >= m) break;
                const int4 j4 = jj[e0 / 4];
                Rows r0, r1;  // two pairs in flight
                load(j4.x, r0);
                load(j4.y, r1);
                add(buf, e0, r0);
                load(j4.z, r0);
                add(buf, e0 + 1, r1);
                load(j4.w, r1);
                add(buf, e0 + 2, r0);
                add(buf, e0 + 3, r1);
            }
        };

        int buf = 0;
        if constexpr (!SEARCH) {
            // indices are loaded two chunks ahead and particles one, so that neither waits for the other's latency
            int jn[EPL], ja[EPL];
            float4 pj[EPL];
            auto indices = [&](int c) {
#pragma unroll
                for (int k = 0; k < EPL; ++k) {
                    const int e = c + k * LPP + sl;
                    ja[k] = e < n ? __ldg(list + e) : -1;
                }
            };
            auto particles = [&]() {
#pragma unroll
                for (int k = 0; k < EPL; ++k) {
                    pj[k] = fetch_particle<D>(a.x, a.pv, a.rho, a.mass, jn[k] >= 0 ? jn[k] : i);
                    if (jn[k] < 0) pj[k].w = 0.f;
                }
            };
            auto advance = [&](int c) {
#pragma unroll
                for (int k = 0; k < EPL; ++k) jn[k] = ja[k];
                indices(c);
                particles();
            };
            indices(0);
            advance(CH);
            for (int c = 0; c < nmax; c += CH, buf ^= 1) {
#pragma unroll
                for (int k = 0; k < EPL; ++k) {
                    float rx, ry, rz;
                    listed_displacement<D, PER>(g, pi, Pos<D>{pj[k].x, pj[k].y, pj[k].z}, rx, ry, rz);
                    put(buf, k * LPP + sl, rx, ry, rz, pj[k].w, jn[k] >= 0 ? jn[k] : i);
                }
                __syncwarp();
                advance(c + 2 * CH);
                drain(buf, nmax - c);
            }
        }
        if constexpr (SEARCH) {
            bool over = ivalid;
            SubgroupSearch<D, PER, LPP> search;
            if (over) search.begin(g, a.bin_offsets, i, pi);
            while (true) {
                over = over && search.more(g, pi);
                if (!__any_sync(kFull, over)) break;
                float rx = 0.f, ry = 0.f, rz = 0.f;
                bool hit = false;
                const int j = over ? search.j + sl : i;
                if (over) {
                    if (j < search.end) {
                        const Pos<D> p = load_pos<D>(a.x, j);
                        hit = displacement<D, PER, false>(g, search.org, p.x, p.y, p.z, rx, ry, rz) < g.h2;
                    }
                    search.j += LPP;
                }
                int m;
                const int slot = compact_slot<LPP>(hit, sg, sl, m);
                const int most = __reduce_max_sync(kFull, m);
                if (most == 0) continue;
                if (!hit) rx = ry = rz = 0.f;
                const float m_j = hit && a.mass ? __ldg(a.mass + j) : 1.0f;
                put(buf, slot, rx, ry, rz, hit ? m_j / __ldg(a.rho + j) : 0.f, hit ? j : i);
                __syncwarp();
                drain(buf, most);
                buf ^= 1;
            }
        }

        if (a.grad_s) {
            float o[4];
            unpack2(ds[0], o[0], o[1]);
            unpack2(ds[1], o[2], o[3]);
            if (!FULL) {
#pragma unroll
                for (int q = 0; q < 4; ++q) o[q] *= vi;
            }
            if (kGrad) {
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    const float T = subgroup_sum<LPP>(tsum[d]);
                    const float4 b = __ldg(reinterpret_cast<const float4 *>(a.gg + (long long)i * a.gg_pitch + d * Cp + fv));
                    o[0] = fmaf(-T, b.x, o[0]); o[1] = fmaf(-T, b.y, o[1]);
                    o[2] = fmaf(-T, b.z, o[2]); o[3] = fmaf(-T, b.w, o[3]);
                }
            }
            if (a.direct && ivalid) {  // upstream that reaches the features unchanged
                const float *z = a.direct + (long long)i * a.direct_pitch;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (kFilled || f0 + q < C) o[q] += __ldg(z + f0 + q);
            }
            if (a.add && ivalid) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (kFilled || f0 + q < C) o[q] += __ldg(a.add + (long long)i * C + f0 + q);
            }
            if (ivalid) store_row4<ROWS>(a.grad_s + (long long)i * C, f0, C, o);
        }
    }
    if (FULL) {
        float lo, hi;
        unpack2(drp, lo, hi);
        const float dr = -subgroup_sum<LPP>(lo + hi) / rhoi;
        float out[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int d = 0; d < D; ++d) out[d] = subgroup_sum<LPP>(dx[d]);
        if (ivalid && sl == 0) {
            if (a.grad_x) {
                if (D == 2) reinterpret_cast<float2 *>(a.grad_x)[i] = make_float2(out[0], out[1]);
                else reinterpret_cast<float4 *>(a.grad_x)[i] = make_float4(out[0], out[1], out[2], 0.f);
            }
            if (a.grad_rho) a.grad_rho[i] = dr;
            // what the density backward gathers per neighbour: position and total upstream of the density
            if (a.pg) a.pg[i] = make_float4(pi.x, pi.y, pi.z, dr + (a.g_rho ? __ldg(a.g_rho + i) : 0.f));
        }
    }
}

template <int D, bool PER, int LPP, int ROWS, int MASK, bool FULL>
__device__ __noinline__ void list_backward_search(const FeatureListBwdArgs &a, const Geom &g, float4 (*s_k)[ListShape<LPP, FULL && D == 3>::kSlots],
                                                  float4 (*s_e)[ListShape<LPP, FULL && D == 3>::kSlots], int4 (*s_j)[ListShape<LPP, FULL && D == 3>::kIndexQuads]) {
    list_backward<D, PER, LPP, ROWS, MASK, FULL, true>(a, g, s_k, s_e, s_j);
}

// Features only: four CTAs with up to 16 features -- 32,768 particles are a wave and a seventh of three CTAs, 48 -> 38 us --
// and three with longer rows, 401 us against 411.
template <int D, bool PER, int LPP, int ROWS, int MASK, bool FULL>
__global__ void __launch_bounds__(kListBackwardWarps<D, FULL> * 32, FULL ? (D == 3 ? 8 : 4) : LPP == 4 ? 4 : 3)
feature_list_backward_kernel(const __grid_constant__ FeatureListBwdArgs a, const __grid_constant__ Geom g) {
    after_previous_kernel();
    using S = ListShape<LPP, FULL && D == 3>;
    constexpr int WARPS = kListBackwardWarps<D, FULL>;
    __shared__ float4 s_k[WARPS][2][S::kSlots];             // -K.x -K.y -K.z W; FULL: r.x r.y r.z v_i W
    __shared__ float4 s_e[FULL ? WARPS : 1][2][S::kSlots];  // FULL: v_i (phi, psi, ., E), v_j / v_i
    __shared__ int4 s_j[WARPS][2][S::kIndexQuads];
    const int warp = threadIdx.x >> 5, total = g.B * g.N;
    const unsigned first = (blockIdx.x * WARPS + warp) * S::PP;
    if (first >= (unsigned)total) return;
    list_backward<D, PER, LPP, ROWS, MASK, FULL, false>(a, g, s_k[warp], s_e[FULL ? warp : 0], s_j[warp]);
    __syncwarp();
    const int i = (int)min(first + (threadIdx.x & 31u) / LPP, (unsigned)total - 1u);
    if (__any_sync(kFull, __ldg(a.pair_cache + (long long)i * a.pair_stride) < 0))
        list_backward_search<D, PER, LPP, ROWS, MASK, FULL>(a, g, s_k[warp], s_e[FULL ? warp : 0], s_j[warp]);
}

// ---------------------------------------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------------------------------------
template <int D, bool PER, int LPP, int ROWS, int MASK>
int launch_list_forward(const Geom &g, const FeatureFwdArgs &a, cudaStream_t st) {
    constexpr int PP = 32 / LPP;
    const auto kernel = feature_list_forward_kernel<D, PER, LPP, ROWS, MASK>;
    const size_t dyn = (MASK & F_PACK) ? (size_t)kListWarps * ((PP * a.zstride + 3) & ~3) * sizeof(float) : 0;
    if (dyn > 0) {
        int rc, unused = 0;
        if ((rc = persistent_ctas(kernel, kListWarps * 32, dyn, &unused)) != NPA_OK) return rc;  // raises the shared-memory limit once
    }
    const long long particles = (long long)g.B * g.N, per_cta = (long long)kListWarps * PP;
    kernel<<<(unsigned)((particles + per_cta - 1) / per_cta), kListWarps * 32, dyn, st>>>(a, g);
    return check_launch("feature_list_forward_kernel");
}

template <int D, bool PER, int LPP, int ROWS>
int launch_list_forward_mask(const Geom &g, int mask, const FeatureFwdArgs &a, cudaStream_t st) {
    switch (mask) {
        case F_BLUR: return launch_list_forward<D, PER, LPP, ROWS, F_BLUR>(g, a, st);
        case F_GRAD: return launch_list_forward<D, PER, LPP, ROWS, F_GRAD>(g, a, st);
        case F_BLUR | F_GRAD: return launch_list_forward<D, PER, LPP, ROWS, F_BLUR | F_GRAD>(g, a, st);
        case F_BLUR | F_GRAD | F_DGRAD: return launch_list_forward<D, PER, LPP, ROWS, F_BLUR | F_GRAD | F_DGRAD>(g, a, st);
        case F_BLUR | F_GRAD | F_MOMENT: return launch_list_forward<D, PER, LPP, ROWS, F_BLUR | F_GRAD | F_MOMENT>(g, a, st);
        case F_GRAD | F_MOMENT | F_CORRECTED: return launch_list_forward<D, PER, LPP, ROWS, F_GRAD | F_MOMENT | F_CORRECTED>(g, a, st);
        case F_BLUR | F_GRAD | F_MOMENT | F_PACK:
            if (a.C > LPP * 4) return fail(NPA_ERR_UNSUPPORTED, "the packed perception sweep supports up to %d features here", LPP * 4);
            return launch_list_forward<D, PER, LPP, ROWS, F_BLUR | F_GRAD | F_MOMENT | F_PACK | F_DGRAD>(g, a, st);
        default: return fail(NPA_ERR_INVALID_ARGUMENT, "unsupported feature forward mask %d", mask);
    }
}

// Lanes per particle: the smallest supported power of two whose lanes cover the features four at a time; wider rows
// (more than 128 features) are walked in slices of 128.
#define NPA_LIST_LPP(C, CALL)                                 \
    do {                                                      \
        if ((C) <= 16) return CALL(4);                        \
        if ((C) <= 32) return CALL(8);                        \
        if ((C) <= 64) return CALL(16);                       \
        return CALL(32);                                      \
    } while (0)
// The counts whose rows fill the lanes of their particle.
__host__ inline bool rows_filled(int C) { return C == 16 || C == 32 || C == 64 || C == 128; }

template <int D, bool PER>
int launch_feature_list_forward_geom(const Geom &g, int mask, const FeatureFwdArgs &args, cudaStream_t st) {
    const uintptr_t bits = (uintptr_t)args.s | (uintptr_t)args.blur | (uintptr_t)args.grad | (uintptr_t)args.vgrad;
    FeatureFwdArgs a = args;
    a.out_vec = (uintptr_t)a.z % 16 == 0;
    if (a.C % 4 == 0 && bits % 16 == 0) {
#define NPA_CALL(L) launch_list_forward_mask<D, PER, L, kRowsFilled>(g, mask, a, st)
        if (rows_filled(a.C)) NPA_LIST_LPP(a.C, NPA_CALL);
#undef NPA_CALL
#define NPA_CALL(L) launch_list_forward_mask<D, PER, L, kRowsVec>(g, mask, a, st)
        NPA_LIST_LPP(a.C, NPA_CALL);
#undef NPA_CALL
    }
#define NPA_CALL(L) launch_list_forward_mask<D, PER, L, kRowsAny>(g, mask, a, st)
    NPA_LIST_LPP(a.C, NPA_CALL);
#undef NPA_CALL
}

template <int D, bool PER, int LPP, int ROWS, bool FULL>
int launch_list_backward_mask(const Geom &g, int mask, const FeatureListBwdArgs &a, cudaStream_t st) {
    constexpr int PP = 32 / LPP, WARPS = kListBackwardWarps<D, FULL>;
    const long long particles = (long long)g.B * g.N, per_cta = (long long)WARPS * PP;
    const unsigned blocks = (unsigned)((particles + per_cta - 1) / per_cta);
    switch (mask) {
        case F_BLUR: feature_list_backward_kernel<D, PER, LPP, ROWS, F_BLUR, FULL><<<blocks, WARPS * 32, 0, st>>>(a, g); break;
        case F_GRAD: feature_list_backward_kernel<D, PER, LPP, ROWS, F_GRAD, FULL><<<blocks, WARPS * 32, 0, st>>>(a, g); break;
        case F_BLUR | F_GRAD: feature_list_backward_kernel<D, PER, LPP, ROWS, F_BLUR | F_GRAD, FULL><<<blocks, WARPS * 32, 0, st>>>(a, g); break;
        default: return fail(NPA_ERR_INVALID_ARGUMENT, "unsupported feature backward mask %d", mask);
    }
    return check_launch("feature_list_backward_kernel");
}

template <int D, bool PER, bool FULL>
int launch_feature_list_backward_geom(const Geom &g, int mask, const FeatureListBwdArgs &a, cudaStream_t st) {
    // the features-only pass reads no feature row, only its output has the caller's layout
    const uintptr_t bits = (FULL ? (uintptr_t)a.s : 0) | (uintptr_t)a.grad_s;
    if (a.C % 4 == 0 && bits % 16 == 0) {
#define NPA_CALL(L) launch_list_backward_mask<D, PER, L, kRowsFilled, FULL>(g, mask, a, st)
        if (rows_filled(a.C) && a.cp == a.C) NPA_LIST_LPP(a.C, NPA_CALL);
#undef NPA_CALL
#define NPA_CALL(L) launch_list_backward_mask<D, PER, L, kRowsVec, FULL>(g, mask, a, st)
        NPA_LIST_LPP(a.C, NPA_CALL);
#undef NPA_CALL
    }
#define NPA_CALL(L) launch_list_backward_mask<D, PER, L, kRowsAny, FULL>(g, mask, a, st)
    NPA_LIST_LPP(a.C, NPA_CALL);
#undef NPA_CALL
}

}  // namespace npa
