// The packed perception sweep of a recorded step, over neighbour lists: blur, gradient, moment matrix, density
// gradient and the perception epilogue, with one fixed association of the sums.
//
// Why fixed: see density_ordered.cu.  The order: pairs in list order, position e of the list (particles whose list
// overflowed -- and, in a recorded step, lists of more than 127 pairs -- are searched and go through in pieces of up to
// 128, e counted from the start of each).
// A feature's sum over the pairs is split by e mod CLS and the partial sums are added pairwise; the moments and the density
// gradient are split by e mod 32 and added pairwise, distance 16 first.  CLS = 32 / (lanes that cover the
// features, four each).
//
// Sixteen lanes own a particle: LPR lanes cover a row, VW features each, and the 16 / LPR groups of them take the classes
// of a block of CLS entries, CPL each, so that a lane keeps CPL partial sums per feature.  The groups' sums meet once per
// particle, halving the features a lane goes on with at each exchange.  A chunk of 32 list entries is turned into pair
// scalars, two per lane (their moments are the partial sums e and e + 16), left in shared memory, and walked by the
// groups.  The first 32 entries of a list are loaded together with its length.
//
// Bound by instruction issue and latency together (~1,700 warp instructions per two particles with 41 pairs, a third of
// them the pairs themselves, half of the issue slots at 14.5 warps per SM).  Measured, B200, us, the sweep with the whole
// warp per particle -> this one: 262,144 particles in 3D, C = 32, ~41 pairs 495 -> 417, with rows that
// fill their lanes (feature_list.cuh) 371; 32,768 in 2D, C = 16, ~31 pairs 36 -> 33.
// Not kept: eight lanes per particle with all classes in registers (420, but 42 in 2D), sixteen with every class of one or two
// features (492), five CTAs per SM in 3D (432, spills).
#pragma once
#include "feature_kernels.cuh"
#include "feature_list.cuh"

namespace npa {

constexpr int kOrderedWarps = 2;    // warps per CTA
constexpr int kOrderedPairs = 127;  // longest list that is read in a recorded step
constexpr int kOrderedRow = 164;    // floats of a packed row: 32 features in 3D

struct OrderedMem {  // of one warp
    union {
        struct {
            float4 ent[132];           // v_j K, v_j W; lists: two particles with 33 slots each
            float4 geo[kListPerWarp];  // search: displacement and index; lists: the indices
        };
        float rows[2 * kOrderedRow];   // the packed rows on their way out
    };
    int4 rng[kMaxRanges];
};

// 3 (h - d)^2 / d with the correctly rounded square root and quotient.
__device__ inline float spiky_phi_rounded(float q, float h) {
    const Root r = root_rounded(q + 1e-12f);
    const float t = fmaxf(h - r.d, 0.0f);
    return quotient_rounded(3.0f * t * t, r);
}

template <int D, bool PER, int VW, int LPR, int CPL, int ROWS>
struct Ordered {
    static constexpr int NM = D * (D + 1) / 2, H = VW / 2;
    static constexpr int G = 16 / LPR, CLS = G * CPL;  // groups of a particle, classes
    static constexpr int U = 4, STEP = U / CPL * CLS;  // rows in flight per lane, entries they stand for
    static constexpr int OWN = VW > G ? VW / G : 1;    // features a lane ends with
    static constexpr bool ALIGNED = ROWS != kRowsAny, FILLED = ROWS == kRowsFilled;
    static __device__ inline int features(const FeatureFwdArgs &a) { return FILLED ? VW * LPR : a.C; }
    float si[VW];
    unsigned long long nsi[H], acc[CPL][1 + D][H];
    float mom[2][NM], dgs[2][3];

    __device__ inline void begin(const float *__restrict__ row, int f, int C) {
        load(row, f, C, si);
#pragma unroll
        for (int h = 0; h < H; ++h) nsi[h] = pack2(-si[2 * h], -si[2 * h + 1]);
#pragma unroll
        for (int c = 0; c < CPL; ++c)
#pragma unroll
            for (int q = 0; q <= D; ++q)
#pragma unroll
                for (int h = 0; h < H; ++h) acc[c][q][h] = 0ull;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
#pragma unroll
            for (int q = 0; q < NM; ++q) mom[k][q] = 0.f;
            dgs[k][0] = dgs[k][1] = dgs[k][2] = 0.f;
        }
    }
    // Lanes beyond the last feature read valid neighbours of it (unused).
    static __device__ inline void load(const float *__restrict__ row, int f, int C, float (&v)[VW]) {
        if (FILLED || (ALIGNED && C % VW == 0)) {
            if constexpr (VW == 4) {
                const float4 t = __ldg(reinterpret_cast<const float4 *>(row + (FILLED ? f : min(f, C - 4))));
                v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
            } else {
                const float2 t = __ldg(reinterpret_cast<const float2 *>(row + (FILLED ? f : min(f, C - 2))));
                v[0] = t.x; v[1] = t.y;
            }
        } else {
#pragma unroll
            for (int q = 0; q < VW; ++q) v[q] = __ldg(row + min(f + q, C - 1));
        }
    }
    // Pair scalars (zero volume and mass: no pair); k: which of the lane's partial sums.
    __device__ inline float4 pair(const Geom &g, int k, float rx, float ry, float rz, float vj, float mj) {
        const float q = sq_norm_fast<D>(rx, ry, rz);
        const float t = fmaxf(g.h2 - q, 0.f);
        const float w = vj * (t * t * t);
        float kv = 0.f;
        if (q > 0.f) {
            const float phi = spiky_phi_rounded(q, g.h);
            kv = vj * phi;
            const float md = mj * phi;
            dgs[k][0] = fmaf(md, rx, dgs[k][0]);
            dgs[k][1] = fmaf(md, ry, dgs[k][1]);
            if (D == 3) dgs[k][2] = fmaf(md, rz, dgs[k][2]);
        }
        mom[k][0] = fmaf(kv * rx, rx, mom[k][0]);
        mom[k][1] = fmaf(kv * rx, ry, mom[k][1]);
        if (D == 2) {
            mom[k][2] = fmaf(kv * ry, ry, mom[k][2]);
        } else {
            mom[k][2] = fmaf(kv * rx, rz, mom[k][2]);
            mom[k][NM > 3 ? 3 : 0] = fmaf(kv * ry, ry, mom[k][NM > 3 ? 3 : 0]);
            mom[k][NM > 3 ? 4 : 0] = fmaf(kv * ry, rz, mom[k][NM > 3 ? 4 : 0]);
            mom[k][NM > 3 ? 5 : 0] = fmaf(kv * rz, rz, mom[k][NM > 3 ? 5 : 0]);
        }
        return make_float4(kv * rx, kv * ry, kv * rz, w);
    }
    // STEP entries from a position that is a multiple of CLS; this group's are CPL in a row of each block of CLS.
    __device__ inline void add(const float4 *__restrict__ ent, const int (&js)[U], const float *__restrict__ s, int f, int C) {
        float r[U][VW];
#pragma unroll
        for (int u = 0; u < U; ++u)
            load(reinterpret_cast<const float *>(reinterpret_cast<const char *>(s) + (unsigned long long)(unsigned)js[u] * ((unsigned)C * 4u)), f, C, r[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float4 e = ent[u / CPL * CLS + u % CPL];
            const unsigned long long w = pack2(e.w, e.w), kd[3] = {pack2(e.x, e.x), pack2(e.y, e.y), pack2(e.z, e.z)};
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const unsigned long long sj = pack2(r[u][2 * h], r[u][2 * h + 1]), df = add2(sj, nsi[h]);
                acc[u % CPL][0][h] = fma2(w, sj, acc[u % CPL][0][h]);
#pragma unroll
                for (int d = 0; d < D; ++d) acc[u % CPL][1 + d][h] = fma2(df, kd[d], acc[u % CPL][1 + d][h]);
            }
        }
    }
    // Sums complete -> the packed row `zs`, vgrad and rho_grad of particle i.  WIDE: the lane's partial sum is one of 32.
    template <bool WIDE>
    __device__ inline void finish(const FeatureFwdArgs &a, const Geom &g, long long i, bool valid, int f, int sl, float *zs) {
        constexpr int L = WIDE ? 32 : 16;
        const int C = features(a);
        float m[NM], dg[3] = {0.f, 0.f, 0.f}, inv[D * D];
#pragma unroll
        for (int q = 0; q < NM; ++q) m[q] = g.c_g * subgroup_sum<L>(WIDE ? mom[0][q] : mom[0][q] + mom[1][q]);
#pragma unroll
        for (int d = 0; d < D; ++d) dg[d] = g.c_g * subgroup_sum<L>(WIDE ? dgs[0][d] : dgs[0][d] + dgs[1][d]);
        // the lane's classes, then group by group: neighbours first
        float val[VW][1 + D];
#pragma unroll
        for (int q = 0; q <= D; ++q)
#pragma unroll
            for (int h = 0; h < H; ++h) {
                if (CPL == 2) acc[0][q][h] = add2(acc[0][q][h], acc[CPL - 1][q][h]);
                unpack2(acc[0][q][h], val[2 * h][q], val[2 * h + 1][q]);
            }
        int have = VW;
#pragma unroll
        for (int o = LPR; o < 16; o <<= 1) {
            if (have > 1) {  // half of the features each
                const bool upper = (sl & o) != 0;
                have /= 2;
#pragma unroll
                for (int v = 0; v < VW / 2; ++v) {
                    if (v >= have) break;
#pragma unroll
                    for (int q = 0; q <= D; ++q) {
                        const float mine = upper ? val[v + have][q] : val[v][q], theirs = upper ? val[v][q] : val[v + have][q];
                        val[v][q] = mine + __shfl_xor_sync(kFull, theirs, o);
                    }
                    si[v] = upper ? si[v + have] : si[v];
                }
                f += upper ? have : 0;
            } else {
#pragma unroll
                for (int q = 0; q <= D; ++q) val[0][q] += __shfl_xor_sync(kFull, val[0][q], o);
            }
        }
        safe_inverse_sym<D>(m, a.inv_tol, inv);
#pragma unroll
        for (int v = 0; v < OWN; ++v) {
            float gr[D], w[D];
#pragma unroll
            for (int d = 0; d < D; ++d) gr[d] = g.c_g * val[v][1 + d];
#pragma unroll
            for (int d = 0; d < D; ++d) {
                float sum = 0.f;
#pragma unroll
                for (int k = 0; k < D; ++k) sum = fmaf(gr[k], inv[k * D + d], sum);
                w[d] = sum;
                val[v][1 + d] = sum;
            }
#pragma unroll
            for (int d = 0; d < D; ++d) w[d] *= a.coef;
            if (a.log_norm_grad) log_normalize<D>(w);
            if (FILLED || f + v < C) {
                zs[f + v] = si[v];
                zs[C + f + v] = g.c_s * val[v][0];
#pragma unroll
                for (int d = 0; d < D; ++d) zs[2 * C + (f + v) * D + d] = w[d];
            }
        }
        if (a.vgrad && valid) {
            float *o = a.vgrad + (i * C + f) * D;
            if (ALIGNED && OWN == 2 && C % 2 == 0) {
                if (FILLED || f < C) {
                    auto at = [&](int e) { return val[e / D][1 + e % D]; };
#pragma unroll
                    for (int k = 0; k < D; ++k) reinterpret_cast<float2 *>(o)[k] = make_float2(at(2 * k), at(2 * k + 1));
                }
            } else {
#pragma unroll
                for (int v = 0; v < OWN; ++v)
                    if (f + v < C) {
#pragma unroll
                        for (int d = 0; d < D; ++d) o[v * D + d] = val[v][1 + d];
                    }
            }
        }
        if (sl == 0) {
            float w[D];
#pragma unroll
            for (int d = 0; d < D; ++d) {
                if (valid && a.rho_grad_out) a.rho_grad_out[i * D + d] = dg[d];
                w[d] = dg[d] * a.dg_scale;
            }
            if (a.log_norm_dg) log_normalize<D>(w);
#pragma unroll
            for (int d = 0; d < D; ++d) zs[2 * C + C * D + d] = w[d];
        }
    }
};

// One particle by the whole warp, through the candidates of its cells (the two halves of the warp sum the features
// alike).  Out of line, so that it costs the walk over lists no registers.
template <int D, bool PER, int VW, int LPR, int CPL, int ROWS>
__device__ __noinline__ void ordered_search(const FeatureFwdArgs &a, const Geom &g, OrderedMem &mem, int i) {
    using O = Ordered<D, PER, VW, LPR, CPL, ROWS>;
    const int lane = threadIdx.x & 31, sl = lane & 15, f = sl % LPR * VW, at = sl / LPR * CPL, C = Ordered<D, PER, VW, LPR, CPL, ROWS>::features(a), sys = i / g.N;
    const Pos<D> pi = load_pos<D>(a.x, i);
    WorkItem it = {i, 1, 0, sys};
    it.cell = sys * g.cells + (int)snapshot_cell(g, a.bin_offsets + (size_t)sys * g.cells, i,
                                                 cell_hash<D>(g, axis_cell(pi.x, g, 0), axis_cell(pi.y, g, 1), D == 3 ? axis_cell(pi.z, g, 2) : 0));
    __syncwarp();
    const int nr = build_ranges<D>(g, a.bin_offsets, it, mem.rng);
    O o;
    o.begin(a.s + (long long)i * C, f, C);
    collect_pairs<D, PER>(g, a.x, pi, mem.rng, nr, mem.geo, [&](int n) {
        __syncwarp();
        const int filled = (n + O::STEP - 1) / O::STEP * O::STEP;  // kListPerWarp is a multiple of STEP
        for (int e = lane; e < filled; e += 32) {
            if (e < n) {
                const float4 ge = mem.geo[e];
                const int j = __float_as_int(ge.w);
                const float mj = a.mass ? __ldg(a.mass + j) : 1.0f;
                mem.ent[e] = o.pair(g, 0, ge.x, ge.y, ge.z, mj / __ldg(a.rho + j), mj);
            } else {
                mem.ent[e] = make_float4(0.f, 0.f, 0.f, 0.f);
                mem.geo[e].w = __int_as_float(i);
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int e = at; e < n; e += O::STEP) {
            int js[O::U];
#pragma unroll
            for (int u = 0; u < O::U; ++u) js[u] = __float_as_int(mem.geo[e + u / CPL * O::CLS + u % CPL].w);
            o.add(mem.ent + e, js, a.s, f, C);
        }
        __syncwarp();
    });
    o.template finish<true>(a, g, i, lane < 16, f, sl, mem.rows);
    __syncwarp();
    for (int q = lane; q < a.zstride; q += 32) a.z[(long long)i * a.zstride + q] = mem.rows[q];
    __syncwarp();
}

template <int D, bool PER, int VW, int LPR, int CPL, int ROWS>
__global__ void __launch_bounds__(kOrderedWarps * 32, D == 2 ? 10 : 8)
packed_ordered_kernel(const __grid_constant__ FeatureFwdArgs a, const __grid_constant__ Geom g) {
    after_previous_kernel();
    using O = Ordered<D, PER, VW, LPR, CPL, ROWS>;
    __shared__ OrderedMem s_mem[kOrderedWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sg = lane >> 4, sl = lane & 15;
    const int total = g.B * g.N, first = (int)((blockIdx.x * kOrderedWarps + warp) * 2u);
    if ((unsigned)first >= (unsigned)total) return;
    OrderedMem &mem = s_mem[warp];
    const bool valid = sg < total - first;
    const int i = valid ? first + sg : total - 1, C = O::features(a), f = sl % LPR * VW, at = sl / LPR * CPL;
    const int32_t *list = a.pair_cache + (long long)i * a.pair_stride;
    const int room = a.vgrad ? min(a.pair_stride - 1, kOrderedPairs) : a.pair_stride - 1;
    const int count = __ldg(list++);
    int ja[2];  // entries one chunk ahead; the first are loaded before the length is known
    auto indices = [&](int c) {
#pragma unroll
        for (int k = 0; k < 2; ++k) ja[k] = c + 16 * k + sl < room ? __ldg(list + c + 16 * k + sl) : 0;
    };
    indices(0);
    const Pos<D> pi = load_pos<D>(a.x, i);
    O o;
    o.begin(a.s + (long long)i * C, f, C);
    const bool search = count < 0 || count > room;
    const int n = search ? 0 : count, nmax = __reduce_max_sync(kFull, n);
    float4 *ent = mem.ent + sg * 33;
    int *idx = reinterpret_cast<int *>(mem.geo) + sg * 36;
    int jn[2];
    float4 pj[2];
    auto particles = [&](int c) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const bool in = c + 16 * k + sl < n;
            jn[k] = in ? ja[k] : i;
            pj[k] = fetch_particle<D>(a.x, a.pv, a.rho, a.mass, jn[k]);
            if (!in) pj[k].w = 0.f;
        }
    };
    particles(0);
#pragma unroll 1
    for (int c = 0; c < nmax; c += 32) {
        indices(c + 32);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (c + 16 * k >= nmax) break;
            float rx, ry, rz;
            listed_displacement<D, PER>(g, pi, Pos<D>{pj[k].x, pj[k].y, pj[k].z}, rx, ry, rz);
            const float mj = c + 16 * k + sl >= n ? 0.f : a.mass ? __ldg(a.mass + jn[k]) : 1.0f;
            ent[16 * k + sl] = o.pair(g, k, rx, ry, rz, pj[k].w, mj);
            idx[16 * k + sl] = jn[k];
        }
        __syncwarp();
        particles(c + 32);
        const int m = min(32, nmax - c);
#pragma unroll 1
        for (int e = at; e < m; e += O::STEP) {  // (entries up to the next multiple of 16 are filled)
            int js[O::U];
#pragma unroll
            for (int u = 0; u < O::U; u += CPL) {
                if constexpr (CPL == 2) {
                    const int2 t = *reinterpret_cast<const int2 *>(idx + e + u / CPL * O::CLS);
                    js[u] = t.x; js[u + 1] = t.y;
                } else {
                    js[u] = idx[e + u * O::CLS];
                }
            }
            o.add(ent + e, js, a.s, f, C);
        }
        __syncwarp();
    }
    const int Z = O::FILLED ? (2 + D) * C + D : a.zstride;
    o.template finish<false>(a, g, i, valid && !search, f, sl, mem.rows + sg * Z);
    __syncwarp();
    // the rows of both particles are one run (8-byte aligned when z is: first is even); the row of a particle that is
    // searched is written again below
    const int floats = min(2, total - first) * Z;
    float *out = a.z + (long long)first * Z;
    if (O::ALIGNED) {
        for (int q = lane; q < floats / 2; q += 32) reinterpret_cast<float2 *>(out)[q] = reinterpret_cast<const float2 *>(mem.rows)[q];
        if ((floats & 1) && lane == 0) out[floats - 1] = mem.rows[floats - 1];
    } else {
        for (int q = lane; q < floats; q += 32) out[q] = mem.rows[q];
    }
    const unsigned again = __ballot_sync(kFull, search && valid);
    if (again & 0x0000ffffu) ordered_search<D, PER, VW, LPR, CPL, ROWS>(a, g, mem, first);
    if (again & 0xffff0000u) ordered_search<D, PER, VW, LPR, CPL, ROWS>(a, g, mem, first + 1);
}

// ROWS (feature_list.cuh): kRowsAny where the addresses of the feature rows, of z or of vgrad do not allow the vector accesses of the
// shape, kRowsFilled where the lanes of a row cover it exactly.
template <int D, bool PER, int VW, int LPR, int CPL>
int launch_packed_ordered_shape(const Geom &g, const FeatureFwdArgs &a, cudaStream_t st) {
    const bool aligned = (a.C % VW != 0 || (uintptr_t)a.s % (VW * 4) == 0) && ((uintptr_t)a.z | (uintptr_t)a.vgrad) % 8 == 0;
    auto kernel = packed_ordered_kernel<D, PER, VW, LPR, CPL, kRowsAny>;
    if (aligned) kernel = packed_ordered_kernel<D, PER, VW, LPR, CPL, kRowsVec>;
    if constexpr (VW == 4) {
        if (aligned && a.C == VW * LPR) kernel = packed_ordered_kernel<D, PER, VW, LPR, CPL, kRowsFilled>;
    }
    const long long particles = (long long)g.B * g.N;
    launch_early(kernel, (unsigned)((particles + 2 * kOrderedWarps - 1) / (2 * kOrderedWarps)), kOrderedWarps * 32, 0, st, a, g);
    return check_launch("packed_ordered_kernel");
}

// Up to 32 features.  The classes: 32 / (lanes that cover a row, four features each); with a count that is not a multiple of
// four, four for up to eight features and one beyond.  They depend on the count alone: rows at an address that vectors
// cannot be loaded from are read float by float into the same sums.
template <int D, bool PER>
int launch_packed_ordered_geom(const Geom &g, const FeatureFwdArgs &a, cudaStream_t st) {
    if (a.C % 4 == 0) {
        if (a.C <= 16) return launch_packed_ordered_shape<D, PER, 4, 4, 2>(g, a, st);
        return launch_packed_ordered_shape<D, PER, 4, 8, 2>(g, a, st);
    }
    if (a.C <= 8) return launch_packed_ordered_shape<D, PER, 2, 4, 1>(g, a, st);
    return launch_packed_ordered_shape<D, PER, 2, 16, 1>(g, a, st);
}

}  // namespace npa
