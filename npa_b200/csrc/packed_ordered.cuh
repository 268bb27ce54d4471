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
// Sixteen lanes own a particle, VW = 1 or 2 features each, and keep the CLS partial sums of their features in
// registers: CLS rows are in flight at a time and nothing is combined across lanes.  A chunk of 32 list entries is
// turned into pair scalars, two per lane (their moments are the partial sums e and e + 16), left in shared memory, and
// walked by the sub-group.  The first 32 entries of a list are loaded together with its length.
#pragma once
#include "feature_kernels.cuh"
#include "feature_list.cuh"
#include <type_traits>

namespace npa {

constexpr int kOrderedWarps = 4;    // warps per CTA
constexpr int kOrderedPairs = 127;  // longest list that is read in a recorded step
constexpr int kOrderedRow = 164;    // floats of a packed row: 32 features in 3D

struct OrderedMem {     // of one warp
    float4 ent[132];    // v_j K, v_j W; lists: two particles with 33 slots each
    float4 geo[kListPerWarp];  // search: displacement and index; lists: the indices
    int4 rng[kMaxRanges];
    float rows[2 * kOrderedRow];
};

// 3 (h - d)^2 / d with the correctly rounded square root and quotient.
__device__ inline float spiky_phi_rounded(float q, float h) {
    const float d = sqrtf(q + 1e-12f);
    const float t = fmaxf(h - d, 0.0f);
    return 3.0f * t * t / d;
}

template <int D, bool PER, int VW, int CLS>
struct Ordered {
    static constexpr int NM = D * (D + 1) / 2;
    static constexpr int U = CLS > 4 ? CLS : 4;  // rows in flight
    using Sum = typename std::conditional<VW == 2, unsigned long long, float>::type;
    float si[VW];
    Sum nsi, acc[CLS][1 + D];
    float mom[2][NM], dgs[2][3];

    __device__ inline void begin(const float *__restrict__ row, int f, int C) {
        load(row, f, C, si);
        if constexpr (VW == 2) nsi = pack2(-si[0], -si[1]);
#pragma unroll
        for (int c = 0; c < CLS; ++c)
#pragma unroll
            for (int q = 0; q <= D; ++q) acc[c][q] = 0;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
#pragma unroll
            for (int q = 0; q < NM; ++q) mom[k][q] = 0.f;
            dgs[k][0] = dgs[k][1] = dgs[k][2] = 0.f;
        }
    }
    // Lanes beyond the last feature read valid neighbours of it (unused).
    static __device__ inline void load(const float *__restrict__ row, int f, int C, float (&v)[VW]) {
        if (VW == 2 && C % 2 == 0) {
            const float2 t = __ldg(reinterpret_cast<const float2 *>(row + min(f, C - 2)));
            v[0] = t.x; v[VW - 1] = t.y;
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
    // U entries from a position that is a multiple of U (so entry u belongs to class u mod CLS).
    __device__ inline void add(const float4 *__restrict__ ent, const int (&js)[U], const float *__restrict__ s, int f, int C) {
        float r[U][VW];
#pragma unroll
        for (int u = 0; u < U; ++u)
            load(reinterpret_cast<const float *>(reinterpret_cast<const char *>(s) + (unsigned long long)(unsigned)js[u] * ((unsigned)C * 4u)), f, C, r[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float4 e = ent[u];
            const float kd[3] = {e.x, e.y, e.z};
            Sum(&to)[1 + D] = acc[u % CLS];
            if constexpr (VW == 2) {
                const unsigned long long sj = pack2(r[u][0], r[u][1]), df = add2(sj, nsi);
                to[0] = fma2(pack2(e.w, e.w), sj, to[0]);
#pragma unroll
                for (int d = 0; d < D; ++d) to[1 + d] = fma2(df, pack2(kd[d], kd[d]), to[1 + d]);
            } else {
                const float df = r[u][0] - si[0];
                to[0] = fmaf(e.w, r[u][0], to[0]);
#pragma unroll
                for (int d = 0; d < D; ++d) to[1 + d] = fmaf(df, kd[d], to[1 + d]);
            }
        }
    }
    // Sums complete -> the packed row `zs`, vgrad and rho_grad of particle i.  WIDE: the lane's partial sum is one of 32.
    template <bool WIDE>
    __device__ inline void finish(const FeatureFwdArgs &a, const Geom &g, long long i, bool valid, int f, int sl, float *zs) {
        constexpr int L = WIDE ? 32 : 16;
        const int C = a.C;
#pragma unroll
        for (int o = 1; o < CLS; o <<= 1)
#pragma unroll
            for (int c = 0; c < CLS; c += 2 * o)
#pragma unroll
                for (int q = 0; q <= D; ++q) {
                    if constexpr (VW == 2) acc[c][q] = add2(acc[c][q], acc[(c + o) % CLS][q]);
                    else acc[c][q] += acc[(c + o) % CLS][q];
                }
        float m[NM], dg[3] = {0.f, 0.f, 0.f}, inv[D * D];
#pragma unroll
        for (int q = 0; q < NM; ++q) m[q] = g.c_g * subgroup_sum<L>(WIDE ? mom[0][q] : mom[0][q] + mom[1][q]);
#pragma unroll
        for (int d = 0; d < D; ++d) dg[d] = g.c_g * subgroup_sum<L>(WIDE ? dgs[0][d] : dgs[0][d] + dgs[1][d]);
        safe_inverse_sym<D>(m, a.inv_tol, inv);
        float val[VW][1 + D];
#pragma unroll
        for (int q = 0; q <= D; ++q) {
            if constexpr (VW == 2) unpack2(acc[0][q], val[0][q], val[VW - 1][q]);
            else val[0][q] = acc[0][q];
        }
#pragma unroll
        for (int v = 0; v < VW; ++v) {
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
            if (f + v < C) {
                zs[f + v] = si[v];
                zs[C + f + v] = g.c_s * val[v][0];
#pragma unroll
                for (int d = 0; d < D; ++d) zs[2 * C + (f + v) * D + d] = w[d];
            }
        }
        if (a.vgrad && valid) {
            float *o = a.vgrad + (i * C + f) * D;
            if (VW == 2 && C % 2 == 0) {
                if (f < C) {
                    float run[VW * D];
#pragma unroll
                    for (int v = 0; v < VW; ++v)
#pragma unroll
                        for (int d = 0; d < D; ++d) run[v * D + d] = val[v][1 + d];
#pragma unroll
                    for (int k = 0; k < D; ++k) reinterpret_cast<float2 *>(o)[k] = make_float2(run[(2 * k) % (VW * D)], run[(2 * k + 1) % (VW * D)]);
                }
            } else {
#pragma unroll
                for (int v = 0; v < VW; ++v)
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
template <int D, bool PER, int VW, int CLS>
__device__ __noinline__ void ordered_search(const FeatureFwdArgs &a, const Geom &g, OrderedMem &mem, int i) {
    using O = Ordered<D, PER, VW, CLS>;
    const int lane = threadIdx.x & 31, sl = lane & 15, f = sl * VW, C = a.C, sys = i / g.N;
    const Pos<D> pi = load_pos<D>(a.x, i);
    WorkItem it = {i, 1, 0, sys};
    it.cell = sys * g.cells + (int)cell_hash<D>(g, axis_cell(pi.x, g, 0), axis_cell(pi.y, g, 1), D == 3 ? axis_cell(pi.z, g, 2) : 0);
    __syncwarp();
    const int nr = build_ranges<D>(g, a.bin_offsets, it, mem.rng);
    O o;
    o.begin(a.s + (long long)i * C, f, C);
    collect_pairs<D, PER>(g, a.x, pi, mem.rng, nr, mem.geo, [&](int n) {
        __syncwarp();
        const int filled = (n + O::U - 1) / O::U * O::U;  // kListPerWarp is a multiple of U
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
        for (int e = 0; e < n; e += O::U) {
            int js[O::U];
#pragma unroll
            for (int u = 0; u < O::U; ++u) js[u] = __float_as_int(mem.geo[e + u].w);
            o.add(mem.ent + e, js, a.s, f, C);
        }
        __syncwarp();
    });
    o.template finish<true>(a, g, i, lane < 16, f, lane, mem.rows);
    __syncwarp();
    for (int q = lane; q < a.zstride; q += 32) a.z[(long long)i * a.zstride + q] = mem.rows[q];
    __syncwarp();
}

template <int D, bool PER, int VW, int CLS>
__global__ void __launch_bounds__(kOrderedWarps * 32, VW == 2 ? 4 : 5)
packed_ordered_kernel(const __grid_constant__ FeatureFwdArgs a, const __grid_constant__ Geom g) {
    using O = Ordered<D, PER, VW, CLS>;
    __shared__ OrderedMem s_mem[kOrderedWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sg = lane >> 4, sl = lane & 15;
    const int total = g.B * g.N, first = (blockIdx.x * kOrderedWarps + warp) * 2;
    if (first >= total) return;
    OrderedMem &mem = s_mem[warp];
    const bool valid = first + sg < total;
    const int i = min(first + sg, total - 1), C = a.C, f = sl * VW;
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
    int4 *idx = reinterpret_cast<int4 *>(mem.geo) + sg * 9;
    int jn[2];
    float4 pj[2];
    float mj[2];
    auto particles = [&](int c) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const bool in = c + 16 * k + sl < n;
            jn[k] = in ? ja[k] : i;
            pj[k] = fetch_particle<D>(a.x, a.pv, a.rho, a.mass, jn[k]);
            mj[k] = !in ? 0.f : a.mass ? __ldg(a.mass + jn[k]) : 1.0f;
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
            ent[16 * k + sl] = o.pair(g, k, rx, ry, rz, pj[k].w, mj[k]);
            reinterpret_cast<int *>(idx)[16 * k + sl] = jn[k];
        }
        __syncwarp();
        particles(c + 32);
        const int m = min(32, nmax - c);
#pragma unroll 1
        for (int e = 0; e < m; e += O::U) {
            int js[O::U];
#pragma unroll
            for (int u = 0; u < O::U; u += 4) {
                const int4 t = idx[(e + u) / 4];
                js[u] = t.x; js[u + 1] = t.y; js[u + 2] = t.z; js[u + 3] = t.w;
            }
            o.add(ent + e, js, a.s, f, C);
        }
        __syncwarp();
    }
    const int Z = a.zstride;
    o.template finish<false>(a, g, i, valid && !search, f, sl, mem.rows + sg * Z);
    __syncwarp();
    // the rows of both particles are one run; the row of a particle that is searched is written again below
    const int floats = min(2, total - first) * Z;
    float *out = a.z + (long long)first * Z;
    for (int q = lane; q < floats; q += 32) out[q] = mem.rows[q];
    const unsigned again = __ballot_sync(kFull, search && valid);
    if (again & 0x0000ffffu) ordered_search<D, PER, VW, CLS>(a, g, mem, first);
    if (again & 0xffff0000u) ordered_search<D, PER, VW, CLS>(a, g, mem, first + 1);
}

template <int D, bool PER, int VW, int CLS>
int launch_packed_ordered_shape(const Geom &g, const FeatureFwdArgs &a, cudaStream_t st) {
    const long long particles = (long long)g.B * g.N;
    packed_ordered_kernel<D, PER, VW, CLS><<<(unsigned)((particles + 2 * kOrderedWarps - 1) / (2 * kOrderedWarps)), kOrderedWarps * 32, 0, st>>>(a, g);
    return check_launch("packed_ordered_kernel");
}

// Up to 32 features.  The classes follow the lanes that cover a row four features each (one each where C is no multiple of four).
template <int D, bool PER>
int launch_packed_ordered_geom(const Geom &g, const FeatureFwdArgs &a, cudaStream_t st) {
    if (a.C % 4 == 0) {
        if (a.C <= 16) return launch_packed_ordered_shape<D, PER, 1, 8>(g, a, st);
        return launch_packed_ordered_shape<D, PER, 2, 4>(g, a, st);
    }
    if (a.C <= 8) return launch_packed_ordered_shape<D, PER, 1, 4>(g, a, st);
    if (a.C <= 16) return launch_packed_ordered_shape<D, PER, 1, 1>(g, a, st);
    return launch_packed_ordered_shape<D, PER, 2, 1>(g, a, st);
}

}  // namespace npa
