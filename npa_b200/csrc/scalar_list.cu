// Density and density gradient over recorded neighbour lists, and the layout change the feature backward reads.
#include "feature_list.cuh"

namespace npa {

// ---------------------------------------------------------------------------------------------------------
// Gather backward of density and / or density gradient.  Four lanes per particle, eight particles per warp; a lane takes
// a 16-byte piece of the list at a time (four entries, whose gathers are all in flight together).  Bound by the L1 tag
// stage: every gathered entry is its own sector, so position and upstream come as one 16-byte record (pg) when the
// feature backward has just written it.
// ---------------------------------------------------------------------------------------------------------
template <int D, bool PER, int MASK>
__global__ void __launch_bounds__(256)
scalar_list_backward_kernel(ScalarListArgs a, Geom g) {
    after_previous_kernel();
    constexpr int LPP = 4;
    const int lane = threadIdx.x & 31, sl = lane % LPP;
    const int total = g.B * g.N;
    const unsigned at = blockIdx.x * (256u / LPP) + threadIdx.x / LPP;  // below 2^31 + 256 / LPP
    if (at - lane / LPP >= (unsigned)total) return;
    const bool ivalid = at < (unsigned)total;
    const int i = ivalid ? (int)at : total - 1;
    const Pos<D> pi = load_pos<D>(a.x, i);
    const float mi = a.mass ? __ldg(a.mass + i) : 1.0f;
    auto upstream = [&](int j) {
        float v = 0.f;
        if (a.g_rho_a) v += __ldg(a.g_rho_a + j);
        if (a.g_rho_b) v += __ldg(a.g_rho_b + j);
        return v;
    };
    float gri = 0.f, gdi[3] = {0.f, 0.f, 0.f};
    if (MASK & S_DENSITY) gri = a.pg ? __ldg(a.pg + i).w : upstream(i);
    if (MASK & S_DGRAD) {
#pragma unroll
        for (int d = 0; d < D; ++d) gdi[d] = __ldg(a.g_dg + (long long)i * D + d);
    }
    float dxs[3] = {0.f, 0.f, 0.f}, dxg[3] = {0.f, 0.f, 0.f};

    auto record = [&](int j) {  // position and density upstream of j
        if (a.pg) return __ldg(a.pg + j);
        const Pos<D> p = load_pos<D>(a.x, j);
        return make_float4(p.x, p.y, p.z, (MASK & S_DENSITY) ? upstream(j) : 0.f);
    };
    auto visit = [&](int j, float grj, float rx, float ry, float rz, float q) {
        if (!(q > 0.f)) return;  // the self or a coincident pair has zero gradient
        const float rv[3] = {rx, ry, rz};
        const float mj = a.mass ? __ldg(a.mass + j) : 1.0f;
        if (MASK & S_DENSITY) {
            const float t = fmaxf(g.h2 - q, 0.f);
            const float w = 6.0f * t * t * (gri * mj + grj * mi);
#pragma unroll
            for (int d = 0; d < D; ++d) dxs[d] = fmaf(w, rv[d], dxs[d]);
        }
        if (MASK & S_DGRAD) {
            const Spiky sp = spiky_distance(q);
            const float phi = spiky_phi(sp, g.h), psi = spiky_psi(sp, g.h);
            float u[3] = {0.f, 0.f, 0.f}, ru = 0.f;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                u[d] = mi * __ldg(a.g_dg + (long long)j * D + d) - mj * gdi[d];
                ru = fmaf(rv[d], u[d], ru);
            }
            const float s = psi * ru;
#pragma unroll
            for (int d = 0; d < D; ++d) dxg[d] += phi * u[d] - s * rv[d];
        }
    };

    const int32_t *row = a.pair_cache + (long long)i * a.pair_stride;
    const int count = ivalid ? __ldg(row) : 0;
    const bool vec = ((a.pair_stride & 3) | ((uintptr_t)a.pair_cache & 15)) == 0;
    for (int w = sl * 4; w <= count; w += LPP * 4) {  // words w..w+3 of the row; word 0 is the count
        int j[4];
        if (vec) {
            const int4 t = __ldg(reinterpret_cast<const int4 *>(row + w));
            j[0] = t.x; j[1] = t.y; j[2] = t.z; j[3] = t.w;
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) j[u] = w + u <= count ? __ldg(row + w + u) : 0;
        }
        float4 p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (w + u == 0 || w + u > count) j[u] = i;  // the self pair adds nothing
            p[u] = record(j[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            float rx, ry, rz;
            listed_displacement<D, PER>(g, pi, Pos<D>{p[u].x, p[u].y, p[u].z}, rx, ry, rz);
            visit(j[u], p[u].w, rx, ry, rz, sq_norm_fast<D>(rx, ry, rz));
        }
    }
    if (count < 0) {  // the list overflowed: the four lanes search the cells
        SubgroupSearch<D, PER, LPP> search;
        search.begin(g, a.bin_offsets, i, pi);
        while (search.more(g, pi)) {
            const int j = search.j + sl;
            if (j < search.end) {
                const float4 p = record(j);
                float rx, ry, rz;
                const float q = displacement<D, PER, false>(g, search.org, p.x, p.y, p.z, rx, ry, rz);
                if (q < g.h2) visit(j, p.w, rx, ry, rz, q);
            }
            search.j += LPP;
        }
    }
    __syncwarp();
    float out[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < D; ++d) out[d] = subgroup_sum<LPP>(g.c_s * dxs[d] + g.c_g * dxg[d]);
    if (ivalid && sl == 0) {
        if (D == 2) {
            float2 *o = reinterpret_cast<float2 *>(a.grad_x) + i;
            float2 v = make_float2(out[0], out[1]);
            if (a.accumulate_x) { const float2 p = *o; v.x += p.x; v.y += p.y; }
            *o = v;
        } else {
            float4 *o = reinterpret_cast<float4 *>(a.grad_x) + i;
            float4 v = make_float4(out[0], out[1], out[2], 0.f);
            if (a.accumulate_x) { const float4 p = *o; v.x += p.x; v.y += p.y; v.z += p.z; }
            *o = v;
        }
    }
}

template <int D, bool PER>
static int launch_scalar_list_geom(const Geom &g, const ScalarListArgs &a, cudaStream_t st) {
    const int mask = ((a.g_rho_a || a.g_rho_b || a.pg) ? S_DENSITY : 0) | (a.g_dg ? S_DGRAD : 0);
    const long long threads = 4ll * g.B * g.N;
    const unsigned blocks = (unsigned)((threads + 255) / 256);
    switch (mask) {
        case S_DENSITY: launch_early(scalar_list_backward_kernel<D, PER, S_DENSITY>, blocks, 256, 0, st, a, g); break;
        case S_DGRAD: launch_early(scalar_list_backward_kernel<D, PER, S_DGRAD>, blocks, 256, 0, st, a, g); break;
        default: launch_early(scalar_list_backward_kernel<D, PER, S_DENSITY | S_DGRAD>, blocks, 256, 0, st, a, g); break;
    }
    return check_launch("scalar_list_backward_kernel");
}

int launch_scalar_list_backward(const Geom &g, const ScalarListArgs &a, cudaStream_t st) {
    if (g.dim == 2) return g.periodic ? launch_scalar_list_geom<2, true>(g, a, st) : launch_scalar_list_geom<2, false>(g, a, st);
    return g.periodic ? launch_scalar_list_geom<3, true>(g, a, st) : launch_scalar_list_geom<3, false>(g, a, st);
}

// ---------------------------------------------------------------------------------------------------------
// Density gradient over lists: eight lanes per particle.  The sums meet in the order of the feature sweep that carries
// the density gradient along (lane partials over entries with equal entry mod 8), so both give the same bits for up to
// 32 features.
// ---------------------------------------------------------------------------------------------------------
template <int D, bool PER>
__global__ void __launch_bounds__(256)
density_gradient_list_kernel(ScalarListArgs a, Geom g) {
    after_previous_kernel();
    constexpr int LPP = 8;
    const int lane = threadIdx.x & 31, sl = lane % LPP;
    const int total = g.B * g.N;
    const unsigned at = blockIdx.x * (256u / LPP) + threadIdx.x / LPP;  // below 2^31 + 256 / LPP
    if (at - lane / LPP >= (unsigned)total) return;
    const bool ivalid = at < (unsigned)total;
    const int i = ivalid ? (int)at : total - 1;
    const Pos<D> pi = load_pos<D>(a.x, i);
    float dg[3] = {0.f, 0.f, 0.f};
    auto visit = [&](int j, float rx, float ry, float rz) {
        const float q = sq_norm_fast<D>(rx, ry, rz);
        if (!(q > 0.f)) return;
        const Spiky sp = spiky_distance(q);
        const float md = (a.mass ? __ldg(a.mass + j) : 1.0f) * spiky_phi(sp, g.h);
        dg[0] = fmaf(md, rx, dg[0]);
        dg[1] = fmaf(md, ry, dg[1]);
        if (D == 3) dg[2] = fmaf(md, rz, dg[2]);
    };
    const int32_t *row = a.pair_cache + (long long)i * a.pair_stride;
    const int count = ivalid ? __ldg(row) : 0;
    for (int e = sl; e < count; e += LPP) {
        const int j = __ldg(row + 1 + e);
        float rx, ry, rz;
        listed_displacement<D, PER>(g, pi, load_pos<D>(a.x, j), rx, ry, rz);
        visit(j, rx, ry, rz);
    }
    if (count < 0) {
        SubgroupSearch<D, PER, LPP> search;
        search.begin(g, a.bin_offsets, i, pi);
        while (search.more(g, pi)) {
            const int j = search.j + sl;
            if (j < search.end) {
                const Pos<D> p = load_pos<D>(a.x, j);
                float rx, ry, rz;
                if (displacement<D, PER, false>(g, search.org, p.x, p.y, p.z, rx, ry, rz) < g.h2) visit(j, rx, ry, rz);
            }
            search.j += LPP;
        }
    }
    __syncwarp();
#pragma unroll
    for (int d = 0; d < D; ++d) dg[d] = g.c_g * subgroup_sum<LPP>(dg[d]);
    if (ivalid && sl == 0) {
#pragma unroll
        for (int d = 0; d < D; ++d) a.rho_grad_out[(long long)i * D + d] = dg[d];
    }
}

int launch_density_gradient_list(const Geom &g, const ScalarListArgs &a, cudaStream_t st) {
    const unsigned blocks = (unsigned)((8ll * g.B * g.N + 255) / 256);
    if (g.dim == 2) {
        if (g.periodic) launch_early(density_gradient_list_kernel<2, true>, blocks, 256, 0, st, a, g);
        else launch_early(density_gradient_list_kernel<2, false>, blocks, 256, 0, st, a, g);
    } else {
        if (g.periodic) launch_early(density_gradient_list_kernel<3, true>, blocks, 256, 0, st, a, g);
        else launch_early(density_gradient_list_kernel<3, false>, blocks, 256, 0, st, a, g);
    }
    return check_launch("density_gradient_list_kernel");
}

// ---------------------------------------------------------------------------------------------------------
// Upstream gradients of a caller, [N, C] and [N, C, D], as the rows the feature backward reads: [N, (1 +) D, cp], the
// axis in front of the features.  One thread per particle and four features; HBM bound (read once, written once).
// ---------------------------------------------------------------------------------------------------------
template <int D, bool VEC>
__global__ void __launch_bounds__(256)
upstream_rows_kernel(const float *__restrict__ g_blur, const float *__restrict__ g_grad, float *__restrict__ rows, long long total, int C, int cp,
                     int with_blur) {
    after_previous_kernel();
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    const int quads = cp / 4;
    if (t >= total * quads) return;
    const long long i = t / quads;
    const int f = (int)(t - i * quads) * 4;
    float *out = rows + i * (long long)((with_blur + (g_grad ? D : 0)) * cp) + f;
    if (with_blur) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        const float *b = g_blur + i * C + f;
        if (VEC) {
            v = __ldg(reinterpret_cast<const float4 *>(b));
        } else {
            if (f < C) v.x = __ldg(b);
            if (f + 1 < C) v.y = __ldg(b + 1);
            if (f + 2 < C) v.z = __ldg(b + 2);
            if (f + 3 < C) v.w = __ldg(b + 3);
        }
        *reinterpret_cast<float4 *>(out) = v;
        out += cp;
    }
    if (g_grad) {
        const float *b = g_grad + (i * C + f) * D;
        float v[4 * D];
        if (VEC) {
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const float4 q = __ldg(reinterpret_cast<const float4 *>(b) + k);
                v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4 * D; ++k) v[k] = f + k / D < C ? __ldg(b + k) : 0.f;
        }
#pragma unroll
        for (int d = 0; d < D; ++d) *reinterpret_cast<float4 *>(out + d * cp) = make_float4(v[d], v[D + d], v[2 * D + d], v[3 * D + d]);
    }
}

int launch_upstream_rows(const Geom &g, int C, const float *g_blur, const float *g_grad, bool with_blur, float *rows, cudaStream_t st) {
    const long long total = (long long)g.B * g.N;
    const int cp = (C + 3) & ~3;
    const unsigned blocks = (unsigned)((total * (cp / 4) + 255) / 256);
    const bool vec = C % 4 == 0 && (((uintptr_t)g_grad | (with_blur ? (uintptr_t)g_blur : 0)) % 16) == 0;
    const int wb = with_blur ? 1 : 0;
    if (g.dim == 2) {
        if (vec) launch_early(upstream_rows_kernel<2, true>, blocks, 256, 0, st, g_blur, g_grad, rows, total, C, cp, wb);
        else launch_early(upstream_rows_kernel<2, false>, blocks, 256, 0, st, g_blur, g_grad, rows, total, C, cp, wb);
    } else {
        if (vec) launch_early(upstream_rows_kernel<3, true>, blocks, 256, 0, st, g_blur, g_grad, rows, total, C, cp, wb);
        else launch_early(upstream_rows_kernel<3, false>, blocks, 256, 0, st, g_blur, g_grad, rows, total, C, cp, wb);
    }
    return check_launch("upstream_rows_kernel");
}

// ---------------------------------------------------------------------------------------------------------
// dispatch of the feature kernels over the four geometries
// ---------------------------------------------------------------------------------------------------------
#define NPA_EXTERN(D, P)                                                                                            \
    extern template int launch_feature_list_forward_geom<D, P>(const Geom &, int, const FeatureFwdArgs &, cudaStream_t); \
    extern template int launch_feature_list_backward_geom<D, P, true>(const Geom &, int, const FeatureListBwdArgs &, cudaStream_t); \
    extern template int launch_feature_list_backward_geom<D, P, false>(const Geom &, int, const FeatureListBwdArgs &, cudaStream_t);
NPA_EXTERN(2, false) NPA_EXTERN(2, true) NPA_EXTERN(3, false) NPA_EXTERN(3, true)
#undef NPA_EXTERN

int launch_feature_list_forward(const Geom &g, int mask, const FeatureFwdArgs &a, cudaStream_t st) {
    if (g.dim == 2)
        return g.periodic ? launch_feature_list_forward_geom<2, true>(g, mask, a, st) : launch_feature_list_forward_geom<2, false>(g, mask, a, st);
    return g.periodic ? launch_feature_list_forward_geom<3, true>(g, mask, a, st) : launch_feature_list_forward_geom<3, false>(g, mask, a, st);
}

int launch_feature_list_backward(const Geom &g, int mask, bool full, const FeatureListBwdArgs &a, cudaStream_t st) {
#define NPA_LB(DD, PP) \
    (full ? launch_feature_list_backward_geom<DD, PP, true>(g, mask, a, st) : launch_feature_list_backward_geom<DD, PP, false>(g, mask, a, st))
    if (g.dim == 2) return g.periodic ? NPA_LB(2, true) : NPA_LB(2, false);
    return g.periodic ? NPA_LB(3, true) : NPA_LB(3, false);
#undef NPA_LB
}

}  // namespace npa
