// Per-particle scalar SPH operators: count, density, density gradient and
// moment matrix, forward and backward, on the warp-per-work-item neighbour
// walk of neighbors.cuh.  Any subset of the four runs fused in one sweep.
//
// Replaces forward_kernel / backward_kernel of the reference for the
// Count, Density, DensityGradient and MomentMatrix computation types
// (sphops/sph_cuda.cu:1418-1812 and 723-1416; pair math at :1160-1184,
// :1236-1264, :1328-1375).  The backward is a gather: particle i accumulates
// the terms of both roles it plays in a pair, so no global atomics are needed.
// The forward sweep can also record each particle's accepted neighbours (the
// neighbour-list cache) so that later sweeps of the same snapshot skip the search.
#include "neighbors.cuh"
#include "ops.cuh"

namespace npa {

// dK/dr applied to u:  J u = phi u - psi (r.u) r.
template <int D>
__device__ inline void apply_jacobian(float phi, float psi, float rx, float ry, float rz,
                                      float ux, float uy, float uz, float &ox, float &oy, float &oz) {
    float ru = rx * ux + ry * uy;
    if (D == 3) ru = fmaf(rz, uz, ru);
    const float s = psi * ru;
    ox = phi * ux - s * rx;
    oy = phi * uy - s * ry;
    oz = D == 3 ? phi * uz - s * rz : 0.f;
}

constexpr int kScalarLpp = 4;                // lanes per particle
constexpr int kScalarPpw = 32 / kScalarLpp;  // particles per warp pass
constexpr unsigned kScalarSubMask = (1u << kScalarLpp) - 1u;

// One warp per work item (several warps share an item when items are scarce).  The warp handles 8
// particles of the item per pass: each particle has a sub-group of 4 lanes that split its
// candidates, every lane adds the contribution of its own accepted pair, and a sub-group shuffle
// reduction yields the sums.  Eight independent particles per warp keep many loads in flight.
// The sweep can record the accepted pairs of each particle (in candidate order) in the
// neighbour-list cache for the sweeps that follow.
template <int D, bool PER, int MASK>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
scalar_forward_kernel(ScalarFwdArgs a, Geom g) {
    __shared__ int4 s_ranges[kWarpsPerCta][kMaxRanges];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int4 *rng = s_ranges[warp];
    const int sub = lane / kScalarLpp, sl = lane % kScalarLpp;
    constexpr bool kSpiky = (MASK & (S_DGRAD | S_MOMENT)) != 0;
    constexpr bool kPoly = (MASK & S_DENSITY) != 0;
    constexpr int kSym = D * (D + 1) / 2;
    const int K = a.pair_stride;

    const int vrows = g.max_blocks * g.split;
    for (int vrow = next_row(a.tickets); vrow < vrows; vrow = next_row(a.tickets)) {
        const int row = vrow / g.split, part = vrow - row * g.split;
        const WorkItem it = load_item(a.block_info, a.bin_offsets, row);
        if (it.count <= 0) break;  // rows after the last work item are zero
        if (part * kScalarPpw >= it.count) continue;
        __syncwarp();
        const int nr = build_ranges<D>(g, a.bin_offsets, it, rng);

        for (int k0 = part * kScalarPpw; k0 < it.count; k0 += g.split * kScalarPpw) {
            const int k = k0 + sub;
            const bool ivalid = k < it.count;
            const long long i = it.first + (ivalid ? k : 0);
            const Pos<D> pi = load_pos<D>(a.x, i);
            int32_t *list = a.pair_cache ? a.pair_cache + i * K + 1 : nullptr;
            float cnt = 0.f, rho = 0.f, dg[3] = {0.f, 0.f, 0.f}, mom[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            int listed = 0;
            for (int r = 0; r < nr; ++r) {
                const int4 rg = rng[r];
                const Origin<D, PER> org = make_origin<D, PER>(g, pi.x, pi.y, pi.z, rg.z);
                for (int j0 = rg.x; j0 < rg.y; j0 += kScalarLpp) {
                    const int j = j0 + sl;
                    float rx = 0.f, ry = 0.f, rz = 0.f, q = 0.f;
                    bool acc = false;
                    if (ivalid && j < rg.y) {
                        const Pos<D> pj = load_pos<D>(a.x, j);
                        q = displacement<D, PER>(g, org, pj.x, pj.y, pj.z, rx, ry, rz);
                        acc = q < g.h2;
                    }
                    if (list) {  // warp-uniform
                        const unsigned bits = (__ballot_sync(kFull, acc) >> (sub * kScalarLpp)) & kScalarSubMask;
                        const int pos = listed + __popc(bits & ((1u << sl) - 1u));
                        if (acc && pos < K - 1) list[pos] = j;
                        listed += __popc(bits);
                    }
                    if (!acc) continue;
                    if (MASK & S_COUNT) cnt += 1.0f;
                    const float mj = (kPoly || kSpiky) ? (a.mass ? __ldg(a.mass + j) : 1.0f) : 0.f;
                    if (kPoly) {
                        const float t = fmaxf(g.h2 - q, 0.f);
                        rho = fmaf(mj, t * t * t, rho);
                    }
                    if (kSpiky && q > 0.f) {
                        const Spiky sp = spiky_distance(q);
                        const float phi = spiky_phi(sp, g.h);
                        if (MASK & S_DGRAD) {
                            const float w = mj * phi;
                            dg[0] = fmaf(w, rx, dg[0]);
                            dg[1] = fmaf(w, ry, dg[1]);
                            if (D == 3) dg[2] = fmaf(w, rz, dg[2]);
                        }
                        if (MASK & S_MOMENT) {
                            const float w = phi * mj / __ldg(a.rho_in + j);
                            mom[0] = fmaf(w * rx, rx, mom[0]);
                            mom[1] = fmaf(w * rx, ry, mom[1]);
                            if (D == 2) {
                                mom[2] = fmaf(w * ry, ry, mom[2]);
                            } else {
                                mom[2] = fmaf(w * rx, rz, mom[2]);
                                mom[3] = fmaf(w * ry, ry, mom[3]);
                                mom[4] = fmaf(w * ry, rz, mom[4]);
                                mom[5] = fmaf(w * rz, rz, mom[5]);
                            }
                        }
                    }
                }
            }
            if (MASK & S_COUNT) cnt = subgroup_sum<kScalarLpp>(cnt);
            if (kPoly) rho = subgroup_sum<kScalarLpp>(rho);
            if (MASK & S_DGRAD) {
#pragma unroll
                for (int d = 0; d < D; ++d) dg[d] = subgroup_sum<kScalarLpp>(dg[d]);
            }
            if (MASK & S_MOMENT) {
#pragma unroll
                for (int d = 0; d < kSym; ++d) mom[d] = subgroup_sum<kScalarLpp>(mom[d]);
            }
            if (ivalid && sl == 0) {
                if (list) list[-1] = listed <= K - 1 ? listed : -1;
                if ((MASK & S_COUNT) && a.count) a.count[i] = cnt;
                if (kPoly && a.rho_out) {
                    const float r = g.c_s * rho;
                    a.rho_out[i] = r;
                    if (a.pv) a.pv[i] = make_float4(pi.x, pi.y, pi.z, (a.mass ? __ldg(a.mass + i) : 1.0f) / r);
                }
                if ((MASK & S_DGRAD) && a.rho_grad) {
#pragma unroll
                    for (int d = 0; d < D; ++d) a.rho_grad[i * D + d] = g.c_g * dg[d];
                }
                if ((MASK & S_MOMENT) && a.moment) {
                    float *o = a.moment + i * (D * D);
                    if (D == 2) {
                        reinterpret_cast<float4 *>(o)[0] =
                            make_float4(g.c_g * mom[0], g.c_g * mom[1], g.c_g * mom[1], g.c_g * mom[2]);
                    } else {
                        o[0] = g.c_g * mom[0]; o[1] = g.c_g * mom[1]; o[2] = g.c_g * mom[2];
                        o[3] = g.c_g * mom[1]; o[4] = g.c_g * mom[3]; o[5] = g.c_g * mom[4];
                        o[6] = g.c_g * mom[2]; o[7] = g.c_g * mom[4]; o[8] = g.c_g * mom[5];
                    }
                }
            }
        }
    }
    release_rows(a.tickets);
}

// Gather backward of density / density gradient / moment matrix by the cell search, same layout (8
// particles per warp pass, 4 lanes each); over neighbour lists it is scalar_list.cu.
template <int D, bool PER, int MASK>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
scalar_backward_kernel(ScalarBwdArgs a, Geom g) {
    __shared__ int4 s_ranges[kWarpsPerCta][kMaxRanges];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int4 *rng = s_ranges[warp];
    const int sub = lane / kScalarLpp, sl = lane % kScalarLpp;
    constexpr bool kSpiky = (MASK & (S_DGRAD | S_MOMENT)) != 0;
    constexpr int DD = D * D;

    const int vrows = g.max_blocks * g.split;
    for (int vrow = next_row(a.tickets); vrow < vrows; vrow = next_row(a.tickets)) {
        const int row = vrow / g.split, part = vrow - row * g.split;
        const WorkItem it = load_item(a.block_info, a.bin_offsets, row);
        if (it.count <= 0) break;
        if (part * kScalarPpw >= it.count) continue;
        __syncwarp();
        const int nr = build_ranges<D>(g, a.bin_offsets, it, rng);

        for (int k0 = part * kScalarPpw; k0 < it.count; k0 += g.split * kScalarPpw) {
            const int k = k0 + sub;
            const bool ivalid = k < it.count;
            const long long i = it.first + (ivalid ? k : 0);
            const Pos<D> pi = load_pos<D>(a.x, i);
            const float mi = a.mass ? __ldg(a.mass + i) : 1.0f;
            float gri = 0.f, gdi[3] = {0.f, 0.f, 0.f}, gmi[DD], vi = 0.f;
            if (MASK & S_DENSITY) {
                if (a.g_rho_a) gri += __ldg(a.g_rho_a + i);
                if (a.g_rho_b) gri += __ldg(a.g_rho_b + i);
            }
            if (MASK & S_DGRAD) {
#pragma unroll
                for (int d = 0; d < D; ++d) gdi[d] = __ldg(a.g_rho_grad + i * D + d);
            }
            if (MASK & S_MOMENT) {
#pragma unroll
                for (int d = 0; d < DD; ++d) gmi[d] = __ldg(a.g_moment + i * DD + d);
                vi = mi / __ldg(a.rho_in + i);
            }
            float dxs[3] = {0.f, 0.f, 0.f};  // poly6 part, scaled by c_s at the end
            float dxg[3] = {0.f, 0.f, 0.f};  // spiky part, scaled by c_g at the end
            float drho = 0.f;

            // contribution of one pair (the self / coincident pair has zero gradient)
            auto visit = [&](long long j, float rx, float ry, float rz, float q) {
                if (!(q > 0.f)) return;
                const float rv[3] = {rx, ry, rz};
                const float mj = a.mass ? __ldg(a.mass + j) : 1.0f;
                if (MASK & S_DENSITY) {
                    float grj = 0.f;
                    if (a.g_rho_a) grj += __ldg(a.g_rho_a + j);
                    if (a.g_rho_b) grj += __ldg(a.g_rho_b + j);
                    const float t = fmaxf(g.h2 - q, 0.f);
                    const float w = 6.0f * t * t * (gri * mj + grj * mi);
#pragma unroll
                    for (int d = 0; d < D; ++d) dxs[d] = fmaf(w, rv[d], dxs[d]);
                }
                if (kSpiky) {
                    const Spiky sp = spiky_distance(q);
                    const float phi = spiky_phi(sp, g.h);
                    const float psi = spiky_psi(sp, g.h);
                    if (MASK & S_DGRAD) {
                        float u[3] = {0.f, 0.f, 0.f}, o[3];
#pragma unroll
                        for (int d = 0; d < D; ++d) u[d] = mi * __ldg(a.g_rho_grad + j * D + d) - mj * gdi[d];
                        apply_jacobian<D>(phi, psi, rv[0], rv[1], rv[2], u[0], u[1], u[2], o[0], o[1], o[2]);
#pragma unroll
                        for (int d = 0; d < D; ++d) dxg[d] += o[d];
                    }
                    if (MASK & S_MOMENT) {
                        const float vj = mj / __ldg(a.rho_in + j);
                        float w[3] = {0.f, 0.f, 0.f}, o[3];
                        float rr = 0.f;  // sum_ab gM_j[a,b] r_a r_b
#pragma unroll
                        for (int p = 0; p < D; ++p) {
                            float kc = 0.f;  // sum_b Cm[p,b] K_b
#pragma unroll
                            for (int b = 0; b < D; ++b) {
                                const float gj = __ldg(a.g_moment + j * DD + p * D + b);
                                const float cm = vj * gmi[p * D + b] + vi * gj;
                                kc = fmaf(cm, phi * rv[b], kc);
                                w[b] = fmaf(rv[p], cm, w[b]);
                                rr = fmaf(gj * rv[p], rv[b], rr);
                            }
                            dxg[p] -= kc;
                        }
                        apply_jacobian<D>(phi, psi, rv[0], rv[1], rv[2], w[0], w[1], w[2], o[0], o[1], o[2]);
#pragma unroll
                        for (int d = 0; d < D; ++d) dxg[d] -= o[d];
                        drho = fmaf(rr, phi, drho);
                    }
                }
            };

            for (int r = 0; r < nr; ++r) {
                const int4 rg = rng[r];
                const Origin<D, PER> org = make_origin<D, PER>(g, pi.x, pi.y, pi.z, rg.z);
                for (int j0 = rg.x; j0 < rg.y; j0 += kScalarLpp) {
                    const int j = j0 + sl;
                    if (!(ivalid && j < rg.y)) continue;
                    const Pos<D> pj = load_pos<D>(a.x, j);
                    float rx, ry, rz;
                    const float q = displacement<D, PER, false>(g, org, pj.x, pj.y, pj.z, rx, ry, rz);
                    if (q < g.h2) visit(j, rx, ry, rz, q);
                }
            }

            float out[3];
#pragma unroll
            for (int d = 0; d < D; ++d) out[d] = subgroup_sum<kScalarLpp>(g.c_s * dxs[d] + g.c_g * dxg[d]);
            if (MASK & S_MOMENT) drho = subgroup_sum<kScalarLpp>(drho);
            if (ivalid && sl == 0) {
                if (a.grad_x) {
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
                if ((MASK & S_MOMENT) && a.grad_rho) a.grad_rho[i] = -g.c_g * (vi * vi / mi) * drho;
            }
        }
    }
    release_rows(a.tickets);
}

// ---------------------------------------------------------------------------
// dispatch: persistent launches (every SM filled to the kernel's occupancy)
// ---------------------------------------------------------------------------
template <typename Kernel, typename Args>
static int launch_persistent(const Geom &g, Kernel kernel, const Args &a, cudaStream_t st, const char *what) {
    const int threads = kWarpsPerCta * 32;
    int ctas = 0;
    int rc = persistent_ctas(kernel, threads, 0, &ctas);
    if (rc != NPA_OK) return rc;
    const int needed = (g.max_blocks * g.split + kWarpsPerCta - 1) / kWarpsPerCta;
    Args b = a;
    if ((rc = acquire_row_tickets(st, &b.tickets)) != NPA_OK) return rc;
    kernel<<<needed < ctas ? needed : ctas, threads, 0, st>>>(b, g);
    return check_launch(what);
}

static bool g_shared_search = true;  // count / density by density_search.cu
void set_scalar_shared_search(bool on) { g_shared_search = on; }
bool scalar_shared_search() { return g_shared_search; }

// The count by the search that shares its candidates: not on Morton grids (its tiles are x-rows of cells), and not for few
// particles on a 3D periodic grid, where most tiles meet an edge of the box and test every pair with its own shifted origin
// (walk / search, ~40 neighbours: 4,096 particles 36 / 48 us, 16,384 48 / 57, 65,536 99 / 108, 131,072 139 / 142, 262,144
// 251 / 217; ~130: 65,536 231 / 201).
static bool count_by_search(const Geom &g) {
    return !g.morton && !(g.periodic && g.dim == 3 && (long long)g.B * g.N < 65536);
}

template <int MASK>
static int launch_scalar_fwd_mask(const Geom &g, const ScalarFwdArgs &a, cudaStream_t st) {
    // the count or the density alone: the search that shares its candidates between particles
    if ((MASK == S_DENSITY || (MASK == S_COUNT && count_by_search(g))) && g_shared_search)
        return launch_density_search(g, MASK == S_COUNT, a, st);
    const char *what = "scalar_forward_kernel";
    if (g.dim == 2) {
        if (g.periodic) return launch_persistent(g, scalar_forward_kernel<2, true, MASK>, a, st, what);
        return launch_persistent(g, scalar_forward_kernel<2, false, MASK>, a, st, what);
    }
    if (g.periodic) return launch_persistent(g, scalar_forward_kernel<3, true, MASK>, a, st, what);
    return launch_persistent(g, scalar_forward_kernel<3, false, MASK>, a, st, what);
}

int launch_scalar_forward(const Geom &g, int mask, const ScalarFwdArgs &a, cudaStream_t st) {
    switch (mask) {
        case S_COUNT: return launch_scalar_fwd_mask<S_COUNT>(g, a, st);
        case S_DENSITY: return launch_scalar_fwd_mask<S_DENSITY>(g, a, st);
        case S_DGRAD: return launch_scalar_fwd_mask<S_DGRAD>(g, a, st);
        case S_MOMENT: return launch_scalar_fwd_mask<S_MOMENT>(g, a, st);
        case S_DENSITY | S_DGRAD: return launch_scalar_fwd_mask<S_DENSITY | S_DGRAD>(g, a, st);
        default:
            if ((mask & ~(S_COUNT | S_DENSITY | S_DGRAD)) == 0)
                return launch_scalar_fwd_mask<S_COUNT | S_DENSITY | S_DGRAD>(g, a, st);
            return fail(NPA_ERR_INVALID_ARGUMENT, "unsupported scalar forward mask %d", mask);
    }
}

template <int MASK>
static int launch_scalar_bwd_mask(const Geom &g, const ScalarBwdArgs &a, cudaStream_t st) {
    const char *what = "scalar_backward_kernel";
    if (g.dim == 2) {
        if (g.periodic) return launch_persistent(g, scalar_backward_kernel<2, true, MASK>, a, st, what);
        return launch_persistent(g, scalar_backward_kernel<2, false, MASK>, a, st, what);
    }
    if (g.periodic) return launch_persistent(g, scalar_backward_kernel<3, true, MASK>, a, st, what);
    return launch_persistent(g, scalar_backward_kernel<3, false, MASK>, a, st, what);
}

int launch_scalar_backward(const Geom &g, int mask, const ScalarBwdArgs &a, cudaStream_t st) {
    switch (mask) {
        case S_DENSITY: return launch_scalar_bwd_mask<S_DENSITY>(g, a, st);
        case S_DGRAD: return launch_scalar_bwd_mask<S_DGRAD>(g, a, st);
        case S_MOMENT: return launch_scalar_bwd_mask<S_MOMENT>(g, a, st);
        case S_DENSITY | S_DGRAD: return launch_scalar_bwd_mask<S_DENSITY | S_DGRAD>(g, a, st);
        default: return fail(NPA_ERR_INVALID_ARGUMENT, "unsupported scalar backward mask %d", mask);
    }
}

}  // namespace npa
