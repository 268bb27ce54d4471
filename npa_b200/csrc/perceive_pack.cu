// Packed perception: the whole per-step perception of an NPA model as two neighbour sweeps that
// write the MLP input row directly, and its backward.
//
// NPA.perceive (models/npa.py:87-137) computes density, blur, the moment-corrected feature
// gradient (gradient_hybrid, sphops/sph.py:474-484: raw @ safe_inv(M) with the gradient of the
// raw operator), the density gradient, then scales by eps/eps0, log-normalises the two gradient
// features and concatenates everything into z[B,N,2C+C*D+D] with a dozen torch kernels that each
// re-read the [B,N,C,D] gradient tensor.  Here sweep 2 applies that per-particle epilogue while
// the sums are still in registers (feature_kernels.cuh, F_PACK) and writes z once; backward turns
// dL/dz into the upstream gradients of blur / gradient / density gradient with one elementwise
// kernel and then runs the ordinary fused backward sweeps.  (In a step whose positions want no gradient
// the product that makes dL/dz writes them: launch_step_rows.)
#include "perceive_backward.cuh"

namespace npa {

// One thread per (particle, feature): dL/dz -> dL/dblur, dL/dgrad; the thread of feature 0 also
// handles the density-gradient part.  ROWS: the rows the backward over neighbour lists reads, blur and the D
// axes of the gradient as cp floats each, `pitch` floats per particle (g_blur = the rows, g_grad unused, columns C..cp-1 zero); otherwise the
// operators' own layouts.
template <int D, bool ROWS>
__global__ void __launch_bounds__(256)
pack_backward_kernel(const float *__restrict__ gz, const float *__restrict__ vgrad, const float *__restrict__ rho_grad,
                     float *__restrict__ g_blur, float *__restrict__ g_grad, float *__restrict__ g_rho_grad,
                     long long particles, int C, int pitch, float coef, float dg_scale, int log_norm_grad, int log_norm_dg) {
    after_previous_kernel();
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    const int cp = ROWS ? (C + 3) & ~3 : C;
    if (t >= particles * cp) return;
    const long long i = t / cp;
    const int f = (int)(t - i * cp);
    const int Z = 2 * C + C * D + D;
    const float *gr = gz + i * Z;
    float *row = ROWS ? g_blur + i * pitch + f : nullptr;
    if (ROWS && f >= C) {
#pragma unroll
        for (int d = 0; d <= D; ++d) row[d * cp] = 0.f;
        return;
    }
    if (ROWS) row[0] = gr[C + f];
    else g_blur[t] = gr[C + f];
    float w[D], gin[D], gout[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
        w[d] = vgrad[(i * C + f) * D + d] * coef;
        gin[d] = gr[2 * C + f * D + d];
    }
    log_normalize_backward<D>(w, gin, log_norm_grad, coef, gout);
#pragma unroll
    for (int d = 0; d < D; ++d) {
        if (ROWS) row[(1 + d) * cp] = gout[d];
        else g_grad[t * D + d] = gout[d];
    }
    if (f == 0 && g_rho_grad) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            w[d] = rho_grad[i * D + d] * dg_scale;
            gin[d] = gr[2 * C + C * D + d];
        }
        log_normalize_backward<D>(w, gin, log_norm_dg, dg_scale, gout);
#pragma unroll
        for (int d = 0; d < D; ++d) g_rho_grad[i * D + d] = gout[d];
    }
}

// grad_s[i][f] += dL/dz[i][f]: the features enter z unchanged as its first C columns.
__global__ void __launch_bounds__(256)
add_direct_kernel(const float *__restrict__ gz, float *__restrict__ grad_s, long long particles, int C, int Z) {
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    if (t >= particles * C) return;
    const long long i = t / C;
    grad_s[t] += gz[i * Z + (t - i * C)];
}

// Differences of root_rounded and quotient_rounded from CUDA's rounded intrinsics.
__global__ void __launch_bounds__(256)
rounding_selftest_kernel(uint32_t first, int step, int count, uint32_t seed, int32_t *__restrict__ mismatches) {
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k >= count) return;
    const float Q = __uint_as_float(first + (uint32_t)k * (uint32_t)step);
    const Root r = root_rounded(Q);
    const float want = __fsqrt_rn(Q);
    uint32_t u = ((uint32_t)k + 1u) * 2654435761u + seed * 40503u;  // scrambled: the mantissa and the exponent of the numerator
    u = (u ^ (u >> 15)) * 0x2c1b3c6du;
    u ^= u >> 12;
    const float n = __fmul_rn(__uint_as_float(0x3f800000u | (u >> 9)), ldexpf(want, (int)(u % 81u) - 40));
    if (r.d != want) atomicAdd(mismatches, 1);
    else if (quotient_rounded(n, r) != __fdiv_rn(n, want)) atomicAdd(mismatches + 1, 1);
}

}  // namespace npa

using namespace npa;

namespace npa {
template <int D, bool PER>
int launch_packed_ordered_geom(const Geom &g, const FeatureFwdArgs &a, cudaStream_t st);
extern template int launch_packed_ordered_geom<2, false>(const Geom &, const FeatureFwdArgs &, cudaStream_t);
extern template int launch_packed_ordered_geom<2, true>(const Geom &, const FeatureFwdArgs &, cudaStream_t);
extern template int launch_packed_ordered_geom<3, false>(const Geom &, const FeatureFwdArgs &, cudaStream_t);
extern template int launch_packed_ordered_geom<3, true>(const Geom &, const FeatureFwdArgs &, cudaStream_t);

static int launch_packed_ordered(const Geom &g, const FeatureFwdArgs &a, cudaStream_t st) {
    if (g.dim == 2) return g.periodic ? launch_packed_ordered_geom<2, true>(g, a, st) : launch_packed_ordered_geom<2, false>(g, a, st);
    return g.periodic ? launch_packed_ordered_geom<3, true>(g, a, st) : launch_packed_ordered_geom<3, false>(g, a, st);
}
}  // namespace npa

extern "C" {

int npa_perceive_features_forward_lists(const npa_grid *gd, int32_t channels, const float *x_bin, const float *mass,
                                        const float *s_bin, float coef, float dg_scale, float inv_tol,
                                        int32_t log_norm_grad, int32_t log_norm_dg, float *rho, float *rho_grad,
                                        float *z, float *vgrad, float *packed, const int32_t *bin_offsets, const int32_t *block_info,
                                        int32_t *pair_cache, int32_t pair_stride, void *stream) {
    Geom g;
    int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    if (!x_bin || !s_bin || !rho || !rho_grad || !z || !bin_offsets || !block_info)
        return fail(NPA_ERR_INVALID_ARGUMENT, "perceive_features_forward: a required pointer is NULL");
    if (channels <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "perceive_features_forward: channels must be positive");
    if (((uintptr_t)x_bin % (g.dim == 2 ? 8 : 16)) || ((uintptr_t)block_info % 16))
        return fail(NPA_ERR_INVALID_ARGUMENT, "perceive_features_forward: positions / block_info are misaligned");
    cudaStream_t st = (cudaStream_t)stream;
    if (pair_cache && (pair_stride < 2 || pair_stride > 513))
        return fail(NPA_ERR_INVALID_ARGUMENT, "perceive_features_forward: pair_stride must be in [2, 513]");
    // The packed sweep meets every pair with its spiky kernel value in hand, so it also sums the density
    // gradient; the first sweep is then the density alone (and the neighbour lists), which the shared-
    // candidate kernel runs in about half the time of the density + density-gradient sweep.  With the
    // cell-tile engine switched on (it has no such sum) the first sweep computes both as before.
    if (packed && ((uintptr_t)packed % 16 || !pair_cache))
        return fail(NPA_ERR_INVALID_ARGUMENT, "perceive_features_forward: packed must be 16-byte aligned and needs neighbour lists");
    const bool in_sweep = !tile_forward_enabled();
    // Over lists the sums have one fixed order, recorded for a backward or not: see density_ordered.cu.
    const bool ordered = pair_cache && in_sweep && channels <= 32;
    ScalarFwdArgs sa = {x_bin, mass, nullptr, nullptr, rho, in_sweep ? nullptr : rho_grad, nullptr, bin_offsets, block_info, pair_cache, pair_stride};
    sa.pv = reinterpret_cast<float4 *>(packed);
    rc = ordered && scalar_shared_search() ? launch_density_ordered(g, sa, st) : launch_scalar_forward(g, in_sweep ? S_DENSITY : (S_DENSITY | S_DGRAD), sa, st);
    if (rc != NPA_OK) return rc;
    FeatureFwdArgs fa = {x_bin, mass, rho, s_bin, nullptr, nullptr, channels, bin_offsets, block_info, nullptr};
    fa.z = z;
    fa.zstride = 2 * channels + channels * g.dim + g.dim;
    fa.vgrad = vgrad;
    fa.rho_grad = in_sweep ? nullptr : rho_grad;
    fa.rho_grad_out = in_sweep ? rho_grad : nullptr;
    fa.coef = coef;
    fa.dg_scale = dg_scale;
    fa.inv_tol = inv_tol;
    fa.log_norm_grad = log_norm_grad;
    fa.log_norm_dg = log_norm_dg;
    fa.pv = sa.pv;
    fa.pair_cache = pair_cache;
    fa.pair_stride = pair_stride;
    fa.pair_cache_valid = pair_cache != nullptr;  // written by the density sweep above
    if (ordered) return launch_packed_ordered(g, fa, st);
    return launch_feature_forward(g, F_BLUR | F_GRAD | F_MOMENT | F_PACK, fa, st);
}

int npa_perceive_features_forward(const npa_grid *gd, int32_t channels, const float *x_bin, const float *mass,
                                  const float *s_bin, float coef, float dg_scale, float inv_tol,
                                  int32_t log_norm_grad, int32_t log_norm_dg, float *rho, float *rho_grad,
                                  float *z, float *vgrad, const int32_t *bin_offsets, const int32_t *block_info,
                                  int32_t *pair_cache, int32_t pair_stride, void *stream) {
    return npa_perceive_features_forward_lists(gd, channels, x_bin, mass, s_bin, coef, dg_scale, inv_tol, log_norm_grad, log_norm_dg, rho,
                                               rho_grad, z, vgrad, nullptr, bin_offsets, block_info, pair_cache, pair_stride, stream);
}

int npa_rounding_selftest(uint32_t first_bits, int32_t step, int32_t count, uint32_t seed, int32_t *device_mismatches, void *stream) {
    if (!device_mismatches || step <= 0 || count <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "rounding_selftest: bad arguments");
    const int64_t last = (int64_t)first_bits + (int64_t)step * (count - 1);
    if (first_bits < (uint32_t)(127 - 66) << 23 || last >= (int64_t)(127 + 66) << 23)
        return fail(NPA_ERR_INVALID_ARGUMENT, "rounding_selftest: operands must lie in [2^-66, 2^66)");
    rounding_selftest_kernel<<<(unsigned)((count + 255) / 256), 256, 0, (cudaStream_t)stream>>>(first_bits, step, count, seed, device_mismatches);
    return check_launch("rounding_selftest_kernel");
}

int64_t npa_lists_backward_scratch_bytes(const npa_grid *gd, int32_t channels) {
    Geom g;
    const int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    if (channels < 0) return fail(NPA_ERR_INVALID_ARGUMENT, "lists_backward_scratch_bytes: channels must not be negative");
    // upstream rows, the density gradient's upstream (rounded up to whole 16-byte records), position + upstream records
    const int64_t n = (int64_t)g.B * g.N, cp = (channels + 3) & ~3;
    const int64_t lists = (1 + g.dim) * cp * 4 + 32, dense = feature_dense_pitch(g.dim, (int)cp) * 4;
    return n * (lists > dense ? lists : dense);
}

static int features_backward_lists(const char *me, const npa_grid *gd, int32_t channels, const float *x_bin, const float *mass,
                                   const float *s_bin, const float *rho, const float *rho_grad, const float *vgrad,
                                   const float *packed, const float *dL_dz, float coef, float dg_scale, int32_t log_norm_grad,
                                   int32_t log_norm_dg, const float *grad_s_add, float *grad_x, float *grad_s, void *scratch,
                                   int64_t scratch_bytes, const int32_t *bin_offsets, const int32_t *pair_cache, int32_t pair_stride, bool binned,
                                   void *stream, const float *dh = nullptr, const void *image = nullptr, int64_t image_bytes = 0) {
    Geom g;
    int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    if (!x_bin || !s_bin || !rho || (!rho_grad && !dh) || !vgrad || (!dL_dz && !dh) || !scratch || !bin_offsets || !pair_cache)
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: a required pointer is NULL", me);
    if (channels <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: channels must be positive", me);
    if (((uintptr_t)x_bin | (uintptr_t)grad_x) % (g.dim == 2 ? 8 : 16) || ((uintptr_t)scratch | (uintptr_t)packed) % 16)
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: positions, packed or scratch are misaligned", me);
    if (pair_stride < 2 || pair_stride > 513) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: pair_stride must be in [2, 513]", me);
    if (scratch_bytes < npa_lists_backward_scratch_bytes(gd, channels))
        return fail(NPA_ERR_SCRATCH_TOO_SMALL, "%s: scratch holds %lld bytes, %lld needed", me, (long long)scratch_bytes,
                    (long long)npa_lists_backward_scratch_bytes(gd, channels));
    if (!grad_x && !grad_s) return NPA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const long long n = (long long)g.B * g.N;
    const int cp = (channels + 3) & ~3;
    const bool dense = binned && packed && !grad_x && feature_dense_covers(g, channels);
    const int pitch = dense ? feature_dense_pitch(g.dim, cp) : (1 + g.dim) * cp;
    float *rows = static_cast<float *>(scratch), *g_dg = rows + n * pitch;
    float4 *pg = reinterpret_cast<float4 *>(g_dg + n * 4);
    const unsigned blocks = (unsigned)((n * cp + 255) / 256);
    // dh: dL/dz has not been formed; its product's epilogue writes the rows (and the features' own part where the density gradient's
    // upstream and the records would lie)
    if (dh) {
        const StepRows out = {vgrad, g_dg, rows, pitch, channels, g.dim, coef, log_norm_grad};
        if ((rc = launch_step_rows(out, dh, n, image, image_bytes, st)) != NPA_OK) return rc;
    } else if (g.dim == 2)
        launch_early(pack_backward_kernel<2, true>, blocks, 256, 0, st, dL_dz, vgrad, rho_grad, rows, nullptr, grad_x ? g_dg : nullptr, n, channels, pitch, coef,
                                                              dg_scale, log_norm_grad, log_norm_dg);
    else
        launch_early(pack_backward_kernel<3, true>, blocks, 256, 0, st, dL_dz, vgrad, rho_grad, rows, nullptr, grad_x ? g_dg : nullptr, n, channels, pitch, coef,
                                                              dg_scale, log_norm_grad, log_norm_dg);
    if ((rc = check_launch("pack_backward_kernel")) != NPA_OK) return rc;
    FeatureListBwdArgs a = {};
    a.x = x_bin; a.mass = mass; a.rho = rho; a.s = s_bin; a.pv = reinterpret_cast<const float4 *>(packed);
    a.gb = rows; a.gg = rows + cp; a.gb_pitch = a.gg_pitch = pitch; a.cp = cp;
    a.direct = dh ? g_dg : dL_dz; a.direct_pitch = dh ? channels : 2 * channels + channels * g.dim + g.dim;  // the features enter z unchanged as its first columns
    a.add = grad_s_add;
    a.g_dg = grad_x ? g_dg : nullptr;
    a.grad_x = grad_x; a.grad_s = grad_s; a.pg = grad_x ? pg : nullptr; a.C = channels;
    a.bin_offsets = bin_offsets; a.pair_cache = pair_cache; a.pair_stride = pair_stride;
    if (dense) return launch_feature_dense_backward(g, a, st);
    if ((rc = launch_feature_list_backward(g, F_BLUR | F_GRAD, grad_x != nullptr, a, st)) != NPA_OK || !grad_x) return rc;
    ScalarListArgs d = {};
    d.x = x_bin; d.mass = mass; d.pg = pg; d.grad_x = grad_x; d.accumulate_x = 1;
    d.bin_offsets = bin_offsets; d.pair_cache = pair_cache; d.pair_stride = pair_stride;
    return launch_scalar_list_backward(g, d, st);
}

int npa_perceive_features_backward_lists(const npa_grid *gd, int32_t channels, const float *x_bin, const float *mass,
                                         const float *s_bin, const float *rho, const float *rho_grad, const float *vgrad,
                                         const float *packed, const float *dL_dz, float coef, float dg_scale, int32_t log_norm_grad,
                                         int32_t log_norm_dg, const float *grad_s_add, float *grad_x, float *grad_s, void *scratch,
                                         int64_t scratch_bytes, const int32_t *bin_offsets, const int32_t *pair_cache, int32_t pair_stride, void *stream) {
    const char *me = "perceive_features_backward_lists";
    return features_backward_lists(me, gd, channels, x_bin, mass, s_bin, rho, rho_grad, vgrad, packed, dL_dz, coef, dg_scale, log_norm_grad, log_norm_dg, grad_s_add, grad_x, grad_s,
                                   scratch, scratch_bytes, bin_offsets, pair_cache, pair_stride, false, stream);
}

int npa_perceive_features_backward_binned(const npa_grid *gd, int32_t channels, const float *x_bin, const float *mass,
                                         const float *s_bin, const float *rho, const float *rho_grad, const float *vgrad,
                                         const float *packed, const float *dL_dz, float coef, float dg_scale, int32_t log_norm_grad,
                                         int32_t log_norm_dg, const float *grad_s_add, float *grad_x, float *grad_s, void *scratch,
                                         int64_t scratch_bytes, const int32_t *bin_offsets, const int32_t *pair_cache, int32_t pair_stride, void *stream) {
    const char *me = "perceive_features_backward_binned";
    return features_backward_lists(me, gd, channels, x_bin, mass, s_bin, rho, rho_grad, vgrad, packed, dL_dz, coef, dg_scale, log_norm_grad, log_norm_dg, grad_s_add, grad_x, grad_s,
                                   scratch, scratch_bytes, bin_offsets, pair_cache, pair_stride, true, stream);
}

int64_t npa_step_perceive_backward_scratch_bytes(const npa_grid *gd, int32_t channels) {
    const int64_t bytes = npa_lists_backward_scratch_bytes(gd, channels);
    return bytes < 0 ? bytes : bytes + (int64_t)gd->batch * gd->particles * channels * 4;
}

int npa_step_perceive_backward(const npa_grid *gd, int32_t channels, const float *dh, const void *rows_image, int64_t rows_image_bytes,
                               const float *x_bin, const float *s_bin, const float *rho, const float *vgrad, const float *packed, float coef,
                               int32_t log_norm_grad, const float *grad_s_add, float *grad_s, void *scratch, int64_t scratch_bytes,
                               const int32_t *bin_offsets, const int32_t *pair_cache, int32_t pair_stride, void *stream) {
    const char *me = "step_perceive_backward";
    if (!step_rows_cover(channels)) return fail(NPA_ERR_UNSUPPORTED, "%s: supports multiples of four up to 32 features, got %d", me, channels);
    if (!dh || !rows_image || !grad_s) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: a required pointer is NULL", me);
    const int64_t need = npa_step_perceive_backward_scratch_bytes(gd, channels);
    if (need < 0) return (int)need;
    if (scratch_bytes < need)
        return fail(NPA_ERR_SCRATCH_TOO_SMALL, "%s: scratch holds %lld bytes, %lld needed", me, (long long)scratch_bytes, (long long)need);
    return features_backward_lists(me, gd, channels, x_bin, nullptr, s_bin, rho, nullptr, vgrad, packed, nullptr, coef, 0.f, log_norm_grad, 0, grad_s_add, nullptr,
                                   grad_s, scratch, scratch_bytes, bin_offsets, pair_cache, pair_stride, true, stream, dh, rows_image, rows_image_bytes);
}

int npa_perceive_features_backward(const npa_grid *gd, int32_t channels, const float *x_bin, const float *mass,
                                   const float *s_bin, const float *rho, const float *rho_grad,
                                   const float *vgrad, const float *dL_dz, float coef, float dg_scale,
                                   int32_t log_norm_grad, int32_t log_norm_dg, float *g_blur_scratch,
                                   float *g_grad_scratch, float *g_rho_grad_scratch, float *grad_rho_scratch,
                                   float *grad_x, float *grad_s, const int32_t *bin_offsets,
                                   const int32_t *block_info, const int32_t *pair_cache, int32_t pair_stride,
                                   void *stream) {
    Geom g;
    int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    if (!x_bin || !s_bin || !rho || !rho_grad || !vgrad || !dL_dz || !g_blur_scratch || !g_grad_scratch)
        return fail(NPA_ERR_INVALID_ARGUMENT, "perceive_features_backward: a required pointer is NULL");
    if (grad_x && (!g_rho_grad_scratch || !grad_rho_scratch))
        return fail(NPA_ERR_INVALID_ARGUMENT, "perceive_features_backward: grad_x needs g_rho_grad_scratch and grad_rho_scratch");
    if (channels <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "perceive_features_backward: channels must be positive");
    if (!grad_x && !grad_s) return NPA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const long long particles = (long long)g.B * g.N;
    const unsigned blocks = (unsigned)((particles * channels + 255) / 256);
    float *grg = grad_x ? g_rho_grad_scratch : nullptr;
    if (g.dim == 2)
        launch_early(pack_backward_kernel<2, false>, blocks, 256, 0, st, dL_dz, vgrad, rho_grad, g_blur_scratch, g_grad_scratch, grg,
                                                        particles, channels, 0, coef, dg_scale, log_norm_grad, log_norm_dg);
    else
        launch_early(pack_backward_kernel<3, false>, blocks, 256, 0, st, dL_dz, vgrad, rho_grad, g_blur_scratch, g_grad_scratch, grg,
                                                        particles, channels, 0, coef, dg_scale, log_norm_grad, log_norm_dg);
    if ((rc = check_launch("pack_backward_kernel")) != NPA_OK) return rc;
    rc = npa_perception_backward(gd, channels, x_bin, mass, s_bin, rho, nullptr, g_blur_scratch, g_grad_scratch, grg,
                                 grad_x, grad_s, grad_rho_scratch, bin_offsets, block_info, pair_cache, pair_stride, stream);
    if (rc != NPA_OK) return rc;
    if (grad_s) {
        add_direct_kernel<<<blocks, 256, 0, st>>>(dL_dz, grad_s, particles, channels,
                                                  2 * channels + channels * g.dim + g.dim);
        rc = check_launch("add_direct_kernel");
    }
    return rc;
}

}  // extern "C"
