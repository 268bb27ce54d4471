// Argument blocks and launch functions of the perception kernels; the glue
// between the C ABI (capi.cu) and the kernel translation units.
#pragma once
#include "common.cuh"

namespace npa {

// Which per-particle scalar operators a sweep computes.
enum { S_COUNT = 1, S_DENSITY = 2, S_DGRAD = 4, S_MOMENT = 8 };
// Which feature operators a sweep computes.
// F_MOMENT (forward only) adds the moment matrix to a blur + gradient sweep.
// F_PACK (forward only, with all three others) applies the perception epilogue per particle and
// writes the packed perception vector instead of the separate tensors.
// Over neighbour lists also: F_DGRAD sums the density gradient (rho_grad_out) and F_CORRECTED (with F_GRAD |
// F_MOMENT) writes gradient . safe_inv(moment) in place of the gradient.
enum { F_BLUR = 1, F_GRAD = 2, F_MOMENT = 4, F_PACK = 8, F_DGRAD = 16, F_CORRECTED = 32 };
bool tile_forward_enabled();  // tile_host.cu: the cell-tile streaming engine is switched on for forward sweeps

struct ScalarFwdArgs {
    const float *x;       // [B,N,P] cell order
    const float *mass;    // [B,N] or NULL (all ones)
    const float *rho_in;  // [B,N], only for S_MOMENT
    float *count;         // [B,N]
    float *rho_out;       // [B,N]
    float *rho_grad;      // [B,N,D]
    float *moment;        // [B,N,D,D]
    const int32_t *bin_offsets;
    const int32_t *block_info;
    int32_t *pair_cache;  // neighbour lists to write ([B*N, pair_stride]) or NULL
    int pair_stride;
    unsigned int *tickets;  // row tickets of this launch (set by the launcher)
    float4 *pv;             // [B*N] out: (x, y, z, m / rho), or NULL (S_DENSITY)
};

struct ScalarBwdArgs {
    const float *x;
    const float *mass;
    const float *rho_in;      // S_MOMENT
    const float *g_rho_a;     // upstream of density output; the two are summed, either may be NULL
    const float *g_rho_b;
    const float *g_rho_grad;  // upstream of density gradient [B,N,D]
    const float *g_moment;    // upstream of moment matrix [B,N,D,D]
    float *grad_x;            // [B,N,P]
    float *grad_rho;          // [B,N], S_MOMENT only
    int accumulate_x;         // add into grad_x instead of overwriting
    const int32_t *bin_offsets;
    const int32_t *block_info;
    unsigned int *tickets;  // row tickets of this launch (set by the launcher)
};

struct FeatureFwdArgs {
    const float *x;
    const float *mass;
    const float *rho;
    const float *s;      // [B,N,C]
    float *blur;         // [B,N,C]
    float *grad;         // [B,N,C,D]
    int C;
    const int32_t *bin_offsets;
    const int32_t *block_info;
    float *moment;       // [B,N,D,D], only with F_MOMENT
    // ---- F_PACK: z[i] = [ s_i | blur_i | lognorm(coef * grad_i @ safe_inv(M_i)) | lognorm(dg_scale * rho_grad_i) ]
    float *z;                // [B,N,zstride], zstride = 2C + C*D + D
    int zstride;
    float *vgrad;            // [B,N,C,D] or NULL: grad_i @ safe_inv(M_i), kept for the backward pass
    const float *rho_grad;   // [B,N,D] density gradient of the same positions, or NULL when rho_grad_out is set
    float *rho_grad_out;     // [B,N,D] or NULL: the packed sweep computes the density gradient itself and writes it here
    float coef, dg_scale, inv_tol;
    int log_norm_grad, log_norm_dg;
    // ---- neighbour list cache (optional): row i = [count | j_0 .. j_{count-1}], count = -1 when the
    // particle has more than pair_stride - 1 neighbours (the reader then searches the cells itself)
    int32_t *pair_cache;     // [B*N, pair_stride] or NULL
    int pair_stride;
    int pair_cache_valid;    // 0: this sweep writes the lists; 1: they are valid, read them instead of searching
    unsigned int *tickets;  // row tickets of this launch (set by the launcher)
    const float4 *pv;        // [B*N] (x, y, z, m / rho) written by the density sweep, or NULL (lists only)
    int out_vec;             // packed rows over lists: z can be stored as vectors (set by the launcher)
};

struct FeatureBwdArgs {
    const float *x;
    const float *mass;
    const float *rho;
    const float *s;
    const float *g_blur;  // [B,N,C]
    const float *g_grad;  // [B,N,C,D]
    float *grad_x;        // [B,N,P] or NULL
    float *grad_s;        // [B,N,C] or NULL
    float *grad_rho;      // [B,N] or NULL
    int C;
    const int32_t *bin_offsets;
    const int32_t *block_info;
    const int32_t *pair_cache;  // neighbour lists written by the forward sweep of the same snapshot, or NULL
    int pair_stride;
    unsigned int *tickets;  // row tickets of this launch (set by the launcher)
};

// Backward of blur and / or gradient over neighbour lists (feature_list.cuh).
struct FeatureListBwdArgs {
    const float *x, *mass, *rho, *s;
    const float4 *pv;         // as above, or NULL
    const float *gb;          // dL/dblur, rows of gb_pitch floats, 16-byte aligned, padded to cp features
    const float *gg;          // dL/dgradient as [N, D, cp] inside rows of gg_pitch floats, 16-byte aligned
    int gb_pitch, gg_pitch, cp;
    const float *direct;      // rows of direct_pitch floats added to grad_s, or NULL
    int direct_pitch;
    const float *add;         // [B,N,C] added to grad_s, or NULL
    int out_vec;              // feature_dense.cu: grad_s and add can be moved in vectors
    const float *g_dg;        // upstream of the density gradient [B,N,D] (its part of grad_x is added), or NULL
    const float *g_rho;       // upstream of the density [B,N], or NULL: only goes into pg
    float *grad_x, *grad_s, *grad_rho;
    float4 *pg;               // [B*N] (x, y, z, g_rho + drho) for the density backward, or NULL
    int C;
    const int32_t *bin_offsets;
    const int32_t *pair_cache;
    int pair_stride;
};

// Backward of density (upstream g_rho_a + g_rho_b, or packed in pg) and density gradient over neighbour lists, and the
// density gradient itself over lists (scalar_list.cu).
struct ScalarListArgs {
    const float *x, *mass, *g_rho_a, *g_rho_b, *g_dg;
    const float4 *pg;
    float *grad_x;
    int accumulate_x;
    float *rho_grad_out;
    const int32_t *bin_offsets, *pair_cache;
    int pair_stride;
};
int launch_scalar_list_backward(const Geom &g, const ScalarListArgs &a, cudaStream_t st);
int launch_density_gradient_list(const Geom &g, const ScalarListArgs &a, cudaStream_t st);
int launch_feature_list_forward(const Geom &g, int mask, const FeatureFwdArgs &a, cudaStream_t st);
int launch_feature_list_backward(const Geom &g, int mask, bool full, const FeatureListBwdArgs &a, cudaStream_t st);
// Features only, blur and gradient, for positions that are those that were binned (feature_dense.cu); what it covers and is faster at.
bool feature_dense_covers(const Geom &g, int C);
int feature_dense_pitch(int dim, int cp);  // floats from particle to particle of the rows (gb and gg in one)
int launch_feature_dense_backward(const Geom &g, const FeatureListBwdArgs &a, cudaStream_t st);
// [N, C(, D)] upstreams -> rows [N, (1 +) D, cp] of `rows` (blur part only when with_blur).
int launch_upstream_rows(const Geom &g, int C, const float *g_blur, const float *g_grad, bool with_blur, float *rows, cudaStream_t st);

// Number of CTAs of a persistent launch of `kernel`: every SM filled to the kernel's occupancy.
// Cached per (device, kernel); the first call also raises the kernel's dynamic shared-memory
// limit to what it needs.  Defined in capi.cu.
int persistent_ctas_impl(const void *kernel, int threads, size_t dyn_smem, int *out);
template <typename Kernel>
int persistent_ctas(Kernel kernel, int threads, size_t dyn_smem, int *out) {
    return persistent_ctas_impl(reinterpret_cast<const void *>(kernel), threads, dyn_smem, out);
}

// Two zeroed words in device memory for the row tickets of one persistent launch (next_row /
// release_rows in neighbors.cuh).  They live in a small array inside the library, handed out round
// robin: launches in one stream are ordered, and launches in different streams get different words
// unless hundreds of launches lie between them.  Launches recorded into a CUDA graph draw from a
// separate half of the array, so a replaying graph never shares words with an eager launch.
// Defined in capi.cu.
int acquire_row_tickets(cudaStream_t st, unsigned int **out);

// The same sweeps on the cell-tile streaming engine (feature_tile.cuh).  *taken = false means the
// engine does not cover this call (nothing was launched) and the gather kernel must run.
template <int D, bool PER>
int launch_feature_tile_forward(const Geom &g, int mask, const FeatureFwdArgs &a, cudaStream_t st, bool *taken);
template <int D, bool PER, bool FULL>
int launch_feature_tile_backward(const Geom &g, int mask, const FeatureBwdArgs &a, cudaStream_t st, bool *taken);

int launch_density_search(const Geom &g, bool count, const ScalarFwdArgs &a, cudaStream_t st);  // density_search.cu
bool scalar_shared_search();  // scalar_ops.cu: count and density run there
int launch_density_ordered(const Geom &g, const ScalarFwdArgs &a, cudaStream_t st);  // density_ordered.cu
int launch_scalar_forward(const Geom &g, int mask, const ScalarFwdArgs &a, cudaStream_t st);
int launch_scalar_backward(const Geom &g, int mask, const ScalarBwdArgs &a, cudaStream_t st);
int launch_feature_forward(const Geom &g, int mask, const FeatureFwdArgs &a, cudaStream_t st);
// full = false differentiates with respect to s only.
int launch_feature_backward(const Geom &g, int mask, bool full, const FeatureBwdArgs &a, cudaStream_t st);

}  // namespace npa
