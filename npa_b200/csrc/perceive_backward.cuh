// What the kernels that take dL/dz apart share: perceive_pack.cu, and the epilogue of dz = dh W1 in mlp_tcgen05.cu.
#pragma once
#include "ops.cuh"

namespace npa {

// Gradient of  f(w) = log(1 + |w|) w / |w|  (symmetric Jacobian) applied to g, times `scale`;
// without log-normalisation f is the identity.
template <int D>
__device__ inline void log_normalize_backward(const float *w, const float *gin, int log_norm, float scale, float *gout) {
    if (!log_norm) {
#pragma unroll
        for (int d = 0; d < D; ++d) gout[d] = scale * gin[d];
        return;
    }
    float n2 = w[0] * w[0] + w[1] * w[1];
    float wg = w[0] * gin[0] + w[1] * gin[1];
    if (D == 3) { n2 += w[2] * w[2]; wg += w[2] * gin[2]; }
    const float n = sqrtf(n2);
    const float l = logf(1.0f + n);
    const float a = l / fmaxf(n, 1e-12f);
    const float b = n > 1e-12f ? (1.0f / ((1.0f + n) * n2) - l / (n2 * n)) : 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) gout[d] = scale * (a * gin[d] + b * wg * w[d]);
}

// mlp_tcgen05.cu: rows of dL/dz = dh W1 taken apart as they leave the tensor cores (StepColumns in weight_image.cuh).
struct StepRows {
    const float *vgrad;  // corrected gradients of the features, [particles, C, D]
    float *direct;       // dL/dz of the features themselves, [particles, C]
    float *rows;         // per particle dL/dblur and the D axes of dL/dgradient, C floats each
    int pitch, C, dim;
    float coef;
    int log_norm;
};
// Rows of whole float4, up to the features of the packed sweep.  dL/dz stored and taken apart by a kernel of its own / as it leaves, with the
// sweep that followed then, us: 32,768 particles in 2D, C = 4 / 16 / 20 / 32: 32.9 / 30.8, 36.9 / 32.8, 47.0 / 43.1, 49.7 / 45.2; 65,536 in 3D
// 81.7 / 78.1, 91.8 / 83.0, 126.0 / 118.9, 137.2 / 126.7 (sections that fill half of their columns gain least).
inline bool step_rows_cover(int channels) { return channels % 4 == 0 && channels > 0 && channels <= 32; }
int launch_step_rows(const StepRows &rows, const float *dh, long long particles, const void *image, int64_t image_bytes, cudaStream_t st);

}  // namespace npa
