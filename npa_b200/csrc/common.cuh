// Shared device/host definitions of the npa_b200 kernels: grid geometry, cell
// hashing, SPH pair kernels and the error plumbing of the C ABI.
//
// Math follows the reference operators as restated by its pure-torch oracle
// (sphops/torch_sph.py:96-162: poly6 (h^2-r^2)^3 with cut-off r^2 < h^2, spiky
// 3(h-d)^2/d * r with d = sqrt(r^2 + 1e-12) inside 0 < r < h) and the cell
// geometry of sphops/utils.cuh:303-524.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/npa_b200.h"

namespace npa {

constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;

// Device-side copy of npa_grid plus everything derived from it, passed by
// value to every kernel (the role of GridConfig, sphops/utils.cuh:303-318).
struct Geom {
    int dim, periodic, morton;
    int g[3];       // cells per axis (1 on unused axes)
    int half[3];    // g / 2: the grid is centred on the origin
    int cells;      // per system
    int B, N, mpb;
    int max_blocks;
    int split;      // warps sharing one work item in the feature kernels (small problems only)
    float inv_eps;  // 1.0f / float(eps): the multiplier pos2cell uses
    float h;        // float(eps)
    float h2;       // float(eps * eps) rounded once from double, as torch does
    float L[3];     // box length per axis = g * eps (rounded from double)
    float Llo[3];   // double(g * eps) - L: the part of the box length fp32 cannot hold
    float invL[3];
    float halfL[3];
    float c_s;      // poly6 normalisation
    float c_g;      // spiky normalisation
};

// Host: validate an npa_grid and derive Geom.  Returns an npa_status.
int make_geom(const npa_grid *in, Geom *out);
// Host: record an error message for npa_last_error() and return `code`.
int fail(int code, const char *fmt, ...);
// Host: convert the last CUDA launch error into a status.
int check_launch(const char *what);

// ---- launches that overlap the end of the kernel before -----------------------
// A small step is a chain of dependent kernels of 2-40 us, and between two of them the GPU stands still for 1-2 us: the end of
// the one, the way of the launch to the SMs, its first instructions.  So the CTAs of a kernel launched by launch_early() may take
// their places as soon as every CTA of the kernel before (of this library, in the same stream) has started; each begins with
// after_previous_kernel(), which waits until that kernel has completed and its writes are visible.  No access to global memory may
// come before it: a kernel launched this way that does not call it would not wait for its inputs at all.  Every kernel waits for the
// one before, so a chain is in order as a whole.  Kernels of others, copies and events wait for complete kernels, as ever.
// Training step of 8 x 4,096 particles in 2D 234 -> 207 us, of 4 x 16,384 in 3D 374 -> 336, inference step of 4,096 72 -> 60.
// Plain launches, because they were slower this way:
//  * feature_list.cuh, forward and backward (rollout of 2 x 262,144 particles 3,116 -> 3,344 us): they live off L1, and a CTA that takes
//    its place early finds the SM divided between L1 and shared memory as the kernel before wanted it;
//  * the reduction of the weight gradients (3D step of 262,144 particles 1,544 -> 1,552 us, its kernel and the one behind it together: it
//    takes room beside the gradient kernel's CTAs that the next kernel would have had);
//  * the hidden gradient of the MLP (3D steps 298 -> 301, 1,428 -> 1,432 us, not explained);
//  * feature_dense.cu (1,428 -> 1,454, not explained further: its rows come through L1 as well).
// Plain and not measured otherwise: the searching sweeps of feature_kernels.cuh and scalar_ops.cu, the cell-tile engine, the paths of
// mlp_gemm.cu and mlp_grad.cu, small conversions.  The density searches, the packed sweep and the sweeps of scalar_list.cu are launched
// early; they were measured within the chains above only.
// While a graph is recorded all launches are plain: its nodes are close already (41.3 us instead of 41.9), and the edges would make
// it 10 % slower to build.
__device__ __forceinline__ void after_previous_kernel() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Such a launch; in clusters of `cluster` blocks where that is more than one.
template <typename... P, typename... A>
inline void launch_cluster(int cluster, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaLaunchAttribute attrs[2];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream; cfg.attrs = attrs;
    if (cudaStreamIsCapturing(stream, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone) {
        attrs[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attrs[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attrs[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attrs[cfg.numAttrs].val.clusterDim.x = cluster;
        attrs[cfg.numAttrs].val.clusterDim.y = attrs[cfg.numAttrs].val.clusterDim.z = 1;
        ++cfg.numAttrs;
    }
    (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);  // an error is check_launch's
}

template <typename... P, typename... A>
inline void launch_early(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
    launch_cluster(1, kernel, grid, block, smem, stream, std::forward<A>(args)...);
}

// ---- cell hashing (sphops/utils.cuh:394-524) -------------------------------

__host__ __device__ inline uint32_t dilate2(uint32_t x) {
    x &= 0x3FFu;
    x = (x | (x << 16)) & 0x0000FFFFu;
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}
__host__ __device__ inline uint32_t dilate3(uint32_t x) {
    x &= 0x3FFu;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}
__host__ __device__ inline uint32_t undilate2(uint32_t x) {
    x &= 0x55555555u;
    x = (x | (x >> 1)) & 0x33333333u;
    x = (x | (x >> 2)) & 0x0F0F0F0Fu;
    x = (x | (x >> 4)) & 0x00FF00FFu;
    x = (x | (x >> 8)) & 0x0000FFFFu;
    return x & 0x3FFu;
}
__host__ __device__ inline uint32_t undilate3(uint32_t x) {
    x &= 0x09249249u;
    x = (x | (x >> 2)) & 0x030C30C3u;
    x = (x | (x >> 4)) & 0x0300F00Fu;
    x = (x | (x >> 8)) & 0x030000FFu;
    x = (x | (x >> 16)) & 0x000003FFu;
    return x;
}

template <int D>
__host__ __device__ inline uint32_t cell_hash(const Geom &g, int cx, int cy, int cz) {
    if (g.morton) {
        if (D == 2) return dilate2((uint32_t)cx) | (dilate2((uint32_t)cy) << 1);
        return dilate3((uint32_t)cx) | (dilate3((uint32_t)cy) << 1) | (dilate3((uint32_t)cz) << 2);
    }
    if (D == 2) return (uint32_t)(cy * g.g[0] + cx);
    return (uint32_t)((cz * g.g[1] + cy) * g.g[0] + cx);
}

template <int D>
__device__ inline void hash_to_cell(const Geom &g, uint32_t hsh, int &cx, int &cy, int &cz) {
    cz = 0;
    if (g.morton) {
        if (D == 2) {
            cx = (int)undilate2(hsh);
            cy = (int)undilate2(hsh >> 1);
        } else {
            cx = (int)undilate3(hsh);
            cy = (int)undilate3(hsh >> 1);
            cz = (int)undilate3(hsh >> 2);
        }
        return;
    }
    cx = (int)(hsh % (uint32_t)g.g[0]);
    if (D == 2) {
        cy = (int)(hsh / (uint32_t)g.g[0]);
    } else {
        cy = (int)((hsh / (uint32_t)g.g[0]) % (uint32_t)g.g[1]);
        cz = (int)(hsh / (uint32_t)(g.g[0] * g.g[1]));
    }
}

__device__ inline int wrap_or_clamp(int c, int n, int periodic) {
    if (periodic) {
        c %= n;
        return c < 0 ? c + n : c;
    }
    return min(max(c, 0), n - 1);
}

// Cell coordinate of one position component: floor(x * (1/eps)) + g/2, then
// the boundary rule (sphops/utils.cuh:426-440).
__device__ inline int axis_cell(float x, const Geom &g, int axis) {
    int c = __float2int_rd(__fmul_rn(x, g.inv_eps)) + g.half[axis];
    return wrap_or_clamp(c, g.g[axis], g.periodic);
}

// ---- pair geometry -----------------------------------------------------------

// General minimum image of one displacement component: used only when the
// image shift could not be known in advance (a particle outside the primary
// box, or an axis with fewer than three cells).
__device__ inline float wrap_general(float r, float L, float Llo, float invL) {
    const float n = rintf(r * invL);
    r = __fmaf_rn(-n, L, r);
    return __fmaf_rn(-n, Llo, r);
}

// r^2 accumulated in the order torch.sum uses on a length-D vector, without
// fused multiply-adds, so that the strict cut-off test r^2 < h^2 agrees with
// the fp32 oracle on borderline pairs.
template <int D>
__device__ inline float sq_norm(float rx, float ry, float rz) {
    float q = __fadd_rn(__fmul_rn(rx, rx), __fmul_rn(ry, ry));
    if (D == 3) q = __fadd_rn(q, __fmul_rn(rz, rz));
    return q;
}

// Same quantity with fused multiply-adds, for kernels whose outputs are continuous in r^2
// (everything except the neighbour count).
template <int D>
__device__ inline float sq_norm_fast(float rx, float ry, float rz) {
    float q = fmaf(ry, ry, rx * rx);
    if (D == 3) q = fmaf(rz, rz, q);
    return q;
}

// Two fp32 lanes in one 64-bit register pair and the packed arithmetic of sm_100 on them: one issue slot per
// two multiply-adds, each lane rounded exactly like the scalar instruction.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Spiky pair factors for 0 < q < h2: phi = 3 (h - d)^2 / d with
// d = sqrt(q + 1e-12), so that K(r) = phi * r; psi = 3 (h^2 - d^2) / d^3 so that
// dK/dr = phi * I - psi * r r^T.
// d and 1 / d come from one reciprocal square root with a Newton step each (tests/test_gpu_neighbour_lists.py holds
// the kernel values of single pairs to the fp64 formula): an IEEE square root and a division or two were half of the
// instructions of the pair-scalar stage of the sweeps over neighbour lists.
struct Spiky {
    float d, inv;  // distance and its reciprocal
};
__device__ inline Spiky spiky_refined(float Q, float y) {  // y: 1 / sqrt(Q) to a few ulps
    y = fmaf(0.5f * y, fmaf(-(Q * y), y, 1.0f), y);
    const float d = Q * y;
    return Spiky{fmaf(0.5f * y, fmaf(-d, d, Q), d), y};
}
__device__ inline Spiky spiky_distance(float q) {
    const float Q = q + 1e-12f;
    return spiky_refined(Q, rsqrtf(Q));
}
// Square root and quotient as IEEE rounds them, without the range checks and branches of the general routines: Newton steps
// whose residuals are exact by fused multiply-add (P. Markstein, IA-64 and Elementary Functions, ch. 8-9).  For
// 2^-66 <= Q < 2^66; npa_rounding_selftest compares them with __fsqrt_rn and __fdiv_rn (tests/test_gpu_rounding.py: every root of
// two binades, 2^17 of each other one, a quotient by each).
struct Root {
    float d, inv;  // sqrt(Q), and 1 / d to within an ulp
};
__device__ inline Root root_rounded(float Q) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(Q));
    const float s = __fmul_rn(Q, y);
    const float d = fmaf(fmaf(-s, s, Q), __fmul_rn(0.5f, y), s);
    return Root{d, fmaf(fmaf(-d, y, 1.0f), y, y)};
}
__device__ inline float quotient_rounded(float n, const Root &r) {  // n / r.d
    const float q = __fmul_rn(n, r.inv);
    return fmaf(fmaf(-r.d, q, n), r.inv, q);
}
__device__ inline float spiky_phi(const Spiky &s, float h) {
    const float t = fmaxf(h - s.d, 0.0f);
    return 3.0f * t * t * s.inv;
}
__device__ inline float spiky_psi(const Spiky &s, float h) {
    // d(phi)/dd / d with phi = 3 max(h-d,0)^2 / d  ==  -3 (h - d)(h + d) / d^3
    const float t = fmaxf(h - s.d, 0.0f);
    return 3.0f * t * (h + s.d) * (s.inv * s.inv * s.inv);
}

// Inverse of a symmetric DxD matrix given by its upper triangle m (row-major order of the
// triangle), identity when |det| < tol: the rule of the reference's safe_inv_sym_mat
// (sphops/sph_cuda.cu:3095-3179).  L is the full DxD inverse, row-major.
template <int D>
__device__ inline void safe_inverse_sym(const float *m, float tol, float *L) {
    if (D == 2) {
        const float det = m[0] * m[2] - m[1] * m[1];
        if (fabsf(det) < tol) {
            L[0] = 1.f; L[1] = 0.f; L[2] = 0.f; L[3] = 1.f;
        } else {
            const float r = 1.0f / det;
            L[0] = m[2] * r; L[1] = -m[1] * r; L[2] = -m[1] * r; L[3] = m[0] * r;
        }
    } else {
        const float a = m[0], b = m[1], c = m[2], d = m[3], e = m[4], f = m[5];
        const float t1 = d * f - e * e, t2 = c * e - b * f, t3 = b * e - c * d;
        const float det = a * t1 + b * t2 + c * t3;
        if (fabsf(det) < tol) {
            L[0] = 1.f; L[1] = 0.f; L[2] = 0.f; L[3] = 0.f; L[4] = 1.f; L[5] = 0.f; L[6] = 0.f; L[7] = 0.f; L[8] = 1.f;
        } else {
            const float r = 1.0f / det;
            const float m01 = t2 * r, m02 = t3 * r, m12 = (b * c - a * e) * r;
            L[0] = t1 * r; L[1] = m01; L[2] = m02;
            L[3] = m01; L[4] = (a * f - c * c) * r; L[5] = m12;
            L[6] = m02; L[7] = m12; L[8] = (a * d - b * b) * r;
        }
    }
}

// w <- log(1 + |w|) * w / max(|w|, 1e-12): the log-normalisation NPA applies to its gradient
// features (models/npa.py:83-85, torch.nn.functional.normalize's epsilon).
template <int D>
__device__ inline void log_normalize(float *w) {
    float n2 = w[0] * w[0] + w[1] * w[1];
    if (D == 3) n2 += w[2] * w[2];
    float sc;
    if (n2 > 1e-18f && n2 < 1e18f) {
        const Root r = root_rounded(n2);
        sc = quotient_rounded(logf(1.0f + r.d), r);
    } else {
        const float n = sqrtf(n2);
        sc = logf(1.0f + n) / fmaxf(n, 1e-12f);
    }
#pragma unroll
    for (int d = 0; d < D; ++d) w[d] *= sc;
}

}  // namespace npa
