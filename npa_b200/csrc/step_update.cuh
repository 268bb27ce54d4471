// What the Euler update's kernels (step_update.cu) and the hidden gradient of a whole step (mlp_hidden_grad.cu) share.
#pragma once
#include "ops.cuh"

namespace npa {

struct StepArgs {
    const float *y;       // [BN, D + C]; the hidden gradient reads only the raw displacements, rows of y_pitch floats
    int y_pitch;
    const float *x_bin;   // [BN, P]
    const float *s_bin;   // [BN, C]
    const float *mask;    // [BN] (0 / 1, or uniforms) or NULL = every particle updates
    int uniforms;         // mask holds uniforms: a particle updates where its value is below `below`
    float below;
    float *x_out;         // [BN, P]
    float *s_out;         // [BN, C]
    const float *g_x_out; // backward: upstream of x_out [BN, P]
    const float *g_s_out; // backward: upstream of s_out [BN, C]
    float *g_y;           // backward: [BN, D + C]
    long long particles;
    int C;
    float alpha, eps, dt;
    int wrap;
};

__device__ inline float mask_value(const StepArgs &a, float m) { return a.uniforms ? (m < a.below ? 1.0f : 0.0f) : m; }

__device__ inline float mask_of(const StepArgs &a, long long i) { return a.mask ? mask_value(a, __ldg(a.mask + i)) : 1.0f; }

// remainder(x + L/2, L) - L/2 with torch's sign convention (result of remainder in [0, L)).
__device__ inline float wrap_axis(float x, float L) {
    const float half = 0.5f * L;
    float r = fmodf(x + half, L);
    if (r < 0.f) r += L;
    return r - half;
}

// A position moved by its raw displacement u, in place.  The reference's order: ((alpha * dx) * eps) / (1 + |dx|), then (dt * dx) * mask.
template <int D>
__device__ inline void step_forward_position(const StepArgs &a, const Geom &g, float m, const float *u, float (&x)[4]) {
    float n2 = 0.f;
#pragma unroll
    for (int d = 0; d < D; ++d) n2 = fmaf(u[d], u[d], n2);
    const float den = 1.0f + sqrtf(n2);
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const float lim = ((a.alpha * u[d]) * a.eps) / den;
        x[d] = x[d] + (a.dt * lim) * m;
        if (a.wrap && g.periodic) x[d] = wrap_axis(x[d], g.L[d]);
    }
}

// Four states.
__device__ inline float4 step_forward_states(const StepArgs &a, float m, const float4 &s, const float *y) {
    return make_float4(s.x + (a.dt * y[0]) * m, s.y + (a.dt * y[1]) * m, s.z + (a.dt * y[2]) * m, s.w + (a.dt * y[3]) * m);
}

// dL/dy of one element.  The limiter f(u) = k u / (1 + |u|), k = alpha * eps, has the Jacobian
//   df_a/du_b = k [ delta_ab / (1 + n) - u_a u_b / (n (1 + n)^2) ],  n = |u|  (second term 0 at n = 0,
// as torch's norm backward); the wrap and the additions are the identity for gradients.
// From the raw displacement u and the upstream g of a position, all components.
template <int D>
__device__ inline void step_backward_position(const StepArgs &a, float m, const float (&u)[D], const float (&g)[D], float (&out)[D]) {
    float n2 = 0.f, gu = 0.f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        n2 = fmaf(u[d], u[d], n2);
        gu = fmaf(u[d], g[d], gu);
    }
    const float n = sqrtf(n2);
    const float k = a.alpha * a.eps * a.dt * m;
    const float inv = 1.0f / (1.0f + n);
#pragma unroll
    for (int d = 0; d < D; ++d) {
        float v = g[d] * inv;
        if (n > 0.f) v -= u[d] * gu * inv * inv / n;
        out[d] = k * v;
    }
}

template <int D>
__device__ inline float step_backward_element(const StepArgs &a, long long i, int c) {
    constexpr int P = D == 2 ? 2 : 4;
    const float m = mask_of(a, i);
    if (c >= D) return a.g_s_out ? (a.dt * m) * __ldg(a.g_s_out + i * a.C + (c - D)) : 0.f;
    if (!a.g_x_out) return 0.f;
    float u[D], g[D], out[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
        u[d] = __ldg(a.y + i * (D + a.C) + d);
        g[d] = __ldg(a.g_x_out + i * P + d);
    }
    step_backward_position<D>(a, m, u, g, out);
    float r = out[0];
#pragma unroll
    for (int d = 1; d < D; ++d) r = c == d ? out[d] : r;
    return r;
}

}  // namespace npa
