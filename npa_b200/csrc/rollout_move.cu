// The move between two steps of a rollout in one pass: x_out = wrap(x + dt v(x)) with v a sum of sine modes.
//
// The seeded velocity field of npa_b200.rollout (amp^T sin(k x + phase), a few modes) and the periodic wrap of
// HashGrid.wrap_positions (sphops/sph.py:107-123).  As tensor operations this is two thin matrix products over the particles
// and eight elementwise passes, 145 us per move of 524,288 particles in 3D; here a thread reads a position and writes it,
// 11 us (floor at the copy rate: 2.6; the sines are the rest).  Products and sums are taken one by one in the order of those
// operations (multiply-adds along the axis, then the phase; multiply-adds along the modes; dt v and the sum rounded apart), so that
// the positions are the same bits: a particle that lies next to a cell's edge must not change cells with the way of computing.
#include "neighbors.cuh"
#include "ops.cuh"

namespace npa {

constexpr int kMoveModes = 64;

struct MoveArgs {
    const float *x;      // [B*N, P]
    const float *k;      // [D, modes]
    const float *phase;  // [modes]
    const float *amp;    // [modes, D]
    float *out;          // [B*N, P], the padding column is left alone
    int modes;
    float dt;
};

template <int D>
__global__ void __launch_bounds__(256) rollout_move_kernel(const __grid_constant__ MoveArgs a, const __grid_constant__ Geom g) {
    after_previous_kernel();
    constexpr int P = D == 2 ? 2 : 4;
    __shared__ float s_k[D * kMoveModes], s_phase[kMoveModes], s_amp[D * kMoveModes];
    for (int q = threadIdx.x; q < D * a.modes; q += blockDim.x) {
        s_k[q] = __ldg(a.k + q);
        s_amp[q] = __ldg(a.amp + q);
    }
    for (int q = threadIdx.x; q < a.modes; q += blockDim.x) s_phase[q] = __ldg(a.phase + q);
    __syncthreads();
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)g.B * g.N) return;
    const Pos<D> p = load_pos<D>(a.x, i);
    const float x[3] = {p.x, p.y, p.z};
    float v[3] = {0.f, 0.f, 0.f};
    for (int m = 0; m < a.modes; ++m) {
        float t = 0.f;
#pragma unroll
        for (int d = 0; d < D; ++d) t = __fmaf_rn(x[d], s_k[d * a.modes + m], t);
        t = sinf(__fadd_rn(t, s_phase[m]));
#pragma unroll
        for (int d = 0; d < D; ++d) v[d] = __fmaf_rn(t, s_amp[m * D + d], v[d]);
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
        float y = __fadd_rn(x[d], __fmul_rn(a.dt, v[d]));
        if (g.periodic) {
            const float half = 0.5f * g.L[d];
            y = __fadd_rn(y, half);
            if (!(y >= 0.f && y < g.L[d])) {
                y = fmodf(y, g.L[d]);
                if (y < 0.f) y = __fadd_rn(y, g.L[d]);
            }
            y = __fsub_rn(y, half);
        }
        a.out[i * P + d] = y;
    }
}

// Two arrays in one launch: the inputs of a recorded step are copied into its buffers before every replay, and two copies of
// a few hundred kilobytes are mostly the gap between them (2.5 us of a step of 42).
__global__ void __launch_bounds__(256) copy_pair_kernel(const float *__restrict__ a, float *__restrict__ a_out, long long na,
                                                        const float *__restrict__ b, float *__restrict__ b_out, long long nb) {
    const long long qa = na / 4, qb = nb / 4, step = (long long)gridDim.x * blockDim.x, t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (long long q = t; q < qa + qb; q += step) {
        const bool second = q >= qa;
        const long long at = second ? q - qa : q;
        reinterpret_cast<float4 *>(second ? b_out : a_out)[at] = __ldg(reinterpret_cast<const float4 *>(second ? b : a) + at);
    }
    if (t < na % 4) a_out[qa * 4 + t] = a[qa * 4 + t];
    if (t < nb % 4) b_out[qb * 4 + t] = b[qb * 4 + t];
}

}  // namespace npa

using namespace npa;

extern "C" int npa_copy_pair(const float *a, float *a_out, int64_t na, const float *b, float *b_out, int64_t nb, void *stream) {
    if (!a || !a_out || !b || !b_out || na < 0 || nb < 0) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_copy_pair: arrays must be non-NULL");
    if (((uintptr_t)a | (uintptr_t)a_out | (uintptr_t)b | (uintptr_t)b_out) % 16)
        return fail(NPA_ERR_INVALID_ARGUMENT, "npa_copy_pair: arrays must be 16-byte aligned");
    const long long blocks = (na / 4 + nb / 4 + 255) / 256;
    copy_pair_kernel<<<(unsigned)(blocks < 1 ? 1 : blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, (cudaStream_t)stream>>>(a, a_out, na, b, b_out, nb);
    return check_launch("copy_pair_kernel");
}

extern "C" int npa_rollout_move(const npa_grid *grid, const float *x, const float *k, const float *phase, const float *amp, int32_t modes, float dt,
                                float *x_out, void *stream) {
    Geom g;
    const int rc = make_geom(grid, &g);
    if (rc != NPA_OK) return rc;
    if (modes < 1 || modes > kMoveModes) return fail(NPA_ERR_UNSUPPORTED, "npa_rollout_move: %d modes are outside 1..%d", modes, kMoveModes);
    if (!x || !k || !phase || !amp || !x_out) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_rollout_move: all arrays must be non-NULL");
    if ((uintptr_t)x % (g.dim == 2 ? 8 : 16)) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_rollout_move: x must be aligned to one position");
    const MoveArgs a = {x, k, phase, amp, x_out, modes, dt};
    const unsigned blocks = (unsigned)(((long long)g.B * g.N + 255) / 256);
    launch_early(g.dim == 2 ? rollout_move_kernel<2> : rollout_move_kernel<3>, blocks, 256, 0, (cudaStream_t)stream, a, g);
    return check_launch("rollout_move_kernel");
}
