// The sum of the weight gradients' partial sums (mlp_grad_tcgen05.cu), and what the host has to know of it: the gradients of a step are
// added up by the launch that puts its gradients back into the order of the inputs (binning.cu).
#pragma once
#include "common.cuh"

namespace npa {

constexpr int kGradHidden = 128;
constexpr int kGradStageRows = 16;  // two k-groups of eight rows
constexpr int kReduceQuads = 32, kReduceRuns = 16, kReduceMost = (148 + kReduceRuns - 1) / kReduceRuns;

struct GradReduce {
    const float *partial;  // [ctas][128][N1p + N2p]
    float *dW1, *dW2, *db1;
    int in_dim, out_dim, N1p, N2p, ctas, stages_per_cta;
    int quads() const { return kGradHidden * ((in_dim + 4) / 4 + (out_dim + 3) / 4); }
    unsigned blocks(int quads_each) const { return (unsigned)((quads() + quads_each - 1) / quads_each); }
};

inline int grad_round16(int v) { return (v + 15) / 16 * 16; }

// Shape of the partial sums, and the stages of rows of a CTA.
inline GradReduce grad_plan(long long rows, int in_dim, int out_dim) {
    GradReduce p = {};
    p.in_dim = in_dim; p.out_dim = out_dim; p.N1p = grad_round16(in_dim + 1); p.N2p = grad_round16(out_dim);
    const long long stages = (rows + kGradStageRows - 1) / kGradStageRows;
    const int ctas = (int)(stages < 148 ? stages : 148);
    p.stages_per_cta = (int)((stages + ctas - 1) / ctas);
    p.ctas = (int)((stages + p.stages_per_cta - 1) / p.stages_per_cta);
    return p;
}

// dW1, db1 and dW2 from the CTAs' partial sums.  A thread takes four neighbouring columns of a hidden unit, as they lie in the partial
// sums, of one run of CTAs: all its loads are in flight at once, and a warp reads 512 bytes in a row of each CTA (by output instead,
// dW2's columns lay a row apart).  The runs meet in shared memory, in order.  Latency bound: 7.6 MB (in = 66, out = 18) or 17 MB (163, 35)
// from L2 in one round trip: 8.4 -> 5.2 us and 9.1 -> 5.7.
template <int QUADS>
__device__ inline void reduce_weight_grads(const GradReduce &a, int block) {
    __shared__ float4 s_sum[kReduceRuns][QUADS];
    const int K1 = a.in_dim, O = a.out_dim, Wp = a.N1p + a.N2p;
    const int q1 = (K1 + 4) / 4, per_unit = q1 + (O + 3) / 4, total = kGradHidden * per_unit;  // quads that hold results
    const int lane = threadIdx.x % QUADS, run = threadIdx.x / QUADS;
    auto column = [&](int q) {  // of the first float of quad q, in the partial sums
        const int u = q % per_unit;
        return (long long)(q / per_unit) * Wp + (u < q1 ? 4 * u : a.N1p + 4 * (u - q1));
    };
    const int quad = min(block * QUADS + lane, total - 1);
    const float *p = a.partial + column(quad);
    const long long step = (long long)kGradHidden * Wp;
    const int each = (a.ctas + kReduceRuns - 1) / kReduceRuns, c0 = run * each, end = min(c0 + each, a.ctas);
    float4 v[kReduceMost];
#pragma unroll
    for (int u = 0; u < kReduceMost; ++u)
        v[u] = u < each && c0 + u < end ? __ldg(reinterpret_cast<const float4 *>(p + (c0 + u) * step)) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 sum = v[0];
#pragma unroll
    for (int u = 1; u < kReduceMost; ++u) {
        sum.x += v[u].x; sum.y += v[u].y; sum.z += v[u].z; sum.w += v[u].w;
    }
    s_sum[run][lane] = sum;
    __syncthreads();
    if (threadIdx.x >= 4 * QUADS) return;
    const int q = block * QUADS + (int)threadIdx.x / 4, part = threadIdx.x % 4;
    if (q >= total) return;
    float out = 0.f;
#pragma unroll
    for (int r = 0; r < kReduceRuns; ++r) out += reinterpret_cast<const float *>(&s_sum[r][threadIdx.x / 4])[part];
    const int j = q / per_unit, u = q - j * per_unit, col = u < q1 ? 4 * u + part : 4 * (u - q1) + part;
    if (u >= q1) {
        if (col < O) a.dW2[(long long)col * kGradHidden + j] = out;
    } else if (col < K1) {
        a.dW1[(long long)j * K1 + col] = out;
    } else if (col == K1) {
        a.db1[j] = out;  // the ones column
    }
}

}  // namespace npa
