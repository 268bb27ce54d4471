// Gradient at the hidden layer of the per-particle MLP, with the ReLU mask applied:
//
//     dh [rows, 128] = (dy [rows, out] . W2 [out, 128])  where h > 0,  else 0
//
// (models/npa.py:63-75: the backward of Linear(128, out, bias=False) followed by the backward of the
// ReLU that produced h).  torch runs it as a thin fp32 GEMM (35 columns of dy) plus a masking pass over
// dh; here it is one pass on the CUDA cores in fp32: dh is written once and h is read once.  The
// product is too thin for the tensor cores to matter (out <= 48 multiply-adds per output element
// against 8 bytes of traffic).
//
// In a whole step dy is the backward of the Euler update (step_update.cuh), made here row by row on the way in and written once for the
// weight gradients, instead of by a launch of its own.
//
// A warp takes eight rows at a time, a lane four hidden units of all of them.  W2 stays in shared memory; dy is staged per warp by columns,
// so that a column's eight rows are two broadcast loads, packed in pairs of rows: seven 128-bit loads and register copies serve 32
// multiply-adds in 16 instructions, products in ascending o.  The upstream of the warp's next rows is copied asynchronously meanwhile.
// Four CTAs per SM (64 registers).  Latency bound, with the multiply-adds at 40 % of their rate and memory at half of the copy rate.
// Measured, B200, us, with the update's backward as a launch of its own and scalar multiply-adds -> this: 262,144 rows, C = 32 in 3D
// 94 + 22 -> 90; 65,536 rows, C = 16 in 3D 20.7 + 6.1 -> 20.4; 32,768 rows, C = 16 in 2D 12.2 + 3.4 -> 11.6.  At three CTAs 96 / 21.3 /
// 12.6; sixteen rows and eight units per lane at two CTAs 106 / 25 / 13.5, and with the signs of h fetched a pass ahead 140 (spills).
#include "step_update.cuh"

namespace npa {

constexpr int kHgHidden = 128;
constexpr int kHgMaxOut = 48;
constexpr int kHgRows = 8;       // rows per warp pass
constexpr int kHgPitch = 12;     // floats of a staged column of dy
constexpr int kHgWarps = 8;
constexpr int kHgThreads = kHgWarps * 32;

template <int V> struct Int {
    static constexpr int value = V;
};

struct HiddenGradArgs {
    const float *dy, *W2, *h;
    float *dh;
    long long rows, w_stride_out, w_stride_in;
    int out_dim;
};

// Shared memory in floats: W2's rows (up to a multiple of four), then per warp the columns of dy, the upstream as it comes (of the states;
// per row that of the position, the raw displacement and the mask) and dy's rows as they go out.
struct HiddenGradMem {
    int columns, w2, raw, small, out, per_warp;
    __host__ __device__ HiddenGradMem(int D, int out_dim) {
        columns = (out_dim + 3) / 4 * 4;
        w2 = columns * kHgHidden;
        raw = columns * kHgPitch;
        small = raw + (D ? kHgRows * ((out_dim - D + 3) / 4 * 4) : 0);
        out = small + (D ? kHgRows * 9 : 0);
        per_warp = out + (D ? (kHgRows * out_dim + 3) / 4 * 4 : 0);
    }
    size_t bytes() const { return (size_t)(w2 + kHgWarps * per_warp) * 4; }
};

// D = 0: dy is given; otherwise the update of D-dimensional positions, whose g_y is written.  VEC: its upstream of the states in float4.
template <int D, bool VEC>
__global__ void __launch_bounds__(kHgThreads, 4) mlp_hidden_grad_kernel(const __grid_constant__ HiddenGradArgs a, const __grid_constant__ StepArgs step) {
    after_previous_kernel();
    extern __shared__ __align__(16) float hg_mem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int O = a.out_dim, S = O - D;
    const HiddenGradMem M(D, O);
    float *w2s = hg_mem, *dys = hg_mem + M.w2 + warp * M.per_warp, *raw = dys + M.raw, *small = dys + M.small, *outd = dys + M.out;
    const long long groups = (a.rows + kHgRows - 1) / kHgRows, stride = (long long)gridDim.x * kHgWarps;
    long long g = (long long)blockIdx.x * kHgWarps + warp;
    auto copy = [](float *to, const float *from, auto bytes) {
        const unsigned at = (unsigned)__cvta_generic_to_shared(to);
        if constexpr (decltype(bytes)::value == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(at), "l"(from) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(at), "l"(from) : "memory");
    };
    auto fetch = [&](long long next) {  // what the update's backward of a group reads
        if (D > 0 && next < groups) {
            constexpr int P = D == 2 ? 2 : 4;
            const long long i0 = next * kHgRows;
            const int n = (int)min((long long)kHgRows, a.rows - i0), r = lane & 7, part = lane >> 3;
            if (VEC && step.g_s_out)  // the upstream of the states is one run, 16-byte aligned
                for (int q = lane; q < n * (S / 4); q += 32) copy(raw + 4 * q, step.g_s_out + i0 * S + 4 * q, Int<16>());
            if (r < n) {  // four lanes to a row: a component each, the last one the mask
                if (part < D && step.g_x_out) copy(small + 4 * r + part, step.g_x_out + (i0 + r) * P + part, Int<4>());
                if (part < D) copy(small + kHgRows * 4 + 4 * r + part, step.y + (i0 + r) * step.y_pitch + part, Int<4>());
                if (part == 3 && step.mask) copy(small + kHgRows * 8 + r, step.mask + i0 + r, Int<4>());
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    fetch(g);
    for (int e = threadIdx.x; e < M.w2; e += kHgThreads) {
        const int o = e / kHgHidden, j = e - o * kHgHidden;
        w2s[e] = o < O ? __ldg(a.W2 + o * a.w_stride_out + j * a.w_stride_in) : 0.f;
    }
    for (int e = O * kHgPitch + lane; e < M.columns * kHgPitch; e += 32) dys[e] = 0.f;
    __syncthreads();

    for (; g < groups; g += stride) {
        const long long r0 = g * kHgRows;
        const int rows = (int)min((long long)kHgRows, a.rows - r0);
        // this pass's rows of h (32 lines) towards L1
        if (lane / 4 < rows) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.h + r0 * kHgHidden + lane * 32));
        if constexpr (D == 0) {
            const float *src = a.dy + r0 * O;  // the rows are contiguous
            for (int e = lane; e < kHgRows * O; e += 32) {
                const int r = e / O, o = e - r * O;
                dys[o * kHgPitch + r] = r < rows ? __ldg(src + e) : 0.f;
            }
            __syncwarp();
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncwarp();
            const int own = lane & 7;
            const float m = own < rows ? step.mask ? mask_value(step, small[kHgRows * 8 + own]) : 1.0f : 0.f, scale = step.dt * m;  // of row `own`
            if (lane < kHgRows) {
                float u[D], gx[D], gp[D];
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    u[d] = small[kHgRows * 4 + 4 * own + d];
                    gx[d] = small[4 * own + d];
                    gp[d] = 0.f;
                }
                if (step.g_x_out && own < rows) step_backward_position<D>(step, m, u, gx, gp);
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    dys[d * kHgPitch + own] = gp[d];
                    outd[own * O + d] = gp[d];
                }
            }
            const int pieces = VEC ? S / 4 : S, row_step = 32 / pieces, piece_step = 32 - row_step * pieces;  // pieces per row
            int row = lane / pieces, piece = lane - row * pieces;
            for (int e = lane; e < ((kHgRows * pieces + 31) & ~31); e += 32) {
                const float k = __shfl_sync(kFull, scale, row & 7);
                if (row < kHgRows) {
                    if constexpr (VEC) {
                        float4 v = step.g_s_out && row < rows ? *reinterpret_cast<const float4 *>(raw + 4 * e) : make_float4(0.f, 0.f, 0.f, 0.f);
                        v.x *= k; v.y *= k; v.z *= k; v.w *= k;
                        float *c = dys + (D + 4 * piece) * kHgPitch + row, *o = outd + row * O + D + 4 * piece;
                        c[0] = v.x; c[kHgPitch] = v.y; c[2 * kHgPitch] = v.z; c[3 * kHgPitch] = v.w;
                        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
                    } else {
                        const float v = row < rows && step.g_s_out ? k * __ldg(step.g_s_out + (r0 + row) * S + piece) : 0.f;
                        dys[(D + piece) * kHgPitch + row] = v;
                        outd[row * O + D + piece] = v;
                    }
                }
                row += row_step;
                piece += piece_step;
                if (piece >= pieces) { piece -= pieces; ++row; }
            }
            __syncwarp();
            fetch(g + stride);
            float *dst = step.g_y + r0 * O;  // 32 O bytes per group: 16-byte aligned when g_y is
            const int floats = rows * O;
            if ((uintptr_t)step.g_y % 16 == 0) {
                for (int q = lane; q < floats / 4; q += 32) reinterpret_cast<float4 *>(dst)[q] = reinterpret_cast<const float4 *>(outd)[q];
                for (int e = (floats & ~3) + lane; e < floats; e += 32) dst[e] = outd[e];
            } else {
                for (int e = lane; e < floats; e += 32) dst[e] = outd[e];
            }
        }
        unsigned long long acc[kHgRows / 2][4];  // rows (2 p, 2 p + 1) of hidden units 4 lane .. 4 lane + 3
#pragma unroll
        for (int p = 0; p < kHgRows / 2; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[p][q] = 0ull;
#pragma unroll 4
        for (int o = 0; o < M.columns; ++o) {
            const float4 w = *reinterpret_cast<const float4 *>(w2s + o * kHgHidden + 4 * lane);
            const ulonglong2 d0 = *reinterpret_cast<const ulonglong2 *>(dys + o * kHgPitch), d1 = *reinterpret_cast<const ulonglong2 *>(dys + o * kHgPitch + 4);
            const unsigned long long d[4] = {d0.x, d0.y, d1.x, d1.y}, ww[4] = {pack2(w.x, w.x), pack2(w.y, w.y), pack2(w.z, w.z), pack2(w.w, w.w)};
#pragma unroll
            for (int p = 0; p < kHgRows / 2; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[p][q] = fma2(d[p], ww[q], acc[p][q]);
        }
        const float4 *hp = reinterpret_cast<const float4 *>(a.h + r0 * kHgHidden) + lane;
        float4 *op = reinterpret_cast<float4 *>(a.dh + r0 * kHgHidden) + lane;
        float4 hv[kHgRows];
#pragma unroll
        for (int r = 0; r < kHgRows; ++r) hv[r] = r < rows ? __ldg(hp + r * (kHgHidden / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < kHgRows; ++r) {
            float lo, hi, v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                unpack2(acc[r / 2][q], lo, hi);
                v[q] = r % 2 ? hi : lo;
            }
            if (!(hv[r].x > 0.f)) v[0] = 0.f;
            if (!(hv[r].y > 0.f)) v[1] = 0.f;
            if (!(hv[r].z > 0.f)) v[2] = 0.f;
            if (!(hv[r].w > 0.f)) v[3] = 0.f;
            if (r < rows) op[r * (kHgHidden / 4)] = make_float4(v[0], v[1], v[2], v[3]);
        }
        __syncwarp();  // the staged rows are overwritten by the next pass
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

template <int D, bool VEC>
static int launch_hidden_grad(const HiddenGradArgs &a, const StepArgs &step, cudaStream_t st) {
    const auto kernel = mlp_hidden_grad_kernel<D, VEC>;
    const size_t bytes = HiddenGradMem(D, a.out_dim).bytes();
    int resident = 0;
    const int rc = persistent_ctas(kernel, kHgThreads, bytes, &resident);
    if (rc != NPA_OK) return rc;
    const long long want = (a.rows + kHgRows * kHgWarps - 1) / (kHgRows * kHgWarps);
    kernel<<<(unsigned)(want < resident ? want : resident), kHgThreads, bytes, st>>>(a, step);
    return check_launch("mlp_hidden_grad_kernel");
}

static int check_hidden_grad(const char *me, const float *W2, const float *h, const float *dh, int64_t rows, int32_t hidden, int32_t out_dim) {
    if (hidden != kHgHidden) return fail(NPA_ERR_UNSUPPORTED, "%s: hidden width must be %d, got %d", me, kHgHidden, hidden);
    if (out_dim <= 0 || out_dim > kHgMaxOut) return fail(NPA_ERR_UNSUPPORTED, "%s: supports out <= %d, got %d", me, kHgMaxOut, out_dim);
    if (rows <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: rows must be positive", me);
    if (!W2 || !h || !dh) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: every pointer must be non-NULL", me);
    if (((uintptr_t)h | (uintptr_t)dh) % 16) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: h and dh must be 16-byte aligned", me);
    return NPA_OK;
}

}  // namespace npa

using namespace npa;

extern "C" {

int npa_mlp_hidden_grad(const float *dy, const float *W2, const float *h, float *dh, int64_t rows, int32_t hidden,
                        int32_t out_dim, int64_t w_stride_out, int64_t w_stride_in, void *stream) {
    const char *me = "npa_mlp_hidden_grad";
    const int rc = check_hidden_grad(me, W2, h, dh, rows, hidden, out_dim);
    if (rc != NPA_OK) return rc;
    if (!dy) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: every pointer must be non-NULL", me);
    if ((uintptr_t)dy % 4) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: dy must be float aligned", me);
    const HiddenGradArgs a = {dy, W2, h, dh, rows, w_stride_out, w_stride_in, out_dim};
    return launch_hidden_grad<0, false>(a, StepArgs{}, (cudaStream_t)stream);
}

int npa_step_hidden_grad(const npa_grid *gd, const float *y, int32_t y_pitch, const float *mask, int32_t uniforms, float update_below, int32_t channels, float alpha,
                         float dt, const float *g_x_out, const float *g_s_out, const float *W2, const float *h, float *g_y, float *dh,
                         int32_t hidden, int64_t w_stride_out, int64_t w_stride_in, void *stream) {
    const char *me = "npa_step_hidden_grad";
    Geom g;
    int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    if (channels <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: channels must be positive, got %d", me, channels);
    const int out_dim = g.dim + channels;
    if ((rc = check_hidden_grad(me, W2, h, dh, (int64_t)g.B * g.N, hidden, out_dim)) != NPA_OK) return rc;
    if (!y || !g_y) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: y and g_y must be non-NULL", me);
    if (y_pitch < g.dim) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: rows of %d floats do not hold a displacement", me, y_pitch);
    StepArgs s = {};
    s.y = y; s.y_pitch = y_pitch; s.mask = mask; s.uniforms = uniforms; s.below = update_below; s.g_x_out = g_x_out; s.g_s_out = g_s_out; s.g_y = g_y;
    s.particles = (long long)g.B * g.N; s.C = channels; s.alpha = alpha; s.eps = g.h; s.dt = dt;
    const HiddenGradArgs a = {nullptr, W2, h, dh, s.particles, w_stride_out, w_stride_in, out_dim};
    cudaStream_t st = (cudaStream_t)stream;
    const bool vec = channels % 4 == 0 && (uintptr_t)g_s_out % 16 == 0;
    if (g.dim == 2) return vec ? launch_hidden_grad<2, true>(a, s, st) : launch_hidden_grad<2, false>(a, s, st);
    return vec ? launch_hidden_grad<3, true>(a, s, st) : launch_hidden_grad<3, false>(a, s, st);
}

}  // extern "C"
