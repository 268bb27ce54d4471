// Wide linear layers of the per-particle MLP on the fifth-generation tensor cores (tcgen05.mma,
// accumulators in tensor memory), at fp32 accuracy.
//
//     C[M, N] = act( A[M, K] . B[K, N] + bias[N] ),    B[k][n] = W[n * stride_n + k * stride_k]
//
// the same contract as npa_linear_tf32x3 (mlp_gemm.cu) for the wide products of the adaptation MLP of
// an NPA model (models/npa.py:63-75): h = relu(z W1^T + b1) and dz = dh W1 with M = B*N particles.
// Each product is three TF32 MMAs on operands split into a TF32 head and tail (a = a_hi + a_lo;
// a.b ~ a_lo b_hi + a_hi b_lo + a_hi b_hi, fp32 accumulation): the dropped a_lo b_lo term is 2^-22
// of the product.
//
// One persistent CTA per SM, warp-specialised, tiles of 128 rows, K walked in chunks of 32 floats
// (one 128-byte swizzle row):
//
//   * 16 producer warps read the rows of A from global memory (coalesced 128-byte row segments, three
//     chunks in flight in registers), split every element and write head and tail into the stage's
//     two K-major 128-byte-swizzled operand tiles;
//   * one lane streams the matching chunk of the weights -- split and swizzled once per call by
//     weight_image_kernel into an image that is copied verbatim -- with one bulk copy per stage;
//   * one lane issues the MMAs (M = 128, N = out_dim rounded up to 16, K = 8 per instruction) into
//     one of two accumulators in tensor memory and commits the stage back to the producers;
//   * eight epilogue warps read a finished accumulator (tcgen05.ld, lane = row, 16 columns at a time),
//     turn the blocks through shared memory and store rows with bias, ReLU and the optional gate
//     applied (float4 when out_dim is a multiple of 4).
//
// The forward of a step ends with the Euler update (step_update.cuh): the epilogue has y's tile in shared memory and writes the updated
// positions and states instead of y, of which the backward only needs the raw displacements.  Measured, B200, us, two kernels -> one:
// 262,144 particles in 3D, C = 32, 142 + 25.5 -> 159; pass of an inference step of 4,096 in 2D 54.2 -> 52.7, of 2,500 in a graph 37.8 -> 35.8.
//
// The backward of a step whose positions want no gradient takes dL/dz = dh W1 apart in the epilogue (umma_store_parts): the weights' columns
// stand in the order of StepColumns, so that an axis of the gradient is a run of columns, and the rows that the feature sweep reads leave
// instead of dL/dz, which went to memory (rows of an odd number of floats) and came back.  Measured, B200, us, with the kernel that took it
// apart before -> this one: 262,144 particles in 3D, C = 32, 97 + 85 -> 124; 65,536, C = 16, 27 + 16 -> 30; 32,768 in 2D 17 + 11 -> 17.5 (a
// training step 1,466 -> 1,422, 304 -> 296, 183 -> 175).  Same products and expressions: the same bits.
//
// Every wait on an mbarrier is bounded in time; a wait that gives up raises a flag that ends all
// roles, the CTA frees its tensor memory and the host reads the reason from a status word.
#include <mutex>

#include "perceive_backward.cuh"
#include "step_update.cuh"
#include "umma.cuh"
#include "weight_image.cuh"

namespace npa {

constexpr int kUmmaRows = 128;
constexpr int kUmmaChunk = kImageChunk;   // floats of K per stage
constexpr int kUmmaProducerWarps = 16;
constexpr int kUmmaEpilogueWarps = 8;     // two per quarter of the accumulator's lanes
constexpr int kUmmaWarpMma = 8, kUmmaWarpWeights = 9, kUmmaWarpProducer0 = 10;
constexpr int kUmmaThreads = (kUmmaWarpProducer0 + kUmmaProducerWarps) * 32;
constexpr int kUmmaMaxStages = 4;
constexpr int kUmmaTmemCols = 512;        // two accumulators of up to 256 columns
constexpr int kUmmaAccStride = 256;
constexpr int kUmmaTileABytes = kUmmaRows * kUmmaChunk * 4;  // one operand tile of A: 16 KB
constexpr int kUmmaEpiPitch = 20;         // floats per staged row of 16 columns: 16-byte aligned, conflict-free float4 writes
constexpr int kUmmaEpiFloats = kUmmaEpilogueWarps * 32 * kUmmaEpiPitch;

constexpr int kUmmaHloCol = 256, kUmmaYCol = 384, kUmmaY2Col = 448;  // two-layer mode: accumulators at 0 / 128, tail of h, the second layer's two accumulators

// D[tmem] (+)= A[tmem] . B[smem]^T: the A operand (128 lanes x 8 columns of 32-bit values) is read from tensor memory.
__device__ inline void umma_tf32_ts(unsigned d_tmem, unsigned a_tmem, uint64_t b_desc, unsigned idesc, int accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

enum { UMMA_STATUS_MMA = 1, UMMA_STATUS_WEIGHTS = 2, UMMA_STATUS_PRODUCER = 4, UMMA_STATUS_EPILOGUE = 8 };

struct UmmaShared {
    uint64_t full[kUmmaMaxStages], empty[kUmmaMaxStages], acc_full[2], acc_empty[2];
    uint64_t h_ready[2], y_full, w2_full, y_written, y_copied;  // two-layer mode only
    uint32_t tmem_base;
    int abort;
    alignas(16) float bias[256];
};

struct UmmaArgs {
    const float *A;      // [M, K], row pitch K
    const float *Wimg;   // [nchunks][head | tail][Np rows x 128 bytes, swizzled]
    const float *bias;   // [N] or NULL
    const float *gate;   // [M, N] or NULL: the output is zero where gate <= 0
    float *C;            // [M, N], row pitch N
    long long M;
    int K, N, Np, nchunks, last_ksteps, stages, stage_bytes, relu;
    unsigned *status;
    // two-layer mode (Y != NULL): Y [M, N2] = C . W2^T with C = the activated output of the first layer kept in
    // tensor memory; N = Np = 128, W2img = [4 chunks][head | tail][N2p rows x 128 bytes, swizzled]
    const float *W2img;
    float *Y;
    int N2, N2p;
    // with the Euler update (D > 0): instead of the rows of the second layer the updated positions and states leave, and
    // into step.y (NULL: nobody wants them) rows of step.y_pitch floats that begin with the raw displacements
    int D;
    StepArgs step;
    Geom g;
    StepRows parts;  // kUmmaParts: where the rows go instead of C
};
constexpr int kUmmaStepQuads = 4;  // float4 of the states per epilogue thread and tile: up to 32 features

__device__ unsigned g_umma_status;

__global__ void weight_image_kernel(const __grid_constant__ ImageJobs jobs) {
    after_previous_kernel();
    write_image_element(jobs, blockIdx.x * blockDim.x + threadIdx.x);
}

enum : int { kUmmaOneLayer = 0, kUmmaTwoLayers = 1, kUmmaStep = 2, kUmmaParts2 = 3, kUmmaParts3 = 4, kUmmaModes = 5 };
constexpr int kUmmaPartPitch = 12;  // floats per staged row of 8 features: float4 writes of eight lanes cover all banks
__host__ __device__ constexpr int umma_epilogue_floats(int mode) {
    return mode == kUmmaParts2 || mode == kUmmaParts3 ? kUmmaEpilogueWarps * 32 * kUmmaPartPitch * (mode == kUmmaParts2 ? 4 : 5) : kUmmaEpiFloats;
}

// The tile of the second layer as the Euler update: the epilogue's threads move four states at a time, the first 128 of them a position.
template <int D>
__device__ __forceinline__ void umma_store_step(const UmmaArgs &a, const float *tile, long long row0, int rows, int e, const float4 (&s_bin)[kUmmaStepQuads],
                                                const float (&m)[kUmmaStepQuads], float m_x, const float4 &x_bin) {
    const StepArgs &st = a.step;
    const int C4 = st.C / 4, W = D + st.C;
#pragma unroll
    for (int k = 0; k < kUmmaStepQuads; ++k) {
        const int q = e + k * kUmmaEpilogueWarps * 32;
        if (q < rows * C4) {
            const int row = q / C4;
            reinterpret_cast<float4 *>(st.s_out)[row0 * C4 + q] = step_forward_states(st, m[k], s_bin[k], tile + row * W + D + 4 * (q - row * C4));
        }
    }
    if (e < rows) {
        const float *u = tile + e * W;
        float x[4] = {x_bin.x, x_bin.y, x_bin.z, x_bin.w};
        step_forward_position<D>(st, a.g, m_x, u, x);
        if (D == 2) {
            reinterpret_cast<float2 *>(st.x_out)[row0 + e] = make_float2(x[0], x[1]);
            if (st.y) reinterpret_cast<float2 *>(const_cast<float *>(st.y))[row0 + e] = make_float2(u[0], u[1]);
        } else {
            reinterpret_cast<float4 *>(st.x_out)[row0 + e] = make_float4(x[0], x[1], x[2], x[3]);
            if (st.y) reinterpret_cast<float4 *>(const_cast<float *>(st.y))[row0 + e] = make_float4(u[0], u[1], u[2], 0.f);
        }
    }
}

// What the update will read of a tile's particles towards L2: the states, positions and mask were last touched before the perception, whose
// rows of z may have taken their place (the kernel for 262,144 particles in 3D: 159 us with it, 167 without; loading them into registers
// ahead of the last pass instead 178, spills).
__device__ __forceinline__ void umma_prefetch_step(const UmmaArgs &a, long long tile, int e) {
    const long long row0 = tile * kUmmaRows;
    const int rows = a.M - row0 < kUmmaRows ? (int)(a.M - row0) : kUmmaRows, P = a.D == 2 ? 2 : 4;
    auto fetch = [](const float *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); };
    if (e * 32 < rows * a.step.C) fetch(a.step.s_bin + row0 * a.step.C + e * 32);  // 256 threads: up to 64 features
    const int f = kUmmaEpilogueWarps * 32 - 1 - e;
    if (f * 32 < rows * P) fetch(a.step.x_bin + row0 * P + f * 32);
    else if (f >= 16 && f < 20 && a.step.mask && (f - 16) * 32 < rows) fetch(a.step.mask + row0 + (f - 16) * 32);
}

// One warp's 32 rows of a tile of dL/dz, columns in the order of StepColumns, as the upstream rows of the perception's backward: eight features
// at a time, every second eight (`first`: 0 or 1); lane = row, four features' gradients through the log-normalisation together, then
// through shared memory so that 32-byte sectors leave whole.  `release` hands the accumulator back.
template <int D, typename Release>
__device__ __forceinline__ void umma_store_parts(const StepRows &p, unsigned taddr, float *stg, long long row0, int nrows, int first, int lane, Release release) {
    const int C = p.C, S = StepColumns::section(C), units = (C + 7) / 8;
    const float *vg = p.vgrad + (row0 + lane) * C * D;
    float v[4 * D];
    auto fetch = [&](int f) {
#pragma unroll
        for (int q = 0; q < D; ++q) {
            const float4 t = lane < nrows ? __ldg(reinterpret_cast<const float4 *>(vg + f * D) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
        }
    };
    if (first >= units) {
        release();
        return;
    }
    fetch(8 * first);
    float *mine = stg + lane * kUmmaPartPitch;
#pragma unroll 1
    for (int u = first; u < units; u += 2) {
        const int f0 = 8 * u, width = min(8, C - f0);
#pragma unroll
        for (int sec = 0; sec < 2; ++sec) {
            unsigned r[8];
            tmem_ld8(taddr + sec * S + f0, r);
            tc_wait_ld();
#pragma unroll
            for (int q = 0; q < 2; ++q)
                *reinterpret_cast<float4 *>(mine + sec * 32 * kUmmaPartPitch + 4 * q) =
                    make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
        }
#pragma unroll 1
        for (int h = 0; h < width; h += 4) {
            unsigned r[D][4];
            float out[D][4], w[4 * D];
#pragma unroll
            for (int d = 0; d < D; ++d) tmem_ld4(taddr + (2 + d) * S + f0 + h, r[d]);
#pragma unroll
            for (int q = 0; q < 4 * D; ++q) w[q] = v[q] * p.coef;
            const int next = h + 4 < width ? f0 + h + 4 : f0 + 16;
            if (next < C) fetch(next);
            tc_wait_ld();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float gin[D], gout[D];
#pragma unroll
                for (int d = 0; d < D; ++d) gin[d] = __uint_as_float(r[d][q]);
                log_normalize_backward<D>(w + q * D, gin, p.log_norm, p.coef, gout);
#pragma unroll
                for (int d = 0; d < D; ++d) out[d][q] = gout[d];
            }
#pragma unroll
            for (int d = 0; d < D; ++d)
                *reinterpret_cast<float4 *>(mine + (2 + d) * 32 * kUmmaPartPitch + h) = make_float4(out[d][0], out[d][1], out[d][2], out[d][3]);
        }
        if (u + 2 >= units) release();
        __syncwarp();
        const int half = 4 * (lane & 1);
        if (half < width) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int row = (lane >> 1) + 16 * i;
                if (row >= nrows) continue;
                const float *from = stg + row * kUmmaPartPitch + half;
                *reinterpret_cast<float4 *>(p.direct + (row0 + row) * C + f0 + half) = *reinterpret_cast<const float4 *>(from);
                float *to = p.rows + (row0 + row) * p.pitch + f0 + half;
#pragma unroll
                for (int sec = 0; sec <= D; ++sec)
                    *reinterpret_cast<float4 *>(to + sec * C) = *reinterpret_cast<const float4 *>(from + (1 + sec) * 32 * kUmmaPartPitch);
            }
        }
        __syncwarp();
    }
}

template <int MODE>
__global__ void __launch_bounds__(kUmmaThreads, 1) linear_umma_kernel(const __grid_constant__ UmmaArgs args) {
    after_previous_kernel();
    // every field is read into a register once: the role loops below must not go back to the parameter block
    const float *__restrict__ A = args.A;
    const float *__restrict__ Wimg = args.Wimg;
    const float *__restrict__ gate = args.gate;
    float *__restrict__ C = args.C;
    unsigned *status = args.status;
    const long long M = args.M;
    const int K = args.K, N = args.N, Np = args.Np, nchunks = args.nchunks, last_ksteps = args.last_ksteps;
    const int stages = args.stages, stage_bytes = args.stage_bytes;
    const bool relu = args.relu != 0;
    constexpr bool fuse = MODE == kUmmaTwoLayers || MODE == kUmmaStep;  // two-layer mode
    constexpr int kParts = MODE == kUmmaParts2 ? 2 : MODE == kUmmaParts3 ? 3 : 0;
    const int N2 = args.N2, N2p = args.N2p;
    const int acc_stride = fuse ? 128 : kUmmaAccStride;
    extern __shared__ uint8_t umma_smem_raw[];
    uint8_t *base = umma_smem_raw + ((1024u - (smem_u32(umma_smem_raw) & 1023u)) & 1023u);
    uint8_t *w2s = base + (size_t)stages * stage_bytes;   // two-layer mode: the whole image of W2, resident
    const int w2_bytes = fuse ? 4 * 2 * N2p * 128 : 0;
    float *epi = (float *)(w2s + w2_bytes);
    float *ytile = epi + umma_epilogue_floats(MODE);                  // two-layer mode: the second layer's tile, rows of N2 floats as in global memory
    UmmaShared *sh = (UmmaShared *)(ytile + (fuse ? ((kUmmaRows * N2 + 3) & ~3) : 0));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&sh->full[s], kUmmaProducerWarps + 1);  // one arrival per producer warp + the weight copy
            mbar_init(&sh->empty[s], 1);                      // the commit of the stage's MMAs
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(&sh->acc_full[q], 1);
            // free again: when every epilogue warp has read it and (two layers) the second layer's MMAs have as well
            mbar_init(&sh->acc_empty[q], fuse ? 1 + kUmmaEpilogueWarps : kUmmaEpilogueWarps);
            mbar_init(&sh->h_ready[q], kUmmaEpilogueWarps);
        }
        mbar_init(&sh->y_full, 1);
        mbar_init(&sh->w2_full, 1);
        mbar_init(&sh->y_written, kUmmaEpilogueWarps);
        mbar_init(&sh->y_copied, kUmmaEpilogueWarps);
        sh->abort = 0;
        mbar_fence_init();
    }
    for (int c = threadIdx.x; c < 256; c += kUmmaThreads) sh->bias[c] = (args.bias && c < N) ? __ldg(args.bias + c) : 0.f;
    if (warp == kUmmaWarpMma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)),
                     "r"(kUmmaTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = sh->tmem_base;

    const long long tiles = (M + kUmmaRows - 1) / kUmmaRows;
    const int ntile = (int)((tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);  // tiles blockIdx.x, + gridDim.x, ...
    const int total = ntile * nchunks;
    bool ok = true;

    if (warp == kUmmaWarpMma) {
        // One lane runs the whole role; stage, phase and descriptors advance by additions only.
        if (lane == 0) {
            // M = 128, N = Np, TF32 x TF32 -> F32, both operands K-major
            const unsigned idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(Np >> 3) << 17) | ((unsigned)(kUmmaRows >> 4) << 24);
            const uint64_t desc0 = umma_desc(smem_u32(base));
            const uint64_t stage16 = (uint64_t)(stage_bytes >> 4), alo16 = kUmmaTileABytes >> 4, bhi16 = (2 * kUmmaTileABytes) >> 4;
            const uint64_t blo16 = bhi16 + (uint64_t)((Np * 128) >> 4);
            int s = 0;
            unsigned ph = 0;
            // second layer of tile t (two-layer mode): Y tile = h . W2^T with h (in place, activated) and its tail in
            // tensor memory; it runs after the first layer of tile t + 1 has been issued, so that the epilogue of
            // tile t overlaps those MMAs
            const unsigned idesc2 = (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(N2p >> 3) << 17) | ((unsigned)(kUmmaRows >> 4) << 24);
            const uint64_t w2desc = umma_desc(smem_u32(w2s));
            auto second_layer = [&](int t) -> bool {
                const int a = t & 1;
                if (t == 0 && !umma_wait(&sh->w2_full, 0, &sh->abort)) return false;
                if (!umma_wait(&sh->h_ready[a], (t >> 1) & 1, &sh->abort)) return false;
                tc_fence_after();
                // two accumulators (the epilogue adds them): consecutive MMAs into one accumulator wait for each other,
                // and at 48 columns that wait is longer than the MMA
                const unsigned dy = tmem + kUmmaYCol, dy2 = tmem + kUmmaY2Col, ah = tmem + a * 128, al = tmem + kUmmaHloCol;
#pragma unroll 1
                for (int ks = 0; ks < 16; ++ks) {
                    const uint64_t b_hi = w2desc + (uint64_t)(((ks >> 2) * 2 * N2p * 128) >> 4) + 2ull * (ks & 3);
                    const uint64_t b_lo = b_hi + (uint64_t)((N2p * 128) >> 4);
                    umma_tf32_ts(dy, al + 8 * ks, b_hi, idesc2, ks != 0);
                    umma_tf32_ts(dy2, ah + 8 * ks, b_hi, idesc2, ks != 0);
                    umma_tf32_ts(dy, ah + 8 * ks, b_lo, idesc2, 1);
                }
                umma_commit(&sh->y_full);
                umma_commit(&sh->acc_empty[a]);  // the accumulator that held h is free when these MMAs are done
                return true;
            };
#pragma unroll 1
            for (int it = 0; it < ntile; ++it) {
                const int acc = it & 1;
                if (!(ok = umma_wait(&sh->acc_empty[acc], ((it >> 1) & 1) ^ 1, &sh->abort))) break;
                tc_fence_after();
                const unsigned d = tmem + acc * acc_stride;
#pragma unroll 1
                for (int c = 0; c < nchunks; ++c) {
                    if (!(ok = umma_wait(&sh->full[s], ph, &sh->abort))) break;
                    tc_fence_after();
                    const uint64_t a_hi = desc0 + stage16 * s, a_lo = a_hi + alo16, b_hi = a_hi + bhi16, b_lo = a_hi + blo16;
                    const int ksteps = c == nchunks - 1 ? last_ksteps : kUmmaChunk / 8;
#pragma unroll
                    for (int ks = 0; ks < kUmmaChunk / 8; ++ks) {
                        if (ks >= ksteps) break;
                        const uint64_t o = 2ull * ks;  // 8 floats = 32 bytes further along K, in 16-byte units
                        umma_tf32(d, a_lo + o, b_hi + o, idesc, (c | ks) != 0);
                        umma_tf32(d, a_hi + o, b_lo + o, idesc, 1);
                        umma_tf32(d, a_hi + o, b_hi + o, idesc, 1);
                    }
                    umma_commit(&sh->empty[s]);
                    if (c == nchunks - 1) umma_commit(&sh->acc_full[acc]);
                    if (++s == stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (!ok) break;
                if (fuse && it >= 1 && !(ok = second_layer(it - 1))) break;
            }
            if (ok && fuse && ntile > 0) ok = second_layer(ntile - 1);
            if (!ok) atomicOr(status, UMMA_STATUS_MMA);
        }
        __syncwarp();
    } else if (warp == kUmmaWarpWeights) {
        if (lane == 0) {
            const unsigned bytes = 2u * Np * 128u;
            const size_t chunk_floats = (size_t)2 * Np * kUmmaChunk;
            int s = 0, c = 0;
            unsigned ph = 1;  // the first pass over the stages finds them free
            if (fuse) {
                mbar_arrive_expect(&sh->w2_full, (unsigned)w2_bytes);
                bulk_copy_g2s(w2s, args.W2img, (unsigned)w2_bytes, &sh->w2_full);
            }
#pragma unroll 1
            for (int q = 0; q < total; ++q) {
                if (!(ok = umma_wait(&sh->empty[s], ph, &sh->abort))) break;
                mbar_arrive_expect(&sh->full[s], bytes);
                bulk_copy_g2s(base + (size_t)s * stage_bytes + 2 * kUmmaTileABytes, Wimg + chunk_floats * c, bytes, &sh->full[s]);
                if (++s == stages) {
                    s = 0;
                    ph ^= 1;
                }
                if (++c == nchunks) c = 0;
            }
            if (!ok) {
                atomicOr(status, UMMA_STATUS_WEIGHTS);
                __nanosleep(20000);  // a copy issued just before the flag was seen lands before the CTA leaves
            }
        }
    } else if (warp >= kUmmaWarpProducer0) {
        const int pw = warp - kUmmaWarpProducer0;  // rows 8 pw .. 8 pw + 7 of every tile
        // the load stream runs two chunks ahead of the store stream; both advance by additions only
        long long l_row0 = (long long)blockIdx.x * kUmmaRows + pw * 8;
        int l_c = 0;
        auto load = [&](float (&v)[8]) {
            const int k = l_c * kUmmaChunk + lane;
            const float *p = A + l_row0 * K + k;
            if (l_row0 + 8 <= M && l_c * kUmmaChunk + kUmmaChunk <= K) {
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = __ldg(p + (long long)j * K);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = (l_row0 + j < M && k < K) ? __ldg(p + (long long)j * K) : 0.f;
            }
            if (++l_c == nchunks) {
                l_c = 0;
                l_row0 += (long long)gridDim.x * kUmmaRows;
            }
        };
        int s = 0;
        unsigned ph = 1;
        auto store = [&](const float (&v)[8]) -> bool {
            if (!umma_wait(&sh->empty[s], ph, &sh->abort)) return false;
            float *hi = (float *)(base + (size_t)s * stage_bytes), *lo = hi + kUmmaRows * kUmmaChunk;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int at = umma_swizzled(pw * 8 + j, lane);
                const float head = __uint_as_float(tf32_head_bits(v[j]));
                hi[at] = head;
                lo[at] = v[j] - head;
            }
            fence_proxy_async();  // the MMA reads these through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->full[s]);
            if (++s == stages) {
                s = 0;
                ph ^= 1;
            }
            return true;
        };
        // Three chunks in flight in three register sets that take turns (no register is copied: a copy
        // would wait for the load it reads and end the overlap).
        float v0[8], v1[8], v2[8];
        if (0 < total) load(v0);
        if (1 < total) load(v1);
#pragma unroll 1
        for (int q = 0; q < total; q += 3) {
            if (q + 2 < total) load(v2);
            if (!(ok = store(v0))) break;
            if (q + 1 >= total) break;
            if (q + 3 < total) load(v0);
            if (!(ok = store(v1))) break;
            if (q + 2 >= total) break;
            if (q + 4 < total) load(v1);
            if (!(ok = store(v2))) break;
        }
        if (!ok && lane == 0) atomicOr(status, UMMA_STATUS_PRODUCER);
    } else {
        // epilogue: warp w reads lanes 32 (w % 4) .. + 31 of the accumulator (= rows of the tile) and every
        // second block of 16 columns; a block goes through shared memory so that rows leave coalesced.
        // Two-layer mode: pass 0 activates the first layer's tile and writes it back in place together with its
        // TF32 tail (the A operand of the second layer; nothing else, so that the second layer can start early),
        // pass 1 stores the activated tile, pass 2 stores the second layer's tile.
        float *stg = epi + warp * 32 * kUmmaEpiPitch;
        const int quarter = warp & 3, first_block = warp >> 2;
        const float neg_inf = -__int_as_float(0x7f800000);
        const unsigned tlane = tmem + ((unsigned)(quarter * 32) << 16);
#pragma unroll 1
        for (int it = 0; it < ntile && ok; ++it) {
            const int acc = it & 1;
            const long long row0 = ((long long)blockIdx.x + (long long)it * gridDim.x) * kUmmaRows + quarter * 32;
            const int nrows = M - row0 < 32 ? (int)(M - row0) : 32;  // may be <= 0 in the last tile
            if constexpr (kParts > 0) {
                const int rows_here = M - (row0 - quarter * 32) < kUmmaRows ? (int)(M - (row0 - quarter * 32)) : kUmmaRows;
                for (int q = (warp * 32 + lane) * 32; q < rows_here * args.parts.C * kParts; q += kUmmaEpilogueWarps * 32 * 32)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(args.parts.vgrad + (row0 - quarter * 32) * args.parts.C * kParts + q));
                if (!(ok = umma_wait(&sh->acc_full[acc], (it >> 1) & 1, &sh->abort))) break;
                tc_fence_after();
                umma_store_parts<kParts>(args.parts, tlane + acc * acc_stride, epi + warp * 32 * kUmmaPartPitch * (2 + kParts), row0, nrows, first_block, lane, [&]() {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh->acc_empty[acc]);
                });
                continue;
            }
            if constexpr (MODE == kUmmaStep) umma_prefetch_step(args, (long long)blockIdx.x + (long long)it * gridDim.x, warp * 32 + lane);
#pragma unroll 1
            for (int pass = fuse ? 0 : 1; pass < (fuse ? 3 : 2); ++pass) {
                // what this pass reads and where it goes
                const bool act_here = fuse && pass == 0;           // bias and activation in registers, written back
                const bool post = !fuse;                            // bias and activation while storing
                float *const out = pass == 2 ? args.Y : C;
                const int ncol = pass == 2 ? N2 : N;
                const int nblocks = (pass == 2 ? N2p : Np) >> 4;
                const unsigned taddr0 = tlane + (pass == 2 ? kUmmaYCol : acc * acc_stride);
                const float lo = (post && relu) ? 0.f : neg_inf;
                const float *gt0 = (post && gate) ? gate : nullptr;
                const bool vec4 = (ncol & 3) == 0 && ((uintptr_t)out & 15) == 0 && (!gt0 || ((uintptr_t)gt0 & 15) == 0);
                if (fuse && pass == 1 && !C) {  // nobody wants the hidden layer: hand the accumulator back
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh->acc_empty[acc]);
                    continue;
                }
                if (pass != 1 || !fuse) {  // pass 1 of the two-layer mode reads what pass 0 of the same thread wrote
                    if (!(ok = umma_wait(pass == 2 ? &sh->y_full : &sh->acc_full[acc], pass == 2 ? it & 1 : (it >> 1) & 1, &sh->abort))) break;
                    tc_fence_after();
                }
                // the previous tile's rows have left the shared-memory tile
                if (fuse && pass == 2 && !(ok = umma_wait(&sh->y_copied, (it & 1) ^ 1, &sh->abort))) break;
                int last_block = first_block;
                while (last_block + 2 < nblocks) last_block += 2;
#pragma unroll 1
                for (int b = first_block; b < nblocks; b += 2) {
                    const int c0 = b << 4;
                    unsigned r[16];
                    tmem_ld16(taddr0 + c0, r);
                    tc_wait_ld();
                    if (pass == 1 && b == last_block) {  // this warp has read its last block: hand its share of the accumulator back
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&sh->acc_empty[acc]);
                    }
                    if (fuse && pass == 2) {
                        // the second layer's tile: the sum of its two accumulators goes into a shared-memory tile laid out
                        // like the tile's rows in global memory (they are contiguous there), copied out linearly below
                        unsigned r2[16];
                        tmem_ld16(tlane + kUmmaY2Col + c0, r2);
                        tc_wait_ld();
                        float *yrow = ytile + (quarter * 32 + lane) * ncol + c0;
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c0 + j < ncol) yrow[j] = __uint_as_float(r[j]) + __uint_as_float(r2[j]);
                        continue;
                    }
                    if (act_here) {
                        unsigned tail[16];
                        float bj[16];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float4 b4 = *(const float4 *)(sh->bias + c0 + 4 * j);
                            bj[4 * j] = b4.x; bj[4 * j + 1] = b4.y; bj[4 * j + 2] = b4.z; bj[4 * j + 3] = b4.w;
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            float v = __uint_as_float(r[j]) + bj[j];
                            if (relu) v = fmaxf(v, 0.f);
                            r[j] = __float_as_uint(v);
                            tail[j] = __float_as_uint(v - __uint_as_float(tf32_head_bits(v)));
                        }
                        tmem_st16(taddr0 + c0, r);                 // the MMA reads the head of these by truncation
                        tmem_st16(tlane + kUmmaHloCol + c0, tail);
                        continue;
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *(float4 *)(stg + lane * kUmmaEpiPitch + 4 * j) = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                                                     __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
                    __syncwarp();
                    if (vec4) {
                        // eight rows x four float4 per instruction; the two rows of a quarter-warp are four staged
                        // rows apart (4 x 20 floats = 16 banks), so that its eight float4 cover all 32 banks
                        const int c4 = 4 * (lane & 3), t = lane >> 2, sub = (t >> 1) + 4 * (t & 1);
                        if (c0 + c4 < ncol) {
                            const float4 bv = post ? *(const float4 *)(sh->bias + c0 + c4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int rr = 8 * i + sub;
                                if (rr < nrows) {
                                    float4 v = *(const float4 *)(stg + rr * kUmmaEpiPitch + c4);
                                    v.x = fmaxf(v.x + bv.x, lo); v.y = fmaxf(v.y + bv.y, lo);
                                    v.z = fmaxf(v.z + bv.z, lo); v.w = fmaxf(v.w + bv.w, lo);
                                    const long long at = (row0 + rr) * ncol + c0 + c4;
                                    if (gt0) {
                                        const float4 gv = __ldg((const float4 *)(gt0 + at));
                                        if (!(gv.x > 0.f)) v.x = 0.f;
                                        if (!(gv.y > 0.f)) v.y = 0.f;
                                        if (!(gv.z > 0.f)) v.z = 0.f;
                                        if (!(gv.w > 0.f)) v.w = 0.f;
                                    }
                                    *(float4 *)(out + at) = v;
                                }
                            }
                        }
                    } else {
                        const int cc = lane & 15, sub = lane >> 4;  // two rows x sixteen columns per instruction
                        if (c0 + cc < ncol) {
                            const float bv = post ? sh->bias[c0 + cc] : 0.f;
                            float *dst = out + (row0 + sub) * ncol + c0 + cc;
                            const float *gt = gt0 ? gt0 + (row0 + sub) * ncol + c0 + cc : nullptr;
                            const float *src = stg + sub * kUmmaEpiPitch + cc;
#pragma unroll 4
                            for (int rr = sub; rr < nrows; rr += 2) {
                                float v = fmaxf(*src + bv, lo);
                                if (gt) {
                                    if (!(__ldg(gt) > 0.f)) v = 0.f;
                                    gt += 2 * ncol;
                                }
                                *dst = v;
                                dst += 2 * ncol;
                                src += 2 * kUmmaEpiPitch;
                            }
                        }
                    }
                    __syncwarp();
                }
                if (fuse && pass == 2) {
                    const int e = warp * 32 + lane;
                    [[maybe_unused]] float4 s_bin[kUmmaStepQuads], x_bin = make_float4(0.f, 0.f, 0.f, 0.f);
                    [[maybe_unused]] float m[kUmmaStepQuads], m_x = 1.f;
                    if constexpr (MODE == kUmmaStep) {  // what the update reads of the tile's particles, while the other warps finish
                        const long long r0 = ((long long)blockIdx.x + (long long)it * gridDim.x) * kUmmaRows;
                        const int here = M - r0 < kUmmaRows ? (int)(M - r0) : kUmmaRows, C4 = args.step.C / 4;
#pragma unroll
                        for (int k = 0; k < kUmmaStepQuads; ++k) {
                            const int q = e + k * kUmmaEpilogueWarps * 32;
                            s_bin[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                            m[k] = 1.f;
                            if (q < here * C4) {
                                s_bin[k] = __ldg(reinterpret_cast<const float4 *>(args.step.s_bin) + r0 * C4 + q);
                                m[k] = mask_of(args.step, r0 + q / C4);
                            }
                        }
                        if (e < here) {
                            m_x = mask_of(args.step, r0 + e);
                            if (args.D == 2) {
                                const float2 v = __ldg(reinterpret_cast<const float2 *>(args.step.x_bin) + r0 + e);
                                x_bin.x = v.x; x_bin.y = v.y;
                            } else {
                                x_bin = __ldg(reinterpret_cast<const float4 *>(args.step.x_bin) + r0 + e);
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh->y_written);
                    if (!(ok = umma_wait(&sh->y_written, it & 1, &sh->abort))) break;
                    // all eight warps copy the tile: (rows that exist) x N2 floats, contiguous and 16-byte aligned in global memory
                    const long long tile_row0 = ((long long)blockIdx.x + (long long)it * gridDim.x) * kUmmaRows;
                    const int rows_here = M - tile_row0 < kUmmaRows ? (int)(M - tile_row0) : kUmmaRows;
                    const int total = rows_here * ncol;
                    float *dst = out + tile_row0 * ncol;
                    if constexpr (MODE == kUmmaStep) {
                        if (args.D == 2) umma_store_step<2>(args, ytile, tile_row0, rows_here, e, s_bin, m, m_x, x_bin);
                        else umma_store_step<3>(args, ytile, tile_row0, rows_here, e, s_bin, m, m_x, x_bin);
                    } else if (((uintptr_t)out & 15) == 0) {
                        for (int q = e; q < total / 4; q += kUmmaEpilogueWarps * 32) ((float4 *)dst)[q] = ((const float4 *)ytile)[q];
                        for (int q = (total & ~3) + e; q < total; q += kUmmaEpilogueWarps * 32) dst[q] = ytile[q];
                    } else {
                        for (int q = e; q < total; q += kUmmaEpilogueWarps * 32) dst[q] = ytile[q];
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh->y_copied);
                }
                if (act_here) {  // h and its tail are in tensor memory: the second layer (and pass 1) may read them
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh->h_ready[acc]);
                }
            }
        }
        if (!ok && lane == 0) atomicOr(status, UMMA_STATUS_EPILOGUE);
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kUmmaWarpMma) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kUmmaTmemCols) : "memory");
    }
}

// Self-test of the bounded waits: warp 0 waits, with a short limit, on an mbarrier that nothing completes
// and raises the flag; warp 1 waits with the full limit on another one and must leave through the flag.
// result[0] = 1 when warp 0 gave up, result[1] = 1 when warp 1 left because of the flag.
__global__ void umma_wait_selftest_kernel(unsigned long long limit_ns, int *result) {
    __shared__ uint64_t bar[2];
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        abort_flag = 0;
        mbar_fence_init();
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    const unsigned long long t0 = global_timer_ns();
    const bool completed = warp == 0 ? umma_wait(&bar[0], 0u, &abort_flag, limit_ns) : umma_wait(&bar[1], 0u, &abort_flag);
    const bool by_flag = global_timer_ns() - t0 < kUmmaWaitNs / 2;
    if ((threadIdx.x & 31) == 0) result[warp] = completed ? 0 : (warp == 0 || by_flag ? 1 : 2);
}

static void (*umma_kernel(int mode))(UmmaArgs) {
    switch (mode) {
        case kUmmaStep: return linear_umma_kernel<kUmmaStep>;
        case kUmmaTwoLayers: return linear_umma_kernel<kUmmaTwoLayers>;
        case kUmmaParts2: return linear_umma_kernel<kUmmaParts2>;
        case kUmmaParts3: return linear_umma_kernel<kUmmaParts3>;
        default: return linear_umma_kernel<kUmmaOneLayer>;
    }
}

// Per-device set-up done once: the address of the status word and the shared-memory limit of the kernel.
struct UmmaDevice {
    unsigned *status = nullptr;
    int smem_limit[kUmmaModes] = {};  // per kernel instantiation
};
static std::mutex g_umma_mutex;
static UmmaDevice g_umma_device[64];

static int umma_device_setup(int smem, int mode, unsigned **status) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return fail(NPA_ERR_CUDA, "npa_linear_tcgen05: cudaGetDevice: %s", cudaGetErrorString(e));
    std::lock_guard<std::mutex> lock(g_umma_mutex);
    UmmaDevice &d = g_umma_device[dev];
    if (!d.status) {
        e = cudaGetSymbolAddress((void **)&d.status, g_umma_status);
        if (e != cudaSuccess) return fail(NPA_ERR_CUDA, "npa_linear_tcgen05: status word: %s", cudaGetErrorString(e));
    }
    if (smem > d.smem_limit[mode]) {
        const auto kernel = umma_kernel(mode);
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return fail(NPA_ERR_CUDA, "npa_linear_tcgen05: raising the shared-memory limit: %s", cudaGetErrorString(e));
        d.smem_limit[mode] = smem;
    }
    *status = d.status;
    return NPA_OK;
}

// Device address of the status word on the current device (also used by mlp_grad_tcgen05.cu).
unsigned *umma_status_word() {
    unsigned *p = nullptr;
    return cudaGetSymbolAddress((void **)&p, g_umma_status) == cudaSuccess ? p : nullptr;
}

static int umma_round16(int v) { return (v + 15) / 16 * 16; }
static int umma_chunks(int k) { return (k + kUmmaChunk - 1) / kUmmaChunk; }

static ImageJob image_job(const float *W, int64_t stride_out, int64_t stride_in, int in_dim, int out_dim, void *img) {
    return ImageJob{W, stride_out, stride_in, in_dim, out_dim, umma_round16(out_dim), umma_chunks(in_dim), static_cast<float *>(img)};
}
static int launch_images(const ImageJobs &jobs, cudaStream_t st) {
    launch_early(weight_image_kernel, (jobs.total() + 255) / 256, 256, 0, st, jobs);
    return check_launch("weight_image_kernel");
}

// The images of both layers, and of W1 as the backward wants it.
static int mlp_images(const char *me, const float *W1, const float *W2, int in_dim, int out_dim, int64_t w1_stride_out, int64_t w1_stride_in,
                      int64_t w2_stride_out, int64_t w2_stride_in, void *scratch, int64_t scratch_bytes, void *dz_image, int64_t dz_image_bytes,
                      ImageJobs *jobs, int features = 0, int dim = 0) {
    const int dz_columns = features > 0 ? StepColumns::total(features, dim) : in_dim;
    if (dz_image && ((uintptr_t)dz_image % 16 || dz_image_bytes < npa_linear_tcgen05_scratch_bytes(kUmmaRows, dz_columns)))
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: dz_image must be 16-byte aligned and hold %lld bytes", me,
                    (long long)npa_linear_tcgen05_scratch_bytes(kUmmaRows, dz_columns));
    if (in_dim <= 0 || out_dim <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: rows, in_dim and out_dim must be positive", me);
    if (in_dim > 1024 || out_dim > 64)
        return fail(NPA_ERR_UNSUPPORTED, "%s: supports in_dim <= 1024 and out_dim <= 64 (hidden width 128), got %d and %d", me, in_dim, out_dim);
    if (!W1 || !W2 || !scratch) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: z, W1, W2, y and scratch must be non-NULL", me);
    if ((uintptr_t)scratch % 16) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: z, h and y must be float aligned, scratch 16-byte aligned", me);
    if (scratch_bytes < npa_mlp_forward_tcgen05_scratch_bytes(in_dim, out_dim))
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: scratch holds %lld bytes, %lld needed", me, (long long)scratch_bytes,
                    (long long)npa_mlp_forward_tcgen05_scratch_bytes(in_dim, out_dim));
    void *w2 = (char *)scratch + npa_linear_tcgen05_scratch_bytes(in_dim, kUmmaRows);
    *jobs = {{image_job(W1, w1_stride_out, w1_stride_in, in_dim, kUmmaRows, scratch),
              image_job(W2, w2_stride_out, w2_stride_in, kUmmaRows, out_dim, w2)}, 2};
    if (dz_image) {
        ImageJob j = image_job(W1, w1_stride_in, w1_stride_out, kUmmaRows, dz_columns, dz_image);
        j.features = features;
        j.dim = dim;
        jobs->job[jobs->count++] = j;
    }
    return NPA_OK;
}

// Stages and shared memory of a single layer whose A, K and N are set.
static int plan_one_layer(UmmaArgs &a, int mode, size_t *smem) {
    a.Np = umma_round16(a.N);
    a.nchunks = umma_chunks(a.K);
    a.last_ksteps = (a.K - (a.nchunks - 1) * kUmmaChunk + 7) / 8;
    a.stage_bytes = 2 * kUmmaTileABytes + 2 * a.Np * 128;
    const int fixed = 1024 + umma_epilogue_floats(mode) * 4 + (int)sizeof(UmmaShared);
    a.stages = (227 * 1024 - fixed) / a.stage_bytes;
    if (a.stages > kUmmaMaxStages) a.stages = kUmmaMaxStages;
    if (a.stages < 2) return fail(NPA_ERR_UNSUPPORTED, "npa_linear_tcgen05: out_dim %d leaves room for fewer than two stages", a.N);
    *smem = (size_t)fixed + (size_t)a.stages * a.stage_bytes;
    return umma_device_setup((int)*smem, mode, &a.status);
}
static int launch_one_layer(const UmmaArgs &a, int mode, size_t smem, cudaStream_t st) {
    const long long tiles = (a.M + kUmmaRows - 1) / kUmmaRows;
    launch_early(umma_kernel(mode), (int)(tiles < 148 ? tiles : 148), kUmmaThreads, smem, st, a);
    return check_launch("linear_umma_kernel");
}

int launch_step_rows(const StepRows &rows, const float *dh, long long particles, const void *image, int64_t image_bytes, cudaStream_t st) {
    const int columns = StepColumns::total(rows.C, rows.dim);
    if (!dh || !image || !rows.vgrad || (uintptr_t)dh % 4 || ((uintptr_t)image | (uintptr_t)rows.vgrad | (uintptr_t)rows.direct | (uintptr_t)rows.rows) % 16 ||
        image_bytes < npa_linear_tcgen05_scratch_bytes(kUmmaRows, columns))
        return fail(NPA_ERR_INVALID_ARGUMENT, "step_perceive_backward: dh, vgrad and an image of %lld bytes must be there, 16-byte aligned",
                    (long long)npa_linear_tcgen05_scratch_bytes(kUmmaRows, columns));
    UmmaArgs a = {};
    a.A = dh; a.Wimg = static_cast<const float *>(image); a.M = particles; a.K = kUmmaRows; a.N = columns; a.parts = rows;
    const int mode = rows.dim == 2 ? kUmmaParts2 : kUmmaParts3;
    size_t smem = 0;
    const int rc = plan_one_layer(a, mode, &smem);
    return rc != NPA_OK ? rc : launch_one_layer(a, mode, smem, st);
}

}  // namespace npa

using namespace npa;

extern "C" {

int64_t npa_linear_tcgen05_scratch_bytes(int32_t in_dim, int32_t out_dim) {
    if (in_dim <= 0 || out_dim <= 0) return 0;
    return (int64_t)umma_chunks(in_dim) * 2 * umma_round16(out_dim) * kUmmaChunk * (int64_t)sizeof(float);
}

// W == NULL: scratch holds the image already (npa_mlp_forward_tcgen05_images made it).
static int linear_tcgen05(const float *A, const float *W, const float *bias, const float *gate, float *C, int64_t rows,
                          int32_t in_dim, int32_t out_dim, int64_t w_stride_out, int64_t w_stride_in, int32_t relu, void *scratch,
                          int64_t scratch_bytes, void *stream) {
    if (rows <= 0 || in_dim <= 0 || out_dim <= 0)
        return fail(NPA_ERR_INVALID_ARGUMENT, "npa_linear_tcgen05: rows, in_dim and out_dim must be positive");
    if (out_dim > 256 || in_dim > 1024)
        return fail(NPA_ERR_UNSUPPORTED, "npa_linear_tcgen05: supports in_dim <= 1024 and out_dim <= 256, got %d and %d", in_dim, out_dim);
    if (!A || !C || !scratch) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_linear_tcgen05: A, W, C and scratch must be non-NULL");
    if ((uintptr_t)A % 4 || (uintptr_t)C % 4 || (uintptr_t)scratch % 16)
        return fail(NPA_ERR_INVALID_ARGUMENT, "npa_linear_tcgen05: A and C must be float aligned, scratch 16-byte aligned");
    if (scratch_bytes < npa_linear_tcgen05_scratch_bytes(in_dim, out_dim))
        return fail(NPA_ERR_INVALID_ARGUMENT, "npa_linear_tcgen05: scratch holds %lld bytes, %lld needed", (long long)scratch_bytes,
                    (long long)npa_linear_tcgen05_scratch_bytes(in_dim, out_dim));
    UmmaArgs a = {};
    a.A = A; a.Wimg = (const float *)scratch; a.bias = bias; a.gate = gate; a.C = C; a.M = rows; a.K = in_dim; a.N = out_dim;
    a.relu = relu;
    size_t smem = 0;
    int rc = plan_one_layer(a, kUmmaOneLayer, &smem);
    if (rc != NPA_OK) return rc;
    if (W) {
        ImageJobs jobs = {{image_job(W, w_stride_out, w_stride_in, in_dim, out_dim, scratch)}, 1};
        if ((rc = launch_images(jobs, (cudaStream_t)stream)) != NPA_OK) return rc;
    }
    return launch_one_layer(a, kUmmaOneLayer, smem, (cudaStream_t)stream);
}

int npa_linear_tcgen05(const float *A, const float *W, const float *bias, const float *gate, float *C, int64_t rows,
                       int32_t in_dim, int32_t out_dim, int64_t w_stride_out, int64_t w_stride_in, int32_t relu, void *scratch,
                       int64_t scratch_bytes, void *stream) {
    if (!W) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_linear_tcgen05: A, W, C and scratch must be non-NULL");
    return linear_tcgen05(A, W, bias, gate, C, rows, in_dim, out_dim, w_stride_out, w_stride_in, relu, scratch, scratch_bytes, stream);
}

int npa_linear_tcgen05_prepared(const float *A, const void *image, int64_t image_bytes, float *C, int64_t rows, int32_t in_dim, int32_t out_dim,
                                void *stream) {
    return linear_tcgen05(A, nullptr, nullptr, nullptr, C, rows, in_dim, out_dim, 0, 0, 0, const_cast<void *>(image), image_bytes, stream);
}

int64_t npa_mlp_forward_tcgen05_scratch_bytes(int32_t in_dim, int32_t out_dim) {
    if (in_dim <= 0 || out_dim <= 0) return 0;
    return npa_linear_tcgen05_scratch_bytes(in_dim, kUmmaRows) + (int64_t)4 * 2 * umma_round16(out_dim) * kUmmaChunk * (int64_t)sizeof(float);
}

int npa_mlp_forward_tcgen05_images(const float *z, const float *W1, const float *b1, const float *W2, float *h, float *y, int64_t rows,
                                   int32_t in_dim, int32_t out_dim, int64_t w1_stride_out, int64_t w1_stride_in, int64_t w2_stride_out,
                                   int64_t w2_stride_in, void *scratch, int64_t scratch_bytes, void *dz_image, int64_t dz_image_bytes,
                                   void *stream) {
    const char *me = "npa_mlp_forward_tcgen05";
    ImageJobs jobs;
    int rc = mlp_images(me, W1, W2, in_dim, out_dim, w1_stride_out, w1_stride_in, w2_stride_out, w2_stride_in, scratch, scratch_bytes, dz_image,
                        dz_image_bytes, &jobs);
    if (rc != NPA_OK) return rc;
    if (rows <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: rows, in_dim and out_dim must be positive", me);
    if (!z || !y) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: z, W1, W2, y and scratch must be non-NULL", me);
    if ((uintptr_t)z % 4 || (uintptr_t)h % 4 || (uintptr_t)y % 4)
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: z, h and y must be float aligned, scratch 16-byte aligned", me);
    if ((rc = launch_images(jobs, (cudaStream_t)stream)) != NPA_OK) return rc;
    return npa_mlp_forward_tcgen05_prepared(z, b1, h, y, rows, in_dim, out_dim, scratch, scratch_bytes, stream);
}

int npa_bin_particles_mlp_images(const npa_grid *grid, int32_t channels, const float *x, const float *s, const int32_t *permutation, float *x_out,
                                 float *s_out, const float *W1, const float *W2, int32_t in_dim, int32_t out_dim, int64_t w1_stride_out,
                                 int64_t w1_stride_in, int64_t w2_stride_out, int64_t w2_stride_in, void *scratch, int64_t scratch_bytes,
                                 void *dz_image, int64_t dz_image_bytes, void *stream) {
    ImageJobs jobs;
    const int rc = mlp_images("npa_bin_particles_mlp_images", W1, W2, in_dim, out_dim, w1_stride_out, w1_stride_in, w2_stride_out, w2_stride_in,
                              scratch, scratch_bytes, dz_image, dz_image_bytes, &jobs);
    if (rc != NPA_OK) return rc;
    return bin_particles_and_images(grid, channels, x, s, permutation, x_out, s_out, jobs, (cudaStream_t)stream);
}

int npa_step_bin(const npa_grid *grid, int32_t channels, const float *x, const float *s, int32_t *permutation, int32_t *bin_offsets, int32_t *block_info,
                 void *grid_scratch, int64_t grid_scratch_bytes, float *x_out, float *s_out, const float *W1, const float *W2, int64_t w1_stride_out,
                 int64_t w1_stride_in, int64_t w2_stride_out, int64_t w2_stride_in, void *scratch, int64_t scratch_bytes, void *dz_image,
                 int64_t dz_image_bytes, int32_t rows, void *stream) {
    const char *me = "npa_step_bin";
    Geom g;
    int rc = make_geom(grid, &g);
    if (rc != NPA_OK) return rc;
    if (rows && !step_rows_cover(channels)) return fail(NPA_ERR_UNSUPPORTED, "%s: rows of multiples of four up to 32 features, got %d", me, channels);
    if (!x || !s || !x_out || !s_out) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: x, s and their outputs must be non-NULL", me);
    ImageJobs jobs;
    rc = mlp_images(me, W1, W2, 2 * channels + channels * g.dim + g.dim, g.dim + channels, w1_stride_out, w1_stride_in, w2_stride_out, w2_stride_in, scratch,
                    scratch_bytes, dz_image, dz_image_bytes, &jobs, rows ? channels : 0, g.dim);
    if (rc != NPA_OK) return rc;
    RowsJob rest = {};
    rc = grid_build_leaving(grid, x, permutation, bin_offsets, block_info, grid_scratch, grid_scratch_bytes, (cudaStream_t)stream, &rest);
    if (rc != NPA_OK) return rc;
    return bin_particles_and_images(grid, channels, x, s, permutation, x_out, s_out, jobs, (cudaStream_t)stream, rest);
}

int64_t npa_step_rows_image_bytes(const npa_grid *gd, int32_t channels) {
    Geom g;
    const int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    return step_rows_cover(channels) ? npa_linear_tcgen05_scratch_bytes(kUmmaRows, StepColumns::total(channels, g.dim)) : 0;
}

int npa_bin_particles_step_images(const npa_grid *grid, int32_t channels, const float *x, const float *s, const int32_t *permutation, float *x_out,
                                  float *s_out, const float *W1, const float *W2, int64_t w1_stride_out, int64_t w1_stride_in, int64_t w2_stride_out,
                                  int64_t w2_stride_in, void *scratch, int64_t scratch_bytes, void *rows_image, int64_t rows_image_bytes, void *stream) {
    const char *me = "npa_bin_particles_step_images";
    Geom g;
    int rc = make_geom(grid, &g);
    if (rc != NPA_OK) return rc;
    if (!rows_image) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: rows_image must be non-NULL", me);
    if (!step_rows_cover(channels)) return fail(NPA_ERR_UNSUPPORTED, "%s: supports multiples of four up to 32 features, got %d", me, channels);
    ImageJobs jobs;
    rc = mlp_images(me, W1, W2, 2 * channels + channels * g.dim + g.dim, g.dim + channels, w1_stride_out, w1_stride_in, w2_stride_out, w2_stride_in, scratch,
                    scratch_bytes, rows_image, rows_image_bytes, &jobs, channels, g.dim);
    if (rc != NPA_OK) return rc;
    return bin_particles_and_images(grid, channels, x, s, permutation, x_out, s_out, jobs, (cudaStream_t)stream);
}

// step != NULL: with the Euler update of D-dimensional positions on the geometry g.
static int mlp_forward(const char *me, const float *z, const float *b1, float *h, float *y, int64_t rows, int32_t in_dim, int32_t out_dim,
                       const void *scratch, int64_t scratch_bytes, const StepArgs *step, const Geom *g, cudaStream_t st) {
    if (rows <= 0 || in_dim <= 0 || out_dim <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: rows, in_dim and out_dim must be positive", me);
    if (in_dim > 1024 || out_dim > 64)
        return fail(NPA_ERR_UNSUPPORTED, "%s: supports in_dim <= 1024 and out_dim <= 64 (hidden width 128), got %d and %d", me, in_dim, out_dim);
    if (!z || (!y && !step) || !scratch) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: z, W1, W2, y and scratch must be non-NULL", me);
    if ((uintptr_t)z % 4 || (uintptr_t)h % 4 || (uintptr_t)y % 4 || (uintptr_t)scratch % 16)
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: z, h and y must be float aligned, scratch 16-byte aligned", me);
    if (scratch_bytes < npa_mlp_forward_tcgen05_scratch_bytes(in_dim, out_dim))
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: scratch holds %lld bytes, %lld needed", me, (long long)scratch_bytes,
                    (long long)npa_mlp_forward_tcgen05_scratch_bytes(in_dim, out_dim));
    UmmaArgs a = {};
    a.A = z; a.Wimg = (const float *)scratch; a.bias = b1; a.gate = nullptr; a.C = h; a.M = rows; a.K = in_dim; a.N = kUmmaRows;
    a.Np = kUmmaRows;  // hidden width 128
    a.nchunks = umma_chunks(in_dim);
    a.last_ksteps = (in_dim - (a.nchunks - 1) * kUmmaChunk + 7) / 8;
    a.stage_bytes = 2 * kUmmaTileABytes + 2 * a.Np * 128;
    a.relu = 1;
    a.Y = y; a.N2 = out_dim; a.N2p = umma_round16(out_dim);
    a.W2img = (const float *)((const char *)scratch + npa_linear_tcgen05_scratch_bytes(in_dim, kUmmaRows));
    const int w2_bytes = 4 * 2 * a.N2p * 128;
    const int fixed = 1024 + kUmmaEpiFloats * 4 + (int)sizeof(UmmaShared) + w2_bytes + ((kUmmaRows * out_dim + 3) & ~3) * 4;
    a.stages = (227 * 1024 - fixed) / a.stage_bytes;
    if (a.stages > kUmmaMaxStages) a.stages = kUmmaMaxStages;
    if (a.stages < 2) return fail(NPA_ERR_UNSUPPORTED, "%s: no room for two stages", me);
    const size_t smem = (size_t)fixed + (size_t)a.stages * a.stage_bytes;
    const int mode = step ? kUmmaStep : kUmmaTwoLayers;
    if (step) {
        a.D = g->dim;
        a.step = *step;
        a.g = *g;
    }
    const int rc = umma_device_setup((int)smem, mode, &a.status);
    if (rc != NPA_OK) return rc;
    const long long tiles = (rows + kUmmaRows - 1) / kUmmaRows;
    const int ctas = (int)(tiles < 148 ? tiles : 148);
    launch_early(umma_kernel(mode), ctas, kUmmaThreads, smem, st, a);
    return check_launch("linear_umma_kernel (two layers)");
}

int npa_mlp_forward_tcgen05_prepared(const float *z, const float *b1, float *h, float *y, int64_t rows, int32_t in_dim, int32_t out_dim,
                                     const void *scratch, int64_t scratch_bytes, void *stream) {
    return mlp_forward("npa_mlp_forward_tcgen05", z, b1, h, y, rows, in_dim, out_dim, scratch, scratch_bytes, nullptr, nullptr, (cudaStream_t)stream);
}

int npa_mlp_step_forward(const npa_grid *gd, const float *z, const float *b1, float *h, int32_t in_dim, const void *scratch, int64_t scratch_bytes,
                         const float *x_bin, const float *s_bin, const float *mask, int32_t uniforms, float update_below, int32_t channels,
                         float alpha, float dt, int32_t wrap, float *displacement, float *x_out, float *s_out, void *stream) {
    const char *me = "npa_mlp_step_forward";
    Geom g;
    const int rc = make_geom(gd, &g);
    if (rc != NPA_OK) return rc;
    if (channels <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: channels must be positive, got %d", me, channels);
    if (channels % 4 != 0 || channels > 4 * 2 * kUmmaStepQuads)
        return fail(NPA_ERR_UNSUPPORTED, "%s: supports multiples of four up to %d features, got %d", me, 4 * 2 * kUmmaStepQuads, channels);
    if (!x_bin || !s_bin || !x_out || !s_out) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: x_bin, s_bin, x_out and s_out must be non-NULL", me);
    if (((uintptr_t)x_bin | (uintptr_t)s_bin | (uintptr_t)x_out | (uintptr_t)s_out | (uintptr_t)displacement) % 16)
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: x_bin, s_bin, displacement, x_out and s_out must be 16-byte aligned", me);
    StepArgs s = {};
    s.y = displacement; s.y_pitch = g.dim == 2 ? 2 : 4; s.x_bin = x_bin; s.s_bin = s_bin; s.mask = mask; s.uniforms = uniforms;
    s.below = update_below; s.x_out = x_out; s.s_out = s_out; s.particles = (long long)g.B * g.N; s.C = channels; s.alpha = alpha; s.eps = g.h;
    s.dt = dt; s.wrap = wrap;
    return mlp_forward(me, z, b1, h, nullptr, s.particles, in_dim, g.dim + channels, scratch, scratch_bytes, &s, &g, (cudaStream_t)stream);
}

int npa_mlp_forward_tcgen05(const float *z, const float *W1, const float *b1, const float *W2, float *h, float *y, int64_t rows,
                            int32_t in_dim, int32_t out_dim, int64_t w1_stride_out, int64_t w1_stride_in, int64_t w2_stride_out,
                            int64_t w2_stride_in, void *scratch, int64_t scratch_bytes, void *stream) {
    if (!h) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_mlp_forward_tcgen05: h must be non-NULL");
    return npa_mlp_forward_tcgen05_images(z, W1, b1, W2, h, y, rows, in_dim, out_dim, w1_stride_out, w1_stride_in, w2_stride_out, w2_stride_in,
                                          scratch, scratch_bytes, nullptr, 0, stream);
}

int npa_linear_tcgen05_wait_selftest(int32_t limit_us, int32_t *device_result, void *stream) {
    if (!device_result) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_linear_tcgen05_wait_selftest: device_result is NULL");
    if (limit_us <= 0 || limit_us > 1000000)
        return fail(NPA_ERR_INVALID_ARGUMENT, "npa_linear_tcgen05_wait_selftest: limit_us must be in (0, 1000000]");
    umma_wait_selftest_kernel<<<1, 64, 0, (cudaStream_t)stream>>>((unsigned long long)limit_us * 1000ull, device_result);
    return check_launch("umma_wait_selftest_kernel");
}

/* Status word of the bounded waits of linear_umma_kernel on the current device (synchronises). */
int npa_linear_tcgen05_status(uint32_t *host_status, int32_t reset) {
    if (!host_status) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_linear_tcgen05_status: host_status must be non-NULL");
    cudaError_t e = cudaMemcpyFromSymbol(host_status, g_umma_status, sizeof(unsigned));
    if (e != cudaSuccess) return fail(NPA_ERR_CUDA, "npa_linear_tcgen05_status: %s", cudaGetErrorString(e));
    if (reset) {
        const unsigned zero = 0;
        e = cudaMemcpyToSymbol(g_umma_status, &zero, sizeof(unsigned));
        if (e != cudaSuccess) return fail(NPA_ERR_CUDA, "npa_linear_tcgen05_status: %s", cudaGetErrorString(e));
    }
    return NPA_OK;
}

}  // extern "C"
