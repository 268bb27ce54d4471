// Weight gradients of the per-particle MLP on the fifth-generation tensor cores.
//
//     dW1 [128, in] = dh^T z,   db1 [128] = sum over rows of dh,   dW2 [out, 128] = dy^T h
//
// (models/npa.py:63-75; the contract of npa_mlp_weight_grad, mlp_grad.cu) as two products whose
// reduction index is the row (particle) index:
//
//     D1 [128, in + 1] = dh^T [z | 1]        D2 [128, out] = h^T dy       (dW2 = D2^T)
//
// with tcgen05.mma kind::tf32, M = 128, K = 8 rows per instruction, both operands MN-major (a row of
// the row-major inputs is contiguous along M / N; 128-byte swizzle on 32-byte units), every product as three TF32 MMAs on operands split
// into head and tail, fp32 accumulators in tensor memory.  The tensor cores truncate when they add
// into the accumulator, and a chain of hundreds of accumulations drifts; so a chain is at most one
// segment of 128 rows (48 accumulations): after each segment the epilogue warps add the accumulators,
// rounding to nearest, into running sums kept in a second region of tensor memory, and the MMAs
// start the next segment from zero.  At the end each CTA writes its sums to global memory and a
// second kernel (in a step the launch of the inverse reorder: mlp_grad_reduce.cuh) adds the CTAs' partial sums in a fixed order: results are
// deterministic.
//
// One persistent CTA per SM with a contiguous slab of rows; stages of 16 rows:
//   * one lane brings the 16 rows of dh, h, z and dy of a stage into a ring of raw stages with four bulk
//     copies (each input's 16 rows are one contiguous, 16-byte aligned block of global memory);
//   * 16 producer warps, one row of the stage each, read the raw row, split it and store head and tail
//     into the stage's swizzled operand tiles (a last, partial stage is read from global memory);
//   * one lane issues the 12 MMAs of a stage and commits the stage back to the producers;
//   * eight epilogue warps drain a finished accumulator set (tcgen05.ld, lane = hidden unit).
// Every wait on an mbarrier is bounded in time; a wait that gives up raises a flag that ends all roles,
// the CTA frees its tensor memory, and the host reads the reason from the status word of
// npa_linear_tcgen05_status (bits 16, 32, 64: MMA lane, producers, epilogue of this kernel).
#include <mutex>

#include "mlp_grad_reduce.cuh"
#include "umma.cuh"

namespace npa {

constexpr int kGradSegmentStages = 8;              // 128 rows per accumulation chain
constexpr int kGradProducerWarps = 16;
constexpr int kGradEpilogueWarps = 8;
constexpr int kGradWarpMma = 8, kGradWarpCopy = 9, kGradWarpProducer0 = 10;
constexpr int kGradThreads = (kGradWarpProducer0 + kGradProducerWarps) * 32;
constexpr int kGradAtomBytes = 512;                // 4 rows x 128 bytes (32 columns)
constexpr int kGradAtomsH = 4;                     // atoms of 32 columns: dh / h
// The rest of the shape: atoms of [z | 1] and of dy, operand stages, raw stages.  Byte offsets inside a stage: [k-group of 8 rows][4-row
// half][atom] per operand part; a raw stage holds 16 rows of dh | h | z | dy, each block contiguous as in global memory.
template <int ATOMS_Z, int ATOMS_Y, int STAGES, int RAW_STAGES>
struct GradShape {
    static constexpr int kAtomsZ = ATOMS_Z, kAtomsY = ATOMS_Y, kStages = STAGES, kRawStages = RAW_STAGES;
    static constexpr int kOffDhHi = 0, kOffDhLo = 8192, kOffHHi = 16384, kOffHLo = 24576, kOffZHi = 32768;
    static constexpr int kOffZLo = kOffZHi + 4 * ATOMS_Z * kGradAtomBytes, kOffYHi = kOffZLo + 4 * ATOMS_Z * kGradAtomBytes;
    static constexpr int kOffYLo = kOffYHi + 4 * ATOMS_Y * kGradAtomBytes, kStageBytes = kOffYLo + 4 * ATOMS_Y * kGradAtomBytes;
    // in + 1 columns of D1 fit the atoms, out of D2
    static constexpr int kMaxIn = ATOMS_Z == 6 ? 175 : 32 * ATOMS_Z - 1, kMaxOut = ATOMS_Y == 2 ? 48 : 32 * ATOMS_Y;
    static constexpr int kRawDh = 0, kRawH = 8192, kRawZ = 16384, kRawY = kRawZ + (kGradStageRows * kMaxIn * 4 + 127) / 128 * 128;
    static constexpr int kRawBytes = (kRawY + kGradStageRows * kMaxOut * 4 + 127) / 128 * 128;
    static_assert(kStageBytes % 1024 == 0 && STAGES <= 4 && RAW_STAGES <= 4, "stages are aligned to the swizzle, and have barriers");
};
using GradWide = GradShape<6, 2, 2, 3>;    // up to 175 columns of z and 48 of dy: 64 KB per stage
using GradNarrow = GradShape<3, 1, 3, 3>;  // up to 95 and 32: 48 KB, a stage more and a quarter fewer stores
// (B200, us, wide -> narrow: 32,768 rows of 66 and 18 20.9 -> 19.6, 65,536 rows of 83 and 19 40.1 -> 37.6.)
constexpr int kGradTmemCols = 512, kGradSumCol = 256, kGradD2Col = 192;  // accumulators at 0 / 192, running sums 256 columns up
constexpr int kGradMaxIn = GradWide::kMaxIn, kGradMaxOut = GradWide::kMaxOut;

enum { GRAD_STATUS_MMA = 16, GRAD_STATUS_PRODUCER = 32, GRAD_STATUS_EPILOGUE = 64 };

struct GradShared {
    uint64_t full[4], empty[4], acc_full, acc_empty;
    uint64_t raw_full[4], raw_empty[4];
    uint32_t tmem_base;
    int abort;
};

struct GradArgs {
    const float *z, *dh, *h, *dy;
    float *partial;          // [ctas][128][N1p + N2p]
    long long M;
    int in_dim, out_dim, N1p, N2p, stages_per_cta, ctas;
    unsigned *status;
};

unsigned *umma_status_word();  // mlp_tcgen05.cu: device address of the status word on the current device

template <typename S>
__global__ void __launch_bounds__(kGradThreads, 1) mlp_grad_umma_kernel(const __grid_constant__ GradArgs args) {
    after_previous_kernel();
    const float *__restrict__ Z = args.z;
    const float *__restrict__ DH = args.dh;
    const float *__restrict__ H = args.h;
    const float *__restrict__ DY = args.dy;
    const long long M = args.M;
    const int K1 = args.in_dim, O = args.out_dim, N1p = args.N1p, N2p = args.N2p;
    unsigned *status = args.status;
    extern __shared__ uint8_t grad_smem_raw[];
    uint8_t *base = grad_smem_raw + ((1024u - (smem_u32(grad_smem_raw) & 1023u)) & 1023u);
    uint8_t *raw = base + S::kStages * S::kStageBytes;
    GradShared *sh = (GradShared *)(raw + S::kRawStages * S::kRawBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::kStages; ++s) {
            mbar_init(&sh->full[s], kGradProducerWarps);
            mbar_init(&sh->empty[s], 1);
        }
        for (int s = 0; s < S::kRawStages; ++s) {
            mbar_init(&sh->raw_full[s], 1);                    // the copy lane's arrival + the bytes of four copies
            mbar_init(&sh->raw_empty[s], kGradProducerWarps);  // every producer warp has read its row
        }
        mbar_init(&sh->acc_full, 1);
        mbar_init(&sh->acc_empty, kGradEpilogueWarps);
        sh->abort = 0;
        mbar_fence_init();
    }
    if (warp == kGradWarpMma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)),
                     "r"(kGradTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = sh->tmem_base;

    // this CTA's slab: stages first_stage .. first_stage + nstage - 1 of 16 rows
    const long long stages_total = (M + kGradStageRows - 1) / kGradStageRows;
    const long long first_stage = (long long)blockIdx.x * args.stages_per_cta;
    const int nstage = (int)(stages_total - first_stage < args.stages_per_cta ? stages_total - first_stage : args.stages_per_cta);
    const int nseg = (nstage + kGradSegmentStages - 1) / kGradSegmentStages;
    // stages whose 16 rows all exist come in by bulk copy; a last, partial stage is read row by row
    const long long rows_left = M - first_stage * kGradStageRows;
    const int nraw = (int)(rows_left / kGradStageRows < nstage ? rows_left / kGradStageRows : nstage);
    bool ok = true;

    if (warp == kGradWarpMma) {
        if (lane == 0) {
            // M = 128, TF32 x TF32 -> F32, both operands MN-major
            const unsigned idesc0 = (1u << 4) | (2u << 7) | (2u << 10) | (1u << 15) | (1u << 16) | ((unsigned)(kGradHidden >> 4) << 24);
            const unsigned idesc1 = idesc0 | ((unsigned)(N1p >> 3) << 17), idesc2 = idesc0 | ((unsigned)(N2p >> 3) << 17);
            const unsigned sbase = smem_u32(base);
            int s = 0, done = 0;
            unsigned ph = 0;
#pragma unroll 1
            for (int seg = 0; seg < nseg; ++seg) {
                if (!(ok = umma_wait(&sh->acc_empty, (seg & 1) ^ 1, &sh->abort))) break;  // the epilogue has read segment seg - 1
                tc_fence_after();
                const unsigned d1 = tmem, d2 = tmem + kGradD2Col;
                const int nst = nstage - done < kGradSegmentStages ? nstage - done : kGradSegmentStages;
#pragma unroll 1
                for (int st = 0; st < nst; ++st) {
                    if (!(ok = umma_wait(&sh->full[s], ph, &sh->abort))) break;
                    tc_fence_after();
                    const unsigned sa = sbase + s * S::kStageBytes;
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk) {
                        const unsigned oh = kk * 2 * kGradAtomsH * kGradAtomBytes, oz = kk * 2 * S::kAtomsZ * kGradAtomBytes;
                        const unsigned oy = kk * 2 * S::kAtomsY * kGradAtomBytes;
                        const uint64_t a1h = umma_desc_mn32(sa + S::kOffDhHi + oh, kGradAtomBytes, kGradAtomsH * kGradAtomBytes);
                        const uint64_t a1l = umma_desc_mn32(sa + S::kOffDhLo + oh, kGradAtomBytes, kGradAtomsH * kGradAtomBytes);
                        const uint64_t b1h = umma_desc_mn32(sa + S::kOffZHi + oz, kGradAtomBytes, S::kAtomsZ * kGradAtomBytes);
                        const uint64_t b1l = umma_desc_mn32(sa + S::kOffZLo + oz, kGradAtomBytes, S::kAtomsZ * kGradAtomBytes);
                        const uint64_t a2h = umma_desc_mn32(sa + S::kOffHHi + oh, kGradAtomBytes, kGradAtomsH * kGradAtomBytes);
                        const uint64_t a2l = umma_desc_mn32(sa + S::kOffHLo + oh, kGradAtomBytes, kGradAtomsH * kGradAtomBytes);
                        const uint64_t b2h = umma_desc_mn32(sa + S::kOffYHi + oy, kGradAtomBytes, S::kAtomsY * kGradAtomBytes);
                        const uint64_t b2l = umma_desc_mn32(sa + S::kOffYLo + oy, kGradAtomBytes, S::kAtomsY * kGradAtomBytes);
                        const int acc = (st | kk) != 0;
                        umma_tf32(d1, a1l, b1h, idesc1, acc);
                        umma_tf32(d1, a1h, b1l, idesc1, 1);
                        umma_tf32(d1, a1h, b1h, idesc1, 1);
                        umma_tf32(d2, a2l, b2h, idesc2, acc);
                        umma_tf32(d2, a2h, b2l, idesc2, 1);
                        umma_tf32(d2, a2h, b2h, idesc2, 1);
                    }
                    umma_commit(&sh->empty[s]);
                    if (++s == S::kStages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (!ok) break;
                umma_commit(&sh->acc_full);
                done += nst;
            }
            if (!ok) atomicOr(status, GRAD_STATUS_MMA);
        }
        __syncwarp();
    } else if (warp == kGradWarpCopy) {
        if (lane == 0) {
            // four bulk copies per stage: the 16 rows of each input are one contiguous, 16-byte aligned block
            const unsigned bz = kGradStageRows * K1 * 4, by = kGradStageRows * O * 4;
            int rs = 0;
            unsigned rphase = 1;  // the first pass finds the raw stages free
#pragma unroll 1
            for (int q = 0; q < nraw; ++q) {
                if (!(ok = umma_wait(&sh->raw_empty[rs], rphase, &sh->abort))) break;
                const long long row = (first_stage + q) * kGradStageRows;
                uint8_t *dst = raw + rs * S::kRawBytes;
                mbar_arrive_expect(&sh->raw_full[rs], 2u * 8192u + bz + by);
                bulk_copy_g2s(dst + S::kRawDh, DH + row * kGradHidden, 8192u, &sh->raw_full[rs]);
                bulk_copy_g2s(dst + S::kRawH, H + row * kGradHidden, 8192u, &sh->raw_full[rs]);
                bulk_copy_g2s(dst + S::kRawZ, Z + row * K1, bz, &sh->raw_full[rs]);
                bulk_copy_g2s(dst + S::kRawY, DY + row * O, by, &sh->raw_full[rs]);
                if (++rs == S::kRawStages) {
                    rs = 0;
                    rphase ^= 1;
                }
            }
            if (!ok) {
                atomicOr(status, GRAD_STATUS_PRODUCER);
                __nanosleep(20000);  // copies issued just before the flag was seen land before the CTA leaves
            }
        }
    } else if (warp >= kGradWarpProducer0) {
        const int pw = warp - kGradWarpProducer0;  // this warp owns row pw of every stage
        const int kk = pw >> 3;                    // its k-group of eight rows
        const int half4 = (pw >> 2) & 1;           // its group of four rows inside the k-group
        const int at = umma_mn32_offset(pw & 3, lane);  // float offset of (row, lane) inside an atom of 32 columns
        int s = 0, rs = 0;
        unsigned phase = 1, rphase = 0;  // operand stages start free; raw stages start empty of data
#pragma unroll 1
        for (int q = 0; q < nstage; ++q) {
            // v[0..3] dh, v[4..7] h, v[8..13] [z | 1 | 0...], v[14..15] dy: column 32 t + lane of this warp's row
            float v[16];
            if (q < nraw) {
                if (!(ok = umma_wait(&sh->raw_full[rs], rphase, &sh->abort))) break;
                const float *r = (const float *)(raw + rs * S::kRawBytes);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    v[t] = r[S::kRawDh / 4 + pw * kGradHidden + 32 * t + lane];
                    v[4 + t] = r[S::kRawH / 4 + pw * kGradHidden + 32 * t + lane];
                }
#pragma unroll
                for (int t = 0; t < S::kAtomsZ; ++t) {
                    const int col = 32 * t + lane;
                    v[8 + t] = col < K1 ? r[S::kRawZ / 4 + pw * K1 + col] : (col == K1 ? 1.f : 0.f);  // the ones column gives db1
                }
#pragma unroll
                for (int t = 0; t < S::kAtomsY; ++t) {
                    const int col = 32 * t + lane;
                    v[14 + t] = col < O ? r[S::kRawY / 4 + pw * O + col] : 0.f;
                }
            } else {
                const long long row = (first_stage + q) * kGradStageRows + pw;
                if (row < M) {
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        v[t] = __ldg(DH + row * kGradHidden + 32 * t + lane);
                        v[4 + t] = __ldg(H + row * kGradHidden + 32 * t + lane);
                    }
#pragma unroll
                    for (int t = 0; t < S::kAtomsZ; ++t) {
                        const int col = 32 * t + lane;
                        v[8 + t] = col < K1 ? __ldg(Z + row * K1 + col) : (col == K1 ? 1.f : 0.f);
                    }
#pragma unroll
                    for (int t = 0; t < S::kAtomsY; ++t) {
                        const int col = 32 * t + lane;
                        v[14 + t] = col < O ? __ldg(DY + row * O + col) : 0.f;
                    }
                } else {
#pragma unroll
                    for (int t = 0; t < 16; ++t) v[t] = 0.f;  // rows behind the end add nothing, not even to db1
                }
            }
            if (!(ok = umma_wait(&sh->empty[s], phase, &sh->abort))) break;
            float *stage = (float *)(base + s * S::kStageBytes);
            auto put = [&](int off_hi, int off_lo, int natoms, int atom, float x) {
                const int f = ((kk * 2 + half4) * natoms + atom) * (kGradAtomBytes / 4) + at;
                const float head = __uint_as_float(tf32_head_bits(x));
                stage[off_hi / 4 + f] = head;
                stage[off_lo / 4 + f] = x - head;
            };
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                put(S::kOffDhHi, S::kOffDhLo, kGradAtomsH, t, v[t]);
                put(S::kOffHHi, S::kOffHLo, kGradAtomsH, t, v[4 + t]);
            }
#pragma unroll
            for (int t = 0; t < S::kAtomsZ; ++t) put(S::kOffZHi, S::kOffZLo, S::kAtomsZ, t, v[8 + t]);
#pragma unroll
            for (int t = 0; t < S::kAtomsY; ++t) put(S::kOffYHi, S::kOffYLo, S::kAtomsY, t, v[14 + t]);
            fence_proxy_async();  // the MMA reads these through the async proxy
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&sh->full[s]);
                if (q < nraw) mbar_arrive(&sh->raw_empty[rs]);  // the raw row has been consumed
            }
            if (q < nraw && ++rs == S::kRawStages) {
                rs = 0;
                rphase ^= 1;
            }
            if (++s == S::kStages) {
                s = 0;
                phase ^= 1;
            }
        }
        if (!ok && lane == 0) atomicOr(status, GRAD_STATUS_PRODUCER);
    } else {
        // epilogue: warp w owns lanes 32 (w % 4) .. + 31 of tensor memory (= hidden units) and every second
        // block of 16 columns.  After each segment it adds the accumulators, rounding to nearest, into running
        // sums that stay in tensor memory (the same thread reads and writes the same cells every time);
        // after the last segment the sums go to this CTA's partial sums in global memory.
        const int quarter = warp & 3, half = warp >> 2;
        const int nb1 = N1p >> 4, nb = nb1 + (N2p >> 4);
        float *prow = args.partial + ((long long)blockIdx.x * kGradHidden + quarter * 32 + lane) * (N1p + N2p);
        const unsigned taddr0 = tmem + ((unsigned)(quarter * 32) << 16);
        int last_block = half;
        while (last_block + 2 < nb) last_block += 2;
#pragma unroll 1
        for (int seg = 0; seg < nseg; ++seg) {
            if (!(ok = umma_wait(&sh->acc_full, seg & 1, &sh->abort, kUmmaWaitNs, 200))) break;
            tc_fence_after();
#pragma unroll 1
            for (int b = half; b < nb; b += 2) {
                const int col = b < nb1 ? b * 16 : kGradD2Col + (b - nb1) * 16;  // column in tensor memory
                unsigned r[16], sum[16];
                tmem_ld16(taddr0 + col, r);
                if (seg > 0) tmem_ld16(taddr0 + kGradSumCol + col, sum);
                tc_wait_ld();
                if (b == last_block) {  // this warp has read its share of the accumulators: hand them back
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh->acc_empty);
                }
                if (seg > 0) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(sum[j]));
                }
                if (seg + 1 < nseg) {
                    tmem_st16(taddr0 + kGradSumCol + col, r);
                } else {
                    float4 *p = (float4 *)(prow + b * 16);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        p[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]),
                                           __uint_as_float(r[4 * j + 3]));
                }
            }
            tc_wait_st();  // the sums are in place before this thread reads them again
        }
        if (!ok && lane == 0) atomicOr(status, GRAD_STATUS_EPILOGUE);
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kGradWarpMma) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kGradTmemCols) : "memory");
    }
}

__global__ void __launch_bounds__(kReduceQuads * kReduceRuns) mlp_grad_umma_reduce_kernel(const __grid_constant__ GradReduce a) {
    after_previous_kernel();
    reduce_weight_grads<kReduceQuads>(a, (int)blockIdx.x);
}


struct GradDevice {
    unsigned *status = nullptr;
    bool smem_set[2] = {false, false};  // per shape
};
static std::mutex g_grad_mutex;
static GradDevice g_grad_device[64];
template <typename S>
constexpr int kGradSmemBytes = 1024 + S::kStages * S::kStageBytes + S::kRawStages * S::kRawBytes + (int)sizeof(GradShared);
static_assert(kGradSmemBytes<GradWide> <= 227 * 1024 && kGradSmemBytes<GradNarrow> <= 227 * 1024, "shared memory of a CTA");

}  // namespace npa

using namespace npa;

extern "C" {

static int weight_grad_partial(const char *me, const float *z, const float *dh, const float *h, const float *dy, int64_t rows, int32_t in_dim, int32_t hidden,
                               int32_t out_dim, float *scratch, int64_t scratch_floats, void *stream);

int64_t npa_mlp_weight_grad_tcgen05_scratch_floats(int64_t rows, int32_t in_dim, int32_t out_dim) {
    if (rows <= 0 || in_dim <= 0 || out_dim <= 0) return 0;
    return (int64_t)148 * kGradHidden * (grad_round16(in_dim + 1) + grad_round16(out_dim));
}

int npa_mlp_weight_grad_tcgen05(const float *z, const float *dh, const float *h, const float *dy, int64_t rows, int32_t in_dim,
                                int32_t hidden, int32_t out_dim, float *scratch, int64_t scratch_floats, float *dW1,
                                float *dW2, float *db1, void *stream) {
    const char *me = "npa_mlp_weight_grad_tcgen05";
    if (!dW1 || !dW2 || !db1) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: every pointer must be non-NULL", me);
    const int rc = weight_grad_partial(me, z, dh, h, dy, rows, in_dim, hidden, out_dim, scratch, scratch_floats, stream);
    if (rc != NPA_OK) return rc;
    GradReduce a = grad_plan(rows, in_dim, out_dim);
    a.partial = scratch; a.dW1 = dW1; a.dW2 = dW2; a.db1 = db1;
    mlp_grad_umma_reduce_kernel<<<a.blocks(kReduceQuads), kReduceQuads * kReduceRuns, 0, (cudaStream_t)stream>>>(a);
    return check_launch("mlp_grad_umma_reduce_kernel");
}

int npa_mlp_weight_grad_tcgen05_partial(const float *z, const float *dh, const float *h, const float *dy, int64_t rows, int32_t in_dim,
                                        int32_t hidden, int32_t out_dim, float *scratch, int64_t scratch_floats, void *stream) {
    return weight_grad_partial("npa_mlp_weight_grad_tcgen05_partial", z, dh, h, dy, rows, in_dim, hidden, out_dim, scratch, scratch_floats, stream);
}

static int weight_grad_partial(const char *me, const float *z, const float *dh, const float *h, const float *dy, int64_t rows, int32_t in_dim, int32_t hidden,
                               int32_t out_dim, float *scratch, int64_t scratch_floats, void *stream) {
    if (hidden != kGradHidden) return fail(NPA_ERR_UNSUPPORTED, "%s: hidden width must be %d, got %d", me, kGradHidden, hidden);
    if (in_dim <= 0 || in_dim > kGradMaxIn || out_dim <= 0 || out_dim > kGradMaxOut)
        return fail(NPA_ERR_UNSUPPORTED, "%s: supports in <= %d and out <= %d, got %d and %d", me, kGradMaxIn, kGradMaxOut, in_dim, out_dim);
    if (rows <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: rows must be positive", me);
    if (!z || !dh || !h || !dy || !scratch) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: every pointer must be non-NULL", me);
    if (((uintptr_t)z | (uintptr_t)dh | (uintptr_t)h | (uintptr_t)dy | (uintptr_t)scratch) % 16)
        return fail(NPA_ERR_INVALID_ARGUMENT, "%s: z, dh, h, dy and scratch must be 16-byte aligned", me);
    const int64_t need = npa_mlp_weight_grad_tcgen05_scratch_floats(rows, in_dim, out_dim);
    if (scratch_floats < need)
        return fail(NPA_ERR_SCRATCH_TOO_SMALL, "%s: scratch has %lld floats, %lld needed", me, (long long)scratch_floats, (long long)need);

    GradArgs a = {};
    a.z = z; a.dh = dh; a.h = h; a.dy = dy; a.partial = scratch;
    a.M = rows; a.in_dim = in_dim; a.out_dim = out_dim;
    const GradReduce plan = grad_plan(rows, in_dim, out_dim);
    a.N1p = plan.N1p; a.N2p = plan.N2p; a.ctas = plan.ctas; a.stages_per_cta = plan.stages_per_cta;

    const bool narrow = in_dim <= GradNarrow::kMaxIn && out_dim <= GradNarrow::kMaxOut;
    const auto kernel = narrow ? mlp_grad_umma_kernel<GradNarrow> : mlp_grad_umma_kernel<GradWide>;
    const int smem = narrow ? kGradSmemBytes<GradNarrow> : kGradSmemBytes<GradWide>;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return fail(NPA_ERR_CUDA, "%s: cudaGetDevice: %s", me, cudaGetErrorString(e));
    {
        std::lock_guard<std::mutex> lock(g_grad_mutex);
        GradDevice &d = g_grad_device[dev];
        if (!d.status && !(d.status = umma_status_word())) return fail(NPA_ERR_CUDA, "%s: no status word", me);
        if (!d.smem_set[narrow]) {
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return fail(NPA_ERR_CUDA, "%s: raising the shared-memory limit: %s", me, cudaGetErrorString(e));
            d.smem_set[narrow] = true;
        }
        a.status = d.status;
    }
    cudaStream_t st = (cudaStream_t)stream;
    launch_early(kernel, a.ctas, kGradThreads, smem, st, a);
    return check_launch("mlp_grad_umma_kernel");
}

}  // extern "C"
