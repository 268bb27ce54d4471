// Backward of blur and gradient with respect to the features, on the tensor cores.
//
//     ds_i = v_i sum_j [ c_s W_ij gB_j - sum_d K_ij,d gG_j,d ] - sum_d T_i,d gG_i,d,      K = c_g phi r,  T = sum_j v_j K
//
// gathers 1 + D rows per pair and does two multiply-adds with each of their floats: over neighbour lists (feature_list.cuh) it is bound by
// the rows on their way through L1, of which neighbouring particles fetch mostly the same ones.  Here a warp takes eight consecutive
// particles, finds the union of their neighbours among the candidates of their cells, and forms
//     ds^T [features, 8 particles]  +=  rows^T [features, 8 neighbours]  .  weights [8 neighbours, 8 particles]
// class by class (blur, then the axes) with mma.sync m16n8k8: a row is loaded once for eight particles, in the layout of the A operand
// (a lane has four, or two, consecutive features of two neighbours), and a lane computes the weights of two neighbours for one particle,
// which is the layout of the B operand: nothing passes through shared memory but the neighbours' positions.  Weights of pairs beyond the
// cut-off are zero; two fifths of the products are of pairs.
//
// Single precision: every operand is split into a TF32 head, rounded to nearest, and a tail of at most twelve bits; three MMAs per product
// (tail . head + head . tail + head . head), four (tail . tail) where the roundings of few neighbours do not outweigh it.  The tensor cores truncate when they accumulate, so a chain is one group of eight neighbours
// (heads 1 + D MMAs, the others apart) and is added to the running sums in single precision.  A product with a zero weight spreads a row
// or a volume that is not finite to particles that are no neighbours of it; a warp whose sums, of the rows or of T, are not finite therefore
// computes its particles again, pair by pair.
//
// Measured, B200, us, lists -> this: 8 x 4,096 particles in 2D, C = 16, 49 neighbours 35 -> 27; 64 x 512 along lines 35 -> 24; 4 x 65,536 in 3D,
// C = 32, 41 neighbours 380 -> 330 (of these the search 121; instructions 220 M, 64 % of the slots, MMAs a quarter of the tensor pipe's time).
// Error against 64 bits (2-norm, 1e-7), lists / this, rows N(0, 1): 2D, 14 neighbours 1.47 / 1.44 (1.48 with three MMAs), 25 1.70 / 1.47, 77
// 2.52 / 1.67; 3D 16 1.66 / 1.62, 39 2.09 / 1.65, 76 2.58 / 1.73; over 80 drawn training cases of 12 and more neighbours at most 0.99 of
// the lists'.  Below ten neighbours up to 1.03 of it (2D, 7: 1.35 / 1.39).  The fourth MMA costs 2D 25.5 -> 26.7 us with 16 features, 36 -> 38
// with 32.  Not kept (3D, against 334 then): sixteen particles per warp (411,
// larger unions and fewer warps); a queue per residue of the neighbour's index, for rows in banks of their own (515); the head by
// cvt.rna (452).
//
// The positions must be those that were binned (a step of the model: they come out of the reorder): particles two cells apart in x share a
// tile, and are beyond each other's cut-off only then.
#include "feature_list.cuh"

namespace npa {

constexpr int kDenseWarps = 4;
constexpr int kDenseTile = 8;    // particles per warp
constexpr int kDenseRing = 64;   // neighbours found and not yet multiplied
// Particles per cell in 2D below which the tails are multiplied as well: uniform particles have 16 neighbours there, clustered ones more.
// Error against the lists', three / four products: 7 neighbours 1.06 / 1.03, 10 1.04 / 1.01, 12 1.01 / 0.99, 14 1.01 / 0.98, 16 0.96 / 0.94, 19 0.94 / 0.92.
// In 3D the sweep begins at 16 (0.97).
constexpr double kDenseTailsBelow = 5.0;

struct DenseMem {  // of one warp
    float4 at[kDenseRing];  // position and volume of a neighbour
    float minus[3][kDenseTile];  // the tile's particles, negated
    int index[kDenseRing];
    int4 rng[kMaxRanges];
};

struct Tf32 {
    unsigned head, tail;
};
__device__ __forceinline__ Tf32 split_tf32(float x) {
    const unsigned head = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;  // nearest (ties away from zero)
    return Tf32{head, __float_as_uint(x - __uint_as_float(head))};
}

__device__ __forceinline__ void mma_m16n8k8(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_m16n8k8_from_zero(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// spiky_distance; in 2D with the instruction for the reciprocal square root of a normal number, which Q >= 1e-12 is.  With it / with rsqrtf, us:
// 8 x 4,096 particles in 2D, C = 16, 26.7 / 28.4, 64 x 512 along lines 23.6 / 24.4, C = 32 38.1 / 40.4; 4 x 65,536 in 3D, C = 32, 344 / 330, C = 16 228 / 234.
template <int D>
__device__ __forceinline__ Spiky dense_distance(float q) {
    if constexpr (D == 3) return spiky_distance(q);
    const float Q = q + 1e-12f;
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(Q));
    return spiky_refined(Q, y);
}

// Weights of one pair: c_s W and -K, zero unless `live`; K itself times the neighbour's volume goes into T.
template <int D, bool PER>
__device__ __forceinline__ void dense_weights(const Geom &g, const Pos<D> &pi, const float4 &c, bool live, float (&w)[1 + D], float (&tsum)[3]) {
    float r[3];
    listed_displacement<D, PER>(g, pi, Pos<D>{c.x, c.y, c.z}, r[0], r[1], r[2]);
    const float q = live ? sq_norm_fast<D>(r[0], r[1], r[2]) : 1.0e30f, t = fmaxf(g.h2 - q, 0.f);
    w[0] = g.c_s * (t * t * t);
    const float phi = q > 0.f ? g.c_g * spiky_phi(dense_distance<D>(q), g.h) : 0.f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const float k = phi * r[d];
        tsum[d] = fmaf(c.w, k, tsum[d]);
        w[1 + d] = -k;
    }
}

// What reaches the features beside the neighbours' terms: the particle's own rows, the direct part of z's gradient and an addend.
template <int D>
__device__ __forceinline__ float dense_finish(const FeatureListBwdArgs &a, long long i, int f, float sum, float vi, const float (&T)[3]) {
    float o = sum * vi;
#pragma unroll
    for (int d = 0; d < D; ++d) o = fmaf(-T[d], __ldg(a.gg + i * a.gg_pitch + d * a.cp + f), o);
    if (a.direct) o += __ldg(a.direct + i * a.direct_pitch + f);
    if (a.add) o += __ldg(a.add + i * a.C + f);
    return o;
}

// The same for VW consecutive features, as vectors (C = cp, grad_s and the addend aligned).
template <int D, int VW>
__device__ __forceinline__ void dense_finish_row(const FeatureListBwdArgs &a, long long i, int f, const float (&sum)[VW], float vi, const float (&T)[3]) {
    float o[VW];
    auto load = [&](const float *p, float (&v)[VW]) {
        if constexpr (VW == 4) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
            const float2 q = __ldg(reinterpret_cast<const float2 *>(p));
            v[0] = q.x; v[1] = q.y;
        }
    };
#pragma unroll
    for (int k = 0; k < VW; ++k) o[k] = sum[k] * vi;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        float v[VW];
        load(a.gg + i * a.gg_pitch + d * a.cp + f, v);
#pragma unroll
        for (int k = 0; k < VW; ++k) o[k] = fmaf(-T[d], v[k], o[k]);
    }
    if (a.direct) {
#pragma unroll
        for (int k = 0; k < VW; ++k) o[k] += __ldg(a.direct + i * a.direct_pitch + f + k);
    }
    if (a.add) {
        float v[VW];
        load(a.add + i * a.C + f, v);
#pragma unroll
        for (int k = 0; k < VW; ++k) o[k] += v[k];
    }
    if constexpr (VW == 4) *reinterpret_cast<float4 *>(a.grad_s + i * a.C + f) = make_float4(o[0], o[1], o[2], o[3]);
    else *reinterpret_cast<float2 *>(a.grad_s + i * a.C + f) = make_float2(o[0], o[1]);
}

// The particles of a tile one after another, a lane per feature, pair by pair.  Out of line: only for sums that are not finite.
template <int D, bool PER>
__device__ __noinline__ void dense_pairwise(const FeatureListBwdArgs &a, const Geom &g, DenseMem &mem, int first, int count) {
    const int lane = threadIdx.x & 31, f = min(lane, a.C - 1);
    for (int i = first; i < first + count; ++i) {
        const float4 own = __ldg(a.pv + i);
        const Pos<D> pi{own.x, own.y, own.z};
        const int sys = i / g.N;
        int cx, cy, cz;
        snapshot_cell_of<D>(g, a.bin_offsets + (size_t)sys * g.cells, i, pi.x, pi.y, pi.z, cx, cy, cz);
        __syncwarp();
        const int nr = build_ranges_span<D>(g, a.bin_offsets, sys, cx, cx, cy, cz, mem.rng);
        float sum = 0.f, T[3] = {0.f, 0.f, 0.f};
        for (int r = 0; r < nr; ++r)
            for (int j = mem.rng[r].x; j < mem.rng[r].y; ++j) {
                const float4 c = __ldg(a.pv + j);
                float rx, ry, rz, w[1 + D];
                listed_displacement<D, PER>(g, pi, Pos<D>{c.x, c.y, c.z}, rx, ry, rz);
                if (!(sq_norm_fast<D>(rx, ry, rz) < g.h2)) continue;
                dense_weights<D, PER>(g, pi, c, true, w, T);
                sum = fmaf(w[0], __ldg(a.gb + (long long)j * a.gb_pitch + f), sum);
#pragma unroll
                for (int d = 0; d < D; ++d) sum = fmaf(w[1 + d], __ldg(a.gg + (long long)j * a.gg_pitch + d * a.cp + f), sum);
            }
        if (lane < a.C) a.grad_s[(long long)i * a.C + lane] = dense_finish<D>(a, i, lane, sum, own.w, T);
    }
}

// A difference of coordinates as the nearest image has it, two at a time (where the length of the box is not exact, neither is this).
__device__ __forceinline__ unsigned long long nearest_image2(unsigned long long r, float L, float invL) {
    const unsigned long long round = pack2(12582912.f, 12582912.f), back = pack2(-12582912.f, -12582912.f);
    const unsigned long long k = add2(fma2(r, pack2(invL, invL), round), back);
    return fma2(k, pack2(-L, -L), r);
}

// Rows are [1 + D][cp] (gb and gg in one).  MT: blocks of sixteen features; FILLED: cp = 16 MT; TAILS: with the products of the tails.
template <int D, bool PER, int MT, bool FILLED, bool TAILS>
__global__ void __launch_bounds__(kDenseWarps * 32, MT == 2 ? 5 : D == 3 ? 6 : 7)
feature_dense_backward_kernel(const __grid_constant__ FeatureListBwdArgs a, const __grid_constant__ Geom g) {
    after_previous_kernel();
    constexpr int VW = 2 * MT;  // consecutive features of a lane
    __shared__ DenseMem s_mem[kDenseWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, t = lane & 3;
    const unsigned below = (1u << lane) - 1u;
    DenseMem &mem = s_mem[warp];
    const int total = g.B * g.N;
    const int first = (int)((blockIdx.x * kDenseWarps + warp) * (unsigned)kDenseTile);
    if ((unsigned)first >= (unsigned)total) return;
    const int here = min(kDenseTile, total - first);
    // lane p looks at particle p: its cell, and who shares its row of cells
    const int ip = first + min(lane, here - 1);
    const float4 mine = __ldg(a.pv + ip);
    const int sys = ip / g.N;
    int cx, cy, cz;
    snapshot_cell_of<D>(g, a.bin_offsets + (size_t)sys * g.cells, ip, mine.x, mine.y, mine.z, cx, cy, cz);
    const int key = (sys * g.g[2] + cz) * g.g[1] + cy;
    // lanes (gr, t) weigh neighbours for particle gr
    const Pos<D> pi{__shfl_sync(kFull, mine.x, gr), __shfl_sync(kFull, mine.y, gr), __shfl_sync(kFull, mine.z, gr)};
    const int cp = FILLED ? 16 * MT : a.cp;
    const char *rows = reinterpret_cast<const char *>(a.gb);  // less than 2^32 bytes
    const unsigned pitch = (unsigned)a.gb_pitch * 4u, f0 = 4u * min(VW * gr, cp - VW);  // (lanes beyond the last feature read valid neighbours of it, unused)
    const float reach = PER ? g.h2 + 4.0e-6f * g.h * fmaxf(fmaxf(g.L[0], g.L[1]), D == 3 ? g.L[2] : 0.f) : g.h2;

    float acc[MT][4], others[MT][4], tsum[3] = {0.f, 0.f, 0.f};  // products of heads; of tails
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[m][q] = others[m][q] = 0.f;

    unsigned left = (1u << here) - 1u;
    while (left) {
        // ---- the particles of one x-row of cells (consecutive, cx ascending), and the candidates around the cells they span
        const int lead = __ffs(left) - 1;
        const unsigned seg = __ballot_sync(kFull, key == __shfl_sync(kFull, key, lead)) & left;
        left &= ~seg;
        const int cx0 = __shfl_sync(kFull, cx, lead), cx1 = __shfl_sync(kFull, cx, 31 - __clz(seg));
        __syncwarp();
        const int nr = build_ranges_span<D>(g, a.bin_offsets, __shfl_sync(kFull, sys, lead), cx0, cx1, __shfl_sync(kFull, cy, lead),
                                            __shfl_sync(kFull, cz, lead), mem.rng);
        const int4 range = lane < nr ? mem.rng[lane] : make_int4(0, 0, 0, 0);
        int incl = range.y - range.x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += v;
        }
        const int candidates = __shfl_sync(kFull, incl, 31);
        __syncwarp();
        if (lane < nr) mem.rng[lane] = make_int4(range.y - incl, incl, 0, 0);  // candidate 0 as if the range began there; end
        if (lane < kDenseTile) {  // particles of other rows have no pair here: they stand where the first one does
            const bool in = seg >> lane & 1u;
            mem.minus[0][lane] = -__shfl_sync(0xffu, mine.x, in ? lane : lead);
            mem.minus[1][lane] = -__shfl_sync(0xffu, mine.y, in ? lane : lead);
            mem.minus[2][lane] = -__shfl_sync(0xffu, mine.z, in ? lane : lead);
        }
        __syncwarp();

        int head = 0, tail = 0;  // places in the ring
        auto group = [&]() {     // eight neighbours
            const int e0 = (head + t) & (kDenseRing - 1), e1 = (head + t + 4) & (kDenseRing - 1);
            const unsigned r0 = (unsigned)mem.index[e0] * pitch + f0, r1 = (unsigned)mem.index[e1] * pitch + f0;
            float v0[1 + D][VW], v1[1 + D][VW];
#pragma unroll
            for (int c = 0; c <= D; ++c) {
                const unsigned o = (unsigned)(c * cp) * 4u;
                if constexpr (VW == 4) {
                    const float4 p = __ldg(reinterpret_cast<const float4 *>(rows + (r0 + o))), q = __ldg(reinterpret_cast<const float4 *>(rows + (r1 + o)));
                    v0[c][0] = p.x; v0[c][1] = p.y; v0[c][2] = p.z; v0[c][3] = p.w;
                    v1[c][0] = q.x; v1[c][1] = q.y; v1[c][2] = q.z; v1[c][3] = q.w;
                } else {
                    const float2 p = __ldg(reinterpret_cast<const float2 *>(rows + (r0 + o))), q = __ldg(reinterpret_cast<const float2 *>(rows + (r1 + o)));
                    v0[c][0] = p.x; v0[c][1] = p.y;
                    v1[c][0] = q.x; v1[c][1] = q.y;
                }
            }
            float w0[1 + D], w1[1 + D], heads[MT][4];
            const bool in = seg >> gr & 1u;
            dense_weights<D, PER>(g, pi, mem.at[e0], in && head + t < tail, w0, tsum);
            dense_weights<D, PER>(g, pi, mem.at[e1], in && head + t + 4 < tail, w1, tsum);
#pragma unroll
            for (int c = 0; c <= D; ++c) {
                const Tf32 b0 = split_tf32(w0[c]), b1 = split_tf32(w1[c]);
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const Tf32 a0 = split_tf32(v0[c][2 * m]), a1 = split_tf32(v0[c][2 * m + 1]);
                    const Tf32 a2 = split_tf32(v1[c][2 * m]), a3 = split_tf32(v1[c][2 * m + 1]);
                    const unsigned ah[4] = {a0.head, a1.head, a2.head, a3.head}, at[4] = {a0.tail, a1.tail, a2.tail, a3.tail};
                    if constexpr (TAILS) mma_m16n8k8(others[m], at, b0.tail, b1.tail);
                    mma_m16n8k8(others[m], at, b0.head, b1.head);
                    if (c == 0) mma_m16n8k8_from_zero(heads[m], ah, b0.head, b1.head);
                    else mma_m16n8k8(heads[m], ah, b0.head, b1.head);
                    mma_m16n8k8(others[m], ah, b0.tail, b1.tail);
                }
            }
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[m][q] += heads[m][q];
            head += 8;
        };

        int piece = 0;
        int4 R = nr > 0 ? mem.rng[0] : make_int4(0, 0, 0, 0);
        auto fetch = [&](int k, int &j) {  // candidate k of the tile
            j = 0;
            if (k >= candidates) return make_float4(0.f, 0.f, 0.f, 0.f);
            while (k >= R.y) R = mem.rng[++piece];
            j = R.x + k;
            return __ldg(a.pv + j);
        };
        int j_next;
        float4 c_next = fetch(lane, j_next);
        for (int k0 = 0; k0 < candidates; k0 += 32) {
            const float4 c = c_next;
            const int j = j_next;
            c_next = fetch(k0 + 32 + lane, j_next);
            float near = 3.0e38f;
            const unsigned long long X = pack2(c.x, c.x), Y = pack2(c.y, c.y), Z = pack2(c.z, c.z);
#pragma unroll
            for (int p = 0; p < kDenseTile; p += 4) {
                const ulonglong2 mx = *reinterpret_cast<const ulonglong2 *>(mem.minus[0] + p), my = *reinterpret_cast<const ulonglong2 *>(mem.minus[1] + p);
                ulonglong2 mz = make_ulonglong2(0ull, 0ull);
                if (D == 3) mz = *reinterpret_cast<const ulonglong2 *>(mem.minus[2] + p);
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    unsigned long long rx = add2(X, v ? mx.y : mx.x), ry = add2(Y, v ? my.y : my.x), rz = 0ull;
                    if (D == 3) rz = add2(Z, v ? mz.y : mz.x);
                    if (PER) {
                        rx = nearest_image2(rx, g.L[0], g.invL[0]);
                        ry = nearest_image2(ry, g.L[1], g.invL[1]);
                        if (D == 3) rz = nearest_image2(rz, g.L[2], g.invL[2]);
                    }
                    unsigned long long q = fma2(ry, ry, mul2(rx, rx));
                    if (D == 3) q = fma2(rz, rz, q);
                    float lo, hi;
                    unpack2(q, lo, hi);
                    near = fminf(near, fminf(lo, hi));
                }
            }
            const bool hit = k0 + lane < candidates && near < reach;
            const unsigned hits = __ballot_sync(kFull, hit);
            if (hit) {
                const int e = (tail + __popc(hits & below)) & (kDenseRing - 1);
                mem.at[e] = c;
                mem.index[e] = j;
            }
            tail += __popc(hits);
            __syncwarp();
#pragma unroll 1
            while (tail - head >= 8) group();
            __syncwarp();
        }
        if (tail > head) {  // the last ones, and the first particle in the places behind them (weight zero)
            if (lane < 8 && lane >= tail - head) {
                const int e = (head + lane) & (kDenseRing - 1);
                mem.at[e] = mine;
                mem.index[e] = first;
            }
            __syncwarp();
            group();
            __syncwarp();
        }
    }

    float probe = 0.f;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            acc[m][q] += others[m][q];
            probe = fmaf(0.f, acc[m][q], probe);
        }
#pragma unroll
    for (int d = 0; d < D; ++d) probe = fmaf(0.f, tsum[d], probe);
    if (__any_sync(kFull, !(probe == 0.f))) {
        dense_pairwise<D, PER>(a, g, mem, first, here);
        return;
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
        tsum[d] += __shfl_xor_sync(kFull, tsum[d], 1);
        tsum[d] += __shfl_xor_sync(kFull, tsum[d], 2);
    }
    // this lane has particles 2 t and 2 t + 1 of the tile, features f .. f + VW - 1
    const int f = VW * gr;
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const int p = 2 * t + w;
        float T[3] = {0.f, 0.f, 0.f}, o[VW];
#pragma unroll
        for (int d = 0; d < D; ++d) T[d] = __shfl_sync(kFull, tsum[d], 4 * p);
        const float v = __shfl_sync(kFull, mine.w, p);
        if (p >= here) continue;  // (no shuffle follows for this particle)
        const long long i = first + p;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int k = 0; k < 2; ++k) o[2 * m + k] = acc[m][2 * k + w];
        if (FILLED && a.out_vec) {
            dense_finish_row<D, VW>(a, i, f, o, v, T);
        } else {
#pragma unroll
            for (int k = 0; k < VW; ++k)
                if (f + k < a.C) a.grad_s[i * a.C + f + k] = dense_finish<D>(a, i, f + k, o[k], v, T);
        }
    }
}

template <int D, bool PER, bool TAILS>
static int launch_dense(const Geom &g, const FeatureListBwdArgs &a, cudaStream_t st) {
    const long long tiles = ((long long)g.B * g.N + kDenseTile - 1) / kDenseTile;
    const unsigned blocks = (unsigned)((tiles + kDenseWarps - 1) / kDenseWarps);
    auto kernel = feature_dense_backward_kernel<D, PER, 2, false, TAILS>;
    if (a.cp == 32) kernel = feature_dense_backward_kernel<D, PER, 2, true, TAILS>;
    else if (a.cp == 16) kernel = feature_dense_backward_kernel<D, PER, 1, true, TAILS>;
    else if (a.cp < 16) kernel = feature_dense_backward_kernel<D, PER, 1, false, TAILS>;
    kernel<<<blocks, kDenseWarps * 32, 0, st>>>(a, g);
    return check_launch("feature_dense_backward_kernel");
}

// A lane's neighbours are four rows at the same feature: an odd number of 32-byte sectors from row to row puts the neighbours of four
// consecutive particles into different banks of L1 (rows of 512 bytes: sixteen wavefronts per load instead of four).
int feature_dense_pitch(int dim, int cp) {
    const int sectors = ((1 + dim) * cp + 7) / 8;
    return 8 * (sectors | 1);
}

// Where it is the faster one, by the mean number of particles per cell of the grid (a tile costs its candidates and the union of its
// neighbours, a list its length) and by the particles in all: a tile is a longer chain than a list, which shows while either kernel is a
// wave or two.  Particles that leave cells empty have more neighbours than the mean tells, and lists that overflow are searched, so that clustered
// ones gain earlier and more; the lines are where uniform ones lose nothing or little.  The kernels alone, lists / this, us, uniform unless said otherwise:
//  * 2D, C = 16: 65,536 particles 2 a cell 17.8 / 18.9, 3 21.3 / 20.6, 4 24.6 / 22.3, 8 37 / 29; along lines 2 a cell 52 / 38, 4 161 / 60; in blobs
//    29 / 24, 86 / 31; 8,192 2 a cell 6.1 / 7.6, 4 8.5 / 8.4, 8 11.1 / 10.0, along lines 16.8 / 13.4, 70 / 19.  The line at 2 costs uniform particles
//    up to 1.5 us below 4 a cell, where the clustered ones, which are what is that thin (12 neighbours of uniform particles are 3.8 a cell), gain 2 to 50.
//  * C = 32: 65,536 2 a cell 27.3 / 27.2, 4 36 / 32; 16,384 10.2 / 9.7, 13.5 / 11.3; 24,000, beyond a wave, 11.1 / 13.3, 15.1 / 13.6; 12,000 2 a cell
//    6.6 / 9.1, 8 12.6 / 13.1; 8,192 5.6 / 8.6, 9.9 / 11.2; along lines 8,192 2 a cell 14.1 / 15.9, 8 68 / 28, in blobs 8.0 / 10.8, 20.7 / 18.4, 12 a cell
//    60 / 23: for few particles from 8 a cell, where lists of clustered ones overflow.
//  * 2D periodic, whose candidates are tested image by image: C = 16, 65,536 7 a cell 34.8 / 34.0, 10 45 / 41; C = 8 8 a cell 35.7 / 36.6, 10 42.3 / 41.0; C = 32 4 a cell
//    37.0 / 35.8; 48,000 C = 16 7 a cell 30.6 / 28.2, C = 32 4 a cell 28.0 / 27.9; 33,000 20.4 / 22.4, 8 a cell 29.7 / 29.1; 24,000 C = 16 10 a cell 19.9 / 22.7,
//    12 22.7 / 24.4.  Fewer particles than 44,000 lose at any uniform density (8,192 12 a cell 14.6 / 17.8, C = 32 12.7 / 18.4): from 12 a cell on that is
//    left so for clustered ones.
//  * 3D, C = 16: 65,536 4 a cell 39.7 / 39.0, 6 52 / 48; 262,144 4 a cell 134 / 138, 5 154 / 152; 32,768 6 a cell 28.5 / 31.7, 8 35.7 / 34.2.  C = 12, whose rows are
//    padded to 16: 65,536 5 a cell 45.3 / 47.7, 6 51.0 / 49.1; 262,144 147 / 157, 169 / 174.
//  * 3D, C = 32: 98,304 4 a cell 77.5 / 83.2, 5 89.1 / 89.6, 6 96.4 / 92.7; C = 20 5 a cell 87.1 / 91.8, 6 95.4 / 94.9.  262,144 C = 32 4 a cell 194 / 195, 4.5
//    215 / 216, C = 20 5 220 / 223.  One wave (20,500) C = 32 6 a cell 27.8 / 26.4, C = 20 7 30.4 / 30.8, 8 35.0 / 32.2; little more (28,000) 8 a cell
//    35.9 / 40.6, 10 43.1 / 45.8; 41,000 8 53.0 / 52.6, 10 63.1 / 60.4, C = 20 52.5 / 54.9, 61.8 / 61.9.  In a ball, where the particles are twice as dense, C = 32: 98,304
//    5 a cell 138 / 128, 262,144 342 / 309, 4 x 65,536 with a radius of 1.05 cells, 4.7 a cell, 380 / 329.
//  * 3D periodic: lists (64 a cell 428 / 463, 8 a cell 76 / 89).
bool feature_dense_covers(const Geom &g, int C) {
    const long long particles = (long long)g.B * g.N;
    if (g.morton || C > 32 || particles * feature_dense_pitch(g.dim, (C + 3) & ~3) >= (1ll << 30)) return false;
    const double per_cell = (double)g.N / g.cells;
    const bool wide = C > 16;  // two blocks of features
    if (g.dim == 2 && !g.periodic) return per_cell >= (wide && particles < 14000 ? 8.0 : 2.0);
    if (g.dim == 2) return per_cell >= (particles < 44000 ? 12.0 : wide ? 4.0 : C > 12 ? 7.0 : 8.0);
    if (g.periodic || particles < 20000) return false;
    if (!wide) return per_cell >= (particles < 40000 ? 8.0 : C > 12 ? 4.0 : 6.0);
    if (particles < 60000) return per_cell >= (particles <= 148 * 5 * kDenseWarps * kDenseTile ? 8.0 : 10.0);
    if (particles < 200000) return per_cell >= (C > 28 ? 5.0 : 6.0);
    return per_cell >= (C > 28 ? 4.5 : 5.0);
}

int launch_feature_dense_backward(const Geom &g, const FeatureListBwdArgs &args, cudaStream_t st) {
    FeatureListBwdArgs a = args;
    a.out_vec = a.C == a.cp && ((uintptr_t)a.grad_s | (uintptr_t)a.add) % 16 == 0;
    if (g.dim == 3) return launch_dense<3, false, false>(g, a, st);
    if ((double)g.N / g.cells < kDenseTailsBelow) return g.periodic ? launch_dense<2, true, true>(g, a, st) : launch_dense<2, false, true>(g, a, st);
    return g.periodic ? launch_dense<2, true, false>(g, a, st) : launch_dense<2, false, false>(g, a, st);
}

}  // namespace npa
