// Differentiable 2D Gaussian splatting of particles into an image, forward and backward.
//
// Replaces splat_particles / splat_particles_batch of the reference (utils/splatting.py:6-113), the
// renderer of its splat loss (losses/splat_loss.py:71-86).  The reference materialises the
// (2r+1)^2 patch of every particle as [N, (2r+1)^2] index / weight tensors and scatter-adds them
// (atomics, run-to-run different sums).  Here both directions are gathers:
//   forward  : a CTA owns a 16x16 pixel tile and multiplies the separable weights of the particles that
//              touch it into it, or adds them pixel by pixel where they are few -- no atomics, fixed order
//              of sums, deterministic;
//   backward : a warp owns a particle and walks its patch, reading the upstream image gradient
//              (L2 resident) and reducing the colour and position gradients with shuffles.
// Pixel of a particle: p = (x - lo) / (hi - lo) * (img - 1) (y flipped when y_up), base = floor(p),
// frac = p - base; weight of pixel base + (dx, dy): g = exp(-((dx - frac_x)^2 + (dy - frac_y)^2) / (2 sigma^2)),
// with normalisation w = g / (1e-8 + sum of g over the whole patch) * norm_scale; out = [sum c w | sum w].
// The patch sum factorises into two 1D sums (the weight is separable).
#include <cooperative_groups.h>
#include "common.cuh"

namespace npa {

namespace cg = cooperative_groups;

constexpr int kSplatTile = 16;
constexpr int kSplatMaxRadius = 64;

struct SplatArgs {
    const float *x;      // [B, N, 2]
    const float *color;  // [B, N, 3]
    float *out;          // [B, img, img, 4]  (r, g, b, density)
    const float *g_out;  // backward: upstream of out
    float *g_x;          // backward: [B, N, 2]
    float *g_color;      // backward: [B, N, 3]
    float *wscale;       // [B, N] scratch: norm_scale / (1e-8 + patch sum) per particle (normalised mode)
    int B, N, img, radius, y_up, normalize;
    float lo, span, sigma, norm_scale;  // span = hi - lo; sigma in pixels
};

struct SplatPoint {
    int cx, cy;
    float fx, fy;
};

// Pixel of a coordinate along one axis, and the fraction beyond it.  Far-away or non-finite positions touch no pixel: they
// are parked outside every tile.
__device__ inline int splat_axis(const SplatArgs &a, float v, int axis, float &frac) {
    const float top = (float)(a.img - 1);
    float p = __fmul_rn(__fdiv_rn(v - a.lo, a.span), top);
    if (axis && a.y_up) p = top - p;
    const float base = floorf(p), lim = 1.0e8f;
    frac = p - base;
    return (base > -lim && base < lim) ? (int)base : -(1 << 30);
}

__device__ inline SplatPoint splat_point(const SplatArgs &a, long long n) {
    const float2 v = __ldg(reinterpret_cast<const float2 *>(a.x) + n);
    SplatPoint p;
    p.cx = splat_axis(a, v.x, 0, p.fx);
    p.cy = splat_axis(a, v.y, 1, p.fy);
    return p;
}

// sum over d = -r..r of exp(-(d - f)^2 / (2 sigma^2)), and of the same times (d - f)
__device__ inline void axis_sums(int r, float f, float inv2s2, float &s0, float &s1) {
    s0 = 0.f; s1 = 0.f;
    for (int d = -r; d <= r; ++d) {
        const float t = (float)d - f;
        const float g = expf(-(t * t) * inv2s2);
        s0 += g;
        s1 = fmaf(g, t, s1);
    }
}

// Normalised mode: the scale of every particle, once (the forward tiles would otherwise redo the
// 2 (2r+1) exponentials for every tile a particle touches).
__global__ void __launch_bounds__(256) splat_scale_kernel(SplatArgs a) {
    after_previous_kernel();
    const long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (n >= (long long)a.B * a.N) return;
    const SplatPoint p = splat_point(a, n);
    const float inv2s2 = 1.0f / (2.0f * a.sigma * a.sigma);
    float sx, sy, unused;
    axis_sums(a.radius, p.fx, inv2s2, sx, unused);
    axis_sums(a.radius, p.fy, inv2s2, sy, unused);
    a.wscale[n] = a.norm_scale / (1e-8f + sx * sy);
}

// A CTA per 16 x 16 pixel tile.  The weight of a particle is a product of a row and a column factor, so a tile's image is
// a product of small matrices over the particles that touch it: sum_n wx_n[px] (wy_n[py] c_n).  4,096 particles at a time are
// culled with a pixel to spare into a list (a thread's hits in a row, threads in order); 64 at a time get their 16 + 16
// factors in shared memory (32 exponentials per particle and tile instead of 256; eight per thread) while the 64 before are
// multiplied; every half warp multiplies every 16th particle into 8 x 2 pixels x 4 channels per thread in packed fp32x2, two
// neighbouring pixels to a pair; the 16 partial images are added in a fixed order.  kCluster: the CTAs of a cluster share the tile,
// each with a slice of the particles, and add their images through distributed shared memory, slices in order.  kTurns: one CTA takes
// the slices one after the other and adds in the same order, so that either gives the same bits.
// Bound by latency (fill of the list, first factors, sum of the partial images) at two blocks per SM: 45 % of the issue slots,
// fp32 pipe 22 %.  8 systems of 4,096 particles, 256 x 256, patches of 41 x 41, us: pixel by pixel 201; list of 1,024
// particles at a time, factors and products between barriers, channels packed (wants every column factor twice) 113; this 86.  64 x 64,
// one system of 8,192: 92 -> 19 (eight slices).  More warps do not fit: 64 sums per thread.
constexpr int kSplatThreads = 256, kSplatCull = 16, kSplatWindow = kSplatThreads * kSplatCull, kSplatChunk = 64, kSplatParts = 16,
              kSplatWarps = kSplatThreads / 32;

struct SplatFactors {
    float wx[kSplatChunk][kSplatTile];
    float pad[4];                       // the row and the column factors that one instruction stores lie on different banks
    float wy[kSplatChunk][kSplatTile];
    float4 c[kSplatChunk];              // scale times (r, g, b, 1)
};
struct SplatLists {
    SplatFactors f[2];
    unsigned short n[kSplatWindow];
};
union SplatShared {
    SplatLists lists;
    float4 part[kSplatWarps][kSplatTile * kSplatTile];
};

// Place of a pixel in a partial image: sixteen lanes store pixels 8 and 32 apart, which all meet on the same banks in a plain
// layout (4,096 tiles with a few particles each: 67 us, so 48).
__device__ inline int part_at(int pixel) { return pixel ^ ((pixel >> 5) & 7); }

enum class SplatSlices { kOne, kCluster, kTurns };

template <SplatSlices SLICES>
__global__ void __launch_bounds__(kSplatThreads, 2) splat_forward_kernel(SplatArgs a, int slices) {
    after_previous_kernel();
    constexpr bool CLUSTER = SLICES == SplatSlices::kCluster, TURNS = SLICES == SplatSlices::kTurns;
    __shared__ SplatShared sh;
    __shared__ int s_count[kSplatWarps];
    __shared__ float4 s_sum[TURNS ? kSplatThreads : 1];  // a pixel's sum over the slices so far (registers are all taken)
    const int tiles = (a.img + kSplatTile - 1) / kSplatTile;
    if (SLICES == SplatSlices::kOne) slices = 1;
    const int mine = CLUSTER ? blockIdx.x % slices : 0, tile = CLUSTER ? blockIdx.x / slices : blockIdx.x;
    const int tx0 = (tile % tiles) * kSplatTile, ty0 = (tile / tiles) * kSplatTile;
    const int b = blockIdx.y, r = a.radius;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int part = tid >> 4, cell = tid & 15, px = (cell & 1) * 8, py = (cell >> 1) * 2;  // pixels px..px+7, py..py+1
    const float inv2s2 = 1.0f / (2.0f * a.sigma * a.sigma);
    unsigned long long acc[2][4][4];  // [row][channel][two pixels]

    // What a thread needs to make eight factors of one axis of a particle: loaded a chunk ahead.
    const int sp = tid >> 2, axis = (tid >> 1) & 1, o0 = (tid & 1) * 8;
    const bool colours = (tid & 3) == 3;
    float pos = 0.f;
    float4 col = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](unsigned window, int off, int count) {
        if (off + sp >= count) return;
        const long long n = (long long)b * a.N + window + sh.lists.n[off + sp];
        pos = __ldg(a.x + n * 2 + axis);
        if (colours) {
            const float *c = a.color + n * 3;
            col = make_float4(__ldg(c), __ldg(c + 1), __ldg(c + 2), a.normalize ? __ldg(a.wscale + n) : 1.0f);
        }
    };
    // Eight factors into buffer f; whether the particle's colour is finite (zero times one that is not is not zero outside the patch).
    auto factors = [&](SplatFactors &f, int off, int count) {
        if (off + sp >= (count + kSplatParts - 1) / kSplatParts * kSplatParts) return false;
        const bool valid = off + sp < count;
        float w[8], frac;
        int at = splat_axis(a, pos, axis, frac);
        at = (axis ? ty0 : tx0) - at + o0;  // offset of the first of the eight from the particle's pixel
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int d = at + k;
            const float t = (float)d - frac;
            w[k] = valid && d >= -r && d <= r ? expf(-(t * t) * inv2s2) : 0.f;
        }
        float4 *o = reinterpret_cast<float4 *>(axis ? &f.wy[sp][o0] : &f.wx[sp][o0]);
        o[0] = make_float4(w[0], w[1], w[2], w[3]);
        o[1] = make_float4(w[4], w[5], w[6], w[7]);
        if (!colours) return false;
        const float4 c = valid ? make_float4(col.w * col.x, col.w * col.y, col.w * col.z, col.w) : make_float4(0.f, 0.f, 0.f, 0.f);
        f.c[sp] = c;
        return !(fabsf(c.x) + fabsf(c.y) + fabsf(c.z) < INFINITY);
    };
    auto multiply = [&](const SplatFactors &f, int padded, bool odd) {
#pragma unroll 1
        for (int q = part; q < padded; q += kSplatParts) {
            const float4 x0 = *reinterpret_cast<const float4 *>(&f.wx[q][px]), x1 = *reinterpret_cast<const float4 *>(&f.wx[q][px + 4]);
            const float2 wy = *reinterpret_cast<const float2 *>(&f.wy[q][py]);
            const float4 c = f.c[q];
            const float cs[4] = {c.x, c.y, c.z, c.w};
            if (odd) {
                const float xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const float w = y ? wy.y : wy.x;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int x = 0; x < 4; ++x) {
                            float lo, hi;
                            unpack2(acc[y][k][x], lo, hi);
                            if (w != 0.f && xs[2 * x] != 0.f) lo = fmaf(xs[2 * x], w * cs[k], lo);
                            if (w != 0.f && xs[2 * x + 1] != 0.f) hi = fmaf(xs[2 * x + 1], w * cs[k], hi);
                            acc[y][k][x] = pack2(lo, hi);
                        }
                }
                continue;
            }
            const unsigned long long xx[4] = {pack2(x0.x, x0.y), pack2(x0.z, x0.w), pack2(x1.x, x1.y), pack2(x1.z, x1.w)};
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const float w = y ? wy.y : wy.x;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float v = w * cs[k];
                    const unsigned long long vv = pack2(v, v);
#pragma unroll
                    for (int x = 0; x < 4; ++x) acc[y][k][x] = fma2(xx[x], vv, acc[y][k][x]);
                }
            }
        }
    };

    const float top = (float)(a.img - 1), per = top / a.span, reach = (float)r + 9.25f;  // patch radius, half a tile, a pixel, rounding
    const float mx = (float)tx0 + 7.5f, my = (float)ty0 + 7.5f;
    const unsigned share = ((unsigned)a.N + slices - 1) / slices;  // (unsigned: a window may end beyond 2^31 particles)
    float4 v;
    for (int slice = mine; slice < (TURNS ? slices : mine + 1); ++slice) {
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int x = 0; x < 4; ++x) acc[y][c][x] = 0ull;
        const unsigned from = slice * share, end = min((unsigned)a.N, from + share);
        for (unsigned n0 = from; n0 < end; n0 += kSplatWindow) {
            unsigned hits = 0;
#pragma unroll 8
            for (int q = 0; q < kSplatCull; ++q) {
                const unsigned n = n0 + q * kSplatThreads + tid;
                if (n < end) {
                    const float2 v = __ldg(reinterpret_cast<const float2 *>(a.x) + (long long)b * a.N + n);
                    const float x = (v.x - a.lo) * per;
                    float y = (v.y - a.lo) * per;
                    if (a.y_up) y = top - y;
                    if (fabsf(x - mx) <= reach && fabsf(y - my) <= reach) hits |= 1u << q;
                }
            }
            int incl = __popc(hits);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (lane == 31) s_count[warp] = incl;
            __syncthreads();  // (also: the window before has read its list and factors)
            int at = incl - __popc(hits), count = 0;
#pragma unroll
            for (int w = 0; w < kSplatWarps; ++w) {
                const int c = s_count[w];
                if (w < warp) at += c;
                count += c;
            }
            for (; hits; hits &= hits - 1) sh.lists.n[at++] = (unsigned short)((__ffs(hits) - 1) * kSplatThreads + tid);
            __syncthreads();
            fetch(n0, 0, count);
            for (int off = 0, buf = 0; off < count; off += kSplatChunk, buf ^= 1) {
                const bool odd = factors(sh.lists.f[buf], off, count);
                fetch(n0, off + kSplatChunk, count);
                const bool any_odd = __syncthreads_or(odd);  // (also: the chunk before the last has left its buffer)
                multiply(sh.lists.f[buf], min(kSplatChunk, (count - off + kSplatParts - 1) / kSplatParts * kSplatParts), any_odd);
            }
        }
        __syncthreads();
        // the two halves of a warp meet by shuffles, the eight warps in shared memory
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                float v[2][4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    unpack2(acc[y][k][x], v[0][k], v[1][k]);
                    v[0][k] += __shfl_xor_sync(0xffffffffu, v[0][k], 16);
                    v[1][k] += __shfl_xor_sync(0xffffffffu, v[1][k], 16);
                }
                // each half stores one of the two pixels
                const int h = lane >> 4;
                sh.part[warp][part_at((py + y) * kSplatTile + px + 2 * x + h)] =
                    make_float4(h ? v[1][0] : v[0][0], h ? v[1][1] : v[0][1], h ? v[1][2] : v[0][2], h ? v[1][3] : v[0][3]);
            }
        __syncthreads();
        v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < kSplatWarps; ++w) {
            const float4 q = sh.part[w][part_at(tid)];
            v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
        }
        // (the next turn's list overwrites the partial images only behind a barrier that follows these reads)
        if (TURNS) {
            const float4 before = slice ? s_sum[tid] : make_float4(0.f, 0.f, 0.f, 0.f);
            v = make_float4(before.x + v.x, before.y + v.y, before.z + v.z, before.w + v.w);
            s_sum[tid] = v;
        }
    }
    int pixel = tid;
    if (CLUSTER) {
        // every CTA of the cluster adds up its share of the pixels, over the slices in order
        cg::cluster_group cluster = cg::this_cluster();
        sh.part[0][part_at(tid)] = v;  // (only this thread reads this place of the first warp's image)
        cluster.sync();
        const int each = kSplatTile * kSplatTile / slices;
        pixel = mine * each + tid;
        if (tid < each) {
            v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int k = 0; k < slices; ++k) {
                const float4 q = cluster.map_shared_rank(&sh.part[0][0], k)[part_at(pixel)];
                v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
            }
        }
        cluster.sync();
        if (tid >= each) return;
    }
    const int ox = tx0 + (pixel % kSplatTile), oy = ty0 + (pixel / kSplatTile);
    if (ox < a.img && oy < a.img) reinterpret_cast<float4 *>(a.out)[((long long)b * a.img + oy) * a.img + ox] = v;
}

// Few particles to a tile: a thread per pixel adds the particles that touch the tile in particle order.  Most of the
// kernel above is fixed cost then (sixteen partial images, two blocks per SM); this one keeps eight blocks per SM.
__global__ void __launch_bounds__(kSplatTile *kSplatTile) splat_forward_sparse_kernel(SplatArgs a) {
    after_previous_kernel();
    constexpr int T = kSplatTile * kSplatTile;
    __shared__ int s_cx[T], s_cy[T];
    __shared__ float s_fx[T], s_fy[T], s_w[T], s_r[T], s_g[T], s_b[T];
    __shared__ int s_warp_count[T / 32];
    const int tiles = (a.img + kSplatTile - 1) / kSplatTile;
    const int tx0 = (blockIdx.x % tiles) * kSplatTile, ty0 = (blockIdx.x / tiles) * kSplatTile;
    const int b = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int px = tx0 + (tid % kSplatTile), py = ty0 + (tid / kSplatTile);
    const int r = a.radius;
    const float inv2s2 = 1.0f / (2.0f * a.sigma * a.sigma);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};

    for (unsigned n0 = 0; n0 < (unsigned)a.N; n0 += T) {
        const unsigned n = n0 + tid;
        bool hit = false;
        SplatPoint p = {0, 0, 0.f, 0.f};
        if (n < (unsigned)a.N) {
            p = splat_point(a, (long long)b * a.N + n);
            hit = p.cx + r >= tx0 && p.cx - r < tx0 + kSplatTile && p.cy + r >= ty0 && p.cy - r < ty0 + kSplatTile;
        }
        // ordered compaction: particles keep their index order in the list
        const unsigned bal = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) s_warp_count[warp] = __popc(bal);
        __syncthreads();
        int base = 0, total = 0;
        for (int w = 0; w < T / 32; ++w) {
            const int c = s_warp_count[w];
            if (w < warp) base += c;
            total += c;
        }
        if (hit) {
            const int slot = base + __popc(bal & ((1u << lane) - 1u));
            const float scale = a.normalize ? __ldg(a.wscale + (long long)b * a.N + n) : 1.0f;
            const float *c = a.color + ((long long)b * a.N + n) * 3;
            s_cx[slot] = p.cx; s_cy[slot] = p.cy; s_fx[slot] = p.fx; s_fy[slot] = p.fy; s_w[slot] = scale;
            s_r[slot] = __ldg(c); s_g[slot] = __ldg(c + 1); s_b[slot] = __ldg(c + 2);
        }
        __syncthreads();
        for (int e = 0; e < total; ++e) {
            const int dx = px - s_cx[e], dy = py - s_cy[e];
            if (dx < -r || dx > r || dy < -r || dy > r) continue;
            const float tx = (float)dx - s_fx[e], ty = (float)dy - s_fy[e];
            const float w = expf(-(tx * tx + ty * ty) * inv2s2) * s_w[e];
            acc[0] = fmaf(s_r[e], w, acc[0]);
            acc[1] = fmaf(s_g[e], w, acc[1]);
            acc[2] = fmaf(s_b[e], w, acc[2]);
            acc[3] += w;
        }
        __syncthreads();
    }
    if (px < a.img && py < a.img)
        reinterpret_cast<float4 *>(a.out)[((long long)b * a.img + py) * a.img + px] =
            make_float4(acc[0], acc[1], acc[2], acc[3]);
}

__device__ inline float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One warp per particle.  With A = c . g_rgb + g_density at a pixel and g the unnormalised weight:
//   dL/dc      = scale * sum g g_rgb
//   dL/dfrac_x = scale / sigma^2 * [ sum A g t_x  -  (sum A g) (T_x S_y) / (1e-8 + S) ]   (normalised)
//              =         1 / sigma^2 * sum A g t_x                                         (plain)
// sums over the pixels of the patch that lie inside the image; S = S_x S_y and T_x = sum g_x t_x over
// the whole patch axis; t_x = dx - frac_x.  floor() passes no gradient, so dL/dp = dL/dfrac.
// The weight is separable: a lane keeps one column of the patch, runs down its rows with the row factors from shared
// memory and applies the column factor once at the end (2 (2r+1) exponentials per particle instead of (2r+1)^2).  The
// last, narrow group of columns is dealt to the lanes several rows at a time.  Bound by the latency of the reads of the upstream
// image (16 bytes per pixel of the patch, from L1 and L2) at 32 warps per SM: with a third of the instructions less (packed sums, three
// columns per lane and two rows at a time) 80-102 us instead of 74, with particles sorted by place (L1 hits 81 %) 83.
// 8 x 4,096 particles, patches of 41 x 41: 158 -> 74 us.
__global__ void __launch_bounds__(256) splat_backward_kernel(SplatArgs a) {
    after_previous_kernel();
    constexpr int kMost = 2 * kSplatMaxRadius + 1;
    __shared__ float2 s_y[8][kMost];  // row factor, row factor times t_y
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long total = (long long)a.B * a.N;
    if (warp >= total) return;
    const int b = (int)(warp / a.N);
    const SplatPoint p = splat_point(a, warp);
    const int r = a.radius, P = 2 * r + 1;
    const float inv2s2 = 1.0f / (2.0f * a.sigma * a.sigma);
    const float *c = a.color + warp * 3;
    const float cr = __ldg(c), cg = __ldg(c + 1), cb = __ldg(c + 2);
    const float4 *img = reinterpret_cast<const float4 *>(a.g_out) + (long long)b * a.img * a.img;
    float sx = 0.f, sy = 0.f, t_x = 0.f, t_y = 0.f;  // the axis sums, spread over the lanes
    for (int k = lane; k < P; k += 32) {
        const float ux = (float)(k - r) - p.fx, uy = (float)(k - r) - p.fy;
        const float ex = expf(-(ux * ux) * inv2s2), ey = expf(-(uy * uy) * inv2s2);
        sx += ex; sy += ey;
        t_x = fmaf(ex, ux, t_x); t_y = fmaf(ey, uy, t_y);
        s_y[w][k] = make_float2(ey, ey * uy);
    }
    __syncwarp();
    // rows of the patch inside the image
    const int k0 = max(0, r - p.cy), k1 = min(P, a.img - p.cy + r);
    float gr = 0.f, gg = 0.f, gb = 0.f, a0 = 0.f, ax = 0.f, ay = 0.f;
    for (int c0 = 0; c0 < P; c0 += 32) {
        const int width = min(32, P - c0), steps = 32 / width;  // lanes: `width` columns x `steps` rows
        const int col = lane % width, row0 = lane / width;
        const int k = c0 + col, x = p.cx + k - r;
        if (row0 >= steps || x < 0 || x >= a.img) continue;
        float sr = 0.f, sg = 0.f, sb = 0.f, sA = 0.f, tA = 0.f;
        const float4 *at = img + (long long)(p.cy - r + k0 + row0) * a.img + x;
#pragma unroll 4
        for (int y = k0 + row0; y < k1; y += steps, at += (long long)steps * a.img) {
            const float4 d = __ldg(at);
            const float2 f = s_y[w][y];
            const float A = fmaf(cr, d.x, fmaf(cg, d.y, fmaf(cb, d.z, d.w)));
            sr = fmaf(f.x, d.x, sr); sg = fmaf(f.x, d.y, sg); sb = fmaf(f.x, d.z, sb);
            sA = fmaf(f.x, A, sA);
            tA = fmaf(f.y, A, tA);
        }
        const float ux = (float)(k - r) - p.fx, ex = expf(-(ux * ux) * inv2s2);
        gr = fmaf(ex, sr, gr); gg = fmaf(ex, sg, gg); gb = fmaf(ex, sb, gb);
        a0 = fmaf(ex, sA, a0);
        ax = fmaf(ex * ux, sA, ax);
        ay = fmaf(ex, tA, ay);
    }
    gr = warp_sum(gr); gg = warp_sum(gg); gb = warp_sum(gb);
    a0 = warp_sum(a0); ax = warp_sum(ax); ay = warp_sum(ay);
    if (a.normalize) { sx = warp_sum(sx); sy = warp_sum(sy); t_x = warp_sum(t_x); t_y = warp_sum(t_y); }
    if (lane != 0) return;
    float scale = 1.0f, gfx = ax, gfy = ay;
    if (a.normalize) {
        const float inv = 1.0f / (1e-8f + sx * sy);
        scale = a.norm_scale * inv;
        gfx = ax - a0 * inv * (t_x * sy);
        gfy = ay - a0 * inv * (sx * t_y);
    }
    const float inv_s2 = 1.0f / (a.sigma * a.sigma);
    const float chain = (float)(a.img - 1) / a.span;
    if (a.g_color) {
        float *o = a.g_color + warp * 3;
        o[0] = scale * gr; o[1] = scale * gg; o[2] = scale * gb;
    }
    if (a.g_x) {
        const float sign_y = a.y_up ? -1.0f : 1.0f;
        reinterpret_cast<float2 *>(a.g_x)[warp] =
            make_float2(scale * inv_s2 * gfx * chain, sign_y * scale * inv_s2 * gfy * chain);
    }
}

// Which forward: by the particles of a tile if they lay evenly over the image, h = N min(1, (patch + 16) / img)^2, so that an image
// does not depend on the batch it is rendered in.  Measured over 220 sizes (images of 64 to 256, patches of 7 to 41, 1 to 16
// systems), sparse / product kernel, us: 16 systems, 256 x 256, patch 21: h = 1.3 12.8 / 48, 11 31 / 57, 21 54 / 65; 1 system, 256 x
// 256, patch 41: h = 13 8.7 / 9.0, 25 11.6 / 9.9, 51 17.3 / 12.7.  The line is at worst 19 % behind the better kernel, 0.7 % on
// average.
static double particles_of_a_tile(const SplatArgs &a) {
    const double reach = (2.0 * a.radius + 1.0 + kSplatTile) / a.img, part = reach < 1.0 ? reach * reach : 1.0;
    return a.N * part;
}
static bool sparse_tiles(const SplatArgs &a) { return particles_of_a_tile(a) < 28.0; }

// CTAs that share a tile, each with a slice of the particles: an image of few tiles leaves most of the 148 SMs idle, a second CTA
// per tile costs the fixed part of one.  By the tiles of an image and the particles of a tile (h above), again not by the batch.
// Measured over images of 64 to 256 pixels, 64 to 8,192 particles and 1 to 16 systems, us with one / two / four / eight slices: 64
// pixels, h = 1458, 1 system 76 / 43 / 27 / 19, 4 systems 76 / 45 / 33 / 35; h = 729, 1 system 43 / 27 / 19 / 15, 8 systems 43 / 31 /
// 32 / 39; h = 364, 16 systems 31 / 32 / 37; 192 pixels, h = 491, 1 system 37 / 27, 4 systems 71 / 71; h = 245, 8 systems 66 / 84; 224
// pixels, h = 440, 1 system 35 / 33, 4 systems 83 / 85.
// What the batch decides is whether a cluster takes the slices or one CTA in turn, with the same bits: once all tiles of the batch
// fill the chip the clusters only repeat the fixed part, up to 45 % of the kernel with eight slices.  us, cluster / in turn: 64 pixels,
// eight slices of 8,192, 16 systems (256 tiles) 97 / 112, 32 181 / 178, 64 353 / 308; 128 pixels, four slices of 8,192, 8 systems (512) 94 / 99,
// 16 174 / 160, 32 334 / 286; 192 pixels, two slices of 8,192, 8 systems (1,152) 132 / 128, 16 245 / 227, of 16,384,
// 8 systems 224 / 232.  Images of four tiles, which are all as full, fill the chip evenly and earlier: 32 pixels, eight slices of 4,096,
// 32 systems 52 / 84, 64 98 / 85.
static int splat_slices(const SplatArgs &a, int tiles) {
    const double h = particles_of_a_tile(a);
    if (tiles <= 64) return h >= 1400.0 ? 8 : h >= 680.0 ? 4 : h >= 340.0 ? 2 : 1;
    return tiles <= 144 && h >= 340.0 ? 2 : 1;
}

static bool slices_in_turn(const SplatArgs &a, int tiles) { return (long long)a.B * tiles >= (tiles <= 4 ? 256 : tiles <= 64 ? 1024 : 1600); }

static int check_splat(const char *name, const SplatArgs &a) {
    if (a.B <= 0 || a.N <= 0 || a.img <= 0) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: batch, particles and img_size must be positive", name);
    if (a.radius < 1 || a.radius > kSplatMaxRadius)
        return fail(NPA_ERR_UNSUPPORTED, "%s: patch radius %d is outside 1..%d", name, a.radius, kSplatMaxRadius);
    if (!(a.sigma > 0.f) || !(a.span != 0.f)) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: sigma must be positive and hi != lo", name);
    if (!a.x || !a.color) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: x and color must be non-NULL", name);
    if ((uintptr_t)a.x % 8) return fail(NPA_ERR_INVALID_ARGUMENT, "%s: x must be 8-byte aligned", name);
    return NPA_OK;
}

}  // namespace npa

using namespace npa;

extern "C" {

int npa_splat_forward(const float *x, const float *color, int32_t batch, int32_t particles, int32_t img_size,
                      double sigma_pixels, int32_t radius, double lo, double hi, int32_t y_up, int32_t normalize,
                      double norm_scale, float *scale_scratch, float *out, void *stream) {
    SplatArgs a = {};
    a.x = x; a.color = color; a.out = out; a.wscale = scale_scratch; a.B = batch; a.N = particles; a.img = img_size; a.radius = radius;
    a.y_up = y_up; a.normalize = normalize; a.lo = (float)lo; a.span = (float)(hi - lo); a.sigma = (float)sigma_pixels;
    a.norm_scale = (float)norm_scale;
    int rc = check_splat("npa_splat_forward", a);
    if (rc != NPA_OK) return rc;
    if (!out || (uintptr_t)out % 16) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_splat_forward: out must be non-NULL and 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    if (normalize) {
        if (!scale_scratch) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_splat_forward: scale_scratch [B*N] is needed when normalize != 0");
        const long long n = (long long)batch * particles;
        launch_early(splat_scale_kernel, (unsigned)((n + 255) / 256), 256, 0, st, a);
        if ((rc = check_launch("splat_scale_kernel")) != NPA_OK) return rc;
    }
    const int tiles = (img_size + kSplatTile - 1) / kSplatTile;
    if (sparse_tiles(a)) {
        launch_early(splat_forward_sparse_kernel, dim3(tiles * tiles, batch), kSplatTile * kSplatTile, 0, st, a);
        return check_launch("splat_forward_sparse_kernel");
    }
    const int slices = splat_slices(a, tiles * tiles);
    if (slices == 1) {
        launch_early(splat_forward_kernel<SplatSlices::kOne>, dim3(tiles * tiles, batch), kSplatThreads, 0, st, a, 1);
        return check_launch("splat_forward_kernel");
    }
    if (slices_in_turn(a, tiles * tiles)) {
        launch_early(splat_forward_kernel<SplatSlices::kTurns>, dim3(tiles * tiles, batch), kSplatThreads, 0, st, a, slices);
        return check_launch("splat_forward_kernel (slices in turn)");
    }
    launch_cluster(slices, splat_forward_kernel<SplatSlices::kCluster>, dim3(slices * tiles * tiles, batch), kSplatThreads, 0, st, a, slices);
    return check_launch("splat_forward_kernel");
}

int npa_splat_backward(const float *x, const float *color, const float *g_out, int32_t batch, int32_t particles,
                       int32_t img_size, double sigma_pixels, int32_t radius, double lo, double hi, int32_t y_up,
                       int32_t normalize, double norm_scale, float *g_x, float *g_color, void *stream) {
    SplatArgs a = {};
    a.x = x; a.color = color; a.g_out = g_out; a.g_x = g_x; a.g_color = g_color; a.B = batch; a.N = particles;
    a.img = img_size; a.radius = radius; a.y_up = y_up; a.normalize = normalize; a.lo = (float)lo; a.span = (float)(hi - lo);
    a.sigma = (float)sigma_pixels; a.norm_scale = (float)norm_scale;
    int rc = check_splat("npa_splat_backward", a);
    if (rc != NPA_OK) return rc;
    if (!g_out || (uintptr_t)g_out % 16) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_splat_backward: g_out must be non-NULL and 16-byte aligned");
    if (g_x && (uintptr_t)g_x % 8) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_splat_backward: g_x must be 8-byte aligned");
    const long long warps = (long long)batch * particles;
    const long long ctas = (warps * 32 + 255) / 256;
    if (ctas >= (1ll << 31)) return fail(NPA_ERR_INVALID_ARGUMENT, "npa_splat_backward: too many particles");
    launch_early(splat_backward_kernel, (unsigned)ctas, 256, 0, (cudaStream_t)stream, a);
    return check_launch("splat_backward_kernel");
}

}  // extern "C"
