// Images of weight matrices as the tensor-memory kernels of the MLP read them (mlp_tcgen05.cu).
#pragma once
#include "common.cuh"
#include "umma.cuh"

namespace npa {

constexpr int kImageChunk = 32;  // floats of K per chunk

// Head and tail images of one or more weight matrices, chunk by chunk, in the layout the MMA reads.  The jobs share one
// launch: a step of a small system waits for its launches, and both layers' images (and the one the backward will
// want) are a few microseconds of work together.  A whole step lets the reorder of its particles make them
// (bin_particles_and_images).
struct ImageJob {
    const float *W;
    long long stride_n, stride_k;
    int K, N, Np, nchunks;
    float *img;
    int features, dim;  // > 0: rows n in the order of StepColumns (below)
    __host__ __device__ int total() const { return nchunks * Np * kImageChunk; }
};
// The columns of z in the order in which the gradient of a step wants them: the features themselves, their blur, then axis by axis the
// gradient, each section rounded up to 16 columns; the density gradient's columns are left out (nothing of a step reads them).
struct StepColumns {
    __host__ __device__ static int section(int features) { return (features + 15) & ~15; }
    __host__ __device__ static int total(int features, int dim) { return (2 + dim) * section(features); }
    // column of z, or -1 for padding
    __host__ __device__ static int column(int n, int features, int dim) {
        const int sec = n / section(features), f = n - sec * section(features);
        return f >= features ? -1 : sec < 2 ? sec * features + f : 2 * features + f * dim + sec - 2;
    }
};
constexpr int kImageJobs = 3;
struct ImageJobs {
    ImageJob job[kImageJobs];
    int count;
    int total() const {
        int n = 0;
        for (int q = 0; q < count; ++q) n += job[q].total();
        return n;
    }
};

// Element `at` of all jobs together; nothing beyond the last.
__device__ inline void write_image_element(const ImageJobs &jobs, int at) {
    for (int q = 0; q < jobs.count; ++q) {
        const ImageJob &j = jobs.job[q];
        const int total = j.total();
        if (at < total) {
            const int Np = j.Np, c = at / (Np * kImageChunk), rem = at - c * Np * kImageChunk;
            const int n = rem / kImageChunk, kk = rem - n * kImageChunk;
            const int k = c * kImageChunk + kk;
            const int row = j.features > 0 ? StepColumns::column(n, j.features, j.dim) : n;
            const float v = (n < j.N && row >= 0 && k < j.K) ? __ldg(j.W + row * j.stride_n + k * j.stride_k) : 0.f;
            const float head = __uint_as_float(tf32_head_bits(v));
            float *chunk = j.img + (size_t)c * 2 * Np * kImageChunk;
            const int to = umma_swizzled(n, kk);
            chunk[to] = head;
            chunk[Np * kImageChunk + to] = v - head;
            return;
        }
        at -= total;
    }
}

// Work list of several small systems that a grid build has left to the launch behind it.
struct RowsJob {
    const int32_t *bin_offsets;
    int4 *block_info;
    const uint32_t *rows_of_system;
    Geom g;
    int systems;  // 0: nothing is left
};
// binning.cu: npa_grid_build; with `rest`, the work list of several systems is left to bin_particles_and_images where it has a launch of its own.
int grid_build_leaving(const npa_grid *grid, const float *x, int32_t *permutation, int32_t *bin_offsets, int32_t *block_info, void *scratch,
                       int64_t scratch_bytes, cudaStream_t stream, RowsJob *rest);
// binning.cu: npa_bin_particles (without masses) whose launch also makes the images, and the work list that `rest` names.
int bin_particles_and_images(const npa_grid *grid, int channels, const float *x, const float *s, const int32_t *permutation, float *x_out,
                             float *s_out, const ImageJobs &jobs, cudaStream_t stream, const RowsJob &rest = {});

}  // namespace npa
