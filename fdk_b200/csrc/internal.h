// internal.h -- declarations shared between translation units of libfdk_b200.
#pragma once
#include <string>

#include "common.h"

namespace fdk {

// FP64 3x4 projection matrix of CalculateProjMat for view angle a (geometry.cpp).
void projection_matrix(const fdk_geometry &g, double a, double *m);

// FDK_ERR_INVALID_ARG for a geometry without positive sizes, pitches and view count, SOD below SID and a known
// window (geometry.cpp).  The kernels that take a geometry rely on it.
int check_geometry(const fdk_geometry *g);

// Device tables of one filter length (filter.cu).
struct FilterTables {
    int W = 0, log2W = 0;
    float2 *tw = nullptr;   // W/2 twiddles exp(-2 pi i k / W)
    float2 *twp = nullptr;  // the FFT passes' twiddles in the order the threads read them (optional)
    float *hb = nullptr;    // H / W, entry i at frequency filter_response_frequency(i, W)
    // the copies go through a private set-up stream that the call waits for (bounded)
    int create(const double *H, int W_);
    void release();
};

// Fill t's device tables (tw and twp where not null, and hb) for response H (device, W taps) on st
// (filter.cu).
int filter_tables_on_device(const float *H, const FilterTables &t, cudaStream_t st);

// Frequency of entry i of FilterTables::hb.  The row filter's transform leaves thread t of W / 16 with
// points p = 16 t + k, k < 16, in bit-reversed order; the table holds them as four planes of four
// points of every thread.  W < 32 is one thread's.
__host__ __device__ inline int filter_response_frequency(int i, int W) {
    const int threads = W / 16;
    int p = W < 32 ? i : 16 * (i / 4 % threads) + 4 * (i / (4 * threads)) + i % 4, f = 0;
    for (int b = 1; b < W; b <<= 1, p >>= 1) f = 2 * f + (p & 1);
    return f;
}

// Twiddle e < 15 of place i in a pass of stride n: 8 of the first of its four stages, then 4, 2, 1; as a
// power of exp(-2 pi i / 16 n).
__host__ __device__ inline int filter_twiddle(int e, int i, int n) {
    int h = 8;
    while (h && e >= h) {
        e -= h;
        h >>= 1;
    }
    return h ? (i + e * n) * (8 / h) : 0;
}

// Fused cosine weight + pad + ramp filter + crop + layout store (filter.cu).
int filter_views(const float *src, int src_pitch, long long src_vstride, void *dst, int dst_pitch,
                 long long dst_vstride, const float *cos, int cos_pitch, const FilterTables &t, int nu, int nv,
                 int pad_n, int n_views, int layout, int dtype, cudaStream_t st, float out_scale = 1.0f,
                 unsigned int *overflow = nullptr);

// Projection-folder files (io.cpp): folder + "img%04d.raw" % file_index, and count views
// (files (first + i) * step + start, sizes checked first) read by `threads` host threads.
std::string proj_file_path(const char *folder, long long file_index);
int read_views(const char *folder, int nu, int nv, long long first, long long count, int step, int start, float *dst,
               int threads);

}  // namespace fdk
