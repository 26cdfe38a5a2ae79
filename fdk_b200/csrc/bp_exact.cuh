// bp_exact.cuh -- backprojection kernel with the reference kernel's arithmetic.
//
// Same per-voxel operations, in the same order and rounding, as cudaFdkBP<TRANSPOSE, false,
// bSymmetric> (cudaBP/backprojectionFDK.cu:50-129, SUBPIXEL :15-48, dotIJKW and the
// mad.rz.ftz blend cudaBP/cudaBpLib.cuh:5-44), so the results are bit-identical; including the
// way each warp takes (U, 1/w) for view s from lane s.  The launch shape
// differs: 256-thread CTAs (32 z-lanes x 8 columns), 64-bit volume offsets (the reference's
// 32-bit `uint offset` wraps beyond 2^32 voxels), and partial last warps stay alive and only skip the
// store.
#pragma once
#include "common.h"
#include "tma_common.cuh"

namespace fdk {

struct BpExactArgs {
    float *vol;          // [x][y][zs] sub-volume, zs extent D
    const float *proj;   // n_proj frames of height x width (pitch = width)
    const float *mats;   // 12 floats per view
    int width, height, n_proj;
    int x0, y0, z0;      // origin of the top slab (minA)
    int nxs, nys, nzz;   // top slab extent; nzz = z count processed per thread column
    long long D;         // storage depth (top + bottom)
};

__device__ __forceinline__ float fma_rz(float a, float b, float c) {
    float d;
    asm("fma.rz.ftz.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ float dot_ijkw(const float4 m, const float4 p) {
    float s = m.w;
    s = fma_rz(m.x, p.x, s);
    s = fma_rz(m.y, p.y, s);
    s = fma_rz(m.z, p.z, s);
    return s;
}

// What one view has in common for a warp (32 z of one column): computed by the view's lane.
template <typename Off>
struct __align__(16) BpExactView {
    f32x2 d, d1;    // fraction of u, and 1 - it, each twice
    f32x2 f2;       // the square of 1 / w, twice
    float f;        // 1 / w
    float v0, vz;   // detector row v = (v0 + vz z) f
    Off off;        // bytes from the view's first sample to detector column u (its frame row or its element)
};
__device__ __forceinline__ float low2f(f32x2 a) { return __uint_as_float((unsigned)a); }

// Cell and fraction of a coordinate: 64-bit offsets come with detectors of any length, whole_part ends at 2^23.
template <typename Off>
__device__ __forceinline__ unsigned cell(float x, float &fraction) {
    if constexpr (sizeof(Off) == 4) return whole_part(x, fraction);
    const float i = floorf(x);
    fraction = x - i;
    return (unsigned)i;
}

// SUBPIXEL at detector row v of a view (zero outside [0, last)): frame rows are detector columns
// (TRANSPOSE: v runs along the row) or detector rows.  `stride`: bytes of a frame row.
template <bool TRANSPOSE, typename Off>
__device__ __forceinline__ float subpixel_exact(const char *view, const BpExactView<Off> &m, Off stride, float v, float last) {
    if (!(v >= 0.f && v < last)) return 0.f;
    float e;
    const unsigned i = cell<Off>(v, e);
    const float e1 = 1.0f - e;
    const Off o = m.off + (TRANSPOSE ? i * (Off)4 : i * stride);
    const float *p0 = reinterpret_cast<const float *>(view + o), *p1 = reinterpret_cast<const float *>(view + (o + stride));
    float x0 = __ldg(p0), x1 = __ldg(p0 + 1), x2 = __ldg(p1), x3 = __ldg(p1 + 1);
    const float d = low2f(m.d), d1 = low2f(m.d1);
    const float dx = TRANSPOSE ? e : d, dx1 = TRANSPOSE ? e1 : d1, dy = TRANSPOSE ? d : e, dy1 = TRANSPOSE ? d1 : e1;
    x0 = fma_rz(x0, dx1, x1 * dx);
    x2 = fma_rz(x2, dx1, x3 * dx);
    return fma_rz(x0, dy1, x2 * dy);
}

// The same for a voxel and its mirror, both rows vv inside [0, last): one packed instruction for the two.
template <bool TRANSPOSE, typename Off>
__device__ __forceinline__ f32x2 subpixel_pair(const char *view, const BpExactView<Off> &m, Off stride, f32x2 vv) {
    const f32x2 r = add2f_rz(vv, pack2f(8388608.f, 8388608.f)), minus = pack2f(-1.f, -1.f);
    const f32x2 e = fma2f(add2f(r, pack2f(-8388608.f, -8388608.f)), minus, vv), e1 = fma2f(e, minus, pack2f(1.f, 1.f));
    f32x2 t[4];
    const auto texels = [&](unsigned bits, float (&x)[4]) {
        const unsigned i = bits - 0x4B000000u;
        const Off o = m.off + (TRANSPOSE ? i * 4u : i * stride);
        const float *p0 = reinterpret_cast<const float *>(view + o), *p1 = reinterpret_cast<const float *>(view + (o + stride));
        x[0] = __ldg(p0), x[1] = __ldg(p0 + 1), x[2] = __ldg(p1), x[3] = __ldg(p1 + 1);
    };
    float x[4], y[4];
    texels((unsigned)r, x);
    texels((unsigned)(r >> 32), y);
#pragma unroll
    for (int k = 0; k < 4; k++) t[k] = pack2f(x[k], y[k]);
    const f32x2 dx = TRANSPOSE ? e : m.d, dx1 = TRANSPOSE ? e1 : m.d1, dy = TRANSPOSE ? m.d : e, dy1 = TRANSPOSE ? m.d1 : e1;
    const f32x2 x0 = fma2f_rz_ftz(t[0], dx1, mul2f(t[1], dx)), x2 = fma2f_rz_ftz(t[2], dx1, mul2f(t[3], dx));
    return fma2f_rz_ftz(x0, dy1, mul2f(x2, dy));
}

// A warp takes 32 z of one voxel column.  Per 32 views, lane s works out all that view s has in common
// for the column (u, its cell and fraction, 1/w and its square, the part of v without z) and leaves it in
// shared memory; the loop over views then reads it with two broadcast loads and is left with v, two
// cells and eight texels.  The first form shuffled (u, 1/w) and formed the rest in every lane: 105
// instructions a view and voxel pair, 87% of the issue slots, 21.85 ms for 512^3 from 96 views; this
// one, with scalar arithmetic, had 72, filled as many slots and 81% of the L1 wavefronts, and took 14.55
// ms; with voxel and mirror in packed registers where both rows are inside (all but the detector's edge)
// 13.72.  Two z runs a thread on one record took 15.3 ms, the view loop unrolled twice 16.0 (both scalar).
// Off: unsigned, or 64 bits for views of 4 GB and more and for more than 2^22 rows or columns (cell).
template <bool SYM, bool TRANSPOSE, typename Off>
__global__ void __launch_bounds__(256, 6) bp_exact_kernel(BpExactArgs a) {
    __shared__ BpExactView<Off> views[8][32];
    const unsigned lane = threadIdx.x;
    const unsigned ii = blockIdx.x * 32 + lane;
    const unsigned jj = blockIdx.y * 8 + threadIdx.y;
    const unsigned kk = blockIdx.z;
    const bool valid = ii < (unsigned)a.nzz && jj < (unsigned)a.nys;
    const float4 ijkw = make_float4((float)(kk + a.x0), (float)(jj + a.y0), (float)(ii + a.z0), 1.f);
    const size_t frame = (size_t)a.width * a.height * sizeof(float);
    const Off stride = (Off)a.width * 4;
    const int nu = TRANSPOSE ? a.height : a.width, nv = TRANSPOSE ? a.width : a.height;
    const float last = (float)(nv - 1);
    BpExactView<Off> *mine = views[threadIdx.y];

    f32x2 sums = 0;  // the voxel's and its mirror's
    const char *view = reinterpret_cast<const char *>(a.proj);
    for (int base = 0; base < a.n_proj; base += 32) {
        const int nb = min(32, a.n_proj - base);
        if ((int)lane < nb) {
            const float4 *m = reinterpret_cast<const float4 *>(a.mats) + (size_t)(base + lane) * 3;
            const float4 m0 = __ldg(m), m1 = __ldg(m + 1), m2 = __ldg(m + 2);
            const float Z = 1.f / dot_ijkw(m2, ijkw);
            const float u = dot_ijkw(m0, ijkw) * Z;
            BpExactView<Off> r;
            r.f2 = pack2f(Z * Z, Z * Z);
            if (u >= 0 && u < nu - 1) {
                float d;
                const unsigned i = cell<Off>(u, d);
                r.off = TRANSPOSE ? i * stride : i * (Off)4;
                r.d = pack2f(d, d);
                r.d1 = pack2f(1.0f - d, 1.0f - d);
                r.f = Z;
                r.v0 = fma_rz(m1.y, ijkw.y, fma_rz(m1.x, ijkw.x, m1.w));
                r.vz = m1.z;
            } else {  // the view adds zeros: v = -1 and its mirror last + 1 are outside too
                r.off = 0;
                r.d = r.d1 = 0;
                r.vz = 0.f;
                r.f = 1.f;
                r.v0 = -1.f;
            }
            mine[lane] = r;
        }
        __syncwarp();
#pragma unroll 1
        for (int s = 0; s < nb; s++, view += frame) {
            const BpExactView<Off> r = mine[s];
            const float v = fma_rz(r.vz, ijkw.z, r.v0) * r.f;
            const float mirror = last - v, f2 = low2f(r.f2);
            if (SYM && sizeof(Off) == 4 && v >= 0.f && v < last && mirror >= 0.f && mirror < last) {
                sums = fma2f_rz_ftz(subpixel_pair<TRANSPOSE>(view, r, stride, pack2f(v, mirror)), r.f2, sums);
            } else {
                float sum, _sum;
                unpack2f(sums, sum, _sum);
                sum = fma_rz(subpixel_exact<TRANSPOSE>(view, r, stride, v, last), f2, sum);
                if (SYM) _sum = fma_rz(subpixel_exact<TRANSPOSE>(view, r, stride, mirror, last), f2, _sum);
                sums = pack2f(sum, _sum);
            }
        }
        __syncwarp();
        // The reference launches at most 32 views; a longer batch is a sequence of 32-view launches, each
        // adding its own partial sum to the volume.
        if (valid) {
            float sum, _sum;
            unpack2f(sums, sum, _sum);
            float *out = a.vol + ((long long)kk * a.nys + jj) * a.D;
            out[ii] += sum;
            if (SYM) out[a.D - 1 - ii] += _sum;
        }
        sums = 0;
    }
}

}  // namespace fdk
