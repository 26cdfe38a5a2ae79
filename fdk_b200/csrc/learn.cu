// learn.cu -- the learned residual row filter and what training it needs (no reference
// counterpart): a small 1D residual network (3 conv layers, 32 channels, kernel 9) refines each
// ramp-filtered row; it is trained on phantoms that this library's own ray-marching forward
// projector generates, with the loss backpropagated through the exact adjoint of BP.
//
// Network, per detector row x (length L = nu), s = the row scale (1 / (SOD^2 AAF): line-integral
// units):
//   a1 = relu(W1 * (s x) + b1)      1 -> 32 channels, kernel 9, zero 'same' padding
//   a2 = relu(W2 * a1 + b2)         32 -> 32
//   o  = W3 * a2 + b3               32 -> 1
//   y  = x + o / s                  residual: zero W3, b3 give plain FDK
// Parameters FP32 (layout W1[32][9], b1[32], W2[32][32][9], b2[32], W3[32][9], b3); activations
// are kept in shared memory as BF16 (forward) and recomputed in the backward pass, so no
// activation tensor touches HBM.  The network's kernels are in nn_tc.cuh.
//
// Training kernels: exact adjoint of the staged backprojection (scatter with the gather's
// bilinear weights and bounds, accumulated per view in a shared-memory box), the volume MSE
// and its gradient, Adam, Poisson transmission noise, an ellipsoid voxelizer, and the
// ROWS -> MIRROR layout change that feeds the backprojection.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <vector>

#include "common.h"
#include "internal.h"
#include "nn_tc.cuh"

namespace fdk {

// --------------------------------------------------------------------------------------------
// Adam (Kingma & Ba), bias-corrected
// --------------------------------------------------------------------------------------------
__global__ void adam_kernel(float *w, const float *g, float *m, float *v, int n, float lr, float b1, float b2, float eps,
                            float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// --------------------------------------------------------------------------------------------
// transmission noise: p -> -log(max(Poisson(I0 exp(-mu p)), 1) / I0) / mu
// --------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    // splitmix64 finaliser
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ double uniform01(unsigned long long &state) {
    state = mix64(state);
    return ((state >> 11) + 0.5) * (1.0 / 9007199254740992.0);
}
// Poisson sample: inversion by sequential search for lambda < 64, otherwise the normal
// approximation with continuity correction (relative error of the variance < 1% there).
__device__ double poisson(double lam, unsigned long long &st) {
    if (lam <= 0.0) return 0.0;
    if (lam < 64.0) {
        const double L = exp(-lam);
        double p = 1.0;
        int k = 0;
        do {
            k++;
            p *= uniform01(st);
        } while (p > L && k < 1000);
        return (double)(k - 1);
    }
    const double u1 = uniform01(st), u2 = uniform01(st);
    const double n = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
    return fmax(0.0, floor(lam + sqrt(lam) * n + 0.5));
}

__global__ void noise_kernel(float *p, long long n, double i0, double mu, unsigned long long seed) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        unsigned long long st = mix64(seed ^ mix64((unsigned long long)i));
        const double lam = i0 * exp(-mu * (double)p[i]);
        const double cnt = fmax(poisson(lam, st), 1.0);
        p[i] = (float)(-log(cnt / i0) / mu);
    }
}

// --------------------------------------------------------------------------------------------
// ellipsoid voxelizer (value at voxel centres), [z][y][x]
// --------------------------------------------------------------------------------------------
struct __align__(16) EllipsoidForm {
    float a[3][3];   // d(l_r / a_r) / dP
    float b[3];      // l_r / a_r at P = 0
    float in, out;   // q below: inside, q above: outside
    float pad[2];
};
struct EllipsoidSet {  // passed by value: no device allocation or copy per call
    EllipsoidForm f[64];
    double e[64 * 16];
};

// A voxel belongs to an ellipsoid when q = sum (l_r / a_r)^2 <= 1 in FP64 (in_ellipsoid).  Nearly every
// voxel is farther from q = 1 than FP32 arithmetic can be wrong, so q is formed in FP32 first and in FP64
// only between the ellipsoid's two limits.  l_r / a_r is an affine form of the voxel's position; with M the
// largest sum of its terms' magnitudes over the volume, FP32 is off by less than 100 2^-24 (1 + M)
// (roundings of the coefficients, position and sums, 8 of M each, times dq = 2 (l/a) d(l/a) over three
// axes).  Four rows of voxels per thread share an ellipsoid's loads: 30 ellipsoids on 256^3 took 2.03 ms
// with three FP64 divisions for each voxel and ellipsoid, 0.32 ms so.
__device__ __forceinline__ bool in_ellipsoid(const double *e, double px, double py, double pz) {
    double q = 0;
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const double l = e[6 + r] * (px - e[0]) + e[9 + r] * (py - e[1]) + e[12 + r] * (pz - e[2]);
        q += l * l / (e[3 + r] * e[3 + r]);
    }
    return q <= 1.0;
}

constexpr int kVoxRows = 4;
// Grid: x and y tiles of 32 x 32 voxels (first_ty: of blockIdx.y = 0), slices.
__global__ void __launch_bounds__(256) voxelize_kernel(const __grid_constant__ EllipsoidSet ell, int n_ell, int nx, int ny, int nz,
                                                     double dx, double dy, double dz, int first_ty, float *out) {
    __shared__ double se[64 * 16];
    __shared__ EllipsoidForm form[64];
    const int t = threadIdx.y * 32 + threadIdx.x;
    for (int i = t; i < n_ell * 16; i += 256) {
        se[i] = ell.e[i];
        reinterpret_cast<float *>(form)[i] = reinterpret_cast<const float *>(ell.f)[i];
    }
    __syncthreads();
    const int x = blockIdx.x * 32 + threadIdx.x, y0 = ((first_ty + blockIdx.y) * 8 + threadIdx.y) * kVoxRows;
    if (x >= nx) return;
    const double px = (x - (nx - 1) / 2.0) * dx;
    const float fx = (float)px;
    float fy[kVoxRows];
#pragma unroll
    for (int j = 0; j < kVoxRows; j++) fy[j] = (float)(-(y0 + j - (ny - 1) / 2.0) * dy);
    for (int z = blockIdx.z; z < nz; z += gridDim.z) {
        const double pz = -(z - (nz - 1) / 2.0) * dz;
        const float fz = (float)pz;
        double v[kVoxRows];
#pragma unroll
        for (int j = 0; j < kVoxRows; j++) v[j] = 0;
        for (int k = 0; k < n_ell; k++) {
            const EllipsoidForm &f = form[k];
            float l[3];
#pragma unroll
            for (int r = 0; r < 3; r++) l[r] = fmaf(f.a[r][0], fx, fmaf(f.a[r][2], fz, f.b[r]));
#pragma unroll
            for (int j = 0; j < kVoxRows; j++) {
                const float l0 = fmaf(f.a[0][1], fy[j], l[0]), l1 = fmaf(f.a[1][1], fy[j], l[1]), l2 = fmaf(f.a[2][1], fy[j], l[2]);
                const float q = fmaf(l0, l0, fmaf(l1, l1, l2 * l2));
                if (q > f.out) continue;
                const double *e = se + 16 * k;
                if (q < f.in || in_ellipsoid(e, px, -(y0 + j - (ny - 1) / 2.0) * dy, pz)) v[j] += e[15];
            }
        }
#pragma unroll
        for (int j = 0; j < kVoxRows; j++)
            if (y0 + j < ny) out[((long long)z * ny + y0 + j) * nx + x] = (float)v[j];
    }
}

// --------------------------------------------------------------------------------------------
// ROWS (views x nv rows x nu) -> MIRROR pairs (views x nu x nv, element (u, v) = (P[v][u], P[nv-1-v][u]))
// --------------------------------------------------------------------------------------------
__global__ void rows_to_mirror_kernel(const float *__restrict__ src, float2 *__restrict__ dst, int nu, int nv) {
    __shared__ float tile[32][33];
    __shared__ float tilem[32][33];
    const long long f = blockIdx.z;
    const float *s = src + f * (long long)nu * nv;
    float2 *d = dst + f * (long long)nu * nv;
    const int u0 = blockIdx.x * 32, v0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int v = v0 + r, u = u0 + threadIdx.x;
        if (u < nu && v < nv) {
            tile[r][threadIdx.x] = s[(long long)v * nu + u];
            tilem[r][threadIdx.x] = s[(long long)(nv - 1 - v) * nu + u];
        }
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int u = u0 + r, v = v0 + threadIdx.x;
        if (u < nu && v < nv) d[(long long)u * nv + v] = make_float2(tile[threadIdx.x][r], tilem[threadIdx.x][r]);
    }
}

// --------------------------------------------------------------------------------------------
// volume MSE: vol in the backprojection's [x][y][z] layout, truth [z][y][x];
// res[z][y][x] = 2 (vol - truth) / N, sum of squared errors in *sse
// --------------------------------------------------------------------------------------------
__device__ double g_sse[2];  // fdk_volume_mse's accumulator; the network kernels' error word, for the same copy

__global__ void mse_kernel(const float *__restrict__ vol, const float *__restrict__ truth, float *res, int nx, int ny,
                           int nz, double *sse) {
    const long long total = (long long)nx * ny * nz;
    double acc = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % nx);
        const int y = (int)((i / nx) % ny);
        const int z = (int)(i / ((long long)nx * ny));
        const float d = vol[((long long)x * ny + y) * nz + z] - truth[i];
        if (res) res[i] = 2.0f * d / (float)total;
        acc += (double)d * d;
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(sse, acc);
    if (blockIdx.x == 0 && threadIdx.x == 0) sse[1] = (double)atomicExch(&nn::g_nn_err, 0u);
}

// --------------------------------------------------------------------------------------------
// exact adjoint of the staged backprojection (FDK_BP_FP32 semantics): for every voxel pair
// (z, nz-1-z) and view, the residual is scattered with the gather's weights -- bilinear, the
// 1/w^2 factor, SUBPIXEL's bounds -- into the view's ROWS-layout gradient.  One CTA: 16 x 16
// columns x 8 top slices and their mirrors; per view, two shared-memory boxes (main rows and
// mirror rows) collect the contributions before they are added to global memory.
//
// Contention: a warp covers 16 x 2 columns.  Per view the 16-wide side is laid along the
// volume axis whose neighbours land on different detector columns (the larger |dU|), so the
// lanes of one shared-memory atomic rarely hit the same address; both thread -> column
// mappings keep their residuals in registers.  The boxes are double-buffered and zeroed by the
// flush that reads them, so each view costs one barrier.
//
// The sums are issue-bound (81% of the slots).  256^3 from 90 views of 256^2: 3.04 ms with four atomics a
// voxel and view and every warp working out each view's footprint; 2.64 with two (a column's row sums
// stay in registers), 2.36 with the footprints of 8 views shared out among the warps, 2.29 with the residuals
// taken as they are (what is not finite goes past the boxes).  Four CTAs per SM (64
// registers) instead of three are slower (2.07 against 1.99 ms on another residual).
//
// Shared-memory float atomics run as load + compare-and-swap loops, so the boxes hold 32-bit
// fixed point and take native integer atomics: per view every contribution w g is scaled by a
// power of two S with |w g| S <= 2^19 for all voxels of the tile (the tile's largest |residual|
// times the largest 1/w^2, found at its corners).  An entry sums at most one term per voxel, so
// it stays below 2048 * 2^19 = 2^30; a column's sum on a row (at most 8 terms, below 2^22) is rounded to
// the nearest 1/S.  The box is laid
// out u-fastest, so the lanes of one atomic (consecutive detector columns) hit consecutive banks.
// --------------------------------------------------------------------------------------------
// Nearest integer of |x| < 2^22: x + 1.5 2^23 has it in its low bits (conversions run at a quarter of the
// FP32 rate).
__device__ __forceinline__ int fixed(float x) { return __float_as_int(__fadd_rn(x, 12582912.f)) - 0x4B400000; }

constexpr int kAdjR = 8, kAdjBU = 48, kAdjBV = 24;  // box: u extent (fastest) x v extent

struct AdjArgs {
    const float *res;   // [z][y][x]
    float *grad;        // views x nv x nu (ROWS)
    const float *mats;  // 12 per view
    int n, nx, ny, nz, nu, nv;
};

struct AdjView {  // a view's footprint of the tile
    int u_lo, v_lo, rows, cols, boxed, swap;
    float scale, inv_scale;
};

// LONG: more than 2^22 detector rows.
template <bool LONG>
__global__ void __launch_bounds__(256, 3) bp_adjoint_kernel(AdjArgs a) {
    __shared__ int box[2][2][kAdjBV * kAdjBU];  // [buffer][main, mirror], fixed point
    __shared__ float warp_max[8];
    __shared__ AdjView views[2][8];
    const int tid = threadIdx.x, lx = tid & 15, ly = tid >> 4;
    const int zt = blockIdx.z * kAdjR, nzz = a.nz / 2;
    // residuals of column (x0 + lx, y0 + ly) [mapping 0] and (x0 + ly, y0 + lx) [mapping 1]
    float rm[2][kAdjR], rr[2][kAdjR];
    bool col_ok[2], lost = false;
#pragma unroll
    for (int mp = 0; mp < 2; mp++) {
        const int xi = blockIdx.x * 16 + (mp ? ly : lx), yi = blockIdx.y * 16 + (mp ? lx : ly);
        col_ok[mp] = xi < a.nx && yi < a.ny;
#pragma unroll
        for (int k = 0; k < kAdjR; k++) {
            const int z = zt + k;
            const bool ok = col_ok[mp] && z < nzz;
            const float g = ok ? a.res[((long long)z * a.ny + yi) * a.nx + xi] : 0.f;
            const float gr = ok ? a.res[((long long)(a.nz - 1 - z) * a.ny + yi) * a.nx + xi] : 0.f;
            rm[mp][k] = g;
            rr[mp][k] = gr;
            lost |= !(g == g) || !(gr == gr);
        }
    }
    // largest |residual| of the tile: the fixed-point range
    float gmax = 0.f;
#pragma unroll
    for (int k = 0; k < kAdjR; k++) gmax = fmaxf(gmax, fmaxf(fabsf(rm[0][k]), fabsf(rr[0][k])));
#pragma unroll
    for (int o = 16; o; o >>= 1) gmax = fmaxf(gmax, __shfl_xor_sync(0xFFFFFFFFu, gmax, o));
    if ((tid & 31) == 0) warp_max[tid >> 5] = gmax;
    for (int i = tid; i < 2 * 2 * kAdjBV * kAdjBU; i += 256) (&box[0][0][0])[i] = 0;
    lost = __syncthreads_or(lost);
    gmax = warp_max[0];
#pragma unroll
    for (int i = 1; i < 8; i++) gmax = fmaxf(gmax, warp_max[i]);
    if (!(gmax > 0.f || lost)) return;  // the tile adds nothing (the whole CTA leaves together)
    // what is not finite has no fixed point: the tile's sums go to the pixels as they are
    const bool fixed_point = gmax <= FLT_MAX && !lost;
    const float zf0 = (float)zt;
    const int warp = tid >> 5;
    for (int s = 0; s < a.n; s++) {
        const float *m = a.mats + 12 * s;
        const int cur = s & 1;
        if ((s & 7) == 0) {
            // the next 8 views' footprints of the tile, one per warp: lanes 4j .. 4j+3 evaluate one corner each (as
            // the gather kernels)
            const int sv = min(s + warp, a.n - 1), corner = tid & 3;
            const float *m = a.mats + 12 * sv;
            const float cx = blockIdx.x * 16 + ((corner & 1) ? 15 : 0), cy = blockIdx.y * 16 + ((corner & 2) ? 15 : 0);
            const float rw = 1.f / fmaf(m[8], cx, fmaf(m[9], cy, m[11]));
            const float U = fmaf(m[0], cx, fmaf(m[1], cy, m[3])) * rw;
            const float vw = fmaf(m[4], cx, fmaf(m[5], cy, m[7]));
            const float va = fmaf(m[6], zf0, vw) * rw, vb = fmaf(m[6], zf0 + kAdjR - 1, vw) * rw;
            float umin = U, umax = U, vmin = fminf(va, vb), vmax = fmaxf(va, vb);
            float wtmax = rw * rw;  // 1/w is largest at a corner (w is linear in x, y)
            const int base = tid & 28;  // lane of this group's corner 0
            const float u0c = __shfl_sync(0xFFFFFFFFu, U, base);
            const float du_x = __shfl_sync(0xFFFFFFFFu, U, base | 1) - u0c;
            const float du_y = __shfl_sync(0xFFFFFFFFu, U, base | 2) - u0c;
#pragma unroll
            for (int o = 1; o <= 2; o <<= 1) {
                umin = fminf(umin, __shfl_xor_sync(0xFFFFFFFFu, umin, o));
                umax = fmaxf(umax, __shfl_xor_sync(0xFFFFFFFFu, umax, o));
                vmin = fminf(vmin, __shfl_xor_sync(0xFFFFFFFFu, vmin, o));
                vmax = fmaxf(vmax, __shfl_xor_sync(0xFFFFFFFFu, vmax, o));
                wtmax = fmaxf(wtmax, __shfl_xor_sync(0xFFFFFFFFu, wtmax, o));
            }
            int ex;
            frexpf(gmax * wtmax * 1.0001f, &ex);  // |w g| <= gmax * wtmax < 2^ex
            const int e = min(19 - ex, 126);
            AdjView v;
            v.u_lo = (int)floorf(umin) - 1;
            v.v_lo = (int)floorf(vmin) - 1;
            v.rows = (int)floorf(umax) + 3 - v.u_lo;  // u, v extents
            v.cols = (int)floorf(vmax) + 3 - v.v_lo;
            v.boxed = v.rows <= kAdjBU && v.cols <= kAdjBV && fixed_point;
            v.swap = fabsf(du_y) > fabsf(du_x) ? 1 : 0;  // 16 lanes along the axis with the larger |dU|
            v.scale = ldexpf(1.f, e);
            v.inv_scale = ldexpf(1.f, -e);
            if ((tid & 31) == 0) views[s >> 3 & 1][warp] = v;
            __syncthreads();
        }
        const AdjView vw = views[s >> 3 & 1][s & 7];
        const int u_lo = vw.u_lo, v_lo = vw.v_lo, mp = vw.swap;
        const bool boxed = vw.boxed;
        const float S = vw.scale;
        int *boxm = box[cur][0], *boxr = box[cur][1];
        float *gv = a.grad + (long long)s * a.nu * a.nv;
        if (mp ? col_ok[1] : col_ok[0]) {
            const float x = (float)(blockIdx.x * 16 + (mp ? ly : lx)), y = (float)(blockIdx.y * 16 + (mp ? lx : ly));
            const float rw = 1.f / fmaf(m[8], x, fmaf(m[9], y, m[11]));
            const float U = fmaf(m[0], x, fmaf(m[1], y, m[3])) * rw;
            const float A = fmaf(m[4], x, fmaf(m[5], y, fmaf(m[6], zf0, m[7]))) * rw;
            const float B = m[6] * rw;
            const float wt = rw * rw;
            if (U >= 0.f && U < (float)(a.nu - 1)) {
                const float fuf = floorf(U);
                const float fu = U - fuf;
                const int u0 = (int)fuf;
                // The column's detector column and weight are its own, and its slices are about one detector
                // row apart: the sums of (1 - fv) g and fv g on the rows vi and vi + 1 stay in registers,
                // and a row leaves when the next slice has moved on, weighted for the two columns.
                const float wa = (1 - fu) * wt, wb = fu * wt;
                int cur = -0x40000000;
                float m0 = 0.f, m1 = 0.f, r0 = 0.f, r1 = 0.f;  // main and mirror, rows cur and cur + 1
                const float sc = boxed ? S : 1.f;
                const int col = u0 - u_lo - v_lo * kAdjBU;
                auto leave = [&](int row, float m, float r) {
                    if (boxed) {
                        const int b = row * kAdjBU + col;
                        atomicAdd(&boxm[b], fixed(wa * m));
                        atomicAdd(&boxm[b + 1], fixed(wb * m));
                        atomicAdd(&boxr[b], fixed(wa * r));
                        atomicAdd(&boxr[b + 1], fixed(wb * r));
                    } else {  // the mirror voxel: the same weights on row nv - 1 - row
                        float *pm = gv + (long long)row * a.nu + u0, *pr = gv + (long long)(a.nv - 1 - row) * a.nu + u0;
                        if (m != 0.f) {
                            atomicAdd(pm, wa * m);
                            atomicAdd(pm + 1, wb * m);
                        }
                        if (r != 0.f) {
                            atomicAdd(pr, wa * r);
                            atomicAdd(pr + 1, wb * r);
                        }
                    }
                };
#pragma unroll
                for (int k = 0; k < kAdjR; k++) {
                    const float v = fmaf(B, (float)k, A);
                    const float vr = (float)(a.nv - 1) - v;
                    const bool mv = v >= 0.f && v < (float)(a.nv - 1);
                    const bool rv = vr >= 0.f && vr < (float)(a.nv - 1);
                    if (!(mv || rv)) continue;
                    // 0 <= v <= nv - 1 here: its whole part by an addition rounded toward zero
                    const float vf = fminf(LONG ? floorf(v) : __fadd_rz(v, 8388608.f) - 8388608.f, (float)(a.nv - 2));
                    const int vi = LONG ? (int)vf : __float_as_int(vf + 8388608.f) - 0x4B000000;
                    const float fv = v - vf;
                    if (vi != cur) {
                        const bool next = vi == cur + 1;
                        if (cur >= 0) {
                            leave(cur, m0, r0);
                            if (!next) leave(cur + 1, m1, r1);
                        }
                        m0 = next ? m1 : 0.f;
                        r0 = next ? r1 : 0.f;
                        m1 = r1 = 0.f;
                        cur = vi;
                    }
                    const float gm = mv ? (mp ? rm[1][k] : rm[0][k]) * sc : 0.f;  // selects, not a dynamic register index
                    const float gr = rv ? (mp ? rr[1][k] : rr[0][k]) * sc : 0.f;
                    m0 = fmaf(1 - fv, gm, m0);
                    m1 = fmaf(fv, gm, m1);
                    r0 = fmaf(1 - fv, gr, r0);
                    r1 = fmaf(fv, gr, r1);
                }
                if (cur >= 0) {
                    leave(cur, m0, r0);
                    leave(cur + 1, m1, r1);
                }
            }
        }
        __syncthreads();
        if (boxed) {
            // flush: entry (c, ru) = (v - v_lo, u - u_lo) holds row v (main) / row nv-1-v (mirror),
            // column u; each entry is zeroed as it is read, ready for view s + 2.  A warp takes every eighth row.
            for (int c = warp; c < vw.cols; c += 8)
                for (int ru = tid & 31; ru < vw.rows; ru += 32) {
                    const int bi = c * kAdjBU + ru;
                    const int qm = boxm[bi], qr = boxr[bi];
                    boxm[bi] = 0;
                    boxr[bi] = 0;
                    const int u = u_lo + ru, v = v_lo + c;
                    if (u < 0 || u >= a.nu || v < 0 || v >= a.nv) continue;
                    if (qm != 0) atomicAdd(&gv[(long long)v * a.nu + u], (float)qm * vw.inv_scale);
                    if (qr != 0) atomicAdd(&gv[(long long)(a.nv - 1 - v) * a.nu + u], (float)qr * vw.inv_scale);
                }
        }
    }
}

}  // namespace fdk

using namespace fdk;

// The status of the network kernels' error word.
static int network_status(unsigned word) {
    if (word) return fail(FDK_ERR_DEVICE_CHECK, "a network kernel's pipeline wait timed out on the device (error word %u)", word);
    return FDK_OK;
}

extern "C" {

int fdk_nn_param_count(void) { return kNParam; }

int fdk_nn_forward(const float *params, const float *x, float *y, int64_t rows, int32_t len, float scale, void *stream) {
    FDK_ABI_BEGIN
    clear_error();
    FDK_CHECK_ARG(params && x && y, "NULL argument");
    FDK_CHECK_ARG(len >= kK && len <= kMaxLen && rows > 0, "row length must be 9..%d", kMaxLen);
    FDK_CUDA(cudaFuncSetAttribute(nn::forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, nn::Fwd::BYTES));
    int sms = 0, dev = 0;
    FDK_CUDA(cudaGetDevice(&dev));
    FDK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int blocks = (int)std::min<long long>(ceil_div(rows, nn::rows_per_step(len)), 2 * sms);  // two resident CTAs per SM
    nn::forward_kernel<<<blocks, nn::THREADS, nn::Fwd::BYTES, (cudaStream_t)stream>>>(params, x, y, len, rows, scale,
                                                                                   bp_wait_ns(), bp_test_withhold());
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
    FDK_ABI_END
}

int fdk_nn_backward(const float *params, const float *x, const float *dy, float *dparams, int64_t rows, int32_t len,
                    float scale, void *stream) {
    FDK_ABI_BEGIN
    clear_error();
    FDK_CHECK_ARG(params && x && dy && dparams, "NULL argument");
    FDK_CHECK_ARG(len >= kK && len <= kMaxLen && rows > 0, "row length must be 9..%d", kMaxLen);
    FDK_CUDA(cudaFuncSetAttribute(nn::backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, nn::Bwd::BYTES));
    int sms = 0, dev = 0;
    FDK_CUDA(cudaGetDevice(&dev));
    FDK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int blocks = (int)std::min<long long>(ceil_div(rows, nn::rows_per_step(len)), sms);
    FDK_CUDA(cudaMemsetAsync(dparams, 0, sizeof(float) * kNParam, (cudaStream_t)stream));
    nn::backward_kernel<<<blocks, nn::Bwd::THREADS, nn::Bwd::BYTES, (cudaStream_t)stream>>>(
        params, x, dy, dparams, len, rows, scale, bp_wait_ns(), bp_test_withhold());
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
    FDK_ABI_END
}

int fdk_nn_check(void *stream) {
    FDK_ABI_BEGIN
    clear_error();
    unsigned *word = nullptr, got = 0;
    FDK_CUDA(cudaGetSymbolAddress((void **)&word, nn::g_nn_err));
    cudaStream_t st = (cudaStream_t)stream;
    FDK_CUDA(cudaMemcpyAsync(&got, word, sizeof(got), cudaMemcpyDeviceToHost, st));
    FDK_CUDA(cudaStreamSynchronize(st));
    if (got) FDK_CUDA(cudaMemsetAsync(word, 0, sizeof(got), st));
    return network_status(got);
    FDK_ABI_END
}

int fdk_adam_step(float *params, const float *grads, float *m, float *v, int64_t n, float lr, float beta1, float beta2,
                  float eps, int64_t t, void *stream) {
    FDK_ABI_BEGIN
    FDK_CHECK_ARG(params && grads && m && v && n > 0 && t > 0, "bad arguments");
    const float c1 = 1.f - powf(beta1, (float)t), c2 = 1.f - powf(beta2, (float)t);
    adam_kernel<<<(int)ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(params, grads, m, v, (int)n, lr, beta1, beta2,
                                                                         eps, c1, c2);
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
    FDK_ABI_END
}

int fdk_transmission_noise(float *dev_views, int64_t n, double i0, double mu, uint64_t seed, void *stream) {
    FDK_ABI_BEGIN
    FDK_CHECK_ARG(dev_views && n > 0 && i0 > 0 && mu > 0, "bad arguments");
    noise_kernel<<<148 * 8, 256, 0, (cudaStream_t)stream>>>(dev_views, n, i0, mu, seed);
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
    FDK_ABI_END
}

int fdk_voxelize(const fdk_geometry *g, const double *ell, int32_t n_ell, float *dev_vol, void *stream) {
    FDK_ABI_BEGIN
    FDK_CHECK_ARG(g && ell && dev_vol && n_ell >= 0 && n_ell <= 64, "bad arguments");
    if (g->nx <= 0 || g->ny <= 0 || g->nz <= 0) return FDK_OK;  // no voxels
    EllipsoidSet set;
    for (int i = 0; i < 16 * n_ell; i++) set.e[i] = ell[i];
    const double half[3] = {0.5 * (g->nx - 1) * g->dx, 0.5 * (g->ny - 1) * g->dy, 0.5 * (g->nz - 1) * g->dz};
    for (int k = 0; k < n_ell; k++) {
        const double *e = ell + 16 * k;
        EllipsoidForm &f = set.f[k];
        double most = 0;
        for (int r = 0; r < 3; r++) {
            double b = 0, m = 0;
            for (int i = 0; i < 3; i++) {
                const double c = e[6 + 3 * i + r] / e[3 + r];
                f.a[r][i] = (float)c;
                b -= c * e[i];
                m += std::fabs(c) * (half[i] + std::fabs(e[i]));
            }
            f.b[r] = (float)b;
            if (!(m <= most)) most = m;
        }
        // The limits hold to first order: up to M 2^-24 = 1/16.  Beyond (an axis of a millionth of the volume, or of
        // 0: not a number) no q is outside them, and FP64 decides.
        const float off = most < (1 << 20) ? (float)(100.0 / 16777216.0 * (1.0 + most)) : INFINITY;
        f.in = 1.f - off;
        f.out = 1.f + off;
    }
    const int64_t tiles_x = ceil_div(g->nx, 32), tiles_y = ceil_div(g->ny, 8 * kVoxRows);
    const unsigned slices = (unsigned)std::min<int64_t>(g->nz, std::max<int64_t>(1, 148 * 8 / (tiles_x * tiles_y)));
    for (int64_t ty = 0; ty < tiles_y; ty += 65535)  // (the grid's limit)
        voxelize_kernel<<<dim3((unsigned)tiles_x, (unsigned)std::min<int64_t>(tiles_y - ty, 65535), slices), dim3(32, 8), 0,
                          (cudaStream_t)stream>>>(set, n_ell, (int)g->nx, (int)g->ny, (int)g->nz, g->dx, g->dy, g->dz,
                                                  (int)ty, dev_vol);
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
    FDK_ABI_END
}

int fdk_rows_to_mirror(const float *dev_rows, void *dev_mirror, int64_t n_views, int32_t nu, int32_t nv, void *stream) {
    FDK_ABI_BEGIN
    FDK_CHECK_ARG(dev_rows && dev_mirror && n_views > 0 && n_views <= 65535 && nu > 0 && nv > 0, "bad arguments");
    const dim3 grid((unsigned)ceil_div(nu, 32), (unsigned)ceil_div(nv, 32), (unsigned)n_views);
    rows_to_mirror_kernel<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>(dev_rows, (float2 *)dev_mirror, nu, nv);
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
    FDK_ABI_END
}

int fdk_volume_mse(const float *dev_vol_xyz, const float *dev_truth, float *dev_res, int32_t nx, int32_t ny, int32_t nz,
                   double *sse_host, void *stream) {
    FDK_ABI_BEGIN
    FDK_CHECK_ARG(dev_vol_xyz && dev_truth && sse_host && nx > 0 && ny > 0 && nz > 0, "bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    // one accumulator per device (a module global), shared by the callers of that device in turn
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    double *d_sse = nullptr;
    FDK_CUDA(cudaGetSymbolAddress((void **)&d_sse, g_sse));
    FDK_CUDA(cudaMemsetAsync(d_sse, 0, 2 * sizeof(double), st));
    mse_kernel<<<148 * 8, 256, 0, st>>>(dev_vol_xyz, dev_truth, dev_res, nx, ny, nz, d_sse);
    FDK_CUDA(cudaGetLastError());
    double got[2] = {};
    FDK_CUDA(cudaMemcpyAsync(got, d_sse, sizeof(got), cudaMemcpyDeviceToHost, st));
    FDK_CUDA(cudaStreamSynchronize(st));
    *sse_host = got[0];
    return network_status((unsigned)got[1]);
    FDK_ABI_END
}

int fdk_bp_adjoint(const fdk_geometry *g, const float *dev_res, const float *dev_mats, int32_t n_views, float *dev_grad,
                   void *stream) {
    FDK_ABI_BEGIN
    FDK_CHECK_ARG(g && dev_res && dev_mats && dev_grad && n_views > 0, "NULL argument");
    FDK_CHECK_ARG(g->nz % 2 == 0, "the slab-pair adjoint needs an even nz");
    AdjArgs a;
    a.res = dev_res;
    a.grad = dev_grad;
    a.mats = dev_mats;
    a.n = n_views;
    a.nx = (int)g->nx;
    a.ny = (int)g->ny;
    a.nz = (int)g->nz;
    a.nu = (int)g->nu;
    a.nv = (int)g->nv;
    const dim3 grid((unsigned)ceil_div(a.nx, 16), (unsigned)ceil_div(a.ny, 16), (unsigned)ceil_div(a.nz / 2, kAdjR));
    if (a.nv > 1 << 22) bp_adjoint_kernel<true><<<grid, 256, 0, (cudaStream_t)stream>>>(a);
    else bp_adjoint_kernel<false><<<grid, 256, 0, (cudaStream_t)stream>>>(a);
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
    FDK_ABI_END
}

}  // extern "C"
