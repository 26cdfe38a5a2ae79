// fproj.cu -- ray-marching forward projector (the reference's genProj kernel_forwardProject,
// genProj/cudaForwardProjection.cu:174-254, with Text3DLinear, genProj/cudaIterType.cuh:232-276).
//
// One thread per detector pixel.  The ray runs from the source to the pixel centre; it is
// clipped to the box spanned by the voxel centres (cuIntersectBox, :28-48), then sampled every
// tStep = min(dx, dy, dz) mm from the entry point (t < t_far), each sample trilinear on the voxel
// grid with texel indices truncated toward zero and clamped to the volume (the reference's
// point-sampled, clamp-addressed 3-D texture read at integer coordinates); the pixel value is
// sum * tStep.  Geometry: for BP view angle a the projector rotates by -a (:426), i.e. the source
// sits at R(a)^T (0, -SOD, 0) and the detector plane at distance SID, consistent with
// CalculateProjMat.  The volume is [z][y][x], x fastest, in the world frame
// X = (x-(nx-1)/2) dx, Y = -(y-(ny-1)/2) dy, Z = -(z-(nz-1)/2) dz.
#include <algorithm>

#include "common.h"
#include "internal.h"
#include "scratch.h"

namespace fdk {

constexpr double kPi = 3.14159265358979323846;

struct FprojArgs {
    const float *vol;
    float *out;
    long long first, n_proj;  // view index of blockIdx.y = 0; views of the scan
    double direction, scan_angle, position_angle;
    int nx, ny, nz, nu, nv;
    int rows;  // ZFAST: detector rows of a block
    float dx, dy, dz, du, dv, sid, sod, off_u, off_v;
};

__device__ __forceinline__ float vox(const FprojArgs &a, int x, int y, int z) {
    x = min(max(x, 0), a.nx - 1);
    y = min(max(y, 0), a.ny - 1);
    z = min(max(z, 0), a.nz - 1);
    return __ldg(a.vol + ((long long)z * a.ny + y) * a.nx + x);
}

// [z][y][x] -> [y][x][z] with one more slice along every axis, a copy of the last (so that the
// upper texel of a clamped sample needs no clamp of its own).  32 x 32 (z, x) tiles; grid (x, z, y).
__global__ void __launch_bounds__(256) fproj_volume_kernel(const float *__restrict__ src, float *__restrict__ dst, int nx,
                                                         int ny, int nz) {
    __shared__ float tile[32][33];
    const int x0 = blockIdx.x * 32, z0 = blockIdx.y * 32, lane = threadIdx.x & 31;
    for (int y = blockIdx.z; y <= ny; y += gridDim.z) {
        for (int r = threadIdx.x >> 5; r < 32; r += 8) {
            const int z = min(z0 + r, nz - 1), x = min(x0 + lane, nx - 1);
            tile[r][lane] = __ldg(src + ((long long)z * ny + min(y, ny - 1)) * nx + x);
        }
        __syncthreads();
        for (int r = threadIdx.x >> 5; r < 32; r += 8)
            if (x0 + r <= nx && z0 + lane <= nz)
                dst[((long long)y * (nx + 1) + x0 + r) * (nz + 1) + z0 + lane] = tile[lane][r];
        __syncthreads();
    }
}

// ZFAST: a.vol is fproj_volume_kernel's copy.  A warp takes up to 32 rows of one detector column:
// the orbit turns about z, so at every view angle its rays climb through neighbouring z of nearly the
// same (x, y), and each of a sample's loads is one or two 128-byte lines.  Lanes along a detector row
// in the [z][y][x] volume fall into one line or into 32 as the view turns, and the L1 data pipe was
// busy 96% of the time: 18.8 to 27.7 ms for 90 views of 256^2 through 256^3, 2.9 ms so, at 85% of the
// issue slots (unrolled 2 or 4 times the same).
template <bool ZFAST, bool WIDE>
__global__ void __launch_bounds__(256) fproj_kernel(FprojArgs a) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    int i, j;  // detector column, row
    if (ZFAST) {
        i = q / a.rows;
        j = blockIdx.z * a.rows + q % a.rows;
    } else {
        j = q / a.nu;
        i = q - j * a.nu;
    }
    if (i >= a.nu || j >= a.nv) return;
    const long long view = blockIdx.y;
    // the view's angle as fdk_view_angles has it, without a table to allocate and copy
    const double deg = __ddiv_rn(__dmul_rn((double)(a.first + view), a.scan_angle), (double)a.n_proj);
    const double ang = -__dadd_rn(__dmul_rn(__ddiv_rn(__dmul_rn(a.direction, deg), 180.0), kPi), a.position_angle);
    const float c = (float)cos(ang), s = (float)sin(ang);
    // source and detector pixel in mm, rotated (cuRotate: x' = x c - y s, y' = x s + y c)
    const float src_y = -a.sod, det_y = a.sid - a.sod;
    const float ox = -src_y * s, oy = src_y * c, oz = 0.f;
    const float cu = (a.nu - 1) / 2.0f + a.off_u, cv = (a.nv - 1) / 2.0f + a.off_v;
    const float umm = ((float)i - cu) * a.du, vmm = (cv - (float)j) * a.dv;
    const float px = umm * c - det_y * s, py = umm * s + det_y * c, pz = vmm;
    float dxr = px - ox, dyr = py - oy, dzr = pz - oz;
    const float inv = rsqrtf(dxr * dxr + dyr * dyr + dzr * dzr);
    dxr *= inv;
    dyr *= inv;
    dzr *= inv;
    // voxel-centre box in mm
    const float bx = (a.nx - 1) / 2.0f * a.dx, by = (a.ny - 1) / 2.0f * a.dy, bz = (a.nz - 1) / 2.0f * a.dz;
    const float ix = 1.0f / dxr, iy = 1.0f / dyr, iz = 1.0f / dzr;
    const float tx0 = (-bx - ox) * ix, tx1 = (bx - ox) * ix;
    const float ty0 = (-by - oy) * iy, ty1 = (by - oy) * iy;
    const float tz0 = (-bz - oz) * iz, tz1 = (bz - oz) * iz;
    const float tnear = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fminf(tz0, tz1));
    const float tfar = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fmaxf(tz0, tz1));
    const float step = fminf(fminf(a.dx, a.dy), a.dz);
    float sum = 0.f;
    if (tfar > tnear) {
        // index-space origin and direction: i = X/dx + cx, j = cy - Y/dy, k = cz - Z/dz
        const float cxv = (a.nx - 1) / 2.0f, cyv = (a.ny - 1) / 2.0f, czv = (a.nz - 1) / 2.0f;
        const float si = ox / a.dx + cxv, sj = cyv - oy / a.dy, sk = czv - oz / a.dz;
        const float vi = dxr / a.dx, vj = -dyr / a.dy, vk = -dzr / a.dz;
        // ZFAST: the last voxel of each axis, and what the 2^23 terms add to a byte offset (mod 2^32)
        const float ux = (float)(a.nx - 1), uy = (float)(a.ny - 1), uz = (float)(a.nz - 1);
        const unsigned bias = 4u * ((0x4B000000u * (a.nx + 1) + 0x4B000000u) * (a.nz + 1) + 0x4B000000u);
        for (float t = tnear; t < tfar; t += step) {
            const float pi = si + vi * t, pj = sj + vj * t, pk = sk + vk * t;
            float fi, fj, fk, c00, c10, c01, c11;
            if constexpr (ZFAST) {
                // Truncation without the conversion pipe: p + 2^23 rounded toward zero holds the whole
                // part of a p >= 0 in its low bits.  Positions a rounding outside the box are clamped
                // for the index and, as above, not for the fraction.
                const float ri = __fadd_rz(fminf(fmaxf(pi, 0.f), ux), 8388608.f);
                const float rj = __fadd_rz(fminf(fmaxf(pj, 0.f), uy), 8388608.f);
                const float rk = __fadd_rz(fminf(fmaxf(pk, 0.f), uz), 8388608.f);
                fi = pi - (ri - 8388608.f);
                fj = pj - (rj - 8388608.f);
                fk = pk - (rk - 8388608.f);
                const unsigned x = __float_as_uint(ri), y = __float_as_uint(rj), z = __float_as_uint(rk);
                const float *p00, *p10, *p01, *p11;
                if constexpr (WIDE) {
                    p00 = a.vol + ((y - 0x4B000000u) * (long long)(a.nx + 1) + (x - 0x4B000000u)) * (a.nz + 1) + (z - 0x4B000000u);
                    p01 = p00 + (long long)(a.nx + 1) * (a.nz + 1);
                    p10 = p00 + a.nz + 1;
                    p11 = p01 + a.nz + 1;
                } else {  // byte offsets below 2^32, the bits of the 2^23 terms taken off at once
                    const unsigned sx = 4u * (a.nz + 1), o = (y * (a.nx + 1) + x) * sx + 4u * z - bias;
                    const unsigned o1 = o + sx * (a.nx + 1);
                    const char *v = reinterpret_cast<const char *>(a.vol);
                    p00 = reinterpret_cast<const float *>(v + o);
                    p01 = reinterpret_cast<const float *>(v + o1);
                    p10 = reinterpret_cast<const float *>(v + (o + sx));
                    p11 = reinterpret_cast<const float *>(v + (o1 + sx));
                }
                c00 = __ldg(p00) * (1 - fk) + __ldg(p00 + 1) * fk;
                c10 = __ldg(p10) * (1 - fk) + __ldg(p10 + 1) * fk;
                c01 = __ldg(p01) * (1 - fk) + __ldg(p01 + 1) * fk;
                c11 = __ldg(p11) * (1 - fk) + __ldg(p11 + 1) * fk;
            } else {
                const int ai = (int)pi, aj = (int)pj, ak = (int)pk;  // truncation, as int3(pos)
                fi = pi - ai;
                fj = pj - aj;
                fk = pk - ak;
                c00 = vox(a, ai, aj, ak) * (1 - fk) + vox(a, ai, aj, ak + 1) * fk;
                c10 = vox(a, ai + 1, aj, ak) * (1 - fk) + vox(a, ai + 1, aj, ak + 1) * fk;
                c01 = vox(a, ai, aj + 1, ak) * (1 - fk) + vox(a, ai, aj + 1, ak + 1) * fk;
                c11 = vox(a, ai + 1, aj + 1, ak) * (1 - fk) + vox(a, ai + 1, aj + 1, ak + 1) * fk;
            }
            const float f0 = c00 * (1 - fj) + c01 * fj, f1 = c10 * (1 - fj) + c11 * fj;
            sum += f0 * (1 - fi) + f1 * fi;
        }
    }
    a.out[(view * a.nv + j) * (long long)a.nu + i] = sum * step;
}

}  // namespace fdk

using namespace fdk;

extern "C" int fdk_forward_project(const fdk_geometry *g, const float *dev_vol, int64_t first, int64_t n,
                                   float *dev_out, void *stream) {
    FDK_ABI_BEGIN
    clear_error();
    FDK_CHECK_ARG(g && dev_vol && dev_out, "NULL argument");
    FDK_CHECK_ARG(first >= 0 && n > 0 && first + n <= g->n_proj && n <= 65535, "view range out of bounds");
    FDK_CHECK_ARG(g->nu * g->nv < (1ll << 31), "detector too large");
    FDK_TRY(check_geometry(g));
    cudaStream_t st = (cudaStream_t)stream;
    FprojArgs a;
    a.vol = dev_vol;
    a.out = dev_out;
    a.first = first;
    a.n_proj = g->n_proj;
    a.direction = (double)g->direction;
    a.scan_angle = g->scan_angle;
    a.position_angle = g->volume_position_angle;
    a.nx = (int)g->nx;
    a.ny = (int)g->ny;
    a.nz = (int)g->nz;
    a.nu = (int)g->nu;
    a.nv = (int)g->nv;
    a.dx = (float)g->dx;
    a.dy = (float)g->dy;
    a.dz = (float)g->dz;
    a.du = (float)g->du;
    a.dv = (float)g->dv;
    a.sid = (float)g->sid;
    a.sod = (float)g->sod;
    a.off_u = (float)g->offset_nu;
    a.off_v = (float)g->offset_nv;
    // The reordered copy costs two passes over the volume (80 us at 256^3, as much as it saves one view
    // of 256^2), and mapping its memory where the pool does not keep that much (2 views through 500^3:
    // 3.4 ms with it, 0.45 without); 90 views through 256^3 take 2.9 ms with it and 19 without.  What it
    // saves grows with the rays and their length, so the line is a number of rays per column of the
    // volume.  Without memory for it the rays read the volume as it is.
    Scratch copy;
    const long long rays = n * g->nu * g->nv, cells = (g->nx + 1) * (g->ny + 1) * (g->nz + 1);
    const bool small = g->nx < (1 << 20) && g->ny < (1 << 20) && g->nz < (1 << 20) && g->nv <= 32 * 65535ll;
    const long long worth = (sizeof(float) * cells <= kScratchKeep ? 2 : 8) * g->nx * g->ny;
    if (small && rays >= worth && copy.alloc(sizeof(float) * cells, st) != FDK_OK) {
        cudaGetLastError();
        clear_error();
    }
    if (copy.p) {
        const dim3 tiles((unsigned)ceil_div(g->nx + 1, 32), (unsigned)ceil_div(g->nz + 1, 32),
                         (unsigned)std::min<int64_t>(g->ny + 1, 65535));
        fproj_volume_kernel<<<tiles, 256, 0, st>>>(dev_vol, static_cast<float *>(copy.p), a.nx, a.ny, a.nz);
        FDK_CUDA(cudaGetLastError());
        a.vol = static_cast<const float *>(copy.p);
        const unsigned parts = (unsigned)ceil_div(g->nv, 32);
        a.rows = (int)ceil_div(g->nv, parts);
        const dim3 grid((unsigned)ceil_div(g->nu * a.rows, 256), (unsigned)n, parts);
        if (cells < (1ll << 30)) fproj_kernel<true, false><<<grid, 256, 0, st>>>(a);
        else fproj_kernel<true, true><<<grid, 256, 0, st>>>(a);
    } else {
        fproj_kernel<false, false><<<dim3((unsigned)ceil_div(g->nu * g->nv, 256), (unsigned)n), 256, 0, st>>>(a);
    }
    FDK_CUDA(cudaGetLastError());
    FDK_TRY(copy.free());
    FDK_CUDA(cudaStreamSynchronize(st));
    return FDK_OK;
    FDK_ABI_END
}
