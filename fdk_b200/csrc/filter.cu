// filter.cu -- fused FDK row filter for sm_100a: cosine pre-weight, constant edge pad,
// ramp/window filter by FFT, crop, and the store in the layout the backprojection reads.
//
// Reference semantics: FilterEngine::Filtering (Filterlib/FilterLib.h:167-196) and the cuFFT
// plugin (FilterlibCufft/cudaFftFilter.cu:14-61, 283-392).  Two detector rows -- row r and its
// mirror row nv-1-r -- are the real and imaginary parts of one complex FFT of length W: with a
// real, even response H the two filtered rows come back as the real and imaginary parts of the
// inverse transform.  Pairing r with nv-1-r is what lets one CTA emit the backprojection's
// mirror-pair layout directly.
//
// FFT: radix-2 decimation in frequency (natural -> bit-reversed order), multiply by H, radix-2
// decimation in time back.  W / 16 threads hold the W points of a row pair in registers, 16 each, and
// run the stages four at a time: the 16 points that differ in four adjacent index bits form a closed
// group (W = 16 x 16 x W/256, 4096 = 16^3).  Calls of few rows take 4 or 8 points a thread instead (launch_filter).
// The samples go from global memory straight into the first pass's registers and from the last
// pass's registers out again, the spectrum is multiplied by H between the forward and the inverse
// half of the innermost pass, and so a row pair crosses shared memory four times in all.  Bound:
// shared-memory wavefronts and FP32 issue about equally (per 512 points and warp some 460
// wavefronts and 1200 FP32 instructions at W = 4096).  Plain butterflies cost an eighth more
// arithmetic than radix-16 ones with their constants folded (32 views of 2048^2 to MIRROR FP32:
// 997 against 973 us) and keep the roundings of a stage-by-stage transform (but for the roots 1 and -i, whose
// rounded tables may add 6e-17 of the other component).
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "common.h"
#include "internal.h"
#include "scratch.h"

namespace fdk {

struct FilterArgs {
    const float *src;   // views of nv rows x nu, row pitch src_pitch, view stride src_vstride
    void *dst;          // output, layout dependent
    const float *cos;   // nv x nu (pitch cos_pitch) or nullptr
    const float2 *tw;   // W/2 twiddles exp(-2 pi i k / W)
    const float2 *twp;  // the passes' twiddles (FilterTables::twp), or nullptr: gathered from tw
    const float *hb;    // W: H / W in the order of the transform's registers (FilterTables)
    int nu, nv, off, pad_n, n_pairs;
    int src_pitch, dst_pitch, cos_pitch;
    long long src_vstride, dst_vstride;
    int layout, half;         // FDK_LAYOUT_*, FP16 output
    int pair_stores;          // MIRROR: dst takes a pair as one store
    float out_scale;          // multiplies every output sample (FP16 range control)
    unsigned int *overflow;   // set to 1 when a scaled FP16 output exceeds the format (or NULL)
};

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a * w, or a * conj(w): one product of each sum rounded, the other fused, written out so that every
// place rounds alike
template <bool CONJ>
__device__ __forceinline__ float2 cmul(float2 a, float2 w) {
    if (CONJ) return make_float2(__fmaf_rn(a.x, w.x, __fmul_rn(a.y, w.y)), __fmaf_rn(a.y, w.x, -__fmul_rn(a.x, w.y)));
    return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.x, w.y, __fmul_rn(a.y, w.x)));
}

// A table load that stays where it is written.  The forward and the inverse half read the same
// twiddles; as plain read-only loads the compiler merges the two and keeps 32 to 64 registers alive
// from one half to the other, as spills to local memory (300 bytes a thread at W = 4096, which
// missed L1 and made two thirds of the kernel's L2 traffic: 1469 against 1139 us for 32 views of
// 2048^2 to MIRROR FP32, with radix-16 butterflies and 512-thread CTAs).
__device__ __forceinline__ float4 load_here(const float4 *p) {
    float4 f;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w) : "l"(p) : "memory");
    return f;
}

// Stages in registers.  A group of R points has R/2 twiddles in its first decimation-in-frequency
// stage, then R/4, and so on: entry j of the stage of half-width h serves the butterflies j mod h.  `w(h, j)`
// gives it; decimation in time runs the same stages backwards with the conjugates.
template <int R, int N, typename Tw>
__device__ __forceinline__ void dif(float2 (&v)[N], int b, Tw w) {
#pragma unroll
    for (int h = R / 2; h; h >>= 1)
#pragma unroll
        for (int j = 0; j < R; j++) {
            if (j & h) continue;
            const float2 x = v[b + j], y = v[b + j + h];
            v[b + j] = cadd(x, y);
            v[b + j + h] = w(std::false_type{}, csub(x, y), h, j & (h - 1));
        }
}
template <int R, int N, typename Tw>
__device__ __forceinline__ void dit(float2 (&v)[N], int b, Tw w) {
#pragma unroll
    for (int h = 1; h < R; h <<= 1)
#pragma unroll
        for (int j = 0; j < R; j++) {
            if (j & h) continue;
            const float2 x = v[b + j], u = w(std::true_type{}, v[b + j + h], h, j & (h - 1));
            v[b + j] = cadd(x, u);
            v[b + j + h] = csub(x, u);
        }
}
// The stages of the last bits (contiguous points): twiddles exp(-2 pi i j / 2h), constants.
struct Roots {
    template <typename Conj>
    __device__ __forceinline__ float2 operator()(Conj, float2 a, int h, int j) const {
        constexpr float c[8] = {1.f, 0.92387953251128674f, 0.70710678118654752f, 0.38268343236508977f,
                                0.f, -0.38268343236508977f, -0.70710678118654752f, -0.92387953251128674f};
        constexpr float s[8] = {0.f, -0.38268343236508977f, -0.70710678118654752f, -0.92387953251128674f,
                                -1.f, -0.92387953251128674f, -0.70710678118654752f, -0.38268343236508977f};
        const int k = j * (8 / h);
        if (k == 0) return a;
        if (k == 4) return Conj::value ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
        return cmul<Conj::value>(a, make_float2(c[k], s[k]));
    }
};

// Passes of a W-point transform by threads of E = 2^LOG2E points: E points over stride W / E, then over W / E^2
// and so on, then RL contiguous ones.
template <int LOG2W, int LOG2E>
struct Fft {
    static constexpr int W = 1 << LOG2W;
    static constexpr int E = LOG2W < LOG2E ? W : 1 << LOG2E;                // points per thread
    static constexpr int TPF = W / E;                                       // threads per transform
    static constexpr int PASSES = LOG2W > LOG2E ? (LOG2W - 1) / LOG2E : 0;  // strided passes
    static constexpr int RL = W >> (PASSES * LOG2E);                        // points of the last pass
    __host__ __device__ static constexpr int stride(int pass) { return W >> ((pass + 1) * LOG2E); }
    // shared-memory slots of one transform: one float2 of padding per 16, so that the contiguous
    // runs of the last pass and the strided ones of the others are (16 points a thread) all free
    // of bank conflicts
    static constexpr int PITCH = W + W / 16;
    // CTAs per SM that the register budget is set for: 1024 threads of 64 registers
    static constexpr int blocks(int g) { return 1024 / (TPF * g) < 16 ? 1024 / (TPF * g) : 16; }
};

// Slot of point p.  Where p = i + q with i < d, d and 16 of which one divides the other, and q a
// multiple of d, it is slot(i) + slot(q): the passes' slots are one address and constants.
__host__ __device__ constexpr int slot(int p) { return p + (p >> 4); }

enum class Twiddles {
    Planes,  // the passes' planes, each pass's loaded as it begins
    Roots,   // gathered from tw, each pass's as it begins
    // All asked for at the start and kept in registers, as are the response and the pads' samples: from the planes
    // with 16 points a thread (pairs by 16-byte loads), else gathered from tw.
    Early
};

// Row pairs (r, nv-1-r), r = G * blockIdx.x + g, g < G, of view blockIdx.y.
template <int LOG2W, int LOG2E, int G, Twiddles TW>
__global__ void __launch_bounds__(Fft<LOG2W, LOG2E>::TPF * G, TW == Twiddles::Early ? 1 : Fft<LOG2W, LOG2E>::blocks(G))
    filter_kernel(const FilterArgs a) {
    using F = Fft<LOG2W, LOG2E>;
    constexpr bool EARLY = TW == Twiddles::Early;
    constexpr int W = F::W, E = F::E, TPF = F::TPF, RL = F::RL, THREADS = TPF * G, PASSES = F::PASSES;
    extern __shared__ __align__(16) float2 fsm[];
    __shared__ float pads[G][4];
    const int g = threadIdx.x / TPF, t = threadIdx.x % TPF;
    const int r0 = blockIdx.x * G;
    const int r1 = min(r0 + g, a.n_pairs - 1), r2 = a.nv - 1 - r1;  // pairs past the last repeat it, unstored
    float2 *buf = fsm + g * F::PITCH;
    // the threads of one transform meet without the rest of the CTA
    auto meet = [&]() {
        if constexpr (TPF <= 32) __syncwarp();
        else if constexpr (G == 1) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(TPF) : "memory");
    };

    // samples t + m TPF of the padded rows
    const long long view = blockIdx.y;
    const float *p1 = a.src + view * a.src_vstride + (long long)r1 * a.src_pitch;
    const float *p2 = a.src + view * a.src_vstride + (long long)r2 * a.src_pitch;
    const float *w1 = a.cos ? a.cos + (long long)r1 * a.cos_pitch : nullptr;
    const float *w2 = a.cos ? a.cos + (long long)r2 * a.cos_pitch : nullptr;
    const int c0 = t - a.off;  // this thread's first column

    // The twiddles of a strided pass: E/2 of its first stage, E/4 of the next and so on, for the thread's place
    // i < n in a block (n: the pass's stride).  In the planes as float4 pairs, pair-major; in tw entry j of the
    // stage of half-width h is root (i + j n) E/2h of the pass's, which are every (TPF / n)-th.
    float2 early[EARLY && PASSES ? PASSES : 1][E], tq[E];
    auto fetch = [&](float2 (&q)[E], int pass) {
        const int n = F::stride(pass), i = t % n;
        if constexpr (TW == Twiddles::Roots || E < 16) {
#pragma unroll
            for (int h = E / 2; h; h >>= 1)
#pragma unroll
                for (int j = 0; j < h; j++) q[E - 2 * h + j] = __ldg(a.tw + (i + j * n) * (E / 2 / h) * (TPF / n));
        } else {
            const float4 *plane = reinterpret_cast<const float4 *>(a.twp + (pass ? W : 0)) + i;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const float4 f = load_here(plane + k * n);
                q[2 * k] = make_float2(f.x, f.y);
                q[2 * k + 1] = make_float2(f.z, f.w);
            }
        }
    };
    // Four neighbouring entries of the response: quad q of the thread's E points (FilterTables)
    auto response = [&](int q) {
        return __ldg(reinterpret_cast<const float4 *>(a.hb) + (t * E % 16) / 4 * (W / 16) + t * E / 16 + q * (W / 16));
    };
    float4 hearly[4];
    constexpr bool PADS_EARLY = EARLY && TPF >= 4;
    float ex[4], ew[4];
    if constexpr (PADS_EARLY) {
        if (t < 4) {
            const float *p = t < 2 ? p1 : p2, *w = t < 2 ? w1 : w2;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k < a.pad_n) {
                    const int c = (t & 1) ? a.nu - 1 - k : k;
                    ex[k] = __ldg(p + c);
                    if (w) ew[k] = __ldg(w + c);
                }
        }
    }
    if constexpr (EARLY) {
#pragma unroll
        for (int p = 0; p < PASSES; p++) fetch(early[p], p);
        if constexpr (W >= 16)
#pragma unroll
            for (int q = 0; q < E / 4; q++) hearly[q] = response(q);
    }
    float2 v[E];
#pragma unroll
    for (int m = 0; m < E; m++)
        if ((unsigned)(c0 + m * TPF) < (unsigned)a.nu)
            v[m] = make_float2(__ldg(p1 + c0 + m * TPF), __ldg(p2 + c0 + m * TPF));
    if (a.cos) {  // rounded products (here and with H): not fused into the first stage's sums
#pragma unroll
        for (int m = 0; m < E; m++)
            if ((unsigned)(c0 + m * TPF) < (unsigned)a.nu)
                v[m] = make_float2(__fmul_rn(v[m].x, __ldg(w1 + c0 + m * TPF)), __fmul_rn(v[m].y, __ldg(w2 + c0 + m * TPF)));
    }
    // the pads: means of the first and last pad_n weighted samples
    if constexpr (PADS_EARLY) {
        if (t < 4) {
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k < a.pad_n) s += w1 ? __fmul_rn(ex[k], ew[k]) : ex[k];
            pads[g][t] = s / (float)a.pad_n;
        }
    } else {
        for (int q = t; q < 4; q += TPF) {
            const float *p = q < 2 ? p1 : p2, *w = q < 2 ? w1 : w2;
            float s = 0.f;
            for (int k = 0; k < a.pad_n; k++) {
                const int c = (q & 1) ? a.nu - 1 - k : k;
                float x = __ldg(p + c);
                if (w) x *= __ldg(w + c);
                s += x;
            }
            pads[g][q] = s / (float)a.pad_n;
        }
    }
    meet();
#pragma unroll
    for (int m = 0; m < E; m++) {
        const int c = c0 + m * TPF;
        if (c < 0) v[m] = make_float2(pads[g][0], pads[g][2]);
        else if (c >= a.nu) v[m] = make_float2(pads[g][1], pads[g][3]);
    }

    auto load_twiddles = [&](int pass) {
        if constexpr (EARLY) {
#pragma unroll
            for (int j = 0; j < E - 1; j++) tq[j] = early[pass][j];
        } else {
            fetch(tq, pass);
        }
    };
    auto loaded = [&](auto conj, float2 x, int h, int j) { return cmul<decltype(conj)::value>(x, tq[E - 2 * h + j]); };
    // the thread's points of the strided passes, slot(k stride) apart, and its run of points of the last pass
    float2 *at[PASSES + 1], *inner = buf + slot(t * E);
#pragma unroll
    for (int p = 0; p < PASSES; p++) at[p] = buf + slot(t / F::stride(p) * (E * F::stride(p))) + slot(t % F::stride(p));

#pragma unroll
    for (int p = 0; p < PASSES; p++) {
        const int n = F::stride(p);
        if (p)
#pragma unroll
            for (int k = 0; k < E; k++) v[k] = at[p][slot(k * n)];
        load_twiddles(p);
        dif<E>(v, 0, loaded);
#pragma unroll
        for (int k = 0; k < E; k++) at[p][slot(k * n)] = v[k];
        meet();
    }
    if constexpr (PASSES > 0)
#pragma unroll
        for (int k = 0; k < E; k++) v[k] = inner[k];
#pragma unroll
    for (int b = 0; b < E; b += RL) dif<RL>(v, b, Roots{});
    if constexpr (W >= 16) {
#pragma unroll
        for (int q = 0; q < E / 4; q++) {
            const float4 h = EARLY ? hearly[q] : response(q);
            v[4 * q] = make_float2(__fmul_rn(v[4 * q].x, h.x), __fmul_rn(v[4 * q].y, h.x));
            v[4 * q + 1] = make_float2(__fmul_rn(v[4 * q + 1].x, h.y), __fmul_rn(v[4 * q + 1].y, h.y));
            v[4 * q + 2] = make_float2(__fmul_rn(v[4 * q + 2].x, h.z), __fmul_rn(v[4 * q + 2].y, h.z));
            v[4 * q + 3] = make_float2(__fmul_rn(v[4 * q + 3].x, h.w), __fmul_rn(v[4 * q + 3].y, h.w));
        }
    } else if constexpr (W > 1) {  // (a single sample is passed through)
#pragma unroll
        for (int k = 0; k < E; k++) {
            const float h = __ldg(a.hb + t * E + k);
            v[k] = make_float2(__fmul_rn(v[k].x, h), __fmul_rn(v[k].y, h));
        }
    }
#pragma unroll
    for (int b = 0; b < E; b += RL) dit<RL>(v, b, Roots{});
    if constexpr (PASSES > 0) {
#pragma unroll
        for (int k = 0; k < E; k++) inner[k] = v[k];
        meet();
    }
#pragma unroll
    for (int p = PASSES - 1; p >= 0; p--) {
        const int n = F::stride(p);
#pragma unroll
        for (int k = 0; k < E; k++) v[k] = at[p][slot(k * n)];
        load_twiddles(p);
        dit<E>(v, 0, loaded);
        if (p) {
#pragma unroll
            for (int k = 0; k < E; k++) at[p][slot(k * n)] = v[k];
            meet();
        }
    }

    bool over = false;
#pragma unroll
    for (int k = 0; k < E; k++) v[k] = make_float2(v[k].x * a.out_scale, v[k].y * a.out_scale);
    if (a.layout == FDK_LAYOUT_ROWS) {
        // v[k] is sample t + k TPF: coalesced rows
        const bool live = r0 + g < a.n_pairs;
#pragma unroll
        for (int k = 0; k < E; k++) {
            const int u = t + k * TPF - a.off;
            if (!live || u < 0 || u >= a.nu) continue;
            const long long o1 = view * a.dst_vstride + (long long)r1 * a.dst_pitch + u;
            const long long o2 = view * a.dst_vstride + (long long)r2 * a.dst_pitch + u;
            if (a.half) {
                over |= !(fabsf(v[k].x) <= 65504.f) || !(fabsf(v[k].y) <= 65504.f);
                static_cast<__half *>(a.dst)[o1] = __float2half_rn(v[k].x);
                if (r2 != r1) static_cast<__half *>(a.dst)[o2] = __float2half_rn(v[k].y);
            } else {
                static_cast<float *>(a.dst)[o1] = v[k].x;
                if (r2 != r1) static_cast<float *>(a.dst)[o2] = v[k].y;
            }
        }
    } else {
        // Columns: the G pairs' samples of one detector column are neighbours in the output, so they
        // go through shared memory and out in runs of G.  Slot (u, g) is rotated within its column
        // so that the 16 columns a half-warp writes fall into different banks.
        constexpr int ROT = G >= 16 ? 1 : 16 / G;
        __syncthreads();  // every transform of the CTA has read its last points
#pragma unroll
        for (int k = 0; k < E; k++) {
            const int u = t + k * TPF - a.off;
            if (u >= 0 && u < a.nu) fsm[u * G + ((g + u / ROT) & (G - 1))] = v[k];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < a.nu * G; i += THREADS) {
            const int u = i / G, q = i & (G - 1), ra = r0 + q, rb = a.nv - 1 - ra;
            if (ra >= a.n_pairs) continue;
            const float2 y = fsm[u * G + ((q + u / ROT) & (G - 1))];
            if (a.half) over |= !(fabsf(y.x) <= 65504.f) || !(fabsf(y.y) <= 65504.f);
            if (a.layout == FDK_LAYOUT_TRANSPOSED) {
                const long long o = view * a.dst_vstride + (long long)u * a.dst_pitch;
                if (a.half) {
                    __half *d = static_cast<__half *>(a.dst) + o;
                    d[ra] = __float2half_rn(y.x);
                    if (rb != ra) d[rb] = __float2half_rn(y.y);
                } else {
                    float *d = static_cast<float *>(a.dst) + o;
                    d[ra] = y.x;
                    if (rb != ra) d[rb] = y.y;
                }
            } else {  // mirror pairs: element (u, v) = (row v, row nv-1-v); ra last, so that the middle row of an
                      // odd nv has its real part first
                const long long o = view * (a.dst_vstride / 2) + (long long)u * a.dst_pitch;
                if (a.half) {
                    __half2 *d = static_cast<__half2 *>(a.dst) + o;
                    const __half x = __float2half_rn(y.x), z = __float2half_rn(y.y);
                    if (a.pair_stores) {
                        d[rb] = __halves2half2(z, x);
                        d[ra] = __halves2half2(x, z);
                    } else {
                        __half *e = reinterpret_cast<__half *>(d);
                        e[2 * rb] = z;
                        e[2 * rb + 1] = x;
                        e[2 * ra] = x;
                        e[2 * ra + 1] = z;
                    }
                } else {
                    float2 *d = static_cast<float2 *>(a.dst) + o;
                    if (a.pair_stores) {
                        d[rb] = make_float2(y.y, y.x);
                        d[ra] = y;
                    } else {
                        float *e = reinterpret_cast<float *>(d);
                        e[2 * rb] = y.y;
                        e[2 * rb + 1] = y.x;
                        e[2 * ra] = y.x;
                        e[2 * ra + 1] = y.y;
                    }
                }
            }
        }
    }
    if (a.overflow && over) atomicOr(a.overflow, 1u);
}

// f(std::integral_constant<int, log2W>) for the run-time length
template <int L = 0, typename Fn>
static int with_length(int log2W, Fn f) {
    if constexpr (L > 12) return fail(FDK_ERR_INVALID_ARG, "filter length 2^%d", log2W);
    else return log2W == L ? f(std::integral_constant<int, L>{}) : with_length<L + 1>(log2W, f);
}

int FilterTables::create(const double *H, int W_) {
    W = W_;
    log2W = 0;
    while ((1 << log2W) < W) log2W++;
    auto root = [&](long long k, int n) {  // exp(-2 pi i k / n)
        const double ang = -2.0 * 3.14159265358979323846 * (double)k / n;
        return make_float2((float)std::cos(ang), (float)std::sin(ang));
    };
    std::vector<float2> t(std::max(1, W / 2));
    for (int k = 0; k < W / 2; k++) t[k] = root(k, W);
    std::vector<float> h(W);
    for (int i = 0; i < W; i++) h[i] = (float)(H[filter_response_frequency(i, W)] / W);
    // the passes' twiddles: 8 + 4 + 2 + 1 per place i < n of a pass of stride n, as 8 planes of pairs, i
    // fastest: entry j of the stage of half-width h is root (i + j n) 8/h of the 16 n
    std::vector<float2> pt;
    auto put = [&](int n) {
        const size_t at = pt.size();
        pt.resize(at + 16 * (size_t)n, make_float2(0.f, 0.f));
        for (int e = 0; e < 15; e++)
            for (int i = 0; i < n; i++) pt[at + ((size_t)(e / 2) * n + i) * 2 + e % 2] = root(filter_twiddle(e, i, n), 16 * n);
    };
    if (W > 16) put(W / 16);
    if (W > 256) put(W / 256);
    if (pt.empty()) pt.push_back(make_float2(1.f, 0.f));
    FDK_CUDA(cudaMalloc(&tw, sizeof(float2) * t.size()));
    FDK_CUDA(cudaMalloc(&hb, sizeof(float) * W));
    FDK_CUDA(cudaMalloc(&twp, sizeof(float2) * pt.size()));
    SetupStream ss;
    FDK_TRY(ss.open());
    FDK_CUDA(cudaMemcpyAsync(tw, t.data(), sizeof(float2) * t.size(), cudaMemcpyHostToDevice, ss.st));
    FDK_CUDA(cudaMemcpyAsync(hb, h.data(), sizeof(float) * W, cudaMemcpyHostToDevice, ss.st));
    FDK_CUDA(cudaMemcpyAsync(twp, pt.data(), sizeof(float2) * pt.size(), cudaMemcpyHostToDevice, ss.st));
    return ss.finish("filter tables");
}

// The tables of a response in device memory, built there: tw[k] and the passes' twiddles from FP64
// sincospi, rounded; either may be null.
__global__ void filter_tables_kernel(const float *__restrict__ H, int W, float2 *tw, float2 *twp, float *hb) {
    auto root = [](long long k, int n) {
        double s, c;
        sincospi(-2.0 * (double)k / (double)n, &s, &c);
        return make_float2((float)c, (float)s);
    };
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < W; k += gridDim.x * blockDim.x) {
        if (tw && k < W / 2) tw[k] = root(k, W);
        if (twp && W > 16) {  // entry k of the first pass's planes, then of the middle pass's
            const int n = W / 16;
            twp[k] = root(filter_twiddle(k / 2 / n * 2 + (k & 1), k / 2 % n, n), W);
            if (W > 256 && k < W / 16) {
                const int m = W / 256;
                twp[W + k] = root(filter_twiddle(k / 2 / m * 2 + (k & 1), k / 2 % m, m), W / 16);
            }
        }
        hb[k] = H[filter_response_frequency(k, W)] / (float)W;
    }
}

int filter_tables_on_device(const float *H, const FilterTables &t, cudaStream_t st) {
    filter_tables_kernel<<<(t.W + 127) / 128, 128, 0, st>>>(H, t.W, t.tw, t.twp, t.hb);
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
}

void FilterTables::release() {
    if (tw) cudaFree(tw);
    if (twp) cudaFree(twp);
    if (hb) cudaFree(hb);
    tw = nullptr;
    twp = nullptr;
    hb = nullptr;
}

template <int LOG2W, int LOG2E, int G, Twiddles TW>
static int launch_group(const FilterArgs &a, int n_views, cudaStream_t st) {
    using F = Fft<LOG2W, LOG2E>;
    const auto kernel = filter_kernel<LOG2W, LOG2E, G, TW>;
    const int smem = (int)sizeof(float2) * std::max(F::TPF > 1 ? F::PITCH * G : 0, a.layout != FDK_LAYOUT_ROWS ? a.nu * G : 0);
    // per device and size, and needed at 48 KB too (the kernel also has static shared memory):
    // cheap, so set on every launch
    if (smem > 40 * 1024) FDK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kernel<<<dim3((unsigned)ceil_div(a.n_pairs, G), n_views), F::TPF * G, smem, st>>>(a);
    FDK_CUDA(cudaGetLastError());
    return FDK_OK;
}

// Transforms per CTA and points per thread.
//
// Calls that fill the chip hold 16 points a thread.  The column layouts write runs of G elements, so they take the
// largest CTA that still fills the SM's 1024 resident threads evenly: 1024 threads at W = 4096 (G = 4, 32-byte
// runs of FP32 pairs: 971 against 1139 us at 512 threads and G = 2, 32 views of 2048^2 to MIRROR FP32; these and
// the next figures with radix-16 butterflies, 2% to 4% below the present ones), 512 below, where G is 4 or more
// anyway (1500 x 1000 to MIRROR FP16 at 512 / 256 threads: 226 / 236 us).  ROWS stores are coalesced at any G, and
// smaller CTAs overlap each other's loads and transforms better (48 views of 1536 x 1024 at 512 / 256 threads:
// 285 / 260 us).
//
// A call of few transforms is one chain of latencies, the longer the more points a thread carries through it: up
// to 2^17 points (pairs x W) 4 a thread are the fastest, to 2^19 8 a thread, all they read asked for at the
// start.  Microseconds of a call (B200, back to back) with 4 / 8 / 16 points a thread, ROWS FP32:
//   rows of 200 (W 256):     33 rows x 2 views 2.4 / 3.4 / 5.1, 1200 rows 3.5 / 4.1 / 5.8, 2400 x 2 7.9 / 6.0 / 6.9
//   rows of 511 (W 512):     256 rows 2.8 / 3.5 / 6.7, 1200 rows 5.5 / 4.8 / 7.2, 2400 x 2 14.4 / 11.4 / 11.1
//   rows of 1000 (W 1024):   256 rows 4.0 / 4.2 / 7.4, 616 rows 7.4 / 6.3 / 7.6, 1200 rows 11.3 / 9.8 / 8.3
//   rows of 2047 (W 2048):   16 rows 6.0 / 5.3 / 7.1, 616 rows 16.1 / 11.8 / 8.8
//   rows of 2048 (W 4096):   16 rows 11.7 / 8.1 / 7.0, 616 rows 33.2 / 22.2 / 12.1
// (W 4096: a CTA of 512 threads or more to a pair is slower than the longer chain.)  From there to 2^21 points small
// CTAs of 16 points a thread fill the SMs more evenly (1200 rows of 1000: 8.3 against 10.1 us), but for the columns of
// longer rows, whose runs would be short (TRANSPOSED 11.7 against 14.6).
static int launch_filter(const FilterArgs &a, int log2W, int n_views, cudaStream_t st) {
    return with_length(log2W, [&](auto l) {
        constexpr int L = decltype(l)::value, W = 1 << L;
        constexpr int TPF = Fft<L, 4>::TPF, TPF4 = Fft<L, 2>::TPF, TPF8 = Fft<L, 3>::TPF;
        constexpr int cols = std::min((L == 12 ? 1024 : 512) / TPF, 64), rows = std::min(256 / TPF, 64);
        constexpr int least = std::max(1, std::min(64 / TPF, 16));  // 64 threads
        constexpr int few4 = std::max(1, std::min(64 / TPF4, 16)), few8 = std::max(1, std::min(128 / TPF8, 16));
        const long long points = (long long)a.n_pairs * n_views * W;
        if constexpr (L <= 10)
            if (points <= 1 << 17) return launch_group<L, 2, few4, Twiddles::Early>(a, n_views, st);
        if constexpr (L <= 11)
            if (points <= (L <= 8 ? 3 << 18 : 1 << 19)) return launch_group<L, 3, few8, Twiddles::Early>(a, n_views, st);
        if (!a.twp) return launch_group<L, 4, least, Twiddles::Roots>(a, n_views, st);
        if constexpr (L == 12)
            if (points <= 1 << 19) return launch_group<L, 4, least, Twiddles::Early>(a, n_views, st);
        const bool by_rows = a.layout == FDK_LAYOUT_ROWS;
        if (points <= 1 << 21 && (by_rows || L <= 8)) return launch_group<L, 4, least, Twiddles::Planes>(a, n_views, st);
        if (by_rows) return launch_group<L, 4, rows, Twiddles::Planes>(a, n_views, st);
        return launch_group<L, 4, cols, Twiddles::Planes>(a, n_views, st);
    });
}

// Shared by the FilterEngine handle, the cuFFT-plugin entry points and the reconstructor.
int filter_views(const float *src, int src_pitch, long long src_vstride, void *dst, int dst_pitch,
                 long long dst_vstride, const float *cos, int cos_pitch, const FilterTables &t, int nu,
                 int nv, int pad_n, int n_views, int layout, int dtype, cudaStream_t st, float out_scale,
                 unsigned int *overflow) {
    FDK_CHECK_ARG(t.hb && t.tw, "filter tables are missing");
    FDK_CHECK_ARG(((uintptr_t)t.hb & 15) == 0 && ((uintptr_t)t.twp & 15) == 0, "filter tables must start on 16-byte boundaries");
    FDK_CHECK_ARG(layout != FDK_LAYOUT_MIRROR || dst_vstride % 2 == 0, "mirror views are whole pairs apart");
    FilterArgs a;
    a.src = src;
    a.dst = dst;
    a.cos = cos;
    a.tw = t.tw;
    a.twp = t.twp;
    a.hb = t.hb;
    a.nu = nu;
    a.nv = nv;
    a.off = (t.W - nu) >> 1;
    a.pad_n = pad_n;
    a.n_pairs = (nv + 1) / 2;
    a.src_pitch = src_pitch;
    a.dst_pitch = dst_pitch;
    a.cos_pitch = cos_pitch;
    a.src_vstride = src_vstride;
    a.dst_vstride = dst_vstride;
    a.layout = layout;
    a.half = dtype == FDK_DTYPE_F16;
    a.pair_stores = ((uintptr_t)dst & (a.half ? 3 : 7)) == 0;
    a.out_scale = out_scale;
    a.overflow = overflow;
    return launch_filter(a, t.log2W, n_views, st);
}

static int check_filter_dims(int64_t nu, int64_t nv, int64_t W, int pad) {
    FDK_CHECK_ARG(nu > 0 && nv > 0, "nu, nv must be positive");
    FDK_CHECK_ARG(W >= nu && W <= 4096 && (W & (W - 1)) == 0, "W=%lld must be a power of two in [nu, 4096]",
                  (long long)W);
    FDK_CHECK_ARG(pad >= 1 && pad <= 4 && pad <= nu, "pad_edge must be 1..4 and <= nu");
    FDK_CHECK_ARG(nv <= 65535 * 2, "nv too large");
    return FDK_OK;
}

// Kernel dst = src * table (kernelCorrect, cudaFftFilter.cu:270-281).
__global__ void correct_kernel(const float *src, float *dst, int pitch, int width, int height, int depth,
                               const float *table, int tpitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    const int z = blockIdx.z;
    if (x >= width || y >= height || z >= depth) return;
    const long long o = ((long long)z * height + y) * pitch + x;
    dst[o] = src[o] * table[(long long)y * tpitch + x];
}

}  // namespace fdk

struct fdk_filter {
    int device = 0;
    int64_t nu = 0, nv = 0, W = 0;
    int pad = 4;
    float *d_cos = nullptr;
    float *d_src = nullptr;
    float *d_dst = nullptr;
    fdk::FilterTables tables;
    cudaStream_t stream = nullptr;
};

using namespace fdk;

extern "C" {

int fdk_filter_create(fdk_filter **out, const float *cos_table, const float *H, int64_t nu, int64_t nv,
                      int64_t W, int32_t pad_edge, int32_t device) {
    FDK_ABI_BEGIN
    clear_error();
    FDK_CHECK_ARG(out != nullptr && H != nullptr, "out or H is NULL");
    *out = nullptr;
    FDK_TRY(check_filter_dims(nu, nv, W, pad_edge));
    DeviceGuard dg(device);
    FDK_TRY(dg.status);
    fdk_filter *h = new fdk_filter();
    h->device = device;
    h->nu = nu;
    h->nv = nv;
    h->W = W;
    h->pad = pad_edge;
    std::vector<double> Hd(H, H + W);
    int s = h->tables.create(Hd.data(), (int)W);
    if (s == FDK_OK && cos_table) {
        SetupStream ss;
        s = ss.open();
        cudaError_t e = cudaSuccess;
        if (s == FDK_OK) e = cudaMalloc(&h->d_cos, sizeof(float) * nu * nv);
        if (s == FDK_OK && e == cudaSuccess)
            e = cudaMemcpyAsync(h->d_cos, cos_table, sizeof(float) * nu * nv, cudaMemcpyHostToDevice, ss.st);
        if (e != cudaSuccess) s = cuda_status(e, "filter cos table", __FILE__, __LINE__);
        if (s == FDK_OK) s = ss.finish("filter cos table");
    }
    if (s == FDK_OK) {
        cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) s = cuda_status(e, "cudaStreamCreate", __FILE__, __LINE__);
    }
    if (s != FDK_OK) {
        fdk_filter_destroy(h);
        return s;
    }
    *out = h;
    return FDK_OK;
    FDK_ABI_END
}

int fdk_filter_filtering(fdk_filter *h, float *src_host, float *dst_host, int32_t transpose) {
    FDK_ABI_BEGIN
    clear_error();
    FDK_CHECK_ARG(h && src_host && dst_host, "NULL argument");
    DeviceGuard dg(h->device);
    FDK_TRY(dg.status);
    const size_t n = (size_t)h->nu * h->nv;
    // FilterCosCorrect (FilterLib.h:8-13): src *= cos, in place on the caller's buffer, in FP32.
    if (h->d_cos) {
        std::vector<float> cos(n);
        FDK_CUDA(cudaMemcpy(cos.data(), h->d_cos, sizeof(float) * n, cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < n; i++) src_host[i] = src_host[i] * cos[i];
    }
    if (!h->d_src) {
        FDK_CUDA(cudaMalloc(&h->d_src, sizeof(float) * n));
        FDK_CUDA(cudaMalloc(&h->d_dst, sizeof(float) * n));
    }
    FDK_CUDA(cudaMemcpyAsync(h->d_src, src_host, sizeof(float) * n, cudaMemcpyHostToDevice, h->stream));
    const int layout = transpose ? FDK_LAYOUT_TRANSPOSED : FDK_LAYOUT_ROWS;
    const int dpitch = transpose ? (int)h->nv : (int)h->nu;
    FDK_TRY(filter_views(h->d_src, (int)h->nu, (long long)n, h->d_dst, dpitch, (long long)n, nullptr, 0,
                         h->tables, (int)h->nu, (int)h->nv, h->pad, 1, layout, FDK_DTYPE_F32, h->stream));
    FDK_CUDA(cudaMemcpyAsync(dst_host, h->d_dst, sizeof(float) * n, cudaMemcpyDeviceToHost, h->stream));
    FDK_CUDA(cudaStreamSynchronize(h->stream));
    return FDK_OK;
    FDK_ABI_END
}

int fdk_filter_run_device(fdk_filter *h, const float *src_dev, void *dst_dev, int64_t n_views, int32_t layout,
                          int32_t out_dtype, float out_scale, void *stream) {
    FDK_ABI_BEGIN
    clear_error();
    FDK_CHECK_ARG(h && src_dev && dst_dev, "NULL argument");
    FDK_CHECK_ARG(n_views > 0 && n_views <= 65535, "n_views out of range");
    FDK_CHECK_ARG(layout >= FDK_LAYOUT_ROWS && layout <= FDK_LAYOUT_MIRROR, "bad layout");
    FDK_CHECK_ARG(out_dtype == FDK_DTYPE_F32 || out_dtype == FDK_DTYPE_F16, "bad dtype");
    DeviceGuard dg(h->device);
    FDK_TRY(dg.status);
    const long long n = (long long)h->nu * h->nv;
    const int dpitch = layout == FDK_LAYOUT_ROWS ? (int)h->nu : (int)h->nv;
    const long long dstride = layout == FDK_LAYOUT_MIRROR ? 2 * n : n;
    return filter_views(src_dev, (int)h->nu, n, dst_dev, dpitch, dstride, h->d_cos, (int)h->nu, h->tables,
                        (int)h->nu, (int)h->nv, h->pad, (int)n_views, layout, out_dtype,
                        (cudaStream_t)stream, out_scale, nullptr);
    FDK_ABI_END
}

int fdk_filter_destroy(fdk_filter *h) {
    if (!h) return FDK_OK;
    {
        DeviceGuard dg(h->device);
        if (h->stream) cudaStreamSynchronize(h->stream);
        h->tables.release();
        if (h->d_cos) cudaFree(h->d_cos);
        if (h->d_src) cudaFree(h->d_src);
        if (h->d_dst) cudaFree(h->d_dst);
        if (h->stream) cudaStreamDestroy(h->stream);
    }
    delete h;
    return FDK_OK;
}

int fdk_correct_image_real32(const fdk_dataref *src, const fdk_dataref *table, fdk_dataref *dst) {
    FDK_ABI_BEGIN
    clear_error();
    FDK_CHECK_ARG(src && table && dst && src->data && table->data && dst->data, "NULL argument");
    FDK_CHECK_ARG(src->pitch == dst->pitch && src->width == dst->width && src->height == dst->height &&
                      src->depth <= dst->depth,
                  "src/dst shapes differ (CorrectImage, cudaFftFilter.cu:286-289)");
    FDK_CHECK_ARG(src->width > 0 && src->height > 0 && src->depth > 0 && src->pitch >= src->width, "bad shape");
    FDK_CHECK_ARG(src->height <= 65535 && src->depth <= 65535, "shape too large");
    const dim3 grid((unsigned)ceil_div(src->width, 128), src->height, src->depth);
    correct_kernel<<<grid, 128, 0, cudaStreamLegacy>>>(src->data, dst->data, src->pitch, src->width, src->height,
                                                       src->depth, table->data, table->pitch);
    FDK_CUDA(cudaGetLastError());
    FDK_CUDA(cudaStreamSynchronize(cudaStreamLegacy));  // synchronous, as the reference
    return FDK_OK;
    FDK_ABI_END
}

int fdk_scratch_trim(void) {
    FDK_ABI_BEGIN
    clear_error();
    cudaMemPool_t pool = nullptr;
    FDK_TRY(scratch_pool(&pool, false));
    if (pool) FDK_CUDA(cudaMemPoolTrimTo(pool, 0));
    return FDK_OK;
    FDK_ABI_END
}

int fdk_filter_row_real32(const fdk_dataref *src, fdk_dataref *dst, const fdk_dataref *filter) {
    FDK_ABI_BEGIN
    clear_error();
    FDK_CHECK_ARG(src && dst && filter && src->data && dst->data && filter->data, "NULL argument");
    FDK_CHECK_ARG(src->width == dst->width && src->height == dst->height && src->depth <= dst->depth,
                  "src/dst shapes differ (FilterRow, cudaFftFilter.cu:302-305)");
    FDK_CHECK_ARG(filter->height == 1 || filter->height == 0, "filter must be one row");
    const int W = filter->width;
    FDK_TRY(check_filter_dims(src->width, src->height, W, 3));
    // The tables are built on the device in a workspace of the library's pool: copying the response to
    // the host, three allocations and the copies back cost more than the filter (48 views of
    // 1536 x 1024: 1073 us of which 240 in the filter kernel; 268 us so).
    FilterTables t;
    t.W = W;
    while ((1 << t.log2W) < W) t.log2W++;
    // The response first: W floats are whole 16-byte words (W >= 4), which the kernel reads it and the
    // passes' planes by.
    const size_t planes = (size_t)W + W / 16;
    Scratch tables;
    FDK_TRY(tables.alloc(sizeof(float) * W + sizeof(float2) * (planes + W / 2), cudaStreamLegacy));
    t.hb = static_cast<float *>(tables.p);
    t.twp = reinterpret_cast<float2 *>(t.hb + W);
    t.tw = t.twp + planes;
    FDK_TRY(filter_tables_on_device(filter->data, t, cudaStreamLegacy));
    FDK_TRY(filter_views(src->data, src->pitch, (long long)src->pitch * src->height, dst->data, dst->pitch,
                         (long long)dst->pitch * dst->height, nullptr, 0, t, src->width, src->height, 3, src->depth,
                         FDK_LAYOUT_ROWS, FDK_DTYPE_F32, cudaStreamLegacy));
    FDK_TRY(tables.free());
    FDK_CUDA(cudaStreamSynchronize(cudaStreamLegacy));  // synchronous, as the reference
    return FDK_OK;
    FDK_ABI_END
}

}  // extern "C"
