// nn_tc.cuh -- the learned row filter's network on the 5th-generation tensor cores (tcgen05).
//
// The middle layer, a 32 -> 32 channel convolution with 9 taps, is 9216 of the network's 9792 multiply-adds
// per position and a contraction over (tap, input channel).  Its operands lie in shared memory as
// [channel / 8][position][8] BF16: 8 positions x 8 channels are one 128-byte core matrix of the
// no-swizzle operand layout, and the next position is 16 bytes on, so that the operand of tap k is
// the same buffer k rows further.  Nothing is gathered, and positions before and after a row are zeros.
//
// FP32 weights stay FP32: each is the sum of three BF16 parts (8 + 8 + 8 mantissa bits, exact), a
// product of two BF16 is exact in the FP32 accumulator, and the parts accumulate in columns of their
// own, which are added in FP32.  Activations are BF16, as the network defines them.
#pragma once
#include <cuda_bf16.h>

#include "common.h"
#include "tma_common.cuh"

namespace fdk {

constexpr int kCh = 32, kK = 9, kHalo = 4;
constexpr int kW1 = 0, kB1 = kW1 + kCh * kK, kW2 = kB1 + kCh, kB2 = kW2 + kCh * kCh * kK, kW3 = kB2 + kCh,
              kB3 = kW3 + kCh * kK, kNParam = kB3 + 1;
constexpr int kMaxLen = 256;  // row length limit: the positions a CTA holds

namespace nn {

constexpr int THREADS = 256;
constexpr int POS = 256;              // positions of one step: whole rows, 4 zeros apart
// Operand buffers: position p is row p + ROW0 of its 8-channel group, runs of 8 positions being whole, aligned
// 128-byte core matrices.  The halo rows after a group (p = 256 .. 259) are rows 0 .. 3 of the next, which
// has none there.
constexpr int ROW0 = 8, PITCH = POS + 2 * kHalo;
constexpr int GROUP = PITCH * 16;     // bytes of a group
constexpr int SPLIT = 3;

// --- tcgen05
__device__ __forceinline__ void tc_alloc(unsigned smem_word, unsigned columns) {  // one warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_word), "r"(columns));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tc_dealloc(unsigned tmem, unsigned columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns));
}
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic shared-memory writes become visible to the tensor core's reads after the next barrier
__device__ __forceinline__ void tc_publish() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// No-swizzle operand descriptor.  The operand is core matrices of 8 rows x 16 bytes, 128 bytes each;
// `lead` and `stride` are the bytes between neighbouring ones along K and along M or N (K-major), or
// along the other way round for an operand whose contiguous 16 bytes run along M or N.
__device__ __forceinline__ unsigned long long tc_desc(unsigned addr, unsigned lead, unsigned stride) {
    return (unsigned long long)((addr >> 4) & 0x3FFFu) | ((unsigned long long)(lead >> 4) << 16) |
           ((unsigned long long)(stride >> 4) << 32) | (1ull << 46);
}
// kind::f16, BF16 operands, FP32 accumulator, M = 128
__host__ __device__ constexpr unsigned tc_instr(int n, bool a_mn_major = false, bool b_mn_major = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) |
           ((unsigned)(n >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
}
// A whole warp runs the issue loops, so that descriptors live in uniform registers, and `leader` (true in
// one lane) issues.  From a branch that one thread takes, every descriptor is moved across register
// files, at over 100 clocks an instruction against the 32 that it computes for.
__device__ __forceinline__ void tc_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned instr,
                                       bool accumulate, unsigned leader) {
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(instr), "r"((unsigned)accumulate), "r"(leader)
        : "memory");
}
__device__ __forceinline__ unsigned tc_leader() {  // converged warp
    unsigned p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p;
}
__device__ __forceinline__ void tc_commit(unsigned bar) {  // the thread that issued
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 consecutive columns of the warp's 32 lanes; tc_ld_wait before the values are used
__device__ __forceinline__ void tc_ld32(unsigned taddr, unsigned (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tc_ld8(unsigned taddr, unsigned (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// x = hi + mid + lo, exactly, as the upper halves of three FP32 words: each part is the leading 8 bits of
// what is left (by masks and subtractions; the conversion instructions run at a quarter of their rate).
__device__ __forceinline__ void split3(float x, unsigned (&o)[SPLIT]) {
    o[0] = __float_as_uint(x) & 0xFFFF0000u;
    const float r = x - __uint_as_float(o[0]);
    o[1] = __float_as_uint(r) & 0xFFFF0000u;
    o[2] = __float_as_uint(r - __uint_as_float(o[1]));
}
// The upper halves of a (low) and b (high)
__device__ __forceinline__ unsigned upper2(unsigned a, unsigned b) { return __byte_perm(a, b, 0x7632); }
__device__ __forceinline__ unsigned pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned *>(&v);
}

// A wait of the CTA ran out: records it and waits, bounded, for the operations the CTA still has in flight
// (fin: a barrier of 32 arrivals used for nothing else) before the caller gives its TMEM back.  A commit covers its
// own thread's operations and any lane of warp 0 may have issued, so that all of them commit.
__device__ __noinline__ void give_up(unsigned fin, unsigned *err) {
    if (threadIdx.x < 32) {
        if (threadIdx.x == 0) atomicOr(err, kErrTimeout);
        tc_commit(fin);
        mbar_wait(fin, 0);
    }
}
// What a CTA that gave up leaves in the outputs it owes.
__device__ __forceinline__ float lost() { return __int_as_float(0x7FFFFFFF); }

// Device-side failures of the network kernels (a bounded wait that ran out), read by fdk_nn_check and fdk_volume_mse.
static __device__ unsigned int g_nn_err;

// The small layers' weights, in the order the position threads read them.
struct Small {
    float w1[kK][kCh];   // [tap][channel]
    float w3[kCh][12];   // [channel][tap], rows of three 16-byte loads
    float b1[kCh], b2[kCh], b3;
};
__device__ __forceinline__ void load_small(Small &s, const float *params) {
    for (int i = threadIdx.x; i < kCh * kK; i += blockDim.x) {
        s.w1[i % kK][i / kK] = params[kW1 + i];
        s.w3[i / kK][i % kK] = params[kW3 + i];
    }
    for (int i = threadIdx.x; i < kCh; i += blockDim.x) {
        s.b1[i] = params[kB1 + i];
        s.b2[i] = params[kB2 + i];
    }
    if (threadIdx.x == 0) s.b3 = params[kB3];
}

// Rows in a step: row i's sample p is position i (L + 4) + p.  The 4 positions between rows are the halo
// of both.
__host__ __device__ inline int rows_per_step(int L) { return max(1, (POS + kHalo) / (L + kHalo)); }
struct Place {
    int row, p;   // row of the step and sample in it
    bool in;      // a sample of a row
};
__device__ __forceinline__ Place place(int m, int L, int rows) {
    const int i = m / (L + kHalo), p = m - i * (L + kHalo);
    return {i, p, i < rows && p < L};
}

// Layer 1 of positions m and m + 128, channel groups G h .. G h + G - 1 of 8, into the operand buffer:
// a1[c] = relu(b1[c] + sum_k W1[c][k] xs[p + k - 4]) in BF16 (xs: position p at p + 4)
template <int G>
__device__ __forceinline__ void layer1(const Small &w, const float *xs, unsigned char *a1, int m, int h, bool in0,
                                       bool in1) {
    float x0[kK], x1[kK];
#pragma unroll
    for (int k = 0; k < kK; k++) {
        x0[k] = xs[m + k];
        x1[k] = xs[m + 128 + k];
    }
#pragma unroll
    for (int g = 0; g < G; g++) {
        float z0[8], z1[8];
        const int c = 8 * (G * h + g);
#pragma unroll
        for (int i = 0; i < 8; i++) z0[i] = z1[i] = w.b1[c + i];
#pragma unroll
        for (int k = 0; k < kK; k++) {
            const float4 wa = *reinterpret_cast<const float4 *>(&w.w1[k][c]);
            const float4 wb = *reinterpret_cast<const float4 *>(&w.w1[k][c + 4]);
            const float wv[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
            for (int i = 0; i < 8; i++) {
                z0[i] = fmaf(wv[i], x0[k], z0[i]);
                z1[i] = fmaf(wv[i], x1[k], z1[i]);
            }
        }
        uint4 o0 = make_uint4(0, 0, 0, 0), o1 = make_uint4(0, 0, 0, 0);
        if (in0)
            o0 = make_uint4(pack2(fmaxf(z0[0], 0.f), fmaxf(z0[1], 0.f)), pack2(fmaxf(z0[2], 0.f), fmaxf(z0[3], 0.f)),
                            pack2(fmaxf(z0[4], 0.f), fmaxf(z0[5], 0.f)), pack2(fmaxf(z0[6], 0.f), fmaxf(z0[7], 0.f)));
        if (in1)
            o1 = make_uint4(pack2(fmaxf(z1[0], 0.f), fmaxf(z1[1], 0.f)), pack2(fmaxf(z1[2], 0.f), fmaxf(z1[3], 0.f)),
                            pack2(fmaxf(z1[4], 0.f), fmaxf(z1[5], 0.f)), pack2(fmaxf(z1[6], 0.f), fmaxf(z1[7], 0.f)));
        uint4 *d = reinterpret_cast<uint4 *>(a1 + (G * h + g) * GROUP + (m + ROW0) * 16);
        d[0] = o0;
        d[128] = o1;
    }
}

// W2 as the B operand of layer 2: [tap][ci / 8][split * 32 + c][ci % 8], N = 96
constexpr int WF_ROWS = SPLIT * kCh, WF_GROUP = WF_ROWS * 16, WF_BYTES = kK * 4 * WF_GROUP;
__device__ __forceinline__ void load_forward_weights(unsigned char *wf, const float *params) {
    for (int i = threadIdx.x; i < kCh * kCh * kK; i += blockDim.x) {
        const int c = i / (kCh * kK), ci = (i / kK) % kCh, k = i % kK;  // params W2[c][ci][k]
        unsigned s[SPLIT];
        split3(params[kW2 + i], s);
#pragma unroll
        for (int j = 0; j < SPLIT; j++)
            *reinterpret_cast<unsigned short *>(wf + (k * 4 + ci / 8) * WF_GROUP + (j * kCh + c) * 16 + (ci % 8) * 2) = s[j] >> 16;
    }
}

// Layer 2's products of all positions into TMEM columns d (tile 0) and d + apart (tile 1), 96 columns
// each (split j of channel c in column 32 j + c).  One warp.
__device__ __forceinline__ void issue_layer2(unsigned d, unsigned a1, unsigned wf, int tiles, int apart, unsigned leader) {
    for (int t = 0; t < tiles; t++) {
        const unsigned long long a = tc_desc(a1 + 2048 * t, GROUP, 128), b = tc_desc(wf, WF_GROUP, 128);
#pragma unroll
        for (int k = 0; k < kK; k++)
#pragma unroll
            for (int s = 0; s < 2; s++)
                tc_mma(d + apart * t, a + (2 * s * GROUP + (ROW0 - kHalo + k) * 16) / 16, b + (k * 4 + 2 * s) * WF_GROUP / 16, tc_instr(WF_ROWS),
                       k | s, leader);
    }
}

// Layer 2 of channel c at one position as one FP32 chain over (input channel, tap): col is the position's
// first tap in the operand buffer.
__device__ __noinline__ float layer2_chain(const float *__restrict__ params, const unsigned char *col, int c) {
    const float *w2 = params + kW2 + c * kCh * kK;
    float z = __ldg(params + kB2 + c);
#pragma unroll 2
    for (int g = 0; g < kCh / 4; g++, w2 += 4 * kK) {  // four input channels at a time
        float wv[4 * kK];
        if (((size_t)params & 15) == 0) {
#pragma unroll
            for (int i = 0; i < kK; i++) {
                const float4 f = __ldg(reinterpret_cast<const float4 *>(w2) + i);
                wv[4 * i] = f.x;
                wv[4 * i + 1] = f.y;
                wv[4 * i + 2] = f.z;
                wv[4 * i + 3] = f.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4 * kK; i++) wv[i] = __ldg(w2 + i);
        }
        uint2 av[kK];
#pragma unroll
        for (int k = 0; k < kK; k++) av[k] = *reinterpret_cast<const uint2 *>(col + (g >> 1) * GROUP + k * 16 + (g & 1) * 8);
#pragma unroll
        for (int ci = 0; ci < 4; ci++)
#pragma unroll
            for (int k = 0; k < kK; k++) {
                const unsigned u = ci < 2 ? av[k].x : av[k].y;
                z = fmaf(wv[ci * kK + k], __uint_as_float(ci & 1 ? u & 0xFFFF0000u : u << 16), z);
            }
    }
    return z;
}

// a2 of this thread's position (lane of quadrant warp % 4, tile warp / 4): relu of layer 2, rounded to
// BF16, zero outside the rows.
//
// Summed in another order, z moves by one or two of its last bits, and where it lies that near to the
// middle of two BF16 values the activation moves by 2^-8 of itself: single outputs then differ by up to
// 1e-3 of the row's size from an FP32 evaluation of the network.  The activations within kNear last
// bits of a middle (one in 5000) are therefore rounded from the FP32 chain.
constexpr unsigned kNear = 8;
__device__ __forceinline__ bool near_middle(float r) { return (__float_as_uint(r) & 0xFFFFu) - (0x8000u - kNear) <= 2 * kNear; }
__device__ __forceinline__ void read_layer2(unsigned d, const Small &w, const float *__restrict__ params,
                                            const unsigned char *a1, bool in, float (&a2)[kCh]) {
    const unsigned warp = threadIdx.x >> 5;
    const unsigned at = d + 128 * (warp >> 2) + ((32 * (warp & 3)) << 16);
    unsigned hi[32], mid[32], lo[32];
    tc_ld32(at, hi);
    tc_ld32(at + 32, mid);
    tc_ld32(at + 64, lo);
    tc_ld_wait();
    unsigned near = 0;
#pragma unroll
    for (int c = 0; c < kCh; c++) {
        const float z = (w.b2[c] + (__uint_as_float(mid[c]) + __uint_as_float(lo[c]))) + __uint_as_float(hi[c]);
        const float r = fmaxf(z, 0.f);
        if (near_middle(r)) near |= 1u << c;
        a2[c] = in ? __bfloat162float(__float2bfloat16_rn(r)) : 0.f;
    }
    for (near = in ? near : 0u; near; near &= near - 1) {
        const int c = __ffs(near) - 1;
        const float z = layer2_chain(params, a1 + (threadIdx.x + ROW0 - kHalo) * 16, c);
        const float r = __bfloat162float(__float2bfloat16_rn(fmaxf(z, 0.f)));
#pragma unroll
        for (int i = 0; i < kCh; i++)
            if (i == c) a2[i] = r;
    }
}

struct Fwd {
    static constexpr int WF = 0, A1 = WF + WF_BYTES, SMALL = A1 + 4 * GROUP + kHalo * 16, XS = SMALL + (int)sizeof(Small) + 12,
                         PART = XS + (PITCH + 8) * 4, BARS = PART + kK * PITCH * 4, BYTES = BARS + 32;  // barriers: layer 2, fin; TMEM word
    static constexpr unsigned COLUMNS = 256;
};
static_assert(Fwd::XS % 16 == 0 && Fwd::PART % 16 == 0 && Fwd::BARS % 8 == 0, "alignment");

// The CTA gave up at step st: its rows from there on.
__device__ __noinline__ void lose_rows(float *y, int L, long long rows, long long st) {
    const int per = rows_per_step(L);
    const Place me = place(threadIdx.x, L, per);
    for (; st * per < rows; st += gridDim.x)
        if (me.in && st * per + me.row < rows) y[(st * per + me.row) * L + me.p] = lost();
}

// y = x + net(x).  23,040 rows of 256: 545 us; FP32 FMAs, register-blocked, took 2283 (69% of the FP32 rate).
// The tensor core is busy for about 2100 clocks of a step's 11,000 (two CTAs share an SM); the rest is
// layers 1 and 3 on the FP32 pipe and the barriers between the phases.  A CTA of 256 threads takes the rows of one step (256 positions) at a time: layer 1 in
// FP32 by (position, 16 channels), layer 2 on the tensor core (two tiles of 128 positions x 96 columns
// x 288), layer 3 in FP32 by position, its 9 taps' partial sums exchanged through shared memory.
// Two CTAs per SM run their phases against each other.
__global__ void __launch_bounds__(THREADS, 2) forward_kernel(const float *__restrict__ params, const float *__restrict__ x,
                                                           float *__restrict__ y, int L, long long rows, float s,
                                                           unsigned long long wait_ns, int withhold) {
    extern __shared__ __align__(128) unsigned char smem[];
    Small &w = *reinterpret_cast<Small *>(smem + Fwd::SMALL);
    float *xs = reinterpret_cast<float *>(smem + Fwd::XS);      // s x, position p at p + 4
    float *part = reinterpret_cast<float *>(smem + Fwd::PART);  // [tap][position + 4]
    const unsigned base = smem_u32(smem), bar = base + Fwd::BARS;
    unsigned *tmem_word = reinterpret_cast<unsigned *>(smem + Fwd::BARS + 16);
    const int t = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, t >> 5, 0);  // uniform
    load_small(w, params);
    load_forward_weights(smem + Fwd::WF, params);
    for (int i = t; i < (Fwd::SMALL - Fwd::A1) / 16; i += THREADS) reinterpret_cast<uint4 *>(smem + Fwd::A1)[i] = make_uint4(0, 0, 0, 0);
    for (int i = t; i < kK * PITCH; i += THREADS) part[i] = 0.f;
    if (t == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 8, 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (t < 32) tc_alloc(smem_u32(tmem_word), Fwd::COLUMNS);
    tc_before();
    __syncthreads();
    tc_after();
    const unsigned d = *tmem_word;
    const int per = rows_per_step(L), tiles = per * (L + kHalo) - kHalo > 128 ? 2 : 1;
    const long long steps = (rows + per - 1) / per;
    const Place me = place(t, L, per), l0 = place(t & 127, L, per), l1 = place((t & 127) + 128, L, per);
    const unsigned stall = withhold && blockIdx.x == 0 ? 1 : 0;
    unsigned phase = 0;
    for (long long st = blockIdx.x; st < steps; st += gridDim.x, phase ^= 1) {
        const long long r0 = st * per;
        const bool live = me.in && r0 + me.row < rows;
        const float xv = live ? x[(r0 + me.row) * L + me.p] : 0.f;
        xs[t + kHalo] = xv * s;
        if (t < kHalo) xs[t] = xs[POS + kHalo + t] = 0.f;
        __syncthreads();
        layer1<2>(w, xs, smem + Fwd::A1, t & 127, t >> 7, l0.in && r0 + l0.row < rows, l1.in && r0 + l1.row < rows);
        tc_publish();
        tc_before();
        __syncthreads();
        if (warp == 0) {
            tc_after();
            const unsigned leader = tc_leader();
            issue_layer2(d, base + Fwd::A1, base + Fwd::WF, tiles, 128, leader);
            if (leader > stall) tc_commit(bar);
            __syncwarp();
        }
        const bool ok = mbar_wait(bar, phase, wait_ns);
        if (__syncthreads_or(!ok)) {
            give_up(bar + 8, &g_nn_err);
            lose_rows(y, L, rows, st);
            break;
        }
        tc_after();
        if (t < 128 * tiles) {
            float a2[kCh];
            read_layer2(d, w, params, smem + Fwd::A1, live, a2);
            float o[kK];
#pragma unroll
            for (int k = 0; k < kK; k++) o[k] = 0.f;
#pragma unroll
            for (int c = 0; c < kCh; c++) {
                const float4 wa = *reinterpret_cast<const float4 *>(&w.w3[c][0]);
                const float4 wb = *reinterpret_cast<const float4 *>(&w.w3[c][4]);
                const float wv[kK] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w, w.w3[c][8]};
#pragma unroll
                for (int k = 0; k < kK; k++) o[k] = fmaf(wv[k], a2[c], o[k]);
            }
#pragma unroll
            for (int k = 0; k < kK; k++) part[k * PITCH + t + kHalo] = o[k];
        }
        tc_before();
        __syncthreads();
        if (live) {
            float o = w.b3;
#pragma unroll
            for (int k = 0; k < kK; k++) o += part[k * PITCH + t + k];
            y[(r0 + me.row) * L + me.p] = xv + o / s;
        }
    }
    tc_before();
    __syncthreads();
    tc_after();
    if (t < 32) tc_dealloc(d, Fwd::COLUMNS);
}


// ---------------------------------------------------------------------------------------------
// Parameter gradient of sum(dy . y).  One CTA of 512 threads per SM takes the rows of a step (256
// positions) at a time, recomputes a1 and a2, and runs every sum over positions or channels on the
// tensor core, out of operand buffers of one shape ([channel / 8][position][8], one after the other, so
// that neighbours form one operand):
//   dz1 = conv^T(W2, dz2)      A = dz2 (positions x c, per part), B = W2, tap k: rows 8 - k further
//   dW2[c][ci][k]              A = [dz2 parts] (96 x positions), B = a1, tap k: rows k further
//   dW3[c][k], db2             A = [a2, dz2 parts] (128 x positions), B = columns d3[q - k + 4], 1
//   dW1[ci][k], db1            A = [dz1 parts], B = columns xs[q + k - 4], 1
// 23,040 rows of 256: 2120 us; FP32 FMAs took 6690.  Of a step's 25,400 clocks the tensor core works 15,400: an
// instruction of M = 128 takes 33 + N / 4 clocks (41 at N = 32, 57 at N = 96; both operand orders,
// swizzled or not), of which the narrow sums over positions need 176 and dz1 108.
//
// FP32 factors (W2, dz2, dz1, d3, xs) are three BF16 parts each, every product of parts is summed
// (those below 2^-24 too, as they cost no extra pass), and the sums of a step, 16 accumulations deep, are
// added to FP32 registers, so that the accumulator's rounding does not grow with the scan.
// ---------------------------------------------------------------------------------------------
struct Bwd {
    static constexpr int THREADS = 512;
    static constexpr int BUF = 4 * GROUP;  // 32 channels of 256 positions
    static constexpr int A2 = 0, DZ2 = A2 + BUF, DZ1 = DZ2 + SPLIT * BUF, A1 = DZ1 + SPLIT * BUF, T1 = A1 + BUF,
                         T3 = T1 + BUF, WF = T3 + BUF, SMALL = WF + WF_BYTES, XS = SMALL + (int)sizeof(Small) + 12,
                         D3 = XS + (PITCH + 8) * 4, BARS = D3 + (PITCH + 8) * 4, BYTES = BARS + 48;
    // TMEM columns: layer 2, then dz1, then dW1 share the first ones
    static constexpr unsigned LAYER2 = 0, DZ1_D = 0, DW1 = 0, DW2 = 192, DW3 = 480, COLUMNS = 512;
    static constexpr int SUM = SPLIT * kCh * (kK * kCh + 1) * 4;  // dW2 of the three parts, at the end
};
static_assert(Bwd::BYTES <= 227 * 1024 && Bwd::SUM <= Bwd::WF && Bwd::XS % 16 == 0 && Bwd::BARS % 8 == 0, "shared memory");

// Eight channels' BF16 parts of one position into the operand buffers of the parts (dst: the group's row)
__device__ __forceinline__ void store_parts(unsigned char *dst, const float (&v)[8]) {
    unsigned p[8][SPLIT];
#pragma unroll
    for (int i = 0; i < 8; i++) split3(v[i], p[i]);
#pragma unroll
    for (int j = 0; j < SPLIT; j++)
        *reinterpret_cast<uint4 *>(dst + j * Bwd::BUF) = make_uint4(upper2(p[0][j], p[1][j]), upper2(p[2][j], p[3][j]),
                                                                  upper2(p[4][j], p[5][j]), upper2(p[6][j], p[7][j]));
}
// A position's row of a column operand: part j of v[k] in column 9 j + k, then a 1
__device__ __forceinline__ void store_columns(unsigned char *dst, const float (&v)[kK]) {
    unsigned col[32];
#pragma unroll
    for (int k = 0; k < kK; k++) {
        unsigned p[SPLIT];
        split3(v[k], p);
#pragma unroll
        for (int j = 0; j < SPLIT; j++) col[9 * j + k] = p[j];
    }
    col[27] = __float_as_uint(1.f);
#pragma unroll
    for (int i = 28; i < 32; i++) col[i] = 0;
#pragma unroll
    for (int g = 0; g < 4; g++)
        *reinterpret_cast<uint4 *>(dst + g * GROUP) =
            make_uint4(upper2(col[8 * g], col[8 * g + 1]), upper2(col[8 * g + 2], col[8 * g + 3]),
                       upper2(col[8 * g + 4], col[8 * g + 5]), upper2(col[8 * g + 6], col[8 * g + 7]));
}
// Sums over positions: D[128][32] (+)= A^T B, A's 16 channel groups and B's 4 from buffer rows ra and rb on
__device__ __forceinline__ void issue_sum(unsigned d, unsigned a, unsigned b, int steps, unsigned leader) {
    const unsigned long long da = tc_desc(a, 128, GROUP), db = tc_desc(b, 128, GROUP);
#pragma unroll
    for (int s = 0; s < POS / 16; s++)
        if (s < steps) tc_mma(d, da + s * 16, db + s * 16, tc_instr(32, true, true), s, leader);
}

__global__ void __launch_bounds__(Bwd::THREADS, 1) backward_kernel(const float *__restrict__ params,
                                                                 const float *__restrict__ x, const float *__restrict__ dy,
                                                                 float *__restrict__ dparams, int L, long long rows, float s,
                                                                 unsigned long long wait_ns, int withhold) {
    extern __shared__ __align__(128) unsigned char smem[];
    Small &w = *reinterpret_cast<Small *>(smem + Bwd::SMALL);
    float *xs = reinterpret_cast<float *>(smem + Bwd::XS);  // s x, position p at p + 4
    float *d3 = reinterpret_cast<float *>(smem + Bwd::D3);  // dL/do = dL/dy / s, position p at p + 4
    const unsigned base = smem_u32(smem), bar_l2 = base + Bwd::BARS, bar_dz1 = bar_l2 + 8, bar_all = bar_l2 + 16, fin = bar_l2 + 24;
    unsigned *tmem_word = reinterpret_cast<unsigned *>(smem + Bwd::BARS + 32);
    const int t = threadIdx.x, lane = t & 31, q = (t >> 5) & 3, r = t >> 7;  // TMEM quadrant; quarter of the CTA
    const bool issuer = __shfl_sync(0xFFFFFFFFu, t >> 5, 0) == 0;  // warp-uniform
    const int m = 128 * (r & 1) + 32 * q + lane, h = r >> 1;               // position, half of the channels
    load_small(w, params);
    load_forward_weights(smem + Bwd::WF, params);
    for (int i = t; i < Bwd::WF / 16; i += Bwd::THREADS) reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0, 0, 0, 0);
    if (t == 0) {
        mbar_init(bar_l2, 1);
        mbar_init(bar_dz1, 1);
        mbar_init(bar_all, 1);
        mbar_init(fin, 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (t < 32) tc_alloc(smem_u32(tmem_word), Bwd::COLUMNS);
    tc_before();
    __syncthreads();
    tc_after();
    const unsigned d = *tmem_word, at = d + ((32 * q) << 16);  // this warp's lanes
    const int per = rows_per_step(L), used = per * (L + kHalo) - kHalo, tiles = used > 128 ? 2 : 1, ksteps = (used + 15) / 16;
    const long long steps = (rows + per - 1) / per;
    const Place me = place(m, L, per), l0 = place(t & 127, L, per), l1 = place((t & 127) + 128, L, per);
    const Place ld = place(t & 255, L, per);

    // FP32 sums of the CTA's steps: dW2 rows (part q, channel lane), columns 72 r .. 72 r + 71 of (tap, ci); the
    // small layers' by quarter 0 (dW3, db2) and 1 (dW1, db1)
    float gw2[72], gk[kK], gb = 0.f, gb3 = 0.f;
#pragma unroll
    for (int i = 0; i < 72; i++) gw2[i] = 0.f;
#pragma unroll
    for (int k = 0; k < kK; k++) gk[k] = 0.f;

    // this thread's sample of a step: of x, or of dy in the upper half of the CTA
    const float *src = t < 256 ? x : dy;
    auto fetch = [&](long long st) {
        const long long row = st * per + ld.row;
        return ld.in && st < steps && row < rows ? __ldg(src + row * L + ld.p) : 0.f;
    };
    float next = fetch(blockIdx.x);
    unsigned phase = 0;
    bool ok = true;
    for (long long st = blockIdx.x; st < steps; st += gridDim.x, phase ^= 1) {
        const long long r0 = st * per;
        const bool live = me.in && r0 + me.row < rows;
        if (t < 256) {
            xs[t + kHalo] = next * s;
            if (t < kHalo) xs[t] = xs[POS + kHalo + t] = 0.f;
        } else {
            const float g = next / s;  // y = x + o / s
            d3[t - 256 + kHalo] = g;
            if (t < 256 + kHalo) d3[t - 256] = d3[POS + kHalo + t - 256] = 0.f;
            gb3 += g;
        }
        next = fetch(st + gridDim.x);
        if (__syncthreads_or(!ok)) break;
        layer1<1>(w, xs, smem + Bwd::A1, t & 127, t >> 7, l0.in && r0 + l0.row < rows, l1.in && r0 + l1.row < rows);
        tc_publish();
        tc_before();
        __syncthreads();
        float win[kK];
        if (issuer) {
            tc_after();
            const unsigned leader = tc_leader();
            issue_layer2(d + Bwd::LAYER2, base + Bwd::A1, base + Bwd::WF, tiles, 96, leader);
            if (leader && !(withhold && blockIdx.x == 0)) tc_commit(bar_l2);
            __syncwarp();
        }
        // while layer 2 runs: the column operands (tap 8 - k of d3's window is d3[p - k + 4])
        if (h) {
#pragma unroll
            for (int k = 0; k < kK; k++) win[k] = xs[m + k];
            store_columns(smem + Bwd::T1 + (m + ROW0) * 16, win);
        }
#pragma unroll
        for (int k = 0; k < kK; k++) win[k] = d3[m + 8 - k];
        if (!h) store_columns(smem + Bwd::T3 + (m + ROW0) * 16, win);
        ok = mbar_wait(bar_l2, phase, wait_ns);
        tc_after();
        // a2 and dz2[c][p] = [a2 > 0] sum_k W3[c][k] d3[p - k + 4], 8 channels at a time
        if ((r & 1) < tiles) {
#pragma unroll 1
            for (int g = 2 * h; g < 2 * h + 2; g++) {
                unsigned hi[8], mid[8], lo[8];
                const unsigned z0 = at + Bwd::LAYER2 + 96 * (r & 1) + 8 * g;
                tc_ld8(z0, hi);
                tc_ld8(z0 + 32, mid);
                tc_ld8(z0 + 64, lo);
                tc_ld_wait();
                unsigned a2[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    float z[2];
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const int c = 2 * i + j;
                        z[j] = (w.b2[8 * g + c] + (__uint_as_float(mid[c]) + __uint_as_float(lo[c]))) + __uint_as_float(hi[c]);
                        z[j] = live ? fmaxf(z[j], 0.f) : 0.f;
                    }
                    a2[i] = pack2(z[0], z[1]);
                }
                float dz[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float *w3 = &w.w3[8 * g + i][0];
                    const float4 wa = *reinterpret_cast<const float4 *>(w3), wb = *reinterpret_cast<const float4 *>(w3 + 4);
                    const float wv[kK] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w, w3[8]};
                    float v = 0.f;
#pragma unroll
                    for (int k = 0; k < kK; k++) v = fmaf(wv[k], win[k], v);
                    dz[i] = (a2[i >> 1] & (i & 1 ? 0xFFFF0000u : 0xFFFFu)) ? v : 0.f;  // a2 > 0
                }
                *reinterpret_cast<uint4 *>(smem + Bwd::A2 + g * GROUP + (m + ROW0) * 16) = make_uint4(a2[0], a2[1], a2[2], a2[3]);
                store_parts(smem + Bwd::DZ2 + g * GROUP + (m + ROW0) * 16, dz);
            }
        }
        tc_publish();
        tc_before();
        if (__syncthreads_or(!ok)) break;
        if (issuer) {
            tc_after();
            const unsigned leader = tc_leader();
            // dz1: the small parts first, so that the large ones' sums meet the fewest roundings
            for (int tile = 0; tile < tiles; tile++)
                for (int i = SPLIT - 1; i >= 0; i--) {
                    const unsigned long long a = tc_desc(base + Bwd::DZ2 + i * Bwd::BUF + 2048 * tile, GROUP, 128);
                    const unsigned long long b = tc_desc(base + Bwd::WF, 128, 512);
#pragma unroll
                    for (int k = 0; k < kK; k++)
#pragma unroll
                        for (int c = 0; c < 2; c++)
                            tc_mma(d + Bwd::DZ1_D + 96 * tile, a + (2 * c * GROUP + (ROW0 + kHalo - k) * 16) / 16,
                                   b + (k * 4 * WF_GROUP + c * 256) / 16, tc_instr(WF_ROWS, false, true),
                                   i < SPLIT - 1 || k || c, leader);
                }
            if (leader) tc_commit(bar_dz1);
            __syncwarp();
            issue_sum(d + Bwd::DW3, base + Bwd::A2 + ROW0 * 16, base + Bwd::T3 + ROW0 * 16, ksteps, leader);
#pragma unroll 1
            for (int k = 0; k < kK; k++)
                issue_sum(d + Bwd::DW2 + 32 * k, base + Bwd::DZ2 + ROW0 * 16, base + Bwd::A1 + (ROW0 - kHalo + k) * 16, ksteps, leader);
        } else {
            ok = mbar_wait(bar_dz1, phase, wait_ns);
            tc_after();
        }
        // dz1[ci][p] = [a1 > 0] of the sums; channel 8 g + i, part j of W2 in column 8 (3 g + j) + i.  The issuing
        // warp is busy to the end of the sums: warp 4, which reads the same TMEM lanes, has its positions too.
        auto backward1 = [&](int tile) {
            const int p = 128 * tile + 32 * q + lane;
#pragma unroll 1
            for (int g = 2 * h; g < 2 * h + 2; g++) {
                unsigned hi[8], mid[8], lo[8];
                const unsigned z0 = at + Bwd::DZ1_D + 96 * tile + 24 * g;
                tc_ld8(z0, hi);
                tc_ld8(z0 + 8, mid);
                tc_ld8(z0 + 16, lo);
                const uint4 a = *reinterpret_cast<const uint4 *>(smem + Bwd::A1 + g * GROUP + (p + ROW0) * 16);
                const unsigned av[4] = {a.x, a.y, a.z, a.w};  // BF16 pairs, none negative: a1 > 0 is any bit set
                tc_ld_wait();
                float dz[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float v = (__uint_as_float(mid[i]) + __uint_as_float(lo[i])) + __uint_as_float(hi[i]);
                    dz[i] = (av[i >> 1] & (i & 1 ? 0xFFFF0000u : 0xFFFFu)) ? v : 0.f;
                }
                store_parts(smem + Bwd::DZ1 + g * GROUP + (p + ROW0) * 16, dz);
            }
        };
        if (!issuer)
#pragma unroll 1
            for (int tile = (t >> 5) == 4 ? 0 : r & 1; tile < min(tiles, (r & 1) + 1); tile++) backward1(tile);
        tc_publish();
        tc_before();
        if (__syncthreads_or(!ok)) break;
        if (issuer) {
            tc_after();
            const unsigned leader = tc_leader();
            issue_sum(d + Bwd::DW1, base + Bwd::DZ1 + ROW0 * 16, base + Bwd::T1 + ROW0 * 16, ksteps, leader);
            if (leader) tc_commit(bar_all);
            __syncwarp();
        }
        ok = mbar_wait(bar_all, phase, wait_ns);
        tc_after();
#pragma unroll
        for (int i = 0; i < 3; i++) {
            unsigned v[3][8];
#pragma unroll
            for (int e = 0; e < 3; e++) tc_ld8(at + Bwd::DW2 + 72 * r + 24 * i + 8 * e, v[e]);
            tc_ld_wait();
#pragma unroll
            for (int e = 0; e < 3; e++)
#pragma unroll
                for (int j = 0; j < 8; j++) gw2[24 * i + 8 * e + j] += __uint_as_float(v[e][j]);
        }
        if (r < 2) {  // warp-uniform: quarter 0 the sums with d3, quarter 1 those with xs
#pragma unroll
            for (int i = 0; i < 4; i++) {
                unsigned v[8];
                tc_ld8(at + (r ? Bwd::DW1 : Bwd::DW3) + 8 * i, v);
                tc_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (8 * i + j < SPLIT * kK) gk[(8 * i + j) % kK] += __uint_as_float(v[j]);
                    else if (8 * i + j == SPLIT * kK) gb += __uint_as_float(v[j]);
                }
            }
        }
        tc_before();
    }
    const bool gave_up = __syncthreads_or(!ok);
    if (gave_up) give_up(fin, &g_nn_err);
    tc_before();
    __syncthreads();
    tc_after();
    if (t < 32) tc_dealloc(d, Bwd::COLUMNS);
    if (gave_up) {
        for (int i = t; i < kNParam; i += Bwd::THREADS) atomicAdd(dparams + i, lost());
        return;
    }

    // dW2: the three parts' rows through shared memory (one float of padding per row), then one add per
    // parameter
    float *sum = reinterpret_cast<float *>(smem);
    constexpr int ROW = kK * kCh + 1;
    if (q < SPLIT)
#pragma unroll
        for (int i = 0; i < 72; i++) sum[(q * kCh + lane) * ROW + 72 * r + i] = gw2[i];
    __syncthreads();
    for (int i = t; i < kCh * kCh * kK; i += Bwd::THREADS) {
        const int c = i / (kCh * kK), ci = (i / kK) % kCh, k = i % kK;
        const float *e = sum + c * ROW + k * kCh + ci;
        atomicAdd(dparams + kW2 + i, e[0] + (e[kCh * ROW] + e[2 * kCh * ROW]));
    }
    if (r == 0) {  // lanes of quadrant 0: a2 channels; quadrants 1 .. 3: the parts of dz2
        if (q == 0) {
#pragma unroll
            for (int k = 0; k < kK; k++) atomicAdd(dparams + kW3 + lane * kK + k, gk[k]);
        } else {
            atomicAdd(dparams + kB2 + lane, gb);
        }
    } else if (r == 1 && q < SPLIT) {  // the parts of dz1
#pragma unroll
        for (int k = 0; k < kK; k++) atomicAdd(dparams + kW1 + lane * kK + k, gk[k]);
        atomicAdd(dparams + kB1 + lane, gb);
    }
    for (int o = 16; o; o >>= 1) gb3 += __shfl_xor_sync(0xFFFFFFFFu, gb3, o);
    if (lane == 0 && t >= 256) atomicAdd(dparams + kB3, gb3);
}

}  // namespace nn
}  // namespace fdk
