// Quantise-on-load: fp16 weights [N][K] -> unsigned codes as bit-planes (the layout abq_pack_int32 writes and the GEMM
// routes read) + fp16 scale + u8 zero point per output channel or per group of input features.
//
// Restates the min/max calibration of the reference's UniformAffineQuantizer (algorithm/quantize/quantizer.py:149-179,
// without learnable clipping) and its code rule (quantizer.py:111-132) in fp32:
//     asymmetric: scale = clamp((max - min) / L, 1e-5, 1e4),  L = 2^bits - 1 (2^bits for 1 and 2 bits, quantizer.py:170-171)
//                 zero  = rint(clamp(-min / scale, -1e4, 1e4))
//     symmetric:  scale = clamp(absmax / (2^(bits-1) - 1), 1e-5, 1e4),  zero = 2^(bits-1) - 1   (quantizer.py:163-167)
//     code = clamp(rint(x / scale) + zero, 0, 2^bits - 1)
// Two deliberate differences, both because `bits` planes hold the codes 0 .. 2^bits - 1 and nothing else: the reference
// lets 1- and 2-bit codes reach 2^bits (its "bit balance", quantizer.py:66-68) and lets the zero point leave the code
// range; here both are clamped into it.  Groups are contiguous runs of `group_size` input features (quantizer.py:116-119).
//
// One CTA per weight row, a thread per run of 32 features (64 bytes, four 16-byte loads; several runs where the row is long).
// What bounds it: the instructions per weight (a division, clamps, conversions and a byte insertion each).  So the range of a
// run is found on pairs of halves, and the quotient is a product with the scale's reciprocal, two values at a time, added to
// 1.5 * 2^23 + zero so that the rounded code is the sum's low half.  It is taken twice, with the reciprocal 2^-22 too
// small and too large: the division's result lies between the two products, so where both round to the same code it does
// too.  A run where they do not (a quotient close to the middle between two codes), or with values out of range of the
// 16-bit halves, is done again with the division: the codes are those of the rule above, always.
//   groups of 1, 2, 4 .. 32 runs: a group's range meets by shuffles, every value is read once
//   one group per row: the ranges meet in shared memory, the values are read again (from L1 / L2)
//   other group sizes: the run ranges stay in shared memory
#include <cuda_fp16.h>

#include "abq_common.cuh"
#include "abq_kernels.h"

namespace abq {

constexpr int kWquantThreads = 128;

__device__ __forceinline__ void load_run(const __half *row, int run, uint32_t (&v)[16])
{
    const uint4 *src = reinterpret_cast<const uint4 *>(row + (size_t)run * 32);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint4 q = __ldg(src + i);
        v[4 * i] = q.x;
        v[4 * i + 1] = q.y;
        v[4 * i + 2] = q.z;
        v[4 * i + 3] = q.w;
    }
}
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }

__device__ __forceinline__ void run_range(const uint32_t (&v)[16], float &lo, float &hi)
{
    __half2 l = as_half2(v[0]), h = l;
#pragma unroll
    for (int i = 1; i < 16; ++i) {
        l = __hmin2(l, as_half2(v[i]));
        h = __hmax2(h, as_half2(v[i]));
    }
    lo = fminf(__low2float(l), __high2float(l));
    hi = fmaxf(__low2float(h), __high2float(h));
}

template <int BITS>
__device__ __forceinline__ void range_to_params(float lo, float hi, int symmetric, float &scale, float &zero)
{
    const int qmax = (1 << BITS) - 1;
    const float levels = BITS <= 2 ? (float)(1 << BITS) : (float)qmax;
    if (symmetric) {
        scale = __fdiv_rn(fmaxf(fabsf(lo), fabsf(hi)), (float)((1 << (BITS - 1)) - 1));
        scale = fminf(fmaxf(scale, 1e-5f), 1e4f);
        zero = (float)((1 << (BITS - 1)) - 1);
    } else {
        scale = __fdiv_rn(__fsub_rn(hi, lo), levels);
        scale = fminf(fmaxf(scale, 1e-5f), 1e4f);
        zero = rintf(fminf(fmaxf(__fdiv_rn(-lo, scale), -1e4f), 1e4f));
        zero = fminf(fmaxf(zero, 0.f), (float)qmax);
    }
}

__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm volatile("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t pair_of(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

// The codes of a run as one word per plane; reach: largest magnitude among the values.
template <int BITS>
__device__ __forceinline__ void quantize_run(const uint32_t (&v)[16], const __half *src, float scale, float zero, float reach, uint32_t (&planes)[BITS])
{
    constexpr uint32_t kTop = ((1u << BITS) - 1u) * 0x00010001u;
    const float magic = 12582912.f + zero;
    const float inv = __frcp_rn(scale);
    const float low = __fmul_rn(inv, 1.f - 2.384185791015625e-7f), high = __fmul_rn(inv, 1.f + 2.384185791015625e-7f); // 2^-22
    const uint64_t low2 = pair_of(low, low), high2 = pair_of(high, high), magic2 = pair_of(magic, magic);
    uint32_t unsure = 0, r[8], c[16]; // c: two codes in 16-bit halves
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 x = __half22float2(as_half2(v[i]));
        const uint64_t x2 = pair_of(x.x, x.y);
        const uint64_t l = fma_pair(x2, low2, magic2), h = fma_pair(x2, high2, magic2);
        const uint32_t l0 = (uint32_t)l, l1 = (uint32_t)(l >> 32);
        unsure |= l0 ^ (uint32_t)h;
        unsure |= l1 ^ (uint32_t)(h >> 32);
        c[i] = __vimin_s16x2_relu(__byte_perm(l0, l1, 0x5410), kTop);
    }
    if (unsure == 0 && __fmul_rn(reach, inv) < 30000.f) { // (16-bit halves hold every code before it is clamped)
#pragma unroll
        for (int s = 0; s < 8; ++s) { // byte y of r[s] holds element 31 - 8y - s of the run
            const uint32_t sel = (s & 1) ? 0x0040u : 0x0062u;
            r[s] = __byte_perm(__byte_perm(c[(31 - s) >> 1], c[(23 - s) >> 1], sel), __byte_perm(c[(15 - s) >> 1], c[(7 - s) >> 1], sel), 0x5410);
        }
        bytes_to_planes<BITS>(r, planes);
    } else {
#pragma unroll
        for (int b = 0; b < BITS; ++b)
            planes[b] = 0;
#pragma unroll 1
        for (int j = 0; j < 32; ++j) { // rare: rolled up, values read again
            float q = __fadd_rn(rintf(__fdiv_rn(__half2float(src[j]), scale)), zero);
            q = fminf(fmaxf(q, 0.f), (float)((1 << BITS) - 1));
#pragma unroll
            for (int b = 0; b < BITS; ++b)
                planes[b] = (planes[b] << 1) | (((uint32_t)(int)q >> b) & 1u);
        }
    }
}

struct WquantArgs {
    const __half *w;
    uint32_t *planes;
    __half *scale;
    uint8_t *zero;
    int N, K, runs_per_group, symmetric;
};

// KIND 0: groups of 1, 2 .. 32 runs; 1: one group per row; 2: anything else
template <int BITS, int KIND>
__global__ void __launch_bounds__(kWquantThreads, 8) quantize_weights_kernel(const WquantArgs a)
{
    extern __shared__ float run_ranges[]; // KIND 2: [2][K / 32], minimum and maximum of every run of this row
    __shared__ float warp_ranges[2][kWquantThreads / 32];
    const int KW = a.K >> 5, rpg = a.runs_per_group;
    const int row = blockIdx.x;
    const __half *src = a.w + (size_t)row * a.K;
    const int groups = KIND == 1 ? 1 : KW / rpg;
    float scale = 0.f, zero = 0.f, reach = 0.f;
    if (KIND == 1) {
        float lo = __int_as_float(0x7fffffff), hi = lo; // NaN: any value takes its place
        for (int run = threadIdx.x; run < KW; run += kWquantThreads) {
            uint32_t v[16];
            load_run(src, run, v);
            float l, h;
            run_range(v, l, h);
            lo = fminf(lo, l);
            hi = fmaxf(hi, h);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if ((threadIdx.x & 31) == 0) {
            warp_ranges[0][threadIdx.x >> 5] = lo;
            warp_ranges[1][threadIdx.x >> 5] = hi;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kWquantThreads / 32; ++i) {
            lo = fminf(lo, warp_ranges[0][i]);
            hi = fmaxf(hi, warp_ranges[1][i]);
        }
        range_to_params<BITS>(lo, hi, a.symmetric, scale, zero);
        reach = fmaxf(fabsf(lo), fabsf(hi));
    } else if (KIND == 2) {
        for (int run = threadIdx.x; run < KW; run += kWquantThreads) {
            uint32_t v[16];
            load_run(src, run, v);
            run_range(v, run_ranges[run], run_ranges[KW + run]);
        }
        __syncthreads();
    }
    for (int base = threadIdx.x & ~31; base < KW; base += kWquantThreads) { // whole warps: shuffles inside
        const int run = base + (threadIdx.x & 31);
        const bool live = run < KW;
        uint32_t v[16];
        load_run(src, live ? run : KW - 1, v);
        const int grp = KIND == 1 ? 0 : run / rpg;
        if (KIND == 0) {
            float lo, hi;
            run_range(v, lo, hi);
            for (int o = 1; o < rpg; o <<= 1) {
                lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
            range_to_params<BITS>(lo, hi, a.symmetric, scale, zero);
            reach = fmaxf(fabsf(lo), fabsf(hi));
        }
        if (!live)
            continue;
        if (KIND == 2) {
            float lo = run_ranges[grp * rpg], hi = run_ranges[KW + grp * rpg];
            for (int j = 1; j < rpg; ++j) {
                lo = fminf(lo, run_ranges[grp * rpg + j]);
                hi = fmaxf(hi, run_ranges[KW + grp * rpg + j]);
            }
            range_to_params<BITS>(lo, hi, a.symmetric, scale, zero);
            reach = fmaxf(fabsf(lo), fabsf(hi));
        }
        uint32_t p[BITS];
        quantize_run<BITS>(v, src + (size_t)run * 32, scale, zero, reach, p);
#pragma unroll
        for (int b = 0; b < BITS; ++b)
            a.planes[((size_t)b * a.N + row) * KW + run] = p[b];
        if (KIND == 1 ? run == 0 : run % rpg == 0) {
            a.scale[(size_t)row * groups + grp] = __float2half_rn(scale);
            a.zero[(size_t)row * groups + grp] = (uint8_t)(int)zero;
        }
    }
}

template <int BITS>
static cudaError_t launch_wquant(const WquantArgs &a, cudaStream_t stream)
{
    const int KW = a.K / 32, rpg = a.runs_per_group;
    if (rpg <= 32 && (rpg & (rpg - 1)) == 0)
        quantize_weights_kernel<BITS, 0><<<a.N, kWquantThreads, 0, stream>>>(a);
    else if (rpg == KW)
        quantize_weights_kernel<BITS, 1><<<a.N, kWquantThreads, 0, stream>>>(a);
    else
        quantize_weights_kernel<BITS, 2><<<a.N, kWquantThreads, (size_t)KW * 8, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t quantize_weights(const __half *w, uint32_t *planes, __half *scale, uint8_t *zero, int N, int K, int bits, int group_size, int symmetric,
                             cudaStream_t stream)
{
    const WquantArgs a = { w, planes, scale, zero, N, K, (group_size > 0 ? group_size : K) / 32, symmetric };
    switch (bits) {
    case 1: return launch_wquant<1>(a, stream);
    case 2: return launch_wquant<2>(a, stream);
    case 3: return launch_wquant<3>(a, stream);
    case 4: return launch_wquant<4>(a, stream);
    case 5: return launch_wquant<5>(a, stream);
    case 6: return launch_wquant<6>(a, stream);
    case 7: return launch_wquant<7>(a, stream);
    case 8: return launch_wquant<8>(a, stream);
    }
    return cudaErrorInvalidValue;
}

} // namespace abq
