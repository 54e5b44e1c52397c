// Tensor-core GEMM that reads the weights as they are stored -- bit-planes -- and expands them inside the kernel
// (route ABQ_ROUTE_I8_UMMA).  The reference multiplies plane pairs with 1-bit MMAs and adds the shifted partial sums
// (engine/mma_any/aq_bmma_kernel.h:109-271, 485-580); here a CTA turns 128 rows x 128 features of the q weight planes into
// int8 codes in shared memory and ONE tcgen05.mma kind::i8 multiplies them, with the same int32 result.
//
// Orientation: the weight rows are the 128 lanes of the accumulator, the tokens its columns (BT = 16 .. 256 of them), so a
// small token count costs a narrow instruction instead of 128 padded rows, the scale and zero point of an epilogue thread are
// registers, and a warp's stores are 32 consecutive features of one token whatever N is.
//
// Roles of a CTA (one per SM, persistent):
//   warp 0      TMA of the activation codes (BT x 128 bytes per K block, 128B swizzle) into a ring of its own, deep enough for the
//               trip to L2 -- and of the weight codes, behind them in the same slot, when they come expanded (Q = 0)
//   warp 1      TMEM allocation; one thread issues the MMAs
//   warp 2      TMA of the weight planes, chunks of 512 (up to 4 bits) or 256 features x 128 rows x q planes, into a ring that
//               starts to fill before the wait on the previous kernel
//   E warps     expanders: groups of four warps (one weight row per thread) take K blocks in turn: q 16-byte loads, the
//               bit-matrix transposition of xbytes.cuh, zero point subtracted, eight 16-byte stores into the swizzled operand tile.
//               The features of a 32-run stay in the order the transposition leaves them; the activation codes are
//               written in the same order (prepare_x_kernel), so nothing is shuffled back
//   EW warps    epilogue: quarter of the lanes x a share of the columns each
// Work: tiles of 128 features x BT tokens.  Either whole tiles are dealt round-robin, or -- where that would leave SMs
// idle -- every CTA takes an equal run of K chunks (stream-K); the pieces of a tile then meet in global scratch: every
// epilogue warp stores its share, counts in on the tile's counter for that share, and the last one adds the pieces in CTA order
// and finishes the outputs.  Nobody waits for another CTA.
// Scale groups (GROUPED): every 64 or 128 features have an accumulator of their own; the epilogue warps drain two per hand-over into
// fp32 while the next two are multiplied.  An accumulator starts from the bits of 1.5 * 2^23 (2^23 for sums that cannot be
// negative), so what comes back is a float already: one packed subtraction and one packed multiply-add per two elements.
// Groups wider than 128 are summed as a whole in one int32 accumulator (beyond that start's bound) and converted once; K is then
// cut between groups only.
#pragma once
#include <cuda.h>
#include <cstring>

#include "abq_common.cuh"
#include "abq_kernels.h"
#include "umma.cuh"
#include "xbytes.cuh"

namespace abq {

struct TcArgs {
    int M, N;
    int bt;                 // tokens per tile
    int m_tiles, n_tiles;
    int k_blocks;           // K / 128
    int chunk_blocks;       // split: K blocks per piece of work (whole plane chunks and whole scale groups)
    int chunks_per_tile;    // ceil(k_blocks / chunk_blocks)
    int split;              // 0: whole tiles, round-robin; 1: equal runs of K chunks
    int range_q, range_r;   // split: chunks per CTA, the first range_r CTAs take one more
    int x_slots, a_slots, ring; // activation codes, expanded weight codes, plane chunks
    void *D;
    const __half *C;
    const __half *w_scale;
    const uint8_t *w_zero;
    const float *x_scale;
    const int *xpart;       // not null: code sums [K block][token]; the epilogue subtracts what the expanders left in the codes times them
    const __half *residual;
    int fold_zero;          // the expanders subtract w_zero (scale groups; widths up to three bits)
    int w_offset;           // signed weights of up to 7 bits: the planes are read as codes that are w_offset too large
    int out_dtype, scale_mode;
    int group_size, scale_groups;
    int magic;              // GROUPED: int -> float by adding a power of two (its bits as int, the same value as float)
    float magic_f;
    uint32_t idesc;
    int *counters;          // split: [tile][epilogue warp], zeroed by prepare_x_kernel
    int *partials;          // split: [CTA][first / last tile][epilogue warp][column][lane]
    int *status;
};

constexpr int kTcRows = 128;                       // weight rows per tile
constexpr int kTcABytes = kTcRows * 128;           // one K block of weight codes
constexpr int kTcRasterM = 16;                     // token tiles walked before the next weight tile
constexpr int kTcMaxX = 8, kTcMaxA = 6, kTcMaxRing = 8;
constexpr int kTcDone = 8;                         // barriers that the multiplied blocks report to in turn
constexpr int kTcBarriers = kTcMaxX + kTcMaxA + 2 * kTcMaxRing + kTcDone + 4;
__host__ __device__ constexpr int tc_chunk_blocks(int q) { return q == 0 ? 1 : (q <= 4 ? 4 : 2); }
__host__ __device__ constexpr int tc_chunk_bytes(int q) { return q * kTcRows * tc_chunk_blocks(q) * 16; }

// The pieces of work of one CTA, in order: the same sequence for every role.
struct TcSegment {
    int tile, m0, n0, k0, k1; // K blocks [k0, k1) of the tile at token m0, feature n0
};
struct TcWalk {
    int x, x1;
    __device__ __forceinline__ explicit TcWalk(const TcArgs &a)
    {
        const int c = blockIdx.x;
        if (a.split) {
            x = c * a.range_q + min(c, a.range_r);
            x1 = x + a.range_q + (c < a.range_r ? 1 : 0);
        } else {
            x = c;
            x1 = a.m_tiles * a.n_tiles;
        }
    }
    __device__ __forceinline__ bool next(const TcArgs &a, TcSegment &s)
    {
        if (x >= x1)
            return false;
        if (a.split) {
            s.tile = x / a.chunks_per_tile;
            const int c0 = x - s.tile * a.chunks_per_tile;
            const int c1 = min(a.chunks_per_tile, c0 + x1 - x);
            s.k0 = c0 * a.chunk_blocks;
            s.k1 = min(c1 * a.chunk_blocks, a.k_blocks);
            x += c1 - c0;
        } else {
            s.tile = x;
            s.k0 = 0;
            s.k1 = a.k_blocks;
            x += gridDim.x;
        }
        const int per_group = kTcRasterM * a.n_tiles;
        const int g = s.tile / per_group, r = s.tile - g * per_group;
        const int gm = min(kTcRasterM, a.m_tiles - g * kTcRasterM);
        const int n = r / gm;
        s.n0 = n * kTcRows;
        s.m0 = (g * kTcRasterM + r - n * gm) * a.bt;
        return true;
    }
};

// first scale group of K block kb
__device__ __forceinline__ int tc_group_of(const TcArgs &a, int kb)
{
    return a.group_size == 128 ? kb : a.group_size == 64 ? 2 * kb : kb * 128 / a.group_size;
}

// A wait whose outcome is the same in every lane (a lane that gave up must not leave the others at a warp barrier).
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, const TcArgs &a, int status_bit)
{
    return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, a.status, status_bit));
}

// ------------------------------------------------------------------------------------------------ expanders
// Order of the features inside a 32-run.  Widths up to three bits: the transposition stops at nibbles, and one byte permute
// per four codes looks the finished byte (code - zero) up in an eight-entry table, which leaves byte y of word 2 s + h
// with feature 31 - (16 h + 4 y + s).  Wider codes come out as bytes: byte y of word s holds feature 31 - 8 y - s.
// (Logic, shifts and permutes run at half rate: what the expansion costs is their number.)
__host__ __device__ constexpr bool tc_table_order(int q) { return q == 2 || q == 3; }

// One thread: Q x 16 bytes of planes (its weight row, 128 features) -> 128 code bytes of the swizzled operand row.
// sub: what is subtracted from every code, one value per 64 features (bytes); without SUB only the table widths do.
template <int Q, bool SUB>
__device__ __forceinline__ void tc_expand_row(const uint32_t (&w)[Q][4], uint8_t *row_base, int row, uint32_t flip, const uint32_t (&sub)[2])
{
    const uint32_t sw = (uint32_t)(row & 7);
    uint32_t table[2][2]; // [64 features][entries 0 .. 3, 4 .. 7]
    if constexpr (tc_table_order(Q)) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            table[h][0] = (0x83828180u - sub[h]) ^ 0x80808080u;
            table[h][1] = (0x87868584u - sub[h]) ^ 0x80808080u;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t p[Q], r[8];
#pragma unroll
        for (int b = 0; b < Q; ++b)
            p[b] = w[b][i];
        if (Q < 8)
            p[Q - 1] ^= flip; // two's complement -> offset codes
        if constexpr (tc_table_order(Q)) {
            uint32_t n[4];
            nibble_fields(p[0], p[1], Q > 2 ? p[Q > 2 ? 2 : 0] : 0u, 0u, false, n);
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                r[2 * s] = __byte_perm(table[i >> 1][0], table[i >> 1][1], n[s]); // (reads the low four nibbles)
                r[2 * s + 1] = __byte_perm(table[i >> 1][0], table[i >> 1][1], n[s] >> 16);
            }
        } else {
            x_bytes<Q>(p, false, r);
            if (SUB && Q < 8) { // both at most 127: the byte's top bit, set beforehand, absorbs the borrow
#pragma unroll
                for (int s = 0; s < 8; ++s)
                    r[s] = ((r[s] | 0x80808080u) - sub[i >> 1]) ^ 0x80808080u;
            }
        }
        *reinterpret_cast<uint4 *>(row_base + (((uint32_t)(2 * i) ^ sw) << 4)) = make_uint4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<uint4 *>(row_base + (((uint32_t)(2 * i + 1) ^ sw) << 4)) = make_uint4(r[4], r[5], r[6], r[7]);
    }
}

// ------------------------------------------------------------------------------------------------ epilogue pieces
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// What an epilogue thread knows about its weight row.
struct TcRow {
    int n;
    bool live;
    float scale;
    int zero;
    __half cscale;
};

// Output (m, row.n) from its exact int32 sum.  MODE 0: int32; 1: fp16 times one fp16 factor (the reference's arithmetic: the
// accumulator rounded to fp16, then an fp16 multiply); 2: channel scale, zero point, per-token scale
template <int MODE>
__device__ __forceinline__ void tc_store_int(const TcArgs &a, const TcRow &row, int m, int v)
{
    const size_t at = (size_t)m * a.N + row.n;
    if (MODE == 0) {
        reinterpret_cast<int *>(a.D)[at] = v;
        return;
    }
    __half h;
    if (MODE == 1) {
        h = __hmul_rn(__int2half_rn(v), row.cscale); // (_rn: never one instruction with the residual's add)
    } else {
        h = __float2half_rn((float)v * row.scale * (a.x_scale ? __ldg(a.x_scale + m) : 1.f));
    }
    if (a.residual)
        h = __hadd(h, a.residual[at]);
    reinterpret_cast<__half *>(a.D)[at] = h;
}
__device__ __forceinline__ void tc_store_float(const TcArgs &a, const TcRow &row, int m, float f)
{
    __half h = __float2half_rn(f * (a.x_scale ? __ldg(a.x_scale + m) : 1.f));
    const size_t at = (size_t)m * a.N + row.n;
    if (a.residual)
        h = __hadd(h, a.residual[at]);
    reinterpret_cast<__half *>(a.D)[at] = h;
}

// Pieces of a split tile: CTA range of the tile and the slot a CTA keeps its piece in.
struct TcPieces {
    int first, last; // CTAs
};
__device__ __forceinline__ int tc_cta_of(const TcArgs &a, int chunk)
{
    const int big = a.range_r * (a.range_q + 1);
    return chunk < big ? chunk / (a.range_q + 1) : a.range_r + (chunk - big) / a.range_q;
}
__device__ __forceinline__ int tc_first_chunk(const TcArgs &a, int cta) { return cta * a.range_q + min(cta, a.range_r); }
__device__ __forceinline__ TcPieces tc_pieces(const TcArgs &a, int tile)
{
    return TcPieces{ tc_cta_of(a, tile * a.chunks_per_tile), tc_cta_of(a, (tile + 1) * a.chunks_per_tile - 1) };
}
// a CTA cuts at most its first and its last tile: slot 0 and 1
__device__ __forceinline__ int *tc_slot(const TcArgs &a, int cta, int tile, int ew, int warps, int cols)
{
    const int which = tc_first_chunk(a, cta) / a.chunks_per_tile == tile ? 0 : 1;
    return a.partials + (((size_t)cta * 2 + which) * warps + ew) * cols * 32;
}

// Counts this warp's piece in; true for the warp whose piece was the last.  Every lane's stores are visible before the count.
__device__ __forceinline__ bool tc_count_in(const TcArgs &a, int tile, int ew, int warps, int pieces)
{
    __threadfence();
    __syncwarp();
    int old = 0;
    if ((threadIdx.x & 31) == 0)
        old = atomicAdd(a.counters + (size_t)tile * warps + ew, 1);
    old = __shfl_sync(0xffffffffu, old, 0);
    __threadfence();
    return old == pieces - 1;
}

// Eight columns of this warp's share, all pieces added in K order (the same sum whichever warp comes last); four pieces' loads are in
// flight at a time.
template <typename T>
__device__ __forceinline__ void tc_add_pieces(const TcArgs &a, int tile, const TcPieces &pc, int ew, int warps, int cols, int c, int lane, T (&v)[8])
{
#pragma unroll
    for (int j = 0; j < 8; ++j)
        v[j] = 0;
    for (int cta = pc.first; cta <= pc.last; cta += 4) {
        T part[4][8];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const T *p = reinterpret_cast<const T *>(tc_slot(a, min(cta + u, pc.last), tile, ew, warps, cols)) + c * 32 + lane;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                part[u][j] = cta + u <= pc.last ? __ldcg(p + j * 32) : (T)0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                v[j] += part[u][j];
    }
}

// One share (cols columns from column c0 on) of a finished int32 accumulator.
// sums: this warp's token sums of the segment (shared memory), or null.
template <int MODE>
__device__ __forceinline__ void tc_epilogue_int(const TcArgs &a, const TcSegment &s, const TcRow &row, uint32_t taddr, int c0, int cols, int ew,
                                                int warps, const int *sums)
{
    constexpr int CH = 16;
    const int lane = threadIdx.x & 31;
    const bool whole = s.k0 == 0 && s.k1 == a.k_blocks;
    const int live = min(cols, a.M - s.m0 - c0); // columns that hold tokens
    if (whole) {
        for (int c = 0; c < live; c += CH) {
            int v[CH];
            tmem_ld16_nowait(taddr + c, v);
            tmem_ld_wait();
            if (sums) {
#pragma unroll
                for (int j = 0; j < CH; ++j)
                    v[j] -= row.zero * sums[c + j];
            }
            if (row.live) {
#pragma unroll
                for (int j = 0; j < CH; ++j)
                    if (c + j < live)
                        tc_store_int<MODE>(a, row, s.m0 + c0 + c + j, v[j]);
            }
        }
        return;
    }
    int *own = tc_slot(a, blockIdx.x, s.tile, ew, warps, cols) + lane;
    for (int c = 0; c < live; c += CH) {
        int v[CH];
        tmem_ld16_nowait(taddr + c, v);
        tmem_ld_wait();
        if (sums) {
#pragma unroll
            for (int j = 0; j < CH; ++j)
                v[j] -= row.zero * sums[c + j];
        }
#pragma unroll
        for (int j = 0; j < CH; ++j)
            __stcg(own + (c + j) * 32, v[j]);
    }
    const TcPieces pc = tc_pieces(a, s.tile);
    if (!tc_count_in(a, s.tile, ew, warps, pc.last - pc.first + 1))
        return;
    for (int c = 0; c < live; c += 8) {
        int v[8];
        tc_add_pieces<int>(a, s.tile, pc, ew, warps, cols, c, lane, v);
        if (row.live) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (c + j < live)
                    tc_store_int<MODE>(a, row, s.m0 + c0 + c + j, v[j]);
        }
    }
}

template <int COLS>
__device__ __forceinline__ void tc_epilogue_float(const TcArgs &a, const TcSegment &s, const TcRow &row, const uint64_t (&facc)[COLS / 2], int c0, int ew,
                                                  int warps)
{
    const int lane = threadIdx.x & 31;
    const int live = min(COLS, a.M - s.m0 - c0);
    if (s.k0 == 0 && s.k1 == a.k_blocks) {
        if (row.live) {
#pragma unroll
            for (int j = 0; j < COLS; j += 2) {
                float lo, hi;
                unpack2(facc[j / 2], lo, hi);
                if (j < live)
                    tc_store_float(a, row, s.m0 + c0 + j, lo);
                if (j + 1 < live)
                    tc_store_float(a, row, s.m0 + c0 + j + 1, hi);
            }
        }
        return;
    }
    float *own = reinterpret_cast<float *>(tc_slot(a, blockIdx.x, s.tile, ew, warps, COLS)) + lane;
#pragma unroll
    for (int j = 0; j < COLS; j += 2) {
        float lo, hi;
        unpack2(facc[j / 2], lo, hi);
        __stcg(own + j * 32, lo);
        __stcg(own + (j + 1) * 32, hi);
    }
    const TcPieces pc = tc_pieces(a, s.tile);
    if (!tc_count_in(a, s.tile, ew, warps, pc.last - pc.first + 1))
        return;
    for (int c = 0; c < live; c += 8) {
        float v[8];
        tc_add_pieces<float>(a, s.tile, pc, ew, warps, COLS, c, lane, v);
        if (row.live) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (c + j < live)
                    tc_store_float(a, row, s.m0 + c0 + c + j, v[j]);
        }
    }
}

// facc[0 .. 16) += scale * (the sums v), whole numbers
__device__ __forceinline__ void tc_scale_add_int(const int (&v)[16], uint64_t scale2, uint64_t *facc)
{
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
        const uint64_t t = pack2(__float_as_uint(__int2float_rn(v[j])), __float_as_uint(__int2float_rn(v[j + 1])));
        facc[j / 2] = fma2(t, scale2, facc[j / 2]);
    }
}
// facc[0 .. 16) += scale * (the sums v): v are accumulators that started from the bits of a power of two, i.e. read as floats they
// are that power plus the sum
__device__ __forceinline__ void tc_scale_add(const int (&v)[16], uint64_t minus_magic2, uint64_t scale2, uint64_t *facc)
{
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
        const uint64_t t = add2(pack2((uint32_t)v[j], (uint32_t)v[j + 1]), minus_magic2);
        facc[j / 2] = fma2(t, scale2, facc[j / 2]);
    }
}

// ------------------------------------------------------------------------------------------------ the kernel
// Q: weight planes (0: the weights come as codes, tmap_w is a byte map like tmap_x).  COLS: columns per epilogue warp with scale
// groups, 0 without.  E, EW: expander and epilogue warps (multiples of 4).
template <int Q, int COLS, int E, int EW>
__global__ void __launch_bounds__((4 + E + EW) * 32, 1)
    tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const TcArgs a)
{
    constexpr bool GROUPED = COLS > 0;
    constexpr int CK = tc_chunk_blocks(Q);
    constexpr int kChunkBytes = tc_chunk_bytes(Q);
    constexpr int kGroups = E / 4 > 0 ? E / 4 : 1;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int x_bytes_slot = a.bt * 128 + (Q > 0 ? 0 : kTcABytes);
    uint8_t *a_ring = smem + (size_t)a.x_slots * x_bytes_slot;
    uint8_t *ring = a_ring + (size_t)a.a_slots * kTcABytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(ring + (size_t)a.ring * kChunkBytes);
    // done[j % kTcDone]: block j of this CTA has been multiplied, i.e. its slots are free and, with scale groups, its accumulator is
    // complete.  One commit per block and one set of barriers for all who wait, at any distance up to kTcDone blocks: a second
    // commit behind the same MMAs holds the issuing thread up until the first has been carried out (about 400 clocks).
    uint64_t *xfull = bars, *afull = xfull + kTcMaxX, *pfull = afull + kTcMaxA, *pempty = pfull + kTcMaxRing, *done = pempty + kTcMaxRing;
    uint64_t *acc_full = done + kTcDone, *acc_empty = acc_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    int *xsums = reinterpret_cast<int *>(bars + kTcBarriers + 2); // [epilogue warp][128], without scale groups
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tmem_cols = (uint32_t)max(32, (GROUPED ? 4 : 2) * a.bt);

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.x_slots; ++s)
            mbar_init(&xfull[s], 1);
        for (int s = 0; s < a.a_slots; ++s)
            mbar_init(&afull[s], 4); // the four warps that expand the block
        for (int s = 0; s < kTcDone; ++s)
            mbar_init(&done[s], 1);
        for (int s = 0; s < a.ring; ++s) {
            mbar_init(&pfull[s], 1);
            mbar_init(&pempty[s], E > 0 ? E : 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], EW);
        }
        fence_mbar_init();
        prefetch_tmap(&tmap_w);
        prefetch_tmap(&tmap_x);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (!(Q > 0 && warp == 2))
        pdl_wait_prior_grid(); // everything but the weight planes comes from (or goes to) what earlier kernels touch

    TcWalk walk(a);
    TcSegment sg;
    bool ok = true;
    if (warp == 0) {
        if (elect_one()) {
            int s = 0, free_at = -a.x_slots; // the block whose end frees the slot
            while (ok && walk.next(a, sg)) {
                for (int kb = sg.k0; kb < sg.k1; ++kb, ++free_at) {
                    if (free_at >= 0)
                        ok = mbar_wait_bounded(&done[free_at % kTcDone], (free_at / kTcDone) & 1, a.status, STATUS_TIMEOUT_PIPE);
                    if (!ok)
                        break;
                    uint8_t *sx = smem + (size_t)s * x_bytes_slot;
                    mbar_arrive_expect_tx(&xfull[s], (uint32_t)x_bytes_slot);
                    tma_load_2d(sx, &tmap_x, kb * 128, sg.m0, &xfull[s]);
                    if (Q == 0)
                        tma_load_2d(sx + a.bt * 128, &tmap_w, kb * 128, sg.n0, &xfull[s]);
                    if (++s == a.x_slots)
                        s = 0;
                }
            }
            // Every copy has landed before the block ends: after a wait that ran out nobody else may be waiting for them.
            for (int i = max(free_at, 0); i < free_at + a.x_slots; ++i)
                mbar_wait_bounded(&xfull[i % a.x_slots], (i / a.x_slots) & 1, a.status, STATUS_TIMEOUT_TMA);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            int s = 0, ph = 0, c = 0, cph = 0, unit = 0, j = 0;
            // (addresses in the descriptors' 16-byte units: this thread's instructions are on the critical path of every block)
            const uint64_t desc0 = make_smem_desc_sw128(0);
            const uint32_t x_base = smem_u32(smem) >> 4, a_base = smem_u32(a_ring) >> 4, x_step = (uint32_t)x_bytes_slot >> 4;
            const int wide = GROUPED && a.group_size > 128 ? a.group_size >> 7 : 0; // K blocks per group, 0: groups of at most one block
            int open = 0;                                                           // wide: blocks that the open group still misses
            while (ok && walk.next(a, sg)) {
                int b = 0;
                uint32_t acc = 0;
                for (int kb = sg.k0; ok && kb < sg.k1; ++kb) {
                    // ungrouped: one accumulator per tile; grouped: two per hand-over (two 64-feature groups of a K block,
                    // or two K blocks), or one per wide group
                    const bool fresh = !GROUPED ? kb == sg.k0 : wide ? open == 0 : a.group_size == 64 || ((kb - sg.k0) & 1) == 0;
                    if (fresh) {
                        open = wide; // (a segment holds whole groups)
                        b = unit & 1;
                        // (grouped: the epilogue hands the accumulators over with the starting value in them, the first time too)
                        ok = mbar_wait_bounded(&acc_empty[b], ((unit >> 1) & 1) ^ (GROUPED ? 0 : 1), a.status, STATUS_TIMEOUT_PIPE);
                        if (!ok)
                            break;
                        ++unit;
                        acc = tmem_base + (uint32_t)(b * (GROUPED ? 2 : 1) * a.bt);
                    }
                    ok = mbar_wait_bounded(&xfull[s], ph, a.status, STATUS_TIMEOUT_TMA);
                    if (Q > 0)
                        ok = ok && mbar_wait_bounded(&afull[c], cph, a.status, STATUS_TIMEOUT_PIPE);
                    if (!ok)
                        break;
                    tmem_fence_after();
                    const uint32_t sx = x_base + s * x_step;
                    const uint64_t db = desc0 + sx, da = desc0 + (Q > 0 ? a_base + c * (kTcABytes >> 4) : sx + a.bt * 8);
                    if (!GROUPED || wide) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_i8(acc, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), a.idesc, !(fresh && k == 0));
                        if (GROUPED ? --open == 0 : kb + 1 == sg.k1)
                            umma_commit(&acc_full[b]);
                    } else if (a.group_size == 64) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_i8(acc + (uint32_t)((k >> 1) * a.bt), da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), a.idesc, 1);
                    } else {
                        const int half = (kb - sg.k0) & 1;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_i8(acc + (uint32_t)(half * a.bt), da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), a.idesc, 1);
                    }
                    umma_commit(&done[j % kTcDone]);
                    ++j;
                    if (Q > 0 && ++c == a.a_slots) {
                        c = 0;
                        cph ^= 1;
                    }
                    if (++s == a.x_slots) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            if (j > 0) // nothing still multiplies, and the last commit has arrived, before the block ends
                mbar_wait_bounded(&done[(j - 1) % kTcDone], ((j - 1) / kTcDone) & 1, a.status, STATUS_TIMEOUT_MMA);
        }
        __syncwarp();
    } else if (warp == 2) {
        if (Q > 0 && elect_one()) {
            int s = 0, ph = 1, n = 0;
            while (ok && walk.next(a, sg)) {
                for (int kb = sg.k0; kb < sg.k1; kb += CK) {
                    ok = mbar_wait_bounded(&pempty[s], ph, a.status, STATUS_TIMEOUT_PIPE);
                    if (!ok)
                        break;
                    mbar_arrive_expect_tx(&pfull[s], kChunkBytes);
                    tma_load_3d(ring + (size_t)s * kChunkBytes, &tmap_w, kb * 4, sg.n0, 0, &pfull[s]);
                    ++n;
                    if (++s == a.ring) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            for (int i = max(n - a.ring, 0); i < n; ++i)
                mbar_wait_bounded(&pfull[i % a.ring], (i / a.ring) & 1, a.status, STATUS_TIMEOUT_TMA);
        }
        __syncwarp();
    } else if (E > 0 && warp >= 4 && warp < 4 + E) {
        if constexpr (Q > 0) {
            const int group = (warp - 4) >> 2;
            const int row = ((warp & 3) << 5) + lane; // of the tile
            const uint32_t flip = a.w_offset ? 0xffffffffu : 0u;
            const uint32_t row_swz = CK == 4 ? (uint32_t)((row >> 1) & 3) : (uint32_t)((row >> 2) & 1);
            int turn = 0, s = 0, free_at = -a.a_slots, c = 0, cph = 0; // whose block it is, its slot, the block whose end frees that, the chunk
            while (ok && walk.next(a, sg)) {
                const int n = sg.n0 + row;
                uint32_t sub[2] = { 0x01010101u * (uint32_t)a.w_offset, 0x01010101u * (uint32_t)a.w_offset };
                const uint8_t *zrow = a.w_zero + (size_t)(n < a.N ? n : 0) * (GROUPED ? a.scale_groups : 1);
                uint32_t z0 = 0, z1 = 0; // GROUPED: zero points of this group's next block
                auto fetch_zero = [&](int kb) {
                    if (GROUPED && a.fold_zero) {
                        const int g = tc_group_of(a, min(kb, sg.k1 - 1));
                        z0 = zrow[g];
                        z1 = a.group_size == 64 ? zrow[g + 1] : z0;
                    }
                };
                if (!GROUPED && a.fold_zero)
                    sub[0] = sub[1] = 0x01010101u * zrow[0]; // (the table widths)
                fetch_zero(sg.k0 + (group >= turn ? group - turn : group - turn + kGroups));
                for (int kb0 = sg.k0; ok && kb0 < sg.k1; kb0 += CK) {
                    const int nk = min(CK, sg.k1 - kb0);
                    ok = tc_wait(&pfull[c], cph, a, STATUS_TIMEOUT_TMA);
                    const uint8_t *chunk = ring + (size_t)c * kChunkBytes + row * (CK * 16);
                    for (int i = 0; ok && i < nk; ++i) {
                        if (turn == group) {
                            uint32_t w[Q > 0 ? Q : 1][4];
#pragma unroll
                            for (int b = 0; b < Q; ++b) {
                                const uint4 v = *reinterpret_cast<const uint4 *>(chunk + b * (kTcRows * CK * 16) + (((uint32_t)i ^ row_swz) << 4));
                                w[b][0] = v.x;
                                w[b][1] = v.y;
                                w[b][2] = v.z;
                                w[b][3] = v.w;
                            }
                            if (GROUPED && a.fold_zero) {
                                sub[0] = 0x01010101u * z0;
                                sub[1] = 0x01010101u * z1;
                                fetch_zero(kb0 + i + kGroups);
                            }
                            if (free_at >= 0)
                                ok = tc_wait(&done[free_at % kTcDone], (free_at / kTcDone) & 1, a, STATUS_TIMEOUT_PIPE);
                            if (ok) {
                                tc_expand_row<Q, GROUPED>(w, a_ring + (size_t)s * kTcABytes + row * 128, row, flip, sub);
                                fence_proxy_async(); // the stores above, before the tensor core reads them
                                __syncwarp();
                                if (lane == 0)
                                    mbar_arrive(&afull[s]);
                            }
                        }
                        ++free_at;
                        if (++turn == kGroups)
                            turn = 0;
                        if (++s == a.a_slots)
                            s = 0;
                    }
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(&pempty[c]);
                    if (++c == a.ring) {
                        c = 0;
                        cph ^= 1;
                    }
                }
            }
        }
    } else if (warp >= 4 + E) {
        const int ew = warp - 4 - E;
        const int quarter = warp & 3; // the TMEM lanes a warp may read
        const int share = ew >> 2;    // which share of the columns
        const uint32_t tlane = tmem_base + ((uint32_t)(quarter * 32) << 16);
        int unit = 0, j = 0; // accumulators (pairs of them with scale groups) and blocks so far
        if constexpr (GROUPED) {
            for (int acc = 0; acc < 4; ++acc)
#pragma unroll
                for (int c = 0; c < COLS; c += 16)
                    tmem_st16(tlane + (uint32_t)(acc * a.bt + share * COLS + c), a.magic);
            tmem_st_wait();
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&acc_empty[0]);
                mbar_arrive(&acc_empty[1]);
            }
        }
        while (ok && walk.next(a, sg)) {
            TcRow row;
            row.n = sg.n0 + quarter * 32 + lane;
            row.live = row.n < a.N;
            row.scale = 1.f;
            row.zero = 0;
            row.cscale = __half();
            if constexpr (!GROUPED) {
                row.zero = tc_table_order(Q) ? 0 : a.w_offset; // (what the expanders have not subtracted)
                if (a.out_dtype != ABQ_OUT_INT32) {
                    if (a.scale_mode == ABQ_SCALE_TENSOR_COMPAT)
                        row.cscale = ld_half(a.C);
                    else if (row.live) {
                        row.scale = __half2float(ld_half(a.w_scale + row.n));
                        if (a.xpart && a.w_zero)
                            row.zero += a.w_zero[row.n];
                    }
                }
                const int cols = a.bt / (EW / 4);
                int *sums = nullptr;
                if (a.xpart) { // while the tile is being multiplied
                    sums = xsums + ew * 128;
                    __syncwarp();
                    for (int c = lane; c < cols; c += 32) {
                        const int m = sg.m0 + share * cols + c;
                        int v = 0;
                        if (m < a.M) {
#pragma unroll 8
                            for (int kb = sg.k0; kb < sg.k1; ++kb)
                                v += __ldg(a.xpart + (size_t)kb * a.M + m);
                        }
                        sums[c] = v;
                    }
                    __syncwarp();
                }
                const int b = unit & 1;
                ok = tc_wait(&acc_full[b], (unit >> 1) & 1, a, STATUS_TIMEOUT_MMA);
                if (!ok)
                    break;
                ++unit;
                tmem_fence_after();
                const uint32_t taddr = tlane + (uint32_t)(b * a.bt + share * cols);
                if (a.out_dtype == ABQ_OUT_INT32)
                    tc_epilogue_int<0>(a, sg, row, taddr, share * cols, cols, ew, EW, sums);
                else if (a.scale_mode == ABQ_SCALE_TENSOR_COMPAT)
                    tc_epilogue_int<1>(a, sg, row, taddr, share * cols, cols, ew, EW, sums);
                else
                    tc_epilogue_int<2>(a, sg, row, taddr, share * cols, cols, ew, EW, sums);
                tmem_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(&acc_empty[b]);
            } else {
                constexpr int CH = 16;
                constexpr int NCH = COLS / CH;
                uint64_t facc[COLS / 2];
#pragma unroll
                for (int j = 0; j < COLS / 2; ++j)
                    facc[j] = 0;
                const bool g64 = a.group_size == 64;
                const uint64_t minus2 = pack2(__float_as_uint(-a.magic_f), __float_as_uint(-a.magic_f));
                const __half *srow = a.w_scale + (size_t)(row.live ? row.n : 0) * a.scale_groups;
                // groups of 64: an even number of them per row, so a K block's two lie in one word -- where the array starts on one
                // (a caller's view into a larger fp16 buffer need not)
                const bool scale_words = (reinterpret_cast<uintptr_t>(a.w_scale) & 3) == 0;
                const int units = a.group_size > 128 ? 0 : g64 ? sg.k1 - sg.k0 : (sg.k1 - sg.k0 + 1) >> 1;
                for (int kb = sg.k0; a.group_size > 128 && kb < sg.k1; kb += a.group_size >> 7, ++unit) {
                    const int b = unit & 1;
                    const uint32_t u0 = __float_as_uint(__half2float(ld_half(srow + tc_group_of(a, kb))));
                    ok = tc_wait(&acc_full[b], (unit >> 1) & 1, a, STATUS_TIMEOUT_MMA);
                    if (!ok)
                        break;
                    tmem_fence_after();
                    const uint32_t taddr = tlane + (uint32_t)(2 * b * a.bt + share * COLS);
#pragma unroll
                    for (int i = 0; i < NCH; ++i) {
                        int v[CH];
                        tmem_ld16_nowait(taddr + (uint32_t)(i * CH), v);
                        tmem_ld_wait();
                        tc_scale_add_int(v, pack2(u0, u0), facc + i * (CH / 2));
                    }
                    tmem_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(&acc_empty[b]);
                }
                // the scale group of accumulator h of unit u (groups of at most a K block)
                auto group_of = [&](int u, int h) { return tc_group_of(a, min(sg.k0 + 2 * u + h, sg.k1 - 1)); };
                auto fetch = [&](int u) -> __half2 {
                    if (g64 && scale_words)
                        return *reinterpret_cast<const __half2 *>(srow + 2 * (sg.k0 + u));
                    const int g0 = g64 ? 2 * (sg.k0 + u) : group_of(u, 0), g1 = g64 ? g0 + 1 : group_of(u, 1);
                    return __halves2half2(ld_half(srow + g0), ld_half(srow + g1));
                };
                __half2 scales = fetch(0);
                for (int u = 0; u < units; ++u, ++unit) {
                    const int b = unit & 1;
                    const uint32_t u0 = __float_as_uint(__low2float(scales)), u1 = __float_as_uint(__high2float(scales));
                    const uint64_t sc[2] = { pack2(u0, u0), pack2(u1, u1) };
                    if (u + 1 < units) // the next unit's scales travel while this one is drained
                        scales = fetch(u + 1);
                    const bool two = g64 || sg.k0 + 2 * u + 1 < sg.k1;
                    j += g64 || !two ? 1 : 2;
                    ok = tc_wait(&done[(j - 1) % kTcDone], ((j - 1) / kTcDone) & 1, a, STATUS_TIMEOUT_MMA); // the unit's last block
                    if (!ok)
                        break;
                    tmem_fence_after();
                    const uint32_t taddr = tlane + (uint32_t)(2 * b * a.bt + share * COLS);
                    int v[2][CH];
                    tmem_ld16_nowait(taddr, v[0]);
#pragma unroll
                    for (int i = 0; i < 2 * NCH; ++i) {
                        if (i >= NCH && !two)
                            break;
                        tmem_ld_wait();
                        const bool more = i + 1 < NCH || (i + 1 < 2 * NCH && two);
                        if (more)
                            tmem_ld16_nowait(taddr + (uint32_t)(((i + 1) / NCH) * a.bt + ((i + 1) % NCH) * CH), v[(i + 1) & 1]);
                        tmem_st16(taddr + (uint32_t)((i / NCH) * a.bt + (i % NCH) * CH), a.magic); // the next group's starting value
                        if (!more) { // everything of this unit sits in registers: the accumulators go back
                            tmem_st_wait();
                            tmem_fence_before();
                            __syncwarp();
                            if (lane == 0)
                                mbar_arrive(&acc_empty[b]);
                        }
                        tc_scale_add(v[i & 1], minus2, sc[i / NCH], facc + (i % NCH) * (CH / 2));
                    }
                }
                if (ok)
                    tc_epilogue_float<COLS>(a, sg, row, facc, share * COLS, ew, EW);
            }
        }
    }

    tmem_fence_before();
    __syncthreads();
    if (warp == 1) {
        tmem_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------ launch
template <int Q, int COLS, int E, int EW>
cudaError_t tc_launch_one(const CUtensorMap &tw, const CUtensorMap &tx, const TcArgs &a, unsigned grid, size_t smem, cudaStream_t stream)
{
    static thread_local SmemOptIn opted;
    cudaError_t e = opted.ensure(tc_kernel<Q, COLS, E, EW>, smem);
    if (e != cudaSuccess)
        return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((4 + E + EW) * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, tc_kernel<Q, COLS, E, EW>, tw, tx, a);
}

// Warps of a launch.  The expansion of a block is one long dependent sequence per thread, so what it needs is warps: as many as the
// registers allow beside the epilogue (whose sums take 32 registers with scale groups; without them eight warps store the columns of a
// tile twice as fast as four).  Over planes, tiles with scale groups end at 64 tokens: 128 would leave four warps for the expansion.
struct TcWarps {
    int expand, epilogue;
};
__host__ __device__ constexpr TcWarps tc_warps(int q, bool grouped, int bt)
{
    return q == 0 ? TcWarps{ 0, 16 } : !grouped ? TcWarps{ 12, 8 } : bt <= 16 ? TcWarps{ 16, 4 } : bt <= 32 ? TcWarps{ 12, 4 } : TcWarps{ 8, 8 };
}

template <int Q, int BT>
cudaError_t tc_launch_grouped(const CUtensorMap &tw, const CUtensorMap &tx, const TcArgs &a, unsigned grid, size_t smem, cudaStream_t stream)
{
    constexpr TcWarps W = tc_warps(Q, true, BT);
    return tc_launch_one<Q, BT * 4 / W.epilogue, W.expand, W.epilogue>(tw, tx, a, grid, smem, stream);
}

template <int Q>
cudaError_t tc_launch_width(const CUtensorMap &tw, const CUtensorMap &tx, const TcArgs &a, bool grouped, unsigned grid, size_t smem, cudaStream_t stream)
{
    if constexpr (Q == 0) {
        return grouped ? tc_launch_grouped<0, 128>(tw, tx, a, grid, smem, stream) : cudaErrorInvalidValue;
    } else {
        if (!grouped) {
            constexpr TcWarps W = tc_warps(Q, false, 0);
            return tc_launch_one<Q, 0, W.expand, W.epilogue>(tw, tx, a, grid, smem, stream);
        }
        switch (a.bt) {
        case 16: return tc_launch_grouped<Q, 16>(tw, tx, a, grid, smem, stream);
        case 32: return tc_launch_grouped<Q, 32>(tw, tx, a, grid, smem, stream);
        case 64: return tc_launch_grouped<Q, 64>(tw, tx, a, grid, smem, stream);
        }
        return cudaErrorInvalidValue;
    }
}

#define ABQ_TC_DECLARE(Q) cudaError_t tc_launch_w##Q(const CUtensorMap &, const CUtensorMap &, const TcArgs &, bool, unsigned, size_t, cudaStream_t);
ABQ_TC_DECLARE(0)
ABQ_TC_DECLARE(1)
ABQ_TC_DECLARE(2)
ABQ_TC_DECLARE(3)
ABQ_TC_DECLARE(4)
ABQ_TC_DECLARE(5)
ABQ_TC_DECLARE(6)
ABQ_TC_DECLARE(7)
ABQ_TC_DECLARE(8)

} // namespace abq
