// Tensor-core GEMM over weight planes (gemm_tc.cuh): planner, activation codes and launch entry.
#include "gemm_tc.cuh"

namespace abq {

// ------------------------------------------------------------------------------------------ activation codes
// Activation planes (or fp16 activations with the wrapper's static quantiser) -> int8 codes [M][K], inside a run of 32 features in
// the order in which tc_kernel expands the weights (tc_table_order); one run per thread.  On request also the code sums per
// token and K block.  Also clears the GEMM's arrival counters: this kernel runs completely before the GEMM touches them.
struct PrepareXArgs {
    const uint32_t *X;
    const float *qscale; // not null: X is fp16
    uint4 *out;
    long runs, plane_words;
    int bits, is_signed;
    int table_order;
    int *xpart; // [K / 128][M] or null
    int M, kw;  // kw = K / 32
    int *counters;
    int n_counters;
};

template <int P>
__device__ __forceinline__ void prepare_x_planes(const PrepareXArgs &a, long idx, uint32_t (&r)[8])
{
    uint32_t p[P];
#pragma unroll
    for (int b = 0; b < P; ++b)
        p[b] = __ldg(a.X + (long)b * a.plane_words + idx);
    x_bytes<P>(p, a.is_signed != 0, r);
}

__global__ void __launch_bounds__(128) prepare_x_kernel(const PrepareXArgs a)
{
    pdl_launch_dependents();
    pdl_wait_prior_grid();
    const long idx = (long)blockIdx.x * 128 + threadIdx.x;
    if (idx < a.n_counters)
        a.counters[idx] = 0;
    if (idx >= a.runs) // (a multiple of four: the lanes of a K block leave together)
        return;
    uint32_t r[8];
    if (a.qscale) {
        x_bytes_from_half(reinterpret_cast<const uint4 *>(a.X) + idx * 4, __float2half(__ldg(a.qscale)), a.bits, r);
    } else {
        switch (a.bits) {
        case 1: prepare_x_planes<1>(a, idx, r); break;
        case 2: prepare_x_planes<2>(a, idx, r); break;
        case 3: prepare_x_planes<3>(a, idx, r); break;
        case 4: prepare_x_planes<4>(a, idx, r); break;
        case 5: prepare_x_planes<5>(a, idx, r); break;
        case 6: prepare_x_planes<6>(a, idx, r); break;
        case 7: prepare_x_planes<7>(a, idx, r); break;
        default: prepare_x_planes<8>(a, idx, r); break;
        }
    }
    if (a.xpart) {
        int sum = 0;
        unsigned usum = 0;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            sum = __dp4a((int)r[s], 0x01010101, sum);
            usum = __dp4a(r[s], 0x01010101u, usum);
        }
        sum = a.is_signed ? sum : (int)usum;
        const uint32_t lanes = 0xfu << (threadIdx.x & 28);
        sum += __shfl_xor_sync(lanes, sum, 1);
        sum += __shfl_xor_sync(lanes, sum, 2);
        if ((idx & 3) == 0) {
            const long m = idx / a.kw;
            a.xpart[((idx - m * a.kw) >> 2) * a.M + m] = sum;
        }
    }
    if (a.table_order) { // byte y of word s = position 8 y + s -> byte y of word 2 s + h = position 16 h + 4 y + s
        uint32_t t[8];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            t[2 * s] = __byte_perm(r[s], r[s + 4], 0x5140);
            t[2 * s + 1] = __byte_perm(r[s], r[s + 4], 0x7362);
        }
#pragma unroll
        for (int s = 0; s < 8; ++s)
            r[s] = t[s];
    }
    a.out[2 * idx] = make_uint4(r[0], r[1], r[2], r[3]);
    a.out[2 * idx + 1] = make_uint4(r[4], r[5], r[6], r[7]);
}

// ------------------------------------------------------------------------------------------ planner
namespace {

struct TcPlan {
    int q, bt, m_tiles, n_tiles, k_blocks, chunk_blocks, chunks_per_tile, split, ctas, x_slots, a_slots, ring;
    int xpart; // the epilogue needs the token sums
    unsigned long long off_x, off_xpart, off_counters, off_partials;
};
static_assert(sizeof(TcPlan) <= sizeof(abq_gemm_state().tmap[2]), "plan words");

constexpr int kTcPlanes = 3, kTcCodes = 4; // tile[2] of a plan: which form of the kernel (0 and 2: umma_kernel, umma2_kernel)
constexpr size_t kTcSmem = 222 * 1024;

size_t tc_smem(int q, int bt, int x_slots, int a_slots, int ring)
{
    return 1024 + (size_t)x_slots * (bt * 128 + (q == 0 ? kTcABytes : 0)) + (size_t)a_slots * kTcABytes + (size_t)ring * tc_chunk_bytes(q) +
           kTcBarriers * 8 + 16 + 4096; // alignment slack, rings, barriers, token sums
}

// Ring depths.  The activation ring covers the trip to L2 (about a microsecond: six to eight narrow blocks, three of 256 tokens), the
// expanded weights only the hand-over to the tensor core, the planes get what is left.
bool tc_buffers(int q, bool grouped, int bt, int *x_slots, int *a_slots, int *ring)
{
    if (q == 0) {
        *x_slots = 6;
        *a_slots = *ring = 0;
        return tc_smem(q, bt, *x_slots, 0, 0) <= kTcSmem;
    }
    const int groups = tc_warps(q, grouped, bt).expand / 4;
    for (int xs = bt <= 32 ? 8 : bt <= 64 ? 6 : bt <= 128 ? 4 : 3; xs >= 2; --xs)
        for (int as = groups >= 3 ? groups : 3; as >= 2; --as)
            for (int r = kTcMaxRing; r >= 2; --r)
                if (tc_smem(q, bt, xs, as, r) <= kTcSmem) {
                    *x_slots = xs;
                    *a_slots = as;
                    *ring = r;
                    return true;
                }
    return false;
}

TcPlan tc_plan_of(const abq_gemm_state *st)
{
    TcPlan P;
    std::memcpy(&P, st->tmap[2], sizeof(P));
    return P;
}

} // namespace

bool tc_plan(abq_gemm_state *st, int sms, const UmmaLayout &L, bool expanded)
{
    const abq_gemm_params &p = st->p;
    const bool grouped = p.scale_mode == ABQ_SCALE_GROUP;
    const int q = expanded ? 0 : p.w_bits;
    TcPlan P = {};
    P.q = q;
    P.k_blocks = p.K / 128;
    const int ck = tc_chunk_blocks(q);
    P.chunk_blocks = ck;
    while (grouped && p.group_size > 128 && P.chunk_blocks % (p.group_size / 128)) // groups wider than 128 stay whole
        P.chunk_blocks += ck;
    P.chunks_per_tile = (P.k_blocks + P.chunk_blocks - 1) / P.chunk_blocks;
    P.n_tiles = (p.N + kTcRows - 1) / kTcRows;
    // Zero points and the offset of signed codes: subtracted by the expanders with scale groups and where that is free (the table
    // widths); otherwise the epilogue subtracts them times the token's code sum.
    const bool has_zero = p.w_zero && p.out_dtype == ABQ_OUT_FP16 && p.scale_mode == ABQ_SCALE_CHANNEL;
    P.xpart = !grouped && q > 0 && (tc_table_order(q) ? has_zero && p.w_signed : has_zero || (p.w_signed && q < 8));
    P.off_x = L.x;
    const size_t end = expanded ? L.end : L.sum; // scratch: everything behind the activation codes
    P.off_xpart = ((expanded ? L.end : L.x + (size_t)p.M * p.K) + 255) & ~(size_t)255;
    P.off_counters = (P.off_xpart + (P.xpart ? (size_t)p.M * P.k_blocks * 4 : 0) + 255) & ~(size_t)255;
    if (P.xpart && P.off_counters > end)
        return false; // (no room for the sums beside the activation codes)
    // (tuning runs and tests; a forced width may be any that exists)
    const int force_bt = env_int("ABQ_TC_BT", 0), force_split = env_int("ABQ_TC_SPLIT", -1);
    // Cost in clocks per SM, fitted to measured launches (N, K = 4096 .. 22016, 20 .. 512 tokens; 2, 4 and 8 bits).  A K block costs the
    // issuing thread about 560 clocks, the expanders 115 per weight bit, with scale groups the drain of its accumulators; a launch
    // about five microseconds plus the last tile's columns; cutting tiles the trip of their pieces through L2, which
    // grows with the columns.
    double best = 0;
    for (int bt = grouped ? 16 : 32; bt <= (q == 0 ? 128 : grouped ? 64 : 256); bt *= 2) {
        if (q == 0 ? bt != 128 : (force_bt ? bt != force_bt : bt > (grouped ? 16 : 32) && p.M <= bt / 2))
            continue;
        const int m_tiles = (p.M + bt - 1) / bt;
        const long tiles = (long)m_tiles * P.n_tiles;
        const double issue = 560 + 1.08 * bt, expand = 115.0 * q;
        double block = issue > expand ? issue : expand;
        if (grouped)
            block = p.group_size == 64 ? 1200 + 10.0 * bt : 900 + 7.0 * bt;
        const double tail = 9500 + 95.0 * bt;
        for (int split = 0; split < 2; ++split) {
            if (force_split >= 0 && split != force_split && q > 0)
                continue;
            const long chunks = tiles * P.chunks_per_tile;
            const long ctas = split ? (chunks < sms ? chunks : sms) : (tiles < sms ? tiles : sms);
            const int ew = tc_warps(q, grouped, bt).epilogue;
            const size_t off_partials = (P.off_counters + (size_t)tiles * ew * 4 + 255) & ~(size_t)255;
            if (split && (q == 0 || tiles >= 8L * sms || off_partials + (size_t)ctas * 2 * kTcRows * bt * 4 > end))
                continue;
            int x_slots, a_slots, ring;
            if (!tc_buffers(q, grouped, bt, &x_slots, &a_slots, &ring))
                continue;
            const double rounds = split && P.chunk_blocks > ck ? (double)((chunks + ctas - 1) / ctas) * P.chunk_blocks : split ? (double)chunks * ck / ctas : (double)((tiles + ctas - 1) / ctas) * P.k_blocks;
            const double t = rounds * block + tail + (split ? 5700.0 + 266.0 * bt : 0);
            if (best == 0 || t < best) {
                best = t;
                P.bt = bt;
                P.m_tiles = m_tiles;
                P.split = split;
                P.ctas = (int)ctas;
                P.x_slots = x_slots;
                P.a_slots = a_slots;
                P.ring = ring;
                P.off_partials = off_partials;
            }
        }
    }
    if (best == 0)
        return false;
    uint8_t *ws = reinterpret_cast<uint8_t *>(p.workspace);
    const uint64_t xd[2] = { (uint64_t)p.K, (uint64_t)p.M }, xs[1] = { (uint64_t)p.K };
    const uint32_t xb[2] = { 128, (uint32_t)P.bt };
    if (!encode_tmap(st->tmap[1], TMAP_U8, 2, ws + P.off_x, xd, xs, xb, TMAP_SWIZZLE_128B))
        return false;
    if (q > 0) {
        const uint64_t KW = (uint64_t)p.K / 32;
        const uint64_t wd[3] = { KW, (uint64_t)p.N, (uint64_t)q }, wst[2] = { KW * 4, KW * 4 * (uint64_t)p.N };
        const uint32_t wb[3] = { (uint32_t)(ck * 4), (uint32_t)kTcRows, (uint32_t)q };
        if (!encode_tmap(st->tmap[0], TMAP_U32, 3, p.W, wd, wst, wb, ck == 4 ? TMAP_SWIZZLE_64B : TMAP_SWIZZLE_32B))
            return false;
    } else {
        const uint64_t wd[2] = { (uint64_t)p.K, (uint64_t)p.N };
        const uint32_t wb[2] = { 128, (uint32_t)kTcRows };
        if (!encode_tmap(st->tmap[0], TMAP_U8, 2, ws + L.w, wd, xs, wb, TMAP_SWIZZLE_128B))
            return false;
    }
    std::memcpy(st->tmap[2], &P, sizeof(P));
    const TcWarps W = tc_warps(q, grouped, P.bt);
    st->grid[0] = P.ctas;
    st->grid[1] = st->grid[2] = 1;
    st->block[0] = (4 + W.expand + W.epilogue) * 32;
    st->block[1] = st->block[2] = 1;
    st->cluster = 1;
    st->shared_mem_size = tc_smem(q, P.bt, P.x_slots, P.a_slots, P.ring);
    st->tile[0] = kTcRows;
    st->tile[1] = P.split;
    st->tile[2] = expanded ? kTcCodes : kTcPlanes;
    st->tile[3] = P.bt;
    return true;
}

static bool tc_folds_zero(const abq_gemm_params &p, const TcPlan &P)
{
    return p.w_zero && p.out_dtype == ABQ_OUT_FP16 && !p.w_signed && (p.scale_mode == ABQ_SCALE_GROUP || (p.scale_mode == ABQ_SCALE_CHANNEL && tc_table_order(P.q)));
}

bool tc_planned(const abq_gemm_state *st) { return st->tile[2] == kTcPlanes || st->tile[2] == kTcCodes; }

bool tc_expanded(const abq_gemm_state *st) { return st->tile[2] == kTcCodes; }

cudaError_t tc_prepare_x(const abq_gemm_state *st, cudaStream_t stream)
{
    const abq_gemm_params &p = st->p;
    const TcPlan P = tc_plan_of(st);
    uint8_t *ws = reinterpret_cast<uint8_t *>(p.workspace);
    PrepareXArgs a;
    a.X = reinterpret_cast<const uint32_t *>(p.X);
    a.qscale = (p.flags & ABQ_FLAG_X_HALF) ? p.x_quant_scale : nullptr;
    a.out = reinterpret_cast<uint4 *>(ws + P.off_x);
    a.runs = a.plane_words = (long)p.M * (p.K / 32);
    a.bits = p.x_bits;
    a.is_signed = p.x_signed;
    a.table_order = tc_table_order(P.q);
    a.xpart = P.xpart ? reinterpret_cast<int *>(ws + P.off_xpart) : nullptr;
    a.M = p.M;
    a.kw = p.K / 32;
    a.counters = reinterpret_cast<int *>(ws + P.off_counters);
    a.n_counters = P.split ? P.m_tiles * P.n_tiles * tc_warps(P.q, p.scale_mode == ABQ_SCALE_GROUP, P.bt).epilogue : 0;
    const long threads = a.runs > a.n_counters ? a.runs : a.n_counters;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((threads + 127) / 128));
    cfg.blockDim = dim3(128);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    // Without ABQ_FLAG_PDL this launch waits for everything before it on the stream, and with it the GEMM behind, which starts on
    // the weights as soon as this kernel runs; with the flag the caller has promised that the weights are complete.
    cfg.numAttrs = (p.flags & ABQ_FLAG_PDL) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, prepare_x_kernel, a);
}

cudaError_t tc_launch(const abq_gemm_state *st, cudaStream_t stream)
{
    const abq_gemm_params &p = st->p;
    const bool grouped = p.scale_mode == ABQ_SCALE_GROUP;
    const TcPlan P = tc_plan_of(st);
    uint8_t *ws = reinterpret_cast<uint8_t *>(p.workspace);
    TcArgs a = {};
    a.M = p.M;
    a.N = p.N;
    a.bt = P.bt;
    a.m_tiles = P.m_tiles;
    a.n_tiles = P.n_tiles;
    a.k_blocks = P.k_blocks;
    a.chunk_blocks = P.chunk_blocks;
    a.chunks_per_tile = P.chunks_per_tile;
    a.split = P.split;
    const int chunks = P.m_tiles * P.n_tiles * P.chunks_per_tile;
    a.range_q = chunks / P.ctas;
    a.range_r = chunks % P.ctas;
    a.x_slots = P.x_slots;
    a.a_slots = P.a_slots;
    a.ring = P.ring;
    a.D = p.D;
    a.C = reinterpret_cast<const __half *>(p.C);
    a.w_scale = reinterpret_cast<const __half *>(p.w_scale);
    a.w_zero = p.w_zero;
    a.x_scale = p.out_dtype == ABQ_OUT_FP16 && p.scale_mode != ABQ_SCALE_TENSOR_COMPAT ? p.x_scale : nullptr;
    a.xpart = P.xpart ? reinterpret_cast<const int *>(ws + P.off_xpart) : nullptr;
    a.residual = reinterpret_cast<const __half *>(p.residual);
    a.fold_zero = tc_folds_zero(p, P);
    a.w_offset = P.q > 0 && p.w_signed && p.w_bits < 8 ? 1 << (p.w_bits - 1) : 0;
    a.out_dtype = p.out_dtype;
    a.scale_mode = p.scale_mode;
    a.group_size = grouped ? p.group_size : 0;
    a.scale_groups = grouped ? p.K / p.group_size : 0;
    // a sum over at most 128 features: below 2^22 in magnitude with one signed operand (255 * 128 * 128), else in [0, 2^23)
    const bool w_codes_signed = p.w_signed || a.fold_zero;
    const bool both_unsigned = !p.x_signed && !w_codes_signed;
    a.magic = both_unsigned ? 0x4b000000 : 0x4b400000;
    a.magic_f = both_unsigned ? 8388608.f : 12582912.f;
    // A = weights: expanded codes of up to 7 bits are always written as signed bytes
    const bool a_signed = P.q == 0 ? w_codes_signed : (P.q < 8 || p.w_signed);
    a.idesc = (2u << 4) | ((a_signed ? 1u : 0u) << 7) | ((p.x_signed ? 1u : 0u) << 10) | ((uint32_t)(P.bt >> 3) << 17) | ((uint32_t)(kTcRows >> 4) << 24);
    a.counters = reinterpret_cast<int *>(ws + P.off_counters);
    a.partials = reinterpret_cast<int *>(ws + P.off_partials);
    a.status = p.status_word;
    CUtensorMap tw, tx;
    std::memcpy(&tw, st->tmap[0], sizeof(tw));
    std::memcpy(&tx, st->tmap[1], sizeof(tx));
    const unsigned grid = (unsigned)P.ctas;
    const size_t smem = st->shared_mem_size;
    switch (P.q) {
    case 0: return tc_launch_w0(tw, tx, a, grouped, grid, smem, stream);
    case 1: return tc_launch_w1(tw, tx, a, grouped, grid, smem, stream);
    case 2: return tc_launch_w2(tw, tx, a, grouped, grid, smem, stream);
    case 3: return tc_launch_w3(tw, tx, a, grouped, grid, smem, stream);
    case 4: return tc_launch_w4(tw, tx, a, grouped, grid, smem, stream);
    case 5: return tc_launch_w5(tw, tx, a, grouped, grid, smem, stream);
    case 6: return tc_launch_w6(tw, tx, a, grouped, grid, smem, stream);
    case 7: return tc_launch_w7(tw, tx, a, grouped, grid, smem, stream);
    case 8: return tc_launch_w8(tw, tx, a, grouped, grid, smem, stream);
    }
    return cudaErrorInvalidValue;
}

} // namespace abq
