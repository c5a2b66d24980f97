// The matrix product of the 32-bit mode on the tensor cores, for the larger matrices and every number of tokens:
//   out[t,n] = sum_k X[t,k] W[n,k] (+ bias[n]), operands and results in 32 bits.
//
// Every operand is cut into three bfloat16 terms, each the rest rounded to nearest, so that nothing is left behind the third (x = h + m + l: the
// scheme of Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations", 2019), and eight
// of the nine products of terms are taken; l l, 2^-34 of a product, is left out.  The tensor core cuts its 32-bit sums instead of rounding them, so it
// is given little to cut: a block of 32 of K has a sum of its own for h h, whose products have 16 bits, and the blocks' sums are added in
// registers, rounded to nearest; the seven small products are summed in a second accumulator over a piece of K, where a lost bit is 2^-8 of
// that, and added behind its last block.  Against 64 bits (2,048 of K, 32-bit FMAs one behind another in brackets, of the result's norm): one term in a row
// 2.5e-8 (2.5e-8), 4 side by side 2.7e-8 (4.2e-8), 4 far apart 4.5e-8 (4.1e-8), 16 3.7e-8 and 6.9e-8 (7.5e-8), all 9.8e-8 (8.1e-7).
// (One accumulator for all products took 2 to 15 % less time, and the whole sum was cut.)
// Results that are not finite (an infinite operand times a term that is zero) and results below 2^-96 are summed again one product behind another,
// as gemm_generic does, and so are those from which more than 2^-26 may be missing where an operand below 2^-110 has lost bits (its terms reach the end of
// the exponents' range: operands of 1e-34 lose 3e-7 of themselves, of 1e-36 3e-5, of 1e-42 everything).  The conversion looks for such operands; only where it
// finds one are a tile's operands read again for what they may have cost.
//
// A row's result does not depend on the rows beside it: a block's sum is the same whatever the tile's width, and K is cut into pieces
// by the matrix's sizes alone (fx_pieces), whose sums are added in order.
//
// What bounds it: a block of 128 features x 192 tokens x 32 of K takes 1,540 cycles of tensor core (eight products for each 32-bit one), 1,670 of
// shared memory (the loads, X's conversion, the products' reads of X) and 2,500 in all.  Few tokens: the warps' chain from a
// block's copy through its conversion (28,672 x 4,096 at one token with a tile a CTA: 139 us, 96 without the conversion, of which 72 are bytes).
// W is the A operand from tensor memory because shared memory would be busy for 1,700 cycles more with its reads.  Tiles of 64 tokens and more have sixteen
// warps that convert and add (192 tokens 16,384 x 2,048 98 us, 100 with eight; 1,152 tokens 513, 535; before the look for tiny operands, which takes 3 to 5 %).
// Microseconds behind a cleared L2, gemm_f32 in brackets: 16,384 x 2,048, 1, 2, 4, 16 tokens 46, 46, 46, 48 (39, 41, 45, 70), 64 59, 187 103; 2,048 x
// 8,192 30, 30, 31, 32 (37, 38, 39, 64), 64 38, 187 64; 28,672 x 4,096 113, 113, 114, 116 (100, 102, 123, 274), 64 195, 187 346.
//
// A CTA has one tile of 128 features x BN tokens or some pieces of K of one or several.  Warp 0 copies 32-bit blocks of both operands by TMA
// (128-byte swizzle) into a ring (and converts X where there are up to 16 tokens), warp 1 issues the MMAs, eight or sixteen warps convert a block (of W a row and half of the block a
// thread, of X a quarter of a row) and add the sums of an earlier block.  Where a tile is one CTA's, its pieces' sums are added as they come; else they go to
// scratch memory and a second kernel adds them: no CTA waits for another, whatever runs beside them.
#include <mutex>

#include "common.cuh"
#include "sm100.cuh"

using namespace sm100;

namespace {

constexpr int FX_BM = 128, FX_BK = 32;
constexpr int FX_PIECES = 16;                   // of K, at most

template <int BN> struct FxCfg {
    static constexpr int W_BYTES = FX_BM * 128, X_BYTES = BN * 128, RAW = W_BYTES + X_BYTES;
    // blocks whose terms are on their way through the tensor core
    static constexpr int DEPTH = BN <= 16 ? 3 : BN <= 32 ? 2 : BN <= 64 ? 4 : 2;
    static constexpr int RING = BN <= 16 ? 5 : BN <= 32 ? 4 : BN <= 64 ? 5 : BN <= 160 ? 4 : 3;
    static constexpr int SMEM = RING * RAW + (DEPTH + (DEPTH + 1) / 2) * X_BYTES + 1024;
    // Tensor memory, 512 columns (256 where two CTAs share an SM): sums of large products of SUMS blocks, of small products of TAILS pieces of K,
    // and W's terms of DEPTH blocks in buffers of 64 columns, 32 for each 16 of K: h, m, l and eight columns that nothing reads (one store
    // of 32 columns a warp takes a third of what three of eight do: 57 -> 38 us at 16,384 x 2,048 and 2 tokens)
    static constexpr int SUMS = BN <= 96 ? 2 : 1, TAILS = BN <= 128 ? 2 : 1;
    static constexpr int T_COL = SUMS * BN, A_COL = T_COL + TAILS * BN;
    static constexpr int TMEM_COLS = A_COL + DEPTH * 64 <= 256 ? 256 : 512;
    static constexpr int CTAS = BN <= 32 ? 2 : 1;                 // of an SM
    // Warps that convert and add; a warp adds the sums of a GROUPS-th of the columns.  Of sixteen half convert W, half X.
    static constexpr int WORKERS = BN < 64 ? 8 : 16, GROUPS = WORKERS / 4, COLS = BN / GROUPS, THREADS = (WORKERS + 2) * 32;
    static constexpr bool X_BY_COPIER = BN <= 16;                 // the warp that copies converts X too
    static constexpr int ARRIVALS = WORKERS + (X_BY_COPIER ? 1 : 0);             // for a block that is converted
    static_assert(A_COL + DEPTH * 64 <= 512 && TMEM_COLS * CTAS <= 512 && SUMS <= DEPTH);
};

struct FxParams {
    const float* x;
    const float* w;
    const void* bias;
    void* out;
    float* scratch;       // [tiles][pieces][slot_cols][128] sums of the pieces of K, where a tile is not one CTA's
    float* lost;          // [tiles][pieces] behind them: fx_lost of a piece
    int* status;
    long long ldx, ldw, ldo;
    int bias_dtype, out_dtype;
    int T, N, K, pieces, first_blocks, tiles, t_tiles, slot_cols;       // first_blocks: of the first of two unequal pieces of K (0: equal ones)
};

// Two numbers in three bfloat16 terms each, the first in the low halves: each term the rest, rounded to nearest; nothing is left behind the third.
__device__ __forceinline__ uint32_t fx_pack(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float fx_low(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float fx_high(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ void fx_split(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = fx_pack(a, b);
    const float ra = a - fx_low(h), rb = b - fx_high(h);
    m = fx_pack(ra, rb);
    l = fx_pack(ra - fx_low(m), rb - fx_high(m));
}
__device__ __forceinline__ float4 fx_lds4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void fx_sts4(uint32_t a, const uint32_t* v) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// 32 columns of this thread's lane; the wait for it comes later.
__device__ __forceinline__ void fx_tmem_st32(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
          "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
          "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void fx_tmem_ld8(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
// N columns of this thread's lane, added to acc.
template <int N> __device__ __forceinline__ void fx_add(float (&acc)[N], uint32_t d) {
    constexpr int STEP = N % 32 == 0 ? 32 : N % 16 == 0 ? 16 : 8;
#pragma unroll
    for (int c = 0; c < N; c += STEP) {
        float v[STEP];
        if constexpr (STEP == 32) tmem_ld32(d + c, v);
        else if constexpr (STEP == 16) tmem_ld16(d + c, v);
        else fx_tmem_ld8(d + c, v);
#pragma unroll
        for (int j = 0; j < STEP; ++j) acc[c + j] += v[j];
    }
}

// A number below this loses bits in its terms: the third one ends at 2^-133, the smallest bfloat16.
constexpr float FX_TINY = 0x1p-110f;
// The smallest magnitude that is not zero, as twice its bits less one, in which zero is the largest number there is: no branch stands in the
// conversion's loop, where one costs what the whole look costs.
constexpr uint32_t FX_TINY_RANK = ((127u - 110u) << 24) - 1u;
__device__ __forceinline__ uint32_t fx_rank(float v) { return 2u * __float_as_uint(v) - 1u; }
__device__ __forceinline__ uint32_t fx_least(uint32_t least, const float4& v) {
    return __vimin3_u32(__vimin3_u32(least, fx_rank(v.x), fx_rank(v.y)), fx_rank(v.z), fx_rank(v.w));
}

// A sum that is not finite or next to nothing, or from which too much may be lost, taken again one product behind another.
__device__ __noinline__ float fx_again(const float* x, const float* w, int K) {
    float v = 0.f;
    for (int k = 0; k < K; ++k) v = fmaf(x[k], w[k], v);
    return v;
}
__device__ __forceinline__ void fx_store(const FxParams& p, int t, int n, float v, float bias, float lost = 0.f) {
    if (!isfinite(v) || (fabsf(v) < 0x1p-96f && v != 0.f) || fabsf(v) < lost) v = fx_again(p.x + size_t(t) * p.ldx, p.w + size_t(n) * p.ldw, p.K);
    gb_store(p.out, p.out_dtype, size_t(t) * p.ldo + n, p.bias ? v + bias : v);
}

// The largest finite magnitude of a row's K numbers and whether one of them loses bits, by a warp into big and tiny.
__device__ __forceinline__ void fx_scan(const float* row, int K, int* big, int* tiny) {
    float most = 0.f;
    bool any = false;
    for (int k = 4 * (threadIdx.x & 31); k < K; k += 128) {
        const float4 v = *reinterpret_cast<const float4*>(row + k);
        const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (fabsf(a[e]) < INFINITY) most = fmaxf(most, fabsf(a[e]));
            any = any || (a[e] != 0.f && fabsf(a[e]) < FX_TINY);
        }
    }
    if (most > 0.f) atomicMax(big, __float_as_int(most));              // not negative: ordered as whole numbers are
    if (any) *tiny = 1;
}
// What may be missing of a sum over k places of K where operands have lost bits, times 2^26: up to 2^-134 of each, times the largest of the
// other operand, as often as there are places.  Results below it are summed again.  By all threads of a block, for all rows from x and w on.
// (A function of its own with values for arguments, called when no sums wait in registers: inlined in front of the stores it cost the block's loop 10 %.)
__device__ __noinline__ float fx_lost(const float* x, long long ldx, int tokens, const float* w, long long ldw, int features, int k) {
    __shared__ int big_w, big_x, tiny_w, tiny_x;
    __syncthreads();
    if (threadIdx.x == 0) big_w = big_x = tiny_w = tiny_x = 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (int i = warp; i < features; i += warps) fx_scan(w + i * ldw, k, &big_w, &tiny_w);
    for (int i = warp; i < tokens; i += warps) fx_scan(x + i * ldx, k, &big_x, &tiny_x);
    __syncthreads();
    return 0x1p-108f * float(k) * ((tiny_w ? __int_as_float(big_x) : 0.f) + (tiny_x ? __int_as_float(big_w) : 0.f));
}
// The results of a whole tile once more, behind their stores.
__device__ __noinline__ void fx_mend(const float* x, long long ldx, int tokens, const float* w, long long ldw, int features, int K, const void* bias,
                                     int bias_dtype, void* out, int out_dtype, long long ldo, int n0, int t0) {
    const float lost = fx_lost(x, ldx, tokens, w, ldw, features, K);
    for (int i = threadIdx.x; i < tokens * FX_BM; i += blockDim.x) {
        const int n = i & (FX_BM - 1), c = i / FX_BM;
        if (n >= features) continue;
        const size_t at = size_t(t0 + c) * ldo + n0 + n;
        const float b = bias ? gb_load(bias, bias_dtype, n0 + n) : 0.f;
        if (fabsf(gb_load(out, out_dtype, at) - b) < 2.f * lost) {                           // (twice: the result may have been rounded to 8 bits)
            const float v = fx_again(x + c * ldx, w + n * ldw, K);
            gb_store(out, out_dtype, at, bias ? v + b : v);
        }
    }
}

template <int BN>
__global__ void __launch_bounds__(FxCfg<BN>::THREADS, FxCfg<BN>::CTAS) gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                                  const __grid_constant__ CUtensorMap map_x, FxParams p) {
    using Cfg = FxCfg<BN>;
    constexpr int RING = Cfg::RING, COLS = Cfg::COLS, WORKERS = Cfg::WORKERS, DEPTH = Cfg::DEPTH, SUMS = Cfg::SUMS, TAILS = Cfg::TAILS;
    // A block's sums are added SUMS blocks later, before that block's terms are stored, so that the buffer is free when those are there; with
    // one buffer behind the next block's terms, while its small products run, and the large ones wait for it.
    constexpr bool LATE = SUMS == 1;
    constexpr bool EARLY = BN <= 64;               // W's terms in registers while the buffer that they go to is still read
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* xs = ring + RING * Cfg::RAW;          // X's terms: rows of 128 bytes, [h | m] of each buffer, then [l of an even buffer | l of an odd one]
    __shared__ uint64_t raw_full[RING], raw_empty[RING], op_full[DEPTH], done[DEPTH], sum_free, tail_free[TAILS];
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag, tiny_seen;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    // This CTA's units, pieces of K of tiles: all of one tile (whole), or some, and then their sums go to scratch memory.  With two unequal pieces
    // (first_blocks) a CTA has the first piece of a tile, or the second ones of several.
    const int blocks = (p.K + FX_BK - 1) / FX_BK;
    const bool whole = gridDim.x == p.tiles;
    auto piece_begin = [&](int i) { return i == 1 && p.first_blocks ? p.first_blocks : i * blocks / p.pieces; };          // i <= 16, blocks < 2^26
    auto piece_blocks = [&](int unit) { const int i = unit % p.pieces; return piece_begin(i + 1) - piece_begin(i); };
    int unit0, count, step = 1;
    if (p.first_blocks && !whole) {
        const int c = blockIdx.x - p.tiles, rest = gridDim.x - p.tiles;
        unit0 = c < 0 ? 2 * blockIdx.x : 2 * int((long long)c * p.tiles / rest) + 1;
        count = c < 0 ? 1 : int((long long)(c + 1) * p.tiles / rest) - int((long long)c * p.tiles / rest);
        step = 2;
    } else {
        const int units = p.tiles * p.pieces;
        unit0 = int((long long)blockIdx.x * units / gridDim.x);
        count = int((long long)(blockIdx.x + 1) * units / gridDim.x) - unit0;
    }
    const int tile0 = unit0 / p.pieces;
    int S = 0;
    for (int i = 0; i < count; ++i) S += piece_blocks(unit0 + i * step);

    if (threadIdx.x == 0) {
        for (int i = 0; i < RING; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], Cfg::ARRIVALS); }
        for (int i = 0; i < DEPTH; ++i) { mbar_init(&op_full[i], Cfg::ARRIVALS); mbar_init(&done[i], 1); }
        mbar_init(&sum_free, WORKERS);
        for (int i = 0; i < TAILS; ++i) mbar_init(&tail_free[i], WORKERS);
        abort_flag = tiny_seen = 0;
        fence_barrier_init();
        prefetch_tensormap(&map_w);
        prefetch_tensormap(&map_x);
    }
    if (warp == 1) {
        tmem_alloc(&tmem_base, Cfg::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    gb_grid_launch_dependents();
    gb_grid_wait();

    constexpr bool TOTAL = BN <= 96;              // a whole tile's pieces are added in registers of their own
    float acc[COLS], total[TOTAL ? COLS : 1];
#pragma unroll
    for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
#pragma unroll
    for (int i = 0; i < (TOTAL ? COLS : 1); ++i) total[i] = 0.f;
    const int quarter = warp & 3, row = quarter * 32 + lane, group = (warp - 2) >> 2, half = group & 1;       // of the workers
    const int mine = group * COLS;

    // X, eight of K (a 16th of the block's rows of 128 bytes: chunk j of its terms) of row r: the terms of block s in buffer b.
    const uint32_t ring_a = smem_u32(ring), xs_a = smem_u32(xs);
    uint32_t least[2] = {0xffffffffu, 0xffffffffu};                             // fx_least of all that this thread has converted
    auto convert_x = [&](uint32_t raw, int b, int r, int j) {
        const uint32_t x = raw + Cfg::W_BYTES, hm = xs_a + b * Cfg::X_BYTES, lo = xs_a + (DEPTH + (b >> 1)) * Cfg::X_BYTES;
        const int sw = r & 7;
        const float4 u = fx_lds4(x + r * 128 + ((2 * j ^ sw) << 4)), v = fx_lds4(x + r * 128 + (((2 * j + 1) ^ sw) << 4));
        least[0] = fx_least(least[0], u);
        least[1] = fx_least(least[1], v);
        uint32_t xh[4], xm[4], xl[4];
        fx_split(u.x, u.y, xh[0], xm[0], xl[0]);
        fx_split(u.z, u.w, xh[1], xm[1], xl[1]);
        fx_split(v.x, v.y, xh[2], xm[2], xl[2]);
        fx_split(v.z, v.w, xh[3], xm[3], xl[3]);
        fx_sts4(hm + r * 128 + ((j ^ sw) << 4), xh);
        fx_sts4(hm + r * 128 + (((j + 4) ^ sw) << 4), xm);
        fx_sts4(lo + r * 128 + (((j + 4 * (b & 1)) ^ sw) << 4), xl);
    };

    if (warp == 0) {
        int unit = unit0, tile = tile0, kb = piece_begin(unit0 - tile0 * p.pieces), left = piece_blocks(unit0);
        auto copy = [&](int slot) {
            uint8_t* dst = ring + slot * Cfg::RAW;
            mbar_expect_tx(&raw_full[slot], Cfg::RAW);
            tma_load_2d(dst, &map_w, kb * FX_BK, tile / p.t_tiles * FX_BM, &raw_full[slot]);
            tma_load_2d(dst + Cfg::W_BYTES, &map_x, kb * FX_BK, tile % p.t_tiles * BN, &raw_full[slot]);
            ++kb;
            if (--left == 0) {
                unit += step;
                tile = unit / p.pieces;
                kb = piece_begin(unit - tile * p.pieces);
                left = piece_blocks(unit);
            }
        };
        if constexpr (!Cfg::X_BY_COPIER) {
            if (elect_one()) {
                for (int s = 0; s < S; ++s) {
                    const int slot = s % RING;
                    if (s >= RING && !mbar_wait(&raw_empty[slot], (s / RING - 1) & 1)) { atomicExch(p.status, 21); abort_flag = 1; break; }
                    copy(slot);
                }
            }
        } else {
            // few tokens: this warp converts X beside its copies, or two of the workers' warps would be later than the others with every block (28,672 x
            // 4,096 at one token 118 -> 114 us; with 32 tokens it would be the last itself: 130 -> 140)
            if (elect_one())
                for (int s = 0; s < S && s < RING; ++s) copy(s);
            for (int s = 0; s < S; ++s) {
                const int b = s % DEPTH, slot = s % RING;
                if (!mbar_wait(&raw_full[slot], (s / RING) & 1) || (s >= DEPTH && !mbar_wait(&done[b], (s / DEPTH - 1) & 1))) {
                    if (lane == 0) atomicExch(p.status, 28);
                    abort_flag = 1;
                    break;
                }
#pragma unroll
                for (int i = 0; i < BN / 8; ++i) convert_x(ring_a + slot * Cfg::RAW, b, (i >> 1) * 16 + (lane >> 1), (lane & 1) * 2 + (i & 1));
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) { mbar_arrive(&raw_empty[slot]); mbar_arrive(&op_full[b]); }
                if (s + RING < S) {
                    bool late = false;
                    if (elect_one()) {
                        late = !mbar_wait(&raw_empty[slot], (s / RING) & 1);
                        if (!late) copy(slot);
                    }
                    if (__any_sync(0xffffffffu, late)) {
                        if (lane == 0) atomicExch(p.status, 21);
                        abort_flag = 1;
                        break;
                    }
                }
            }
            if (min(least[0], least[1]) < FX_TINY_RANK) tiny_seen = 1;
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = instr_desc_bf16(FX_BM, BN);
            const uint32_t xa = smem_u32(xs);
            int piece = 0, piece_end = piece_blocks(unit0), more = 0;         // pieces before this one; whether it has begun
            for (int s = 0; s < S; ++s) {
                const int b = s % DEPTH, tail = piece % TAILS;
                if (!mbar_wait(&op_full[b], (s / DEPTH) & 1)) { atomicExch(p.status, 22); abort_flag = 1; break; }
                // (two buffers for small products: the piece before the last has been read before this block's terms are there, if not LATE)
                if (LATE && !more && piece >= TAILS && !mbar_wait(&tail_free[tail], (piece / TAILS - 1) & 1)) {
                    atomicExch(p.status, 26);
                    abort_flag = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + s % SUMS * BN, t = tmem + Cfg::T_COL + tail * BN, a = tmem + Cfg::A_COL + b * 64;
                const uint32_t xh = xa + b * Cfg::X_BYTES, xm = xh + 64, xl = xa + (DEPTH + (b >> 1)) * Cfg::X_BYTES + (b & 1) * 64;
                auto two = [&](uint32_t to, int term, uint32_t xt, uint32_t add) {             // both steps of 16 of K
#pragma unroll
                    for (int k = 0; k < 2; ++k) mma_f16_a_tmem(to, a + k * 32 + term * 8, smem_desc_sw128(xt + k * 32), idesc, k ? 1u : add);
                };
                two(t, 2, xm, more);
                two(t, 1, xl, 1u);
                two(t, 1, xm, 1u);
                two(t, 2, xh, 1u);
                two(t, 0, xl, 1u);
                two(t, 1, xh, 1u);
                two(t, 0, xm, 1u);
                if (LATE && s > 0) {
                    if (!mbar_wait(&sum_free, (s - 1) & 1)) { atomicExch(p.status, 27); abort_flag = 1; break; }
                    tc_fence_after();
                }
                two(d, 0, xh, 0u);
                mma_commit(&done[b]);
                more = 1;
                if (s + 1 == piece_end) {
                    more = 0;
                    ++piece;
                    piece_end += piece_blocks(unit0 + piece * step);
                }
            }
        }
    } else {
        const uint32_t lane_base = uint32_t(quarter * 32) << 16;
        int unit = unit0, done_units = 0, piece_end = piece_blocks(unit0);      // the piece whose blocks are being added, and those before it
        const bool does_w = WORKERS == 8 || warp < 10, does_x = !Cfg::X_BY_COPIER && (WORKERS == 8 || warp >= 10);
        const int xw = (warp - 2) & 7;
        // block s: its sums and, behind a piece's last block, those of the piece's small products
        auto add = [&](int s) {
            if (!mbar_wait(&done[s % DEPTH], (s / DEPTH) & 1)) {
                if (lane == 0) atomicExch(p.status, 23);
                abort_flag = 1;
                return false;
            }
            tc_fence_after();
            fx_add<COLS>(acc, tmem + lane_base + s % SUMS * BN + mine);
            if (LATE) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sum_free);
            }
            if (s + 1 == piece_end) {
                const int tail = done_units % TAILS;
                fx_add<COLS>(acc, tmem + lane_base + Cfg::T_COL + tail * BN + mine);
                if (LATE) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&tail_free[tail]);
                }
                const int tile = unit / p.pieces, piece = unit - tile * p.pieces, t0 = tile % p.t_tiles * BN, cols = min(BN, p.T - t0);
                if (!whole) {
                    float* to = p.scratch + size_t(unit) * (p.slot_cols * FX_BM) + row;
#pragma unroll
                    for (int c = 0; c < COLS; ++c) {
                        if (mine + c < cols) __stcg(to + size_t(mine + c) * FX_BM, acc[c]);
                        acc[c] = 0.f;
                    }
                } else if constexpr (TOTAL) {
#pragma unroll
                    for (int c = 0; c < COLS; ++c) {
                        total[c] = piece ? total[c] + acc[c] : acc[c];
                        acc[c] = 0.f;
                    }
                } else if (p.pieces > 1) {
                    // no registers for a second set of sums: they wait in the result's place, which is 32 bits wide then
                    const int n = tile / p.t_tiles * FX_BM + row;
                    float* to = reinterpret_cast<float*>(p.out) + size_t(t0 + mine) * p.ldo + n;
                    const int m = n < p.N ? cols - mine : 0;
#pragma unroll
                    for (int c0 = 0; c0 < COLS; c0 += 8) {
                        float v[8];
#pragma unroll
                        for (int c = 0; c < 8; ++c) v[c] = piece && c0 + c < m ? __ldcg(to + (c0 + c) * p.ldo) : 0.f;
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            if (piece) acc[c0 + c] = v[c] + acc[c0 + c];
                            if (done_units + 1 < count) {
                                if (c0 + c < m) __stcg(to + (c0 + c) * p.ldo, acc[c0 + c]);
                                acc[c0 + c] = 0.f;
                            }
                        }
                    }
                }
                ++done_units;
                unit += step;
                piece_end += piece_blocks(unit);
            }
            return true;
        };
        for (int s = 0; s < S + SUMS; ++s) {
            const int b = s % DEPTH, slot = s % RING;
            uint32_t terms[32];                                                 // h, m, l
            const uint32_t raw = ring_a + slot * Cfg::RAW;
            // W: a row a thread, 16 of K
            auto split_w = [&] {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = fx_lds4(raw + row * 128 + (((half * 4 + c) ^ (row & 7)) << 4));
                    least[c & 1] = fx_least(least[c & 1], v);
                    fx_split(v.x, v.y, terms[2 * c], terms[8 + 2 * c], terms[16 + 2 * c]);
                    fx_split(v.z, v.w, terms[2 * c + 1], terms[9 + 2 * c], terms[17 + 2 * c]);
                }
#pragma unroll
                for (int i = 24; i < 32; ++i) terms[i] = 0;
            };
            if (s < S) {
                if (!mbar_wait(&raw_full[slot], (s / RING) & 1)) {
                    if (lane == 0) atomicExch(p.status, 24);
                    abort_flag = 1;
                    break;
                }
                if (EARLY && does_w) split_w();
            }
            if (!LATE && s >= SUMS && !add(s - SUMS)) break;
            if (s < S) {
                // (the tensor core has read this block's buffers: what lies SUMS <= DEPTH blocks back has been added; LATE: 2 = DEPTH blocks)
                if (!EARLY && does_w) split_w();
                if (does_w) fx_tmem_st32(tmem + lane_base + Cfg::A_COL + b * 64 + half * 32, terms);
                if (does_x) {
                    // X: eight of K a thread; the rows of a quarter of a warp are four apart, so that their 64 bytes lie in both halves
                    const int j = lane & 3, sub = (lane >> 3) + (lane & 4);
#pragma unroll
                    for (int r0 = 0; r0 < BN; r0 += 64)
                        if (BN - r0 >= 64 || r0 + xw * 8 + sub < BN) convert_x(raw, b, r0 + xw * 8 + sub, j);
                    fence_proxy_async();
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { mbar_arrive(&raw_empty[slot]); mbar_arrive(&op_full[b]); }
            }
            if (LATE && s >= 1 && !add(s - 1)) break;
        }
        if (min(least[0], least[1]) < FX_TINY_RANK) tiny_seen = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, Cfg::TMEM_COLS);
    if (abort_flag) return;
    if (!whole) {
        for (int i = 0, unit = unit0; i < count; ++i, unit += step) {
            float lost = 0.f;
            if (tiny_seen) {
                const int tile = unit / p.pieces, piece = unit - tile * p.pieces, n0 = tile / p.t_tiles * FX_BM, t0 = tile % p.t_tiles * BN;
                const int k0 = piece_begin(piece) * FX_BK, k1 = min(p.K, piece_begin(piece + 1) * FX_BK);
                lost = fx_lost(p.x + t0 * p.ldx + k0, p.ldx, min(BN, p.T - t0), p.w + n0 * p.ldw + k0, p.ldw, min(FX_BM, p.N - n0), k1 - k0);
            }
            if (threadIdx.x == 0) p.lost[unit] = lost;
        }
        return;
    }

    const int n0 = tile0 / p.t_tiles * FX_BM, t0 = tile0 % p.t_tiles * BN, n = n0 + row, cols = min(BN, p.T - t0);
    if (warp >= 2 && n < p.N) {
        const float bias = p.bias ? gb_load(p.bias, p.bias_dtype, n) : 0.f;
#pragma unroll
        for (int c = 0; c < COLS; ++c)
            if (mine + c < cols) fx_store(p, t0 + mine + c, n, TOTAL ? total[TOTAL ? c : 0] : acc[c], bias);
    }
    if (tiny_seen)
        fx_mend(p.x + t0 * p.ldx, p.ldx, cols, p.w + n0 * p.ldw, p.ldw, min(FX_BM, p.N - n0), p.K, p.bias, p.bias_dtype, p.out, p.out_dtype, p.ldo, n0, t0);
}

// The sums of the pieces of tiles that were not one CTA's, added in order: a feature a thread, tokens 2 gridDim.y apart.
__global__ void __launch_bounds__(2 * FX_BM) gemm_f32_tc_merge_kernel(FxParams p, int bn) {
    gb_grid_launch_dependents();
    gb_grid_wait();
    __shared__ float lost_s;
    const int tile = blockIdx.x, row = threadIdx.x & (FX_BM - 1);
    const int n = tile / p.t_tiles * FX_BM + row, t0 = tile % p.t_tiles * bn, cols = min(bn, p.T - t0);
    if (threadIdx.x < 32) {                            // one warp asks (by all of them it was 20 us at 2,048 x 2,048 and 187 tokens)
        const float lost = gb_warp_sum(threadIdx.x < p.pieces ? __ldcg(p.lost + tile * p.pieces + threadIdx.x) : 0.f);
        if (threadIdx.x == 0) lost_s = lost;
    }
    const float bias = p.bias && n < p.N ? gb_load(p.bias, p.bias_dtype, n) : 0.f;
    const size_t slot = size_t(p.slot_cols) * FX_BM;
    bool first = true;                                 // every thread's first round, with a token or without: the barrier stands in it
    for (int c = 2 * blockIdx.y + (threadIdx.x >> 7); first || c < cols; c += 2 * gridDim.y) {
        const float* from = p.scratch + size_t(tile) * p.pieces * slot + size_t(c) * FX_BM + row;
        float v[FX_PIECES];
#pragma unroll
        for (int i = 0; i < FX_PIECES; ++i) v[i] = i < p.pieces && c < cols ? __ldcg(from + i * slot) : 0.f;
        float sum = v[0];
#pragma unroll
        for (int i = 1; i < FX_PIECES; ++i)
            if (i < p.pieces) sum += v[i];
        if (first) __syncthreads();                    // lost_s, while the first sums are on their way
        first = false;
        if (n < p.N && c < cols) fx_store(p, t0 + c, n, sum, bias, lost_s);
    }
}

int* g_status_host = nullptr;
int* g_status_dev = nullptr;

int ensure_status() {
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (g_status_dev) return 0;
    if (cudaHostAlloc(&g_status_host, sizeof(int), cudaHostAllocMapped) != cudaSuccess)
        return gb_fail("gb_gemm_f32_tc: cannot allocate the status word");
    *g_status_host = 0;
    if (cudaHostGetDevicePointer(&g_status_dev, g_status_host, 0) != cudaSuccess)
        return gb_fail("gb_gemm_f32_tc: cannot map the status word");
    return 0;
}

constexpr int MAX_DEVICES = 64;

template <int BN> int launch_fx(const CUtensorMap& mw, const CUtensorMap& mx, const FxParams& p, int ctas, cudaStream_t stream) {
    static bool configured[MAX_DEVICES] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return gb_fail("gb_gemm_f32_tc: no usable current device");
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(gemm_f32_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, FxCfg<BN>::SMEM) != cudaSuccess)
            return gb_fail("gb_gemm_f32_tc: cannot get %d bytes of shared memory", FxCfg<BN>::SMEM);
        configured[dev] = true;
    }
    gb_launch(gemm_f32_tc_kernel<BN>, dim3(ctas), dim3(FxCfg<BN>::THREADS), FxCfg<BN>::SMEM, stream, mw, mx, p);
    GB_LAUNCH_OK("gb_gemm_f32_tc");
    if (ctas != p.tiles) {
        int slices = 1280 / p.tiles;                                 // a token a thread, or a few: up to eight blocks an SM
        slices = slices > (p.slot_cols + 1) / 2 ? (p.slot_cols + 1) / 2 : slices > 0 ? slices : 1;
        gb_launch(gemm_f32_tc_merge_kernel, dim3(p.tiles, slices), dim3(2 * FX_BM), 0, stream, p, BN);
        GB_LAUNCH_OK("gb_gemm_f32_tc (merge)");
    }
    return 0;
}

// Pieces of K whose sums are added at the end, in order.  A function of the matrix alone: whatever the tokens beside it, a
// row's result is the same sums in the same order.  As many as give every SM two of a step with a single tile of tokens, of at
// least four blocks each.  More tiles than that makes two of leave SMs with one of them: there K has two unequal pieces, so that a tile's first is a
// CTA's and the places left share the second ones (28,672 x 4,096 at one token: 224 whole tiles 139 us, 103 and 25 blocks 113; equal pieces of a fifth
// 116, but a prompt's tile has to add them: 330 -> 375 us at 187 tokens, with two 346).
struct FxPieces { int n, first_blocks, shares; };          // shares: second pieces of a CTA, at most
FxPieces fx_pieces(int N, int K, int sms) {
    const int tiles = (N + FX_BM - 1) / FX_BM, blocks = (K + FX_BK - 1) / FX_BK, rest = 2 * sms - tiles;
    if (tiles > sms && rest > 0) {
        const int q = (tiles + rest - 1) / rest, first = (blocks * q + q) / (q + 1);
        if (blocks - first >= 4 && 10 * first <= 9 * blocks) return {2, first, q};
        return {1, 0, 0};
    }
    int n = 2 * sms / tiles;
    if (n > FX_PIECES) n = FX_PIECES;
    if (n > blocks / 4) n = blocks / 4;
    return {n > 1 ? n : 1, 0, 0};
}
// The tile and the number of CTAs that take the least time: rounds over the device times blocks of K times a block's time, with what a CTA
// takes beside its blocks, and where tiles are not one CTA's each the merge behind and the bytes that go there and back.  A block's time as
// measured at 16,384 x 2,048, microseconds.  The scratch memory of a launch is bounded (FX_SCRATCH floats); one CTA's tile needs none.
struct FxCut { int bn, pieces, first_blocks, ctas; long long tiles, scratch; };
constexpr long long FX_SCRATCH = 8LL << 20;
FxCut fx_cut(int T, int N, int K, int out_dtype, int sms) {
    static const int BNS[7] = {16, 32, 64, 96, 128, 160, 192};
    static const double BLOCK[7] = {0.9, 1.0, 0.8, 0.87, 0.97, 1.12, 1.3};
    const FxPieces cut = fx_pieces(N, K, sms);
    const int blocks = (K + FX_BK - 1) / FX_BK, pieces = cut.n;
    FxCut best = {16, pieces, cut.first_blocks, 0, 0, 0};
    double least = 1e300;
    for (int i = 0; i < 7; ++i) {
        const int bn = BNS[i];
        const long long tiles = (long long)((N + FX_BM - 1) / FX_BM) * ((T + bn - 1) / bn), places = (bn <= 32 ? 2LL : 1LL) * sms;
        if (bn <= 96 || pieces == 1 || out_dtype == GB_F32) {       // wider ones keep a piece's sums in a 32-bit result
            const double cost = double((tiles + places - 1) / places) * (blocks * BLOCK[i] + 4.0);
            if (cost < least) { least = cost; best = {bn, pieces, cut.first_blocks, int(tiles), tiles, 0}; }
        }
        const long long scratch = tiles * pieces * ((T < bn ? T : bn) * FX_BM + 1);
        for (int each = 1; each < pieces && !cut.first_blocks; ++each) {                   // pieces a CTA
            const int sharers = (pieces + each - 1) / each;
            if (tiles * sharers > places || scratch > FX_SCRATCH) continue;
            const double cost = each * ((blocks + pieces - 1) / pieces) * BLOCK[i] + 8.0 + 2e-6 * scratch;
            if (cost < least) { least = cost; best = {bn, pieces, 0, int(tiles * sharers), tiles, scratch}; }
        }
        if (cut.first_blocks && bn <= 32 && T <= bn && scratch <= FX_SCRATCH) {
            const double second = cut.shares * (blocks - cut.first_blocks + 0.33), cost = (second > cut.first_blocks ? second : cut.first_blocks) * BLOCK[i] + 8.0 + 2e-6 * scratch;
            if (cost < least) { least = cost; best = {bn, pieces, cut.first_blocks, int(places), tiles, scratch}; }
        }
    }
    return best;
}

}  // namespace

GB_API int gb_gemm_f32_tc_status() { return g_status_host ? *g_status_host : 0; }
GB_API int gb_gemm_f32_tc_status_clear() {
    if (g_status_host) *g_status_host = 0;
    return 0;
}

// Whether gb_gemm_f32_tc takes these operands: 32-bit rows that start on 16 bytes.
GB_API int gb_gemm_f32_tc_supported(const void* X, long long ldx, const void* W, long long ldw, int K) {
    return K > 0 && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(W) & 15) == 0;
}

// Floats of scratch that a launch of these sizes needs (0: every tile is one CTA's); never more than gb_gemm_f32_tc_scratch_max.
GB_API long long gb_gemm_f32_tc_scratch_floats(int T, int N, int K, int out_dtype, int sms) {
    return T > 0 && N > 0 && K > 0 && sms > 0 ? fx_cut(T, N, K, out_dtype, sms).scratch : 0;
}
GB_API long long gb_gemm_f32_tc_scratch_max() { return FX_SCRATCH; }

// scratch: gb_gemm_f32_tc_scratch_floats floats.
GB_API int gb_gemm_f32_tc(const float* X, long long ldx, const float* W, long long ldw, const void* bias, int bias_dtype, void* out,
                          int out_dtype, long long ldo, int T, int N, int K, float* scratch, int sms, cudaStream_t stream) {
    GB_REQUIRE(gb_is_dtype(out_dtype) && (!bias || gb_is_dtype(bias_dtype)), "gb_gemm_f32_tc: bad dtype");
    GB_REQUIRE(T >= 0 && N > 0 && K > 0 && ldx >= K && ldw >= K && ldo >= N && sms > 0,
               "gb_gemm_f32_tc: bad sizes T=%d N=%d K=%d ldx=%lld ldw=%lld ldo=%lld", T, N, K, ldx, ldw, ldo);
    GB_REQUIRE(gb_gemm_f32_tc_supported(X, ldx, W, ldw, K), "gb_gemm_f32_tc: rows must start on 16 bytes (K=%d, pitches %lld and %lld)", K, ldx, ldw);
    if (T == 0) return 0;
    if (ensure_status()) return 1;
    const FxCut cut = fx_cut(T, N, K, out_dtype, sms);
    GB_REQUIRE(cut.scratch == 0 || scratch, "gb_gemm_f32_tc: T=%d N=%d K=%d needs scratch memory", T, N, K);
    GB_REQUIRE(cut.tiles * cut.pieces < (1LL << 31), "gb_gemm_f32_tc: T=%d N=%d is more work than one launch numbers", T, N);
    FxParams p;
    p.x = X; p.w = W; p.bias = bias; p.out = out; p.scratch = scratch; p.status = g_status_dev;
    p.ldx = ldx; p.ldw = ldw; p.ldo = ldo; p.bias_dtype = bias_dtype; p.out_dtype = out_dtype; p.T = T; p.N = N; p.K = K;
    p.pieces = cut.pieces; p.first_blocks = cut.first_blocks; p.tiles = int(cut.tiles); p.t_tiles = (T + cut.bn - 1) / cut.bn; p.slot_cols = T < cut.bn ? T : cut.bn;
    p.lost = cut.scratch ? scratch + cut.tiles * cut.pieces * p.slot_cols * FX_BM : nullptr;
    CUtensorMap mw, mx;
    if (tensor_map_f32_2d(W, N, K, ldw, FX_BM, &mw)) return 1;
    if (tensor_map_f32_2d(X, T, K, ldx, cut.bn, &mx)) return 1;
    const int ctas = cut.ctas;
    switch (cut.bn) {
        case 16: return launch_fx<16>(mw, mx, p, ctas, stream);
        case 32: return launch_fx<32>(mw, mx, p, ctas, stream);
        case 64: return launch_fx<64>(mw, mx, p, ctas, stream);
        case 96: return launch_fx<96>(mw, mx, p, ctas, stream);
        case 128: return launch_fx<128>(mw, mx, p, ctas, stream);
        case 160: return launch_fx<160>(mw, mx, p, ctas, stream);
        default: return launch_fx<192>(mw, mx, p, ctas, stream);
    }
}
