// The matrix product of the 32-bit mode on the tensor cores, for more tokens than gemm_f32's few:
//   out[t,n] = sum_k X[t,k] W[n,k] (+ bias[n]), operands and results in 32 bits.
//
// Every operand is cut into three bfloat16 terms of eight bits each (x = h + m + l, exactly: 24 bits by truncation), and
// six of the nine products of terms are taken: hh, hm, mh, hl, lh, mm.  What is left out is 2^-23 of a product and less.
// The tensor core's own 32-bit additions are not relied on for long sums: a block of 32 of K is summed there (its ten small
// products first, so that only two additions meet a sum of full size), and the blocks' sums are added one behind another
// in registers, rounded to nearest.  Against 64 bits the result is 2 to 10 times closer than one thread's ascending sum (K = 256 1.2e-7
// of the result's norm against 2.8e-7, 2048 1.4e-7 and 8.1e-7, 8192 1.6e-7 and 1.6e-6).  Results that are not finite (an infinite
// operand times a term that is zero) and results below 2^-96 (the terms of operands of that size reach the end of the exponents' range: operands
// of 1e-34 would give 6e-7, of 1e-36 5e-5) are summed again one product behind another, as gemm_generic does; an exact zero stays.
//
// A row's result does not depend on the rows beside it: a block's sum is the same whatever the tile's width, and K is cut into pieces
// by the matrix's sizes alone (fx_pieces), whose sums are added in order.
//
// What bounds it: a block of 128 features x 192 tokens x 32 of K takes 1,150 cycles of tensor core (six products for each 32-bit
// one) and 2,300 in all: the warps' chain from a block's copy through its conversion (W's terms into tensor memory, X's into
// shared memory) and the sums of an earlier block.  Without the sums it takes 15 % less, without X's conversion 15 %, with one product
// instead of six 1 %.  W is the A operand from tensor memory because shared memory would be busy for 1,700 cycles with its reads beside X's.
// Microseconds, gemm_f32 in brackets: 187 tokens 16,384 x 2,048 84 (390), 2,048 x 8,192 45 (414), 3,072 x 2,048 26 (123), 2,048 x 2,048 22
// (114 at 100 tokens); 2 tokens 35 (27), 22 (42), 12.6 (12.3), 10.8 (14.5), where two CTAs an SM each stream their share of W; 1 to 16 tokens are the same.
//
// A CTA has one tile of 128 features x BN tokens and some pieces of K.  Warp 0 copies 32-bit blocks of both operands by TMA
// (128-byte swizzle) into a ring, warp 1 issues the MMAs, eight warps convert a block (of W a row and half of the block a
// thread, of X a quarter of a row) and add the sums of an earlier block (half of the columns each).  Where CTAs share a tile they are all
// resident, wait for one another (bounded) and finish a share of the tokens each.
#include <mutex>

#include "common.cuh"
#include "sm100.cuh"

using namespace sm100;

namespace {

constexpr int FX_BM = 128, FX_BK = 32, FX_THREADS = 320, FX_WORKERS = 256;

template <int BN> struct FxCfg {
    static constexpr int W_BYTES = FX_BM * 128, X_BYTES = BN * 128, RAW = W_BYTES + X_BYTES;
    // blocks on their way through the tensor core: terms and sums of DEPTH of them (512 columns of tensor memory in all, 256 where two CTAs share an SM)
    static constexpr int DEPTH = BN <= 16 ? 3 : BN <= 32 ? 2 : BN <= 64 ? 4 : BN <= 96 ? 3 : 2;
    static constexpr int RING = BN <= 16 ? 5 : BN <= 32 ? 4 : BN <= 64 ? 5 : BN <= 160 ? 4 : 3;
    static constexpr int SMEM = RING * RAW + (DEPTH + (DEPTH + 1) / 2) * X_BYTES + 1024;
    // W's terms in tensor memory: DEPTH buffers of 64 columns, 32 for each 16 of K: h, m, l and eight columns that nothing reads (one store
    // of 32 columns a warp takes a third of what three of eight do: 57 -> 38 us at 16,384 x 2,048 and 2 tokens)
    static constexpr int A_COL = DEPTH * BN;
    static constexpr int TMEM_COLS = DEPTH * (BN + 64) <= 256 ? 256 : 512;
    static constexpr int CTAS = BN <= 32 ? 2 : 1;                 // of an SM
};

struct FxParams {
    const float* x;
    const float* w;
    const void* bias;
    void* out;
    float* scratch;       // [tiles][pieces][BN][128] sums of the pieces of K
    int* counters;        // [tiles], zero between launches
    int* status;
    long long ldx, ldw, ldo;
    int bias_dtype, out_dtype;
    int T, N, K, pieces, sharers, t_tiles;
};

// Two numbers in three bfloat16 terms each, the first in the low halves.
__device__ __forceinline__ void fx_split(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    const uint32_t ha = __float_as_uint(a), hb = __float_as_uint(b);
    h = __byte_perm(ha, hb, 0x7632);
    const float ra = a - __uint_as_float(ha & 0xffff0000u), rb = b - __uint_as_float(hb & 0xffff0000u);
    const uint32_t ma = __float_as_uint(ra), mb = __float_as_uint(rb);
    m = __byte_perm(ma, mb, 0x7632);
    const float la = ra - __uint_as_float(ma & 0xffff0000u), lb = rb - __uint_as_float(mb & 0xffff0000u);
    l = __byte_perm(__float_as_uint(la), __float_as_uint(lb), 0x7632);
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
__device__ __forceinline__ void fx_workers_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// A sum that is not finite or next to nothing, taken again one product behind another.
__device__ __noinline__ float fx_again(const float* x, const float* w, int K) {
    float v = 0.f;
    for (int k = 0; k < K; ++k) v = fmaf(x[k], w[k], v);
    return v;
}
__device__ __forceinline__ void fx_store(const FxParams& p, int t, int n, float v, float bias) {
    if (!isfinite(v) || (fabsf(v) < 0x1p-96f && v != 0.f)) v = fx_again(p.x + size_t(t) * p.ldx, p.w + size_t(n) * p.ldw, p.K);
    gb_store(p.out, p.out_dtype, size_t(t) * p.ldo + n, p.bias ? v + bias : v);
}

template <int BN>
__global__ void __launch_bounds__(FX_THREADS, FxCfg<BN>::CTAS) gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                                  const __grid_constant__ CUtensorMap map_x, FxParams p) {
    using Cfg = FxCfg<BN>;
    constexpr int RING = Cfg::RING, HALF = BN / 2, DEPTH = Cfg::DEPTH;
    constexpr bool EARLY = BN <= 64;               // W's terms in registers while the buffer that they go to is still read
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* xs = ring + RING * Cfg::RAW;          // X's terms: rows of 128 bytes, [h | m] of each buffer, then [l of an even buffer | l of an odd one]
    __shared__ uint64_t raw_full[RING], raw_empty[RING], op_full[DEPTH], done[DEPTH];
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag, all_there;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int tile = blockIdx.x / p.sharers, me = blockIdx.x - tile * p.sharers;
    const int n0 = tile / p.t_tiles * FX_BM, t0 = (tile % p.t_tiles) * BN;
    const int blocks = (p.K + FX_BK - 1) / FX_BK;
    // this CTA's pieces of K, and their blocks
    const int piece0 = me * p.pieces / p.sharers, piece1 = (me + 1) * p.pieces / p.sharers;
    // one CTA's two pieces: the second stays in registers (and one CTA's only piece does)
    const bool keep = p.sharers == 1 && p.pieces <= 2;
    auto piece_begin = [&](int i) { return int((long long)i * blocks / p.pieces); };
    const int b0 = piece_begin(piece0), S = piece_begin(piece1) - b0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < RING; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 8); }
        for (int i = 0; i < DEPTH; ++i) { mbar_init(&op_full[i], 8); mbar_init(&done[i], 1); }
        abort_flag = 0;
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

    float acc[HALF];
#pragma unroll
    for (int i = 0; i < HALF; ++i) acc[i] = 0.f;
    const int quarter = warp & 3, row = quarter * 32 + lane, half = warp >= 6 ? 1 : 0;       // of the workers
    const int cols = min(BN, p.T - t0), mine = half * HALF;

    if (warp == 0) {
        if (elect_one()) {
            for (int s = 0; s < S; ++s) {
                const int slot = s % RING;
                if (s >= RING && !mbar_wait(&raw_empty[slot], (s / RING - 1) & 1)) { atomicExch(p.status, 21); abort_flag = 1; break; }
                uint8_t* dst = ring + slot * Cfg::RAW;
                mbar_expect_tx(&raw_full[slot], Cfg::RAW);
                tma_load_2d(dst, &map_w, (b0 + s) * FX_BK, n0, &raw_full[slot]);
                tma_load_2d(dst + Cfg::W_BYTES, &map_x, (b0 + s) * FX_BK, t0, &raw_full[slot]);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = instr_desc_bf16(FX_BM, BN);
            const uint32_t xa = smem_u32(xs);
            for (int s = 0; s < S; ++s) {
                const int b = s % DEPTH;
                if (!mbar_wait(&op_full[b], (s / DEPTH) & 1)) { atomicExch(p.status, 22); abort_flag = 1; break; }
                tc_fence_after();
                const uint32_t d = tmem + b * BN, a = tmem + Cfg::A_COL + b * 64;
                const uint32_t xh = xa + b * Cfg::X_BYTES, xm = xh + 64, xl = xa + (DEPTH + (b >> 1)) * Cfg::X_BYTES + (b & 1) * 64;
                uint32_t more = 0;
                auto two = [&](int term, uint32_t xt) {             // both steps of 16 of K
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        mma_f16_a_tmem(d, a + k * 32 + term * 8, smem_desc_sw128(xt + k * 32), idesc, more);
                        more = 1;
                    }
                };
                two(1, xm);
                two(2, xh);
                two(0, xl);
                two(1, xh);
                two(0, xm);
                two(0, xh);
                mma_commit(&done[b]);
            }
        }
    } else {
        const uint32_t ring_a = smem_u32(ring), xs_a = smem_u32(xs);
        const uint32_t lane_base = uint32_t(quarter * 32) << 16;
        int piece = piece0, piece_end = piece_begin(piece0 + 1) - b0;           // the piece whose blocks are being added
        for (int s = 0; s < S + DEPTH; ++s) {
            const int b = s % DEPTH, slot = s % RING;
            uint32_t terms[32];                                                 // h, m, l
            const uint32_t raw = ring_a + slot * Cfg::RAW;
            // W: a row a thread, 16 of K
            auto split_w = [&] {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = fx_lds4(raw + row * 128 + (((half * 4 + c) ^ (row & 7)) << 4));
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
                if (EARLY) split_w();
            }
            if (s >= DEPTH) {
                if (!mbar_wait(&done[b], (s / DEPTH - 1) & 1)) {
                    if (lane == 0) atomicExch(p.status, 23);
                    abort_flag = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + lane_base + b * BN + mine;
                constexpr int STEP = HALF % 32 == 0 ? 32 : HALF % 16 == 0 ? 16 : 8;
#pragma unroll
                for (int c = 0; c < HALF; c += STEP) {
                    float v[STEP];
                    if constexpr (STEP == 32) tmem_ld32(d + c, v);
                    else if constexpr (STEP == 16) tmem_ld16(d + c, v);
                    else fx_tmem_ld8(d + c, v);
#pragma unroll
                    for (int j = 0; j < STEP; ++j) acc[c + j] += v[j];
                }
                if (s - DEPTH + 1 == piece_end && !(keep && piece + 1 == p.pieces)) {        // a piece is complete
                    float* to = p.scratch + (size_t(tile) * p.pieces + piece) * (BN * FX_BM) + row;
#pragma unroll
                    for (int c = 0; c < HALF; ++c) {
                        if (mine + c < cols) __stcg(to + size_t(mine + c) * FX_BM, acc[c]);
                        acc[c] = 0.f;
                    }
                    ++piece;
                    piece_end = piece_begin(min(piece + 1, p.pieces)) - b0;
                }
            }
            if (s < S) {
                if (!EARLY) split_w();
                fx_tmem_st32(tmem + lane_base + Cfg::A_COL + b * 64 + half * 32, terms);
                // X: eight of K a thread; the rows of a quarter of a warp are four apart, so that their 64 bytes lie in both halves
                const int j = lane & 3, sub = (lane >> 3) + (lane & 4);
                const uint32_t x = raw + Cfg::W_BYTES, hm = xs_a + b * Cfg::X_BYTES, lo = xs_a + (DEPTH + (b >> 1)) * Cfg::X_BYTES;
#pragma unroll
                for (int r0 = 0; r0 < BN; r0 += 64) {
                    const int r = r0 + (warp - 2) * 8 + sub, sw = r & 7;
                    if (BN - r0 >= 64 || r < BN) {
                        const float4 u = fx_lds4(x + r * 128 + ((2 * j ^ sw) << 4)), v = fx_lds4(x + r * 128 + (((2 * j + 1) ^ sw) << 4));
                        uint32_t xh[4], xm[4], xl[4];
                        fx_split(u.x, u.y, xh[0], xm[0], xl[0]);
                        fx_split(u.z, u.w, xh[1], xm[1], xl[1]);
                        fx_split(v.x, v.y, xh[2], xm[2], xl[2]);
                        fx_split(v.z, v.w, xh[3], xm[3], xl[3]);
                        fx_sts4(hm + r * 128 + ((j ^ sw) << 4), xh);
                        fx_sts4(hm + r * 128 + (((j + 4) ^ sw) << 4), xm);
                        fx_sts4(lo + r * 128 + (((j + 4 * (b & 1)) ^ sw) << 4), xl);
                    }
                }
                fence_proxy_async();
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { mbar_arrive(&raw_empty[slot]); mbar_arrive(&op_full[b]); }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, Cfg::TMEM_COLS);
    if (abort_flag) return;
    if (warp < 2) return;

    const int n = n0 + row;
    const float bias = p.bias && n < p.N ? gb_load(p.bias, p.bias_dtype, n) : 0.f;
    if (keep) {
        if (p.pieces == 2) {                            // what this thread has stored itself
            const float* first = p.scratch + size_t(tile) * 2 * (BN * FX_BM) + row;
#pragma unroll
            for (int c = 0; c < HALF; ++c)
                if (mine + c < cols) acc[c] = __ldcg(first + size_t(mine + c) * FX_BM) + acc[c];
        }
        if (n < p.N) {
#pragma unroll
            for (int c = 0; c < HALF; ++c)
                if (mine + c < cols) fx_store(p, t0 + mine + c, n, acc[c], bias);
        }
        return;
    }
    __threadfence();
    fx_workers_sync();
    if (p.sharers > 1) {
        if (threadIdx.x == 64) {
            atomicAdd(&p.counters[tile], 1);
            int seen = 0;
            uint64_t start = 0;
            for (uint32_t i = 0;; ++i) {
                asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(p.counters + tile) : "memory");
                if (seen >= p.sharers) break;
                __nanosleep(40);
                if ((i & 255) == 255) {
                    const uint64_t now = global_timer_ns();
                    if (start == 0) start = now;
                    else if (now - start > WAIT_NS) break;
                }
            }
            all_there = seen >= p.sharers;
            if (!all_there) atomicExch(p.status, 25);
        }
        fx_workers_sync();
        if (!all_there) return;
    }
    const int c_lo = me * cols / p.sharers, c_hi = (me + 1) * cols / p.sharers;
    const float* base = p.scratch + size_t(tile) * p.pieces * (BN * FX_BM) + row;
    for (int c0 = c_lo + half * 4; c0 < c_hi; c0 += 8) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s0 = 0; s0 < p.pieces; s0 += 8) {
            float ld[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    ld[i][j] = s0 + i < p.pieces && c0 + j < c_hi ? __ldcg(base + (size_t(s0 + i) * BN + c0 + j) * FX_BM) : 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] += ld[i][j];
        }
        if (n < p.N) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (c0 + j < c_hi) fx_store(p, t0 + c0 + j, n, v[j], bias);
        }
    }
    if (p.sharers > 1) {
        // the last of the tile's CTAs to have read the others' sums puts the counter back for the next launch
        fx_workers_sync();
        if (threadIdx.x == 64 && atomicAdd(&p.counters[tile], 1) == 2 * p.sharers - 1) p.counters[tile] = 0;
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

template <int BN> int launch_fx(const CUtensorMap& mw, const CUtensorMap& mx, const FxParams& p, int ctas, cudaStream_t stream) {
    constexpr int MAX_DEVICES = 64;
    static bool configured[MAX_DEVICES] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return gb_fail("gb_gemm_f32_tc: no usable current device");
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(gemm_f32_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, FxCfg<BN>::SMEM) != cudaSuccess)
            return gb_fail("gb_gemm_f32_tc: cannot get %d bytes of shared memory", FxCfg<BN>::SMEM);
        configured[dev] = true;
    }
    gb_launch(gemm_f32_tc_kernel<BN>, dim3(ctas), dim3(FX_THREADS), FxCfg<BN>::SMEM, stream, mw, mx, p);
    GB_LAUNCH_OK("gb_gemm_f32_tc");
    return 0;
}

// Pieces of K whose sums are added at the end, in order.  A function of the matrix alone: whatever the tokens beside it, a
// row's result is the same sums in the same order.  As many as give every SM two of a step with a single tile of tokens, of at
// least four blocks each.
int fx_pieces(int N, int K, int sms) {
    const int tiles = (N + FX_BM - 1) / FX_BM, blocks = (K + FX_BK - 1) / FX_BK;
    int n = 2 * sms / tiles;
    if (n > 16) n = 16;
    if (n > blocks / 4) n = blocks / 4;
    return n > 1 ? n : 1;
}
// The tile and the number of CTAs on each that take the least time: rounds over the device times blocks of K times a block's
// time, with what a CTA takes beside its blocks, and a merge.  A block's time as measured at 16,384 x 2,048, microseconds.
struct FxCut { int bn, pieces, sharers; long long tiles; };
FxCut fx_cut(int T, int N, int K, int sms, bool may_share, int n_counters) {
    static const int BNS[7] = {16, 32, 64, 96, 128, 160, 192};
    static const double BLOCK[7] = {0.85, 0.95, 0.65, 0.75, 0.85, 1.0, 1.15};
    const int blocks = (K + FX_BK - 1) / FX_BK, pieces = fx_pieces(N, K, sms);
    FxCut best = {16, pieces, 1, 0};
    double least = 1e300;
    for (int i = 0; i < 7; ++i) {
        const long long tiles = (long long)((N + FX_BM - 1) / FX_BM) * ((T + BNS[i] - 1) / BNS[i]), resident = (BNS[i] <= 32 ? 2LL : 1LL) * sms;
        for (int sharers = 1; sharers <= pieces; ++sharers) {
            if (sharers > 1 && (!may_share || tiles * sharers > resident || tiles > n_counters)) break;
            const int each = (pieces + sharers - 1) / sharers * ((blocks + pieces - 1) / pieces);
            const double cost = double((tiles * sharers + resident - 1) / resident) * (each * BLOCK[i] + 4.0) + (sharers > 1 ? 3.0 : 0.0);
            if (cost < least) { least = cost; best = {BNS[i], pieces, sharers, tiles}; }
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

// Floats of scratch that a launch of these sizes needs, with counters or without (0: K is one piece).
GB_API long long gb_gemm_f32_tc_scratch_floats(int T, int N, int K, int sms, int n_counters) {
    const FxCut c = fx_cut(T, N, K, sms, n_counters > 0, n_counters);
    return c.pieces > 1 ? c.tiles * c.pieces * c.bn * FX_BM : 0;
}

// scratch: gb_gemm_f32_tc_scratch_floats floats, counters: n_counters zeroed ints (left zero), null with n_counters 0: no two CTAs share a tile.
GB_API int gb_gemm_f32_tc(const float* X, long long ldx, const float* W, long long ldw, const void* bias, int bias_dtype, void* out,
                          int out_dtype, long long ldo, int T, int N, int K, float* scratch, int* counters, int n_counters, int sms,
                          cudaStream_t stream) {
    GB_REQUIRE(gb_is_dtype(out_dtype) && (!bias || gb_is_dtype(bias_dtype)), "gb_gemm_f32_tc: bad dtype");
    GB_REQUIRE(T >= 0 && N > 0 && K > 0 && ldx >= K && ldw >= K && ldo >= N && sms > 0,
               "gb_gemm_f32_tc: bad sizes T=%d N=%d K=%d ldx=%lld ldw=%lld ldo=%lld", T, N, K, ldx, ldw, ldo);
    GB_REQUIRE(gb_gemm_f32_tc_supported(X, ldx, W, ldw, K), "gb_gemm_f32_tc: rows must start on 16 bytes (K=%d, pitches %lld and %lld)", K, ldx, ldw);
    if (T == 0) return 0;
    if (ensure_status()) return 1;
    const FxCut cut = fx_cut(T, N, K, sms, counters && n_counters > 0, counters ? n_counters : 0);
    GB_REQUIRE(cut.pieces == 1 || scratch, "gb_gemm_f32_tc: N=%d K=%d needs scratch memory", N, K);
    GB_REQUIRE(cut.tiles * cut.sharers < (1LL << 31), "gb_gemm_f32_tc: T=%d N=%d is more work than one launch numbers", T, N);
    FxParams p;
    p.x = X; p.w = W; p.bias = bias; p.out = out; p.scratch = scratch; p.counters = counters; p.status = g_status_dev;
    p.ldx = ldx; p.ldw = ldw; p.ldo = ldo; p.bias_dtype = bias_dtype; p.out_dtype = out_dtype; p.T = T; p.N = N; p.K = K;
    p.pieces = cut.pieces; p.sharers = cut.sharers; p.t_tiles = (T + cut.bn - 1) / cut.bn;
    CUtensorMap mw, mx;
    if (tensor_map_f32_2d(W, N, K, ldw, FX_BM, &mw)) return 1;
    if (tensor_map_f32_2d(X, T, K, ldx, cut.bn, &mx)) return 1;
    const int ctas = int(cut.tiles * cut.sharers);
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
