// The matrix product of the 32-bit mode for rows that start on 16 bytes and matrices that are too small for the tensor cores
// (gemm_f32_tc.cu) or a head: out[t,n] = sum_k X[t,k] W[n,k] (+ bias[n]),
// every product and sum a 32-bit FMA, every output summed by one thread in ascending k.  That is gemm_generic.cu's sum,
// bit for bit, whatever the sizes, so a row's result does not depend on the rows beside it; only the loads differ.
//
// Few tokens (gemm_f32_few_kernel): the time is the weights' way from memory, and one output's chain of K additions, each
// waiting for the one before.  Every CTA has the same few rows of W with all of K, copied asynchronously as far ahead as
// shared memory allows; a thread has one row and one to four tokens.  On 2,048 x 8,192 at 2 tokens gemm_generic's 64-row
// tiles kept 32 SMs busy, each with one load in flight per thread: 645 us, here 38 (16,384 x 2,048: 223 and 29; a head of
// 128,256 x 2,048: 1,188 and 180, where its bytes take 160).
// More tokens (gemm_f32_tile_kernel): bound by the FMA pipes; tiles of 64 features by 16 to 64 tokens, chosen so that the
// tiles fill the device, 4 x 2 to 4 x 8 outputs a thread, operands copied asynchronously three blocks of K ahead (a block
// is multiplied in a fifth of the time that memory takes to answer).  At 144 tokens 16,384 x 2,048 takes 265 us (gemm_generic
// 602), 2,048 x 8,192 225 (613).  Eight blocks ahead, twice the threads with half the outputs each, and operands loaded a
// step ahead were no faster: 63 to 69 us instead of 65 at 3,072 x 2,048 and 144 tokens.
#include "common.cuh"

namespace {

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// ------------------------------------------------------------------------------------------------------ few tokens
constexpr int FF_THREADS = 256, FF_KC = 128, FF_LD = FF_KC + 4, FF_MAX_T = 16, FF_MAX_ROWS = 64;
constexpr int FF_RING = 3 * (FF_MAX_ROWS + FF_MAX_T) * FF_LD * 4;      // the most shared memory of a CTA

// 16 bytes of shared memory, loaded where it stands in the program.
__device__ __forceinline__ float4 ff_lds(unsigned a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}

// TT: tokens of a thread.  STAGES: chunks of K in the ring.  rows: features of a tile; CTA c takes tiles c, c + CTAs, ...
template <int TT, int STAGES>
__global__ void __launch_bounds__(FF_THREADS, 2) gemm_f32_few_kernel(const float* __restrict__ X, long long ldx, const float* __restrict__ W,
                                                                     long long ldw, const void* __restrict__ bias, int bias_dtype,
                                                                     void* __restrict__ out, int out_dtype, long long ldo, int T, int N,
                                                                     int K, int rows, int tiles) {
    extern __shared__ float4 ff_smem[];
    float* smem = reinterpret_cast<float*>(ff_smem);
    const int stage_floats = (rows + T) * FF_LD;
    const int chunks = (K + FF_KC - 1) / FF_KC;
    const int n_items = ((tiles - 1 - int(blockIdx.x)) / int(gridDim.x) + 1) * chunks;
    const int tid = threadIdx.x, piece = (tid & 31) * 4;                 // a warp copies one row's 512 bytes
    gb_grid_launch_dependents();
    gb_grid_wait();
    int c_item = 0, c_chunk = 0, c_stage = 0, c_n0 = int(blockIdx.x) * rows;      // the next item to be copied
    // The warps that add have their hands full; where they are few, the others copy (2,048 x 8,192 48 -> 37 us).
    const int adders = (rows * ((T + TT - 1) / TT) + 31) >> 5;
    const int first = adders <= FF_THREADS / 128 ? adders : 0, copiers = FF_THREADS / 32 - first, warp = tid >> 5;
    auto copy = [&] {
        if (warp >= first && c_item < n_items) {
            const int n0 = c_n0, k = c_chunk * FF_KC + piece;
            float* s = smem + c_stage * stage_floats;
            for (int r = warp - first; r < rows + T; r += copiers) {
                const bool is_w = r < rows;
                const bool valid = k < K && (!is_w || n0 + r < N);
                const float* src = is_w ? W + size_t(valid ? n0 + r : 0) * ldw : X + size_t(r - rows) * ldx;
                cp_async16(s + r * FF_LD + piece, src + (valid ? k : 0), valid);
            }
            ++c_item;
            if (++c_chunk == chunks) { c_chunk = 0; c_n0 += int(gridDim.x) * rows; }
            if (++c_stage == STAGES) c_stage = 0;
        }
        cp_async_commit();                                               // a group per item, empty ones too
    };
    for (int i = 0; i < STAGES - 1; ++i) copy();
    const int r = tid % rows, t0 = tid / rows * TT;
    const bool mine = t0 < T;
    float acc[TT];
    int chunk = 0, stage = 0, n = int(blockIdx.x) * rows + r;
    for (int item = 0; item < n_items; ++item) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                                                 // this item is there, and the one before is read
        copy();
        const float* s = smem + stage * stage_floats;
        if (++stage == STAGES) stage = 0;
        if (mine) {
            if (chunk == 0) {
#pragma unroll
                for (int j = 0; j < TT; ++j) acc[j] = 0.f;
            }
            const unsigned wa = unsigned(__cvta_generic_to_shared(s + r * FF_LD));
            unsigned xa[TT];
#pragma unroll
            for (int j = 0; j < TT; ++j) xa[j] = unsigned(__cvta_generic_to_shared(s + (rows + min(t0 + j, T - 1)) * FF_LD));
            // Sixteen steps of K at a time, the next sixteen's operands in registers while these are added: a step is one addition
            // behind another (4.2 cycles), and with the loads left to the compiler, next to their uses, it took 8.3.
            float4 wv[2][4], xv[2][TT][4];
            auto fetch = [&](int g, int buf) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    wv[buf][c] = ff_lds(wa + g * 64 + c * 16);
#pragma unroll
                    for (int j = 0; j < TT; ++j) xv[buf][j][c] = ff_lds(xa[j] + g * 64 + c * 16);
                }
            };
            auto add = [&](int buf) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int j = 0; j < TT; ++j) {
                        const float4 w = wv[buf][c], x = xv[buf][j][c];
                        acc[j] = fmaf(x.x, w.x, acc[j]);
                        acc[j] = fmaf(x.y, w.y, acc[j]);
                        acc[j] = fmaf(x.z, w.z, acc[j]);
                        acc[j] = fmaf(x.w, w.w, acc[j]);
                    }
            };
            fetch(0, 0);
#pragma unroll
            for (int g = 0; g < FF_KC / 16; g += 2) {
                fetch(g + 1, 1);
                add(0);
                if (g + 2 < FF_KC / 16) fetch(g + 2, 0);
                add(1);
            }
        }
        if (++chunk == chunks) {
            chunk = 0;
            if (mine && n < N) {
                const float b = bias ? gb_load(bias, bias_dtype, n) : 0.f;
#pragma unroll
                for (int j = 0; j < TT; ++j)
                    if (t0 + j < T) gb_store(out, out_dtype, size_t(t0 + j) * ldo + n, bias ? acc[j] + b : acc[j]);
            }
            n += int(gridDim.x) * rows;
        }
    }
}

// ----------------------------------------------------------------------------------------------------- more tokens
constexpr int FT_BN = 64, FT_BK = 32, FT_LD = FT_BK + 4, FT_THREADS = 128, FT_STAGES = 4;

// MT: tokens of a thread (8 * MT of a tile); a thread has 4 features.
template <int MT>
__global__ void __launch_bounds__(FT_THREADS) gemm_f32_tile_kernel(const float* __restrict__ X, long long ldx, const float* __restrict__ W,
                                                                   long long ldw, const void* __restrict__ bias, int bias_dtype,
                                                                   void* __restrict__ out, int out_dtype, long long ldo, int T, int N,
                                                                   int K) {
    constexpr int BM = 8 * MT, STAGE = (FT_BN + BM) * FT_LD;
    extern __shared__ float4 ft_smem[];
    float* smem = reinterpret_cast<float*>(ft_smem);                 // stages of W [64][36], X [BM][36]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int n0 = blockIdx.x * FT_BN, t0 = blockIdx.y * BM;
    const int blocks = (K + FT_BK - 1) / FT_BK;
    gb_grid_launch_dependents();
    gb_grid_wait();
    // eight threads copy a row's 32 entries of the block
    auto copy = [&](int kb) {
        if (kb < blocks) {
            float* s = smem + (kb % FT_STAGES) * STAGE;
            const int piece = (tid & 7) * 4, k = kb * FT_BK + piece;
#pragma unroll
            for (int i = 0; i < FT_BN / 16; ++i) {
                const int row = (tid >> 3) + 16 * i, n = n0 + row;
                const bool valid = n < N && k < K;
                cp_async16(s + row * FT_LD + piece, W + (valid ? size_t(n) * ldw + k : 0), valid);
            }
#pragma unroll
            for (int i = 0; i < (BM + 15) / 16; ++i) {
                const int row = (tid >> 3) + 16 * i, t = t0 + row;
                const bool valid = t < T && k < K;
                if (row < BM) cp_async16(s + (FT_BN + row) * FT_LD + piece, X + (valid ? size_t(t) * ldx + k : 0), valid);
            }
        }
        cp_async_commit();                                           // a group per block, empty ones too
    };
    float acc[MT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int i = 0; i < FT_STAGES - 1; ++i) copy(i);
    for (int kb = 0; kb < blocks; ++kb) {
        cp_async_wait<FT_STAGES - 2>();
        __syncthreads();                                             // this block is there, and the one before is read
        copy(kb + FT_STAGES - 1);
        const float* ws = smem + (kb % FT_STAGES) * STAGE + tx * FT_LD;                    // features tx, tx + 16, ...
        const float* xs = smem + (kb % FT_STAGES) * STAGE + (FT_BN + ty * MT) * FT_LD;
#pragma unroll
        for (int kk = 0; kk < FT_BK; kk += 4) {
            float4 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * 16 * FT_LD + kk);
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(xs + i * FT_LD + kk);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int n = n0 + tx + 16 * j;
        if (n >= N) continue;
        const float bv = bias ? gb_load(bias, bias_dtype, n) : 0.f;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int t = t0 + ty * MT + i;
            if (t < T) gb_store(out, out_dtype, size_t(t) * ldo + n, bias ? acc[i][j] + bv : acc[i][j]);
        }
    }
}

int sm_count() {
    static int sms = 0;
    if (!sms) {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) sms = n;
    }
    return sms > 0 ? sms : 1;
}

template <int TT, int STAGES>
int launch_f32_few(int grid, size_t smem, cudaStream_t stream, const float* X, long long ldx, const float* W, long long ldw,
                   const void* bias, int bias_dtype, void* out, int out_dtype, long long ldo, int T, int N, int K, int rows, int tiles) {
    constexpr int MAX_DEVICES = 64;
    static bool configured[MAX_DEVICES] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return gb_fail("gb_gemm_f32: no usable current device");
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(gemm_f32_few_kernel<TT, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, FF_RING) != cudaSuccess)
            return gb_fail("gb_gemm_f32: cannot get %d bytes of shared memory", FF_RING);
        configured[dev] = true;
    }
    gb_launch(gemm_f32_few_kernel<TT, STAGES>, dim3(grid), dim3(FF_THREADS), smem, stream, X, ldx, W, ldw, bias, bias_dtype, out, out_dtype,
              ldo, T, N, K, rows, tiles);
    GB_LAUNCH_OK("gb_gemm_f32");
    return 0;
}

template <int MT>
int launch_f32_tile(dim3 grid, cudaStream_t stream, const float* X, long long ldx, const float* W, long long ldw, const void* bias,
                    int bias_dtype, void* out, int out_dtype, long long ldo, int T, int N, int K) {
    constexpr int MAX_DEVICES = 64;
    constexpr size_t SMEM = size_t(FT_STAGES) * (FT_BN + 8 * MT) * FT_LD * 4;
    static bool configured[MAX_DEVICES] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return gb_fail("gb_gemm_f32: no usable current device");
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(gemm_f32_tile_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SMEM)) != cudaSuccess)
            return gb_fail("gb_gemm_f32: cannot get %zu bytes of shared memory", SMEM);
        configured[dev] = true;
    }
    gb_launch(gemm_f32_tile_kernel<MT>, grid, dim3(FT_THREADS), SMEM, stream, X, ldx, W, ldw, bias, bias_dtype, out, out_dtype, ldo, T, N, K);
    GB_LAUNCH_OK("gb_gemm_f32");
    return 0;
}

}  // namespace

// Whether gb_gemm_f32 takes these operands: 32-bit rows that start on 16 bytes.
GB_API int gb_gemm_f32_supported(const void* X, long long ldx, const void* W, long long ldw, int K) {
    return K > 0 && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(W) & 15) == 0;
}

GB_API int gb_gemm_f32(const float* X, long long ldx, const float* W, long long ldw, const void* bias, int bias_dtype, void* out,
                       int out_dtype, long long ldo, int T, int N, int K, cudaStream_t stream) {
    GB_REQUIRE(gb_is_dtype(out_dtype) && (!bias || gb_is_dtype(bias_dtype)), "gb_gemm_f32: bad dtype");
    GB_REQUIRE(T >= 0 && N > 0 && K > 0 && ldx >= K && ldw >= K && ldo >= N,
               "gb_gemm_f32: bad sizes T=%d N=%d K=%d ldx=%lld ldw=%lld ldo=%lld", T, N, K, ldx, ldw, ldo);
    GB_REQUIRE(gb_gemm_f32_supported(X, ldx, W, ldw, K), "gb_gemm_f32: rows must start on 16 bytes (K=%d, pitches %lld and %lld)", K, ldx, ldw);
    if (T == 0) return 0;
    const int sms = sm_count();
    if (T <= FF_MAX_T) {
        // two CTAs an SM, or one where that leaves each fewer rows than there are tokens to copy beside them
        int ctas = 2 * sms;
        if ((N + ctas - 1) / ctas < T) ctas = sms;
        int rounds = 1;
        while ((N + (long long)rounds * ctas - 1) / ((long long)rounds * ctas) > FF_MAX_ROWS) ++rounds;
        const int rows = int((N + (long long)rounds * ctas - 1) / ((long long)rounds * ctas)), tiles = (N + rows - 1) / rows;
        // A token a thread where two warps hold them all (2,048 x 8,192 at 4 tokens 41 us, 60 with four a thread), else up to
        // four: the row's operands are then read once for all (a head of 128,256 x 2,048 at 4 tokens 219 us, 265 with one).
        int tt = 1;
        while (tt < 4 && rows * ((T + tt - 1) / tt) > 64) tt *= 2;
        const int grid = tiles < ctas ? tiles : ctas;
        // as deep a ring as lets two CTAs share an SM: what is on its way has to cover memory's latency
        const size_t stage = size_t(rows + T) * FF_LD * sizeof(float);
        const int stages = 12 * stage <= 104 * 1024 ? 12 : 6 * stage <= 104 * 1024 ? 6 : 3;
#define FF_LAUNCH(TT, ST) \
    return launch_f32_few<TT, ST>(grid, ST * stage, stream, X, ldx, W, ldw, bias, bias_dtype, out, out_dtype, ldo, T, N, K, rows, tiles)
#define FF_STAGED(TT)                  \
    do {                               \
        if (stages == 12) FF_LAUNCH(TT, 12); \
        if (stages == 6) FF_LAUNCH(TT, 6);   \
        FF_LAUNCH(TT, 3);              \
    } while (0)
        if (tt == 1) FF_STAGED(1);
        if (tt == 2) FF_STAGED(2);
        FF_STAGED(4);
#undef FF_STAGED
#undef FF_LAUNCH
    }
    // the tile whose rounds over the device take the least time; a narrow tile's thread reads more operands per FMA
    static const int MTS[4] = {2, 4, 6, 8};
    static const double COST[4] = {1.4, 1.1, 1.0, 0.97};
    int best = 0;
    double least = 1e300;
    for (int i = 0; i < 4; ++i) {
        const long long tiles = (long long)((N + FT_BN - 1) / FT_BN) * ((T + 8 * MTS[i] - 1) / (8 * MTS[i]));
        const double cost = double((tiles + sms - 1) / sms) * MTS[i] * COST[i];
        if (cost < least) { least = cost; best = i; }
    }
    const int bm = 8 * MTS[best];
    const dim3 grid((N + FT_BN - 1) / FT_BN, (T + bm - 1) / bm);
    GB_REQUIRE(grid.y <= 65535, "gb_gemm_f32: T=%d is too many rows for one launch", T);
    switch (best) {
        case 0: return launch_f32_tile<2>(grid, stream, X, ldx, W, ldw, bias, bias_dtype, out, out_dtype, ldo, T, N, K);
        case 1: return launch_f32_tile<4>(grid, stream, X, ldx, W, ldw, bias, bias_dtype, out, out_dtype, ldo, T, N, K);
        case 2: return launch_f32_tile<6>(grid, stream, X, ldx, W, ldw, bias, bias_dtype, out, out_dtype, ldo, T, N, K);
        default: return launch_f32_tile<8>(grid, stream, X, ldx, W, ldw, bias, bias_dtype, out, out_dtype, ldo, T, N, K);
    }
}
