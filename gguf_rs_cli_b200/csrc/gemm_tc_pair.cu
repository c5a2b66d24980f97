// The tensor-core product of gemm_tc.cu for steps of many tokens, with two CTAs on two SMs per output tile of
// 256 features x up to 256 tokens (tcgen05 cta_group::2; the width that wastes least of the last round over the device is
// chosen per product).  Each CTA of the pair loads its 128 features of W and its half of the tile's
// tokens of X for every block of K (32 KB a stage instead of the 48 KB a lone CTA needs for 128 x 256:
// a third less traffic from L2 into shared memory, and room for 6 stages), one thread of the even CTA (the
// leader) issues the MMAs for both, each CTA's TMEM gets its 128 features of the result, and each CTA's four
// epilogue warps finish those with the code the other kernel uses.
//
// Barriers: loads of both CTAs count their bytes on the leader's `full` barriers; the leader's MMA thread
// frees a stage in both CTAs and announces a finished accumulator to both with one multicast commit; the
// epilogue warps of both CTAs arrive on the leader's `acc_empty`.  Every wait is bounded (status word as in
// gemm_tc.cu); the cluster barriers at the start and at the end are reached by every thread on every path.
#include "gemm_tc.cuh"

using namespace sm100;

namespace {

constexpr int PBN = 256;                    // most tokens per tile
constexpr int PHALF = PBN / 2;              // most tokens a CTA loads
constexpr int PSTAGES = 6;
constexpr int PSTAGE_BYTES = A_BYTES + PHALF * BK * 2;         // per CTA
constexpr int POUT_CHUNK = 16 * BM * 2;      // a staged piece of the result: 16 tokens x 128 features of bf16
constexpr int POUT_RING = 4;                // pieces in flight to global memory
constexpr int PSMEM = PSTAGES * PSTAGE_BYTES + POUT_RING * POUT_CHUNK + 1024;
constexpr int PTMEM_COLS = 2 * PBN;         // two accumulators
constexpr int PMAX_DEVICES = 64;

struct PairUnit {
    int n0, t0;                             // first feature and first token of the tile
};
// Tiles in the order of gemm_tc.cu's units: token tiles in groups of TILE_GROUP, inside a group feature tile
// by feature tile with the group's token tiles innermost.
__device__ __forceinline__ PairUnit pair_unit_of(int u, int feature_tiles, int token_tiles, int bn) {
    const int per_group = TILE_GROUP * feature_tiles;
    const int group = u / per_group, r = u - group * per_group;
    const int group_start = group * TILE_GROUP;
    const int group_size = min(TILE_GROUP, token_tiles - group_start);
    const int ft = r / group_size;
    PairUnit w;
    w.n0 = ft * (2 * BM);
    w.t0 = (group_start + (r - ft * group_size)) * bn;
    return w;
}

template <bool STAGED>
__global__ void __launch_bounds__(TC_THREADS, 1) gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                     const __grid_constant__ CUtensorMap map_x,
                                                                     const __grid_constant__ CUtensorMap map_o, TcParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* out_ring = ring + PSTAGES * PSTAGE_BYTES;
    __shared__ uint64_t full_bar[PSTAGES], empty_bar[PSTAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base;
    __shared__ float rstd_s[PBN];
    __shared__ float part_s[128];
    __shared__ float ssq_s[4][PBN];

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();               // 0: leader
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int kb_total = (p.K + BK - 1) / BK;
    const int feature_tiles = (p.N + 2 * BM - 1) / (2 * BM);
    const int bn = p.pair_tile;                             // tokens of a tile, a multiple of 16 up to PBN
    const int token_tiles = (p.T + bn - 1) / bn;
    const int n_units = feature_tiles * token_tiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < PSTAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
        fence_barrier_init();
        prefetch_tensormap(&map_w);
        prefetch_tensormap(&map_x);
    }
    if (warp == 1) {
        tmem_alloc_pair(&tmem_base, PTMEM_COLS);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    cluster_sync_all();                             // both CTAs' barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_d = tmem_base;
    gb_grid_launch_dependents();

    if (warp == 0) {
        if (elect_one()) {
            // ---- producer (both CTAs): this CTA's half of W's and of X's rows for every stage
            gb_grid_wait();
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int u = pair; u < n_units && ok; u += n_pairs) {
                const PairUnit w = pair_unit_of(u, feature_tiles, token_tiles, bn);
                // several products in one launch: the tile's tokens belong to one of them, whose features lie
                // that many times N further down in W
                const int w_first = p.group_t > 0 ? (w.t0 / p.group_t) * p.N : 0;
                for (int kb = 0; kb < kb_total; ++kb) {
                    if (!mbar_wait(&empty_bar[stage], phase ^ 1)) { atomicExch(p.status, 1); ok = false; break; }
                    if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * A_BYTES + bn * BK * 2);
                    uint8_t* a = ring + stage * PSTAGE_BYTES;
                    tma_load_2d_pair(a, &map_w, kb * BK, w_first + w.n0 + int(rank) * BM, &full_bar[stage]);
                    tma_load_2d_pair(a + A_BYTES, &map_x, kb * BK, w.t0 + int(rank) * (bn >> 1), &full_bar[stage]);
                    if (++stage == PSTAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            // ---- MMA issue (leader): 256 x bn x 16 per instruction over the pair
            const uint32_t idesc = instr_desc_bf16(2 * BM, bn);
            const uint64_t ring_desc = smem_desc_sw128(smem_u32(ring));        // an address further on is added in units of 16 bytes
            int stage = 0, j = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int u = pair; u < n_units && ok; u += n_pairs, ++j) {
                const int buf = j & 1;
                if (!mbar_wait(&acc_empty[buf], ((j >> 1) & 1) ^ 1)) { atomicExch(p.status, 4); ok = false; break; }
                tc_fence_after();
                const uint32_t acc = tmem_d + buf * PBN;
                for (int kb = 0; kb < kb_total; ++kb) {
                    if (!mbar_wait(&full_bar[stage], phase)) { atomicExch(p.status, 2); ok = false; break; }
                    tc_fence_after();
                    const uint64_t a = ring_desc + uint64_t(stage) * (PSTAGE_BYTES >> 4), b = a + (A_BYTES >> 4);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        mma_f16_pair(acc, a + k * (UMMA_K * 2 >> 4), b + k * (UMMA_K * 2 >> 4), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    mma_commit_pair(&empty_bar[stage]);
                    if (++stage == PSTAGES) { stage = 0; phase ^= 1; }
                }
                mma_commit_pair(&acc_full[buf]);
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue (both CTAs): this CTA's 128 features of the tile, warp w reads TMEM lanes 32*(w%4) .. +31
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        gb_grid_wait();
        int j = 0, piece = 0;
        for (int u = pair; u < n_units; u += n_pairs, ++j) {
            const PairUnit w = pair_unit_of(u, feature_tiles, token_tiles, bn);
            const int buf = j & 1;
            const int n0 = w.n0 + int(rank) * BM;
            const int n = n0 + row;
            const int cols = min(bn, p.T - w.t0);
            if (p.row_ssq) tc_token_scales<PBN>(p, w.t0, cols, row, rstd_s, part_s);
            const bool waited = mbar_wait(&acc_full[buf], (j >> 1) & 1);
            if (!waited) {
                if (lane == 0) atomicExch(p.status, 3);
                break;
            }
            tc_fence_after();
            const uint32_t taddr = tmem_d + (uint32_t(quarter * 32) << 16) + buf * PBN;
            float bias = 0.f;
            if (p.bias && n < p.N) bias = gb_load(p.bias, p.bias_dtype, n);
            if constexpr (STAGED) {
                // bf16 results: 16 tokens at a time into a ring of shared-memory pieces [token][feature], each
                // sent on its way by one TMA store (the scattered 2-byte stores from registers would take as
                // long as the tile's multiplications)
                for (int c0 = 0; c0 < cols; c0 += 16, ++piece) {
                    float v[16];
                    tmem_ld16(taddr + c0, v);
                    if (p.row_ssq) {
#pragma unroll
                        for (int jj = 0; jj < 16; ++jj) v[jj] *= rstd_s[min(c0 + jj, PBN - 1)];
                    }
                    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(out_ring + (piece % POUT_RING) * POUT_CHUNK);
                    if (threadIdx.x == 64) tma_store_source_free<POUT_RING - 1>();      // the piece's last store has read it
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (!p.swiglu) {
#pragma unroll
                        for (int jj = 0; jj < 16; ++jj) dst[jj * BM + row] = __float2bfloat16_rn(v[jj] + bias);
                    } else {
                        // even rows are gate features, odd rows the matching up features (see tc_finish_chunk)
                        const bool odd = lane & 1;
                        float other[8];
#pragma unroll
                        for (int jj = 0; jj < 8; ++jj) other[jj] = __shfl_xor_sync(0xffffffffu, odd ? v[jj] : v[8 + jj], 1);
#pragma unroll
                        for (int jj = 0; jj < 8; ++jj) {
                            const float gte = odd ? other[jj] : v[jj], up = odd ? v[8 + jj] : other[jj];
                            dst[((odd ? 8 : 0) + jj) * (BM / 2) + (row >> 1)] = __float2bfloat16_rn(gb_gate_act(gte, p.swiglu) * up);
                        }
                    }
                    fence_proxy_async();
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (threadIdx.x == 64 && waited)
                        tma_store_2d(&map_o, p.swiglu ? (n0 >> 1) : n0, w.t0 + c0, dst);
                }
            } else {
                for (int c0 = 0; c0 < cols; c0 += 16) {
                    float v[16];
                    tmem_ld16(taddr + c0, v);
                    tc_finish_chunk<PBN>(p, n0, w.t0, n, row, lane, quarter, bias, waited, c0, cols, v, rstd_s, ssq_s);
                }
                // where the last tile's features end in its first half, the other CTA has none: no sums to write, and no room for them
                if (p.resid_x && n0 < p.N) tc_write_ssq<PBN>(p, n0, w.t0, row, 0, cols, ssq_s);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(&acc_empty[buf], 0);      // the leader may overwrite this accumulator
        }
        if (STAGED && threadIdx.x == 64) tma_store_done();
    }
    // nobody leaves while its partner may still read its shared memory or arrive on its barriers
    tc_fence_before();
    cluster_sync_all();
    if (warp == 1) tmem_dealloc_pair(tmem_d, PTMEM_COLS);
}

}  // namespace

// A tuning aid (process-wide): > 0: tokens of every tile, in the steps that the MMA and the output's pieces of 16 tokens allow.
static int g_pair_tile = 0;
GB_API int gb_gemm_tc_set_pair_tile(int bn) {
    GB_REQUIRE(bn == 0 || (bn >= 32 && bn <= PBN && bn % 16 == 0), "gb_gemm_tc_set_pair_tile: %d is no multiple of 16 from 32 to %d", bn, PBN);
    g_pair_tile = bn;
    return 0;
}

// Raises the kernel's shared-memory limit on the current device, on its first call there; 0: done.
static int pair_ready(int* dev) {
    static bool configured[PMAX_DEVICES] = {};
    if (cudaGetDevice(dev) != cudaSuccess || *dev < 0 || *dev >= PMAX_DEVICES) return gb_fail("gb_gemm_tc: no usable current device");
    if (!configured[*dev]) {
        if (cudaFuncSetAttribute(gemm_tc_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PSMEM) != cudaSuccess ||
            cudaFuncSetAttribute(gemm_tc_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PSMEM) != cudaSuccess) {
            cudaGetLastError();
            return gb_fail("gb_gemm_tc: cannot get %d bytes of shared memory", PSMEM);
        }
        configured[*dev] = true;
    }
    return 0;
}

// How many pairs of CTAs of this kernel the current device holds at once (0 if it cannot be asked; then it is asked again).  The
// question is refused for more shared memory than the kernel's limit, so that comes first.
GB_API int gb_gemm_tc_pair_slots() {
    static int slots[PMAX_DEVICES] = {};
    int dev = 0;
    if (pair_ready(&dev)) return 0;
    if (slots[dev] == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2);
        cfg.blockDim = dim3(TC_THREADS);
        cfg.dynamicSmemBytes = PSMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_tc_pair_kernel<true>, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
        slots[dev] = n;
    }
    return slots[dev];
}

static long long pair_slots(int sms) {
    const int n = gb_gemm_tc_pair_slots();
    return n > 0 ? n : sms / 2;
}

// Tokens of a tile: the width whose rounds over the device take the least time.  A 256 x bn tile over K takes a time
// proportional to bn down to about 176 and hardly less below (512 x 4096 x 4096, one round: 29.5 us at 256, 23.6 at 176, 22.2 at 160,
// 21.4 at 128: what is left is the loads' pace), and a narrower one reads W more often, so 176 is the narrowest.  2048 x 6144 x 4096:
// four rounds of 176 74 us, three of 240 80, three of 256 84; 7001 x 4096 x 14336: seven rounds of 224 639, seven of 256 726;
// 512 x 4096 x 14336: one round of 176 58, of 256 84.  Of equal costs the widest.
int gemm_tc_pair_tile(int T, int N, int sms) {
    if (g_pair_tile > 0) return g_pair_tile;
    const long long ft = (N + 2 * BM - 1) / (2 * BM), slots = pair_slots(sms);
    int best = PBN;
    long long least = -1;
    for (int bn = PBN; bn >= 176; bn -= 16) {
        const long long units = ft * ((T + bn - 1) / bn), cost = (units + slots - 1) / slots * bn;
        if (least < 0 || cost < least) { least = cost; best = bn; }
    }
    return best;
}

int gemm_tc_pair_launch(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap* mo, const void* params,
                        cudaStream_t stream) {
    const TcParams& p = *static_cast<const TcParams*>(params);
    int dev = 0;
    if (pair_ready(&dev)) return 1;
    long long units = (long long)((p.N + 2 * BM - 1) / (2 * BM)) * ((p.T + p.pair_tile - 1) / p.pair_tile);
    long long slots = pair_slots(p.sms);                                // pairs that can be resident at once
    long long rounds = (units + slots - 1) / slots;
    long long pairs = (units + rounds - 1) / rounds;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = PSMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gb_pdl_enabled() ? 2 : 1;
    if (mo)
        cudaLaunchKernelEx(&cfg, gemm_tc_pair_kernel<true>, mw, mx, *mo, p);
    else
        cudaLaunchKernelEx(&cfg, gemm_tc_pair_kernel<false>, mw, mx, mx, p);
    GB_LAUNCH_OK("gb_gemm_tc (pair)");
    return 0;
}
