// Weight-gradient GEMM of the INT2 linear path for sm_100a, plain and fused with the hysteresis update: dW[N,K] = Gq[M,N]^T . Xq[M,K]
// by tcgen05.mma kind::i8, both operands MN-major by TMA, int32 accumulators in tensor memory.
//
// Persistent CTA pairs (cta_group::2) walk output tiles of 256 x 256, each CTA loading 128 columns of either operand and keeping its 128
// rows of the sums; problems of few tiles run on single CTAs with tiles of 128 x 128.  Warp roles:
//   warp 0      TMA producer: both operands of every 128-token block, through a ring of six shared-memory stages of 32 KB
//   warp 1      allocates tensor memory; one lane (of the pair's leader) issues the MMAs and commits them to the ring's barriers
//   warps 2-    epilogue: tcgen05.ld of one of two accumulators while the MMAs fill the other; twelve warps, three per quarter of
//               the tensor-memory lanes, in the plain kernel; sixteen, four per quarter, in the fused one, which its
//               integer instructions bind (two neighbouring 32-column chunks a warp)
//
// A pair's SM takes 32 KB of operands per block of 512 MMA cycles, a single CTA with a tile of 128 x 256 took 48 KB, which at 16 TB/s from
// L2 was its bound.  Fused launch, cold L2, single CTAs / pairs, us: 4096 tokens 4096 -> 11008 137 / 130, 4096 -> 4096 67 / 61, 8192 tokens
// 4096 -> 11008 261 / 229, 16384 tokens 4096 -> 16384 713 / 700.  What binds the fused kernel below 4096 tokens is the
// update's integer instructions (512 tokens 4096 -> 4096: 37 us for 33 us of them; common.cuh has what they took before).
//
// Every wait on an mbarrier is bounded: when it gives up, the kernel records a code in *status, lets its
// outstanding copies land, frees tensor memory and returns.
#include <cuda.h>

#include <atomic>

#include "common.cuh"
#include "epilogue.cuh"
#include "tc_ptx.cuh"

namespace el {

enum { MODE_DW = 2 };
enum { EPI_SCALE = 0, EPI_HYST = 1 };

namespace tc {

constexpr int BM = 128;            // rows of an output tile (UMMA M)
constexpr int BK = 128;            // reduction depth per stage (bytes of int8)
constexpr int UMMA_K = 32;         // reduction depth of one kind::i8 instruction
constexpr int WARP_TMA = 0, WARP_MMA = 1;
__host__ __device__ constexpr int epi_warps(int epi) { return epi == EPI_HYST ? 16 : 12; }
__host__ __device__ constexpr int num_threads(int epi) { return (2 + epi_warps(epi)) * 32; }

constexpr int A_BYTES = BM * BK;                       // 16 KB
constexpr int STAGES = 6;
constexpr int STAGE_BYTES = A_BYTES + 128 * BK;        // a pair's CTAs hold 128 of the 256 columns each
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;

struct Params {
    int R, C, D;                    // output rows, output columns, reduction depth
    int tiles_r, tiles_c, k_blocks;     // tiles_r counts tiles of 128 rows, of 256 for pairs
    int band_rows;                  // row tiles per band of the tile order (see tile_coords)
    EpiParams epi;
    int vec_ok;                     // output rows keep 16-byte alignment
    int32_t* status;
    // hysteresis epilogue
    uint8_t* Wp;
    uint8_t* Hp;
    int pK, pH;
    HystParams hp;
    uint32_t idx_base;
};

// Tile order: bands of `band_rows` row tiles; inside a band the column tiles follow one another and the band's row tiles run
// fastest.  Both operands are streamed along the reduction, and the tiles of a round walk the tokens together: with bands of 2048
// rows a round is near square and needs 2048 + 2368 operand columns, where a round of one or two column tiles needs all rows'
// columns, more than L2 holds from about 6000 tokens on.  Row-fastest / banded (single CTAs, 128 x 256 tiles), us: 6144 tokens 4096 ->
// 11008 223 / 208, 8192 tokens 318 / 294, 65536 tokens 4096 -> 16384 3460 / 2800; 4096 tokens and layers with fewer rows the same.
constexpr int DW_BAND_ROWS = 16;       // of 128
__device__ __forceinline__ void tile_coords(int t, const Params& p, int& tr, int& tc) {
    const int per_band = p.band_rows * p.tiles_c;
    const int band = t / per_band, in = t - band * per_band;
    const int first = band * p.band_rows;
    const int rows_here = min(p.band_rows, p.tiles_r - first);
    tc = in / rows_here;
    tr = first + (in - tc * rows_here);
}

// ---- the kernel ----------------------------------------------------------------------------------------------

template <bool PAIR, int EPI>
__global__ void __launch_bounds__(num_threads(EPI), 1)
gemm_dw_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Params p) {
    constexpr int BN = PAIR ? 256 : 128, TM = PAIR ? 2 * BM : BM;      // output tile: TM x BN
    constexpr uint32_t TMEM_COLS = 2 * BN;     // two accumulators of BN int32 columns (256 or 512: powers of two)

    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    // stage s: [A 16K][B 16K]
    const uint32_t bars = smem_base + STAGES * STAGE_BYTES;
    uint8_t* bars_gen = smem_gen + STAGES * STAGE_BYTES;
    auto bar_full = [&](int s) { return bars + 8u * s; };
    auto bar_empty = [&](int s) { return bars + 8u * (STAGES + s); };
    auto bar_tfull = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto bar_tempty = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };
    volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(bars_gen + 8 * (2 * STAGES + 4));

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int num_tiles = p.tiles_r * p.tiles_c;
    const int rank = PAIR ? (int)cluster_ctarank() : 0;         // 0 = leader: its "full" and "tempty" barriers are used
    const int first_tile = PAIR ? blockIdx.x >> 1 : blockIdx.x, tile_step = PAIR ? gridDim.x >> 1 : gridDim.x;
    auto wait = [&](uint32_t bar, uint32_t parity, int code) {  // whole warp; arrivals of a pair come from both CTAs
        return PAIR ? mbar_wait_cluster_warp(bar, parity, p.status, code) : mbar_wait_warp(bar, parity, p.status, code);
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bar_full(s), 1);
            mbar_init(bar_empty(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(bar_tfull(a), 1);
            mbar_init(bar_tempty(a), (PAIR ? 2 : 1) * epi_warps(EPI));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == WARP_MMA) {     // both CTAs of a pair take part in the allocation
        const uint32_t holder = smem_u32((const void*)tmem_holder);
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(holder), "r"(TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(holder), "r"(TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();          // the peer's barriers are initialised before anything signals them
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    bool failed = false;

    if (warp == WARP_TMA) {
        // ================= producer =================
        griddep_wait();
        int s = 0;
        uint32_t ph = 0;
        for (int t = first_tile; t < num_tiles && !failed; t += tile_step) {
            int tr, tc;
            tile_coords(t, p, tr, tc);
            const int r0 = tr * TM + rank * BM, c0 = tc * BN + rank * 128;
            for (int kb = 0; kb < p.k_blocks; ++kb) {
                if (!wait(bar_empty(s), ph ^ 1u, 1)) { failed = true; break; }
                if (elect_one()) {
                    const uint32_t sa = smem_base + s * STAGE_BYTES, sb = sa + A_BYTES;
                    const int d0 = kb * BK;
                    if (rank == 0) mbar_expect_tx(bar_full(s), (PAIR ? 2 : 1) * STAGE_BYTES);
                    if (PAIR) {
                        const uint32_t bar = mapa_u32(bar_full(s), 0);
                        tma_load_2d_pair(sa, &tmA, bar, r0, d0);                 // Gq  [128 m-rows x 128 n]
                        tma_load_2d_pair(sb, &tmB, bar, c0, d0);                 // Xq  [128 m-rows x 128 k]
                    } else {
                        tma_load_2d(sa, &tmA, bar_full(s), r0, d0);
                        tma_load_2d(sb, &tmB, bar_full(s), c0, d0);
                    }
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp == WARP_MMA) {
        // ================= MMA issuer =================
        if (rank == 0) {
            constexpr uint32_t idesc = make_idesc(1, 1, BN, TM);
            int s = 0;
            uint32_t ph = 0;
            int it = 0;
            for (int t = first_tile; t < num_tiles && !failed; t += tile_step, ++it) {
                const int acc = it & 1;
                const uint32_t acc_ph = (uint32_t)(it >> 1) & 1u;
                if (!wait(bar_tempty(acc), acc_ph ^ 1u, 2)) { failed = true; break; }
                tcgen05_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
                for (int kb = 0; kb < p.k_blocks; ++kb) {
                    if (!wait(bar_full(s), ph, 3)) { failed = true; break; }
                    tcgen05_fence_after();
                    if (elect_one()) {
                        const uint32_t sa = smem_base + s * STAGE_BYTES, sb = sa + A_BYTES;
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k) {
                            // MN-major: step 32 reduction rows of 128 bytes
                            const uint64_t da = make_desc(sa + k * 4096, 16384), db = make_desc(sb + k * 4096, 16384);
                            if (PAIR) umma_i8_pair(d_tmem, da, db, idesc, (kb | k) != 0);
                            else umma_i8(d_tmem, da, db, idesc, (kb | k) != 0);
                        }
                        if (PAIR) umma_commit_pair(bar_empty(s));
                        else umma_commit(bar_empty(s));
                    }
                    __syncwarp();
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
                if (!failed && elect_one()) {
                    if (PAIR) umma_commit_pair(bar_tfull(acc));
                    else umma_commit(bar_tfull(acc));
                }
                __syncwarp();
            }
        }
    } else {
        // ================= epilogue =================
        // the warps of a quarter of the tensor-memory lanes take the 32-column chunks round-robin
        constexpr int EPI_SPLIT = epi_warps(EPI) / 4;
        const int quarter = warp & 3;                 // the tensor-memory lanes this warp may read
        const int sub = (warp - 2) >> 2;              // 0 for warps 2-5, 1 for 6-9, 2 for 10-13, 3 for 14-17
        const int row_in_tile = quarter * 32 + lane;
        griddep_wait();
        const float hyst_scale = EPI == EPI_HYST ? epi_row_scale(p.epi, 0) : 0.0f;      // g_absmax/127 (one scale for the tensor)
        HystParams hp;                                // with the step taken from device memory when the launch says so
        if (EPI == EPI_HYST) hp = hyst_resolve_step(p.hp);
        int it = 0;
        for (int t = first_tile; t < num_tiles && !failed; t += tile_step, ++it) {
            int tr, tc;
            tile_coords(t, p, tr, tc);
            const int r0 = tr * TM + rank * BM, c0 = tc * BN;
            const int acc = it & 1;
            const uint32_t acc_ph = (uint32_t)(it >> 1) & 1u;
            const int row = r0 + row_in_tile;
            const bool row_ok = row < p.R;
            // Fused update: the packed weights and counters of this warp's chunks do not depend on the accumulator, so they
            // are requested before the wait for it and arrive while the tile's MMAs still run.
            constexpr int HYST_CHUNKS = EPI == EPI_HYST ? BN / 32 / EPI_SPLIT : 1;      // 2, or 1 for narrow tiles: neighbours
            uint2 w_pre[HYST_CHUNKS];
            uint4 h_pre[HYST_CHUNKS];
            if (EPI == EPI_HYST) {
#pragma unroll
                for (int i = 0; i < HYST_CHUNKS; ++i) {
                    const int c = sub * HYST_CHUNKS + i;
                    const int col0 = c0 + c * 32;
                    if (row_ok && col0 < p.C) {     // K % 32 == 0: a chunk is inside or outside as a whole
                        w_pre[i] = *reinterpret_cast<const uint2*>(p.Wp + (size_t)row * p.pK + (col0 >> 2));
                        h_pre[i] = *reinterpret_cast<const uint4*>(p.Hp + (size_t)row * p.pH + (col0 >> 1));
                    }
                }
            }
            if (!mbar_wait_warp(bar_tfull(acc), acc_ph, p.status, 5)) { failed = true; break; }
            tcgen05_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN);
            if (EPI == EPI_SCALE) {
                const float sc = row_ok ? epi_row_scale(p.epi, row) : 0.0f;
#pragma unroll 1
                for (int c = sub; c < BN / 32; c += EPI_SPLIT) {
                    uint32_t v[32];
                    tmem_ld32(taddr + c * 32, v);
                    tmem_ld_wait();
                    const int col0 = c0 + c * 32;
                    if (row_ok && col0 < p.C) epi_store_chunk32(p.epi, row, col0, p.C, v, sc, p.vec_ok != 0);
                }
            } else {
                // weight-gradient tile -> hysteresis update of 32 weights of row `row` per chunk
                // (not unrolled: the update is 17 KB of code, and two copies of it ran out of the instruction cache)
#pragma unroll 1
                for (int i = 0; i < HYST_CHUNKS; ++i) {
                    const int c = sub * HYST_CHUNKS + i;
                    uint32_t v[32];
                    tmem_ld32(taddr + c * 32, v);
                    tmem_ld_wait();
                    const int col0 = c0 + c * 32;
                    if (row_ok && col0 < p.C) {
                        uint32_t w[2] = {w_pre[0].x, w_pre[0].y};
                        uint32_t h[4] = {h_pre[0].x, h_pre[0].y, h_pre[0].z, h_pre[0].w};
                        const uint32_t idx0 = p.idx_base + (uint32_t)row * (uint32_t)p.C + (uint32_t)col0;
                        if ((p.idx_base & 31u) == 0) hyst_update_chunk32<true, true>(v, hyst_scale, w, h, idx0, hp);     // C % 32 == 0
                        else hyst_update_chunk32<true, false>(v, hyst_scale, w, h, idx0, hp);
                        *reinterpret_cast<uint2*>(p.Wp + (size_t)row * p.pK + (col0 >> 2)) = make_uint2(w[0], w[1]);
                        *reinterpret_cast<uint4*>(p.Hp + (size_t)row * p.pH + (col0 >> 1)) = make_uint4(h[0], h[1], h[2], h[3]);
                    }
#pragma unroll
                    for (int k = 0; k + 1 < HYST_CHUNKS; ++k) w_pre[k] = w_pre[k + 1], h_pre[k] = h_pre[k + 1];
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_cluster_relaxed(mapa_u32(bar_tempty(acc), 0));     // only tensor memory was read
                else mbar_arrive(bar_tempty(acc));
            }
        }
    }

    // ---- teardown ------------------------------------------------------------------------------------------------
    if (p.status != nullptr && *reinterpret_cast<volatile int32_t*>(p.status) != 0) {
        // a wait gave up somewhere: give copies and MMAs still in flight time to land before the CTA's
        // shared and tensor memory are released
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();          // both CTAs are done with each other's shared and tensor memory
    if (warp == WARP_MMA) {
        tcgen05_fence_after();
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// ---- host side -------------------------------------------------------------------------------------------------

template <bool PAIR, int EPI>
static int launch_t(const CUtensorMap& tmA, const CUtensorMap& tmB, Params& p, cudaStream_t st) {
    static std::atomic<int> max_ctas[64];       // co-resident CTAs (of pairs) per device; 0 = not yet queried
    int dev = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return EL_ERR_DEVICE;
    constexpr int TM = PAIR ? 2 * BM : BM, BN = PAIR ? 256 : 128, BAND = DW_BAND_ROWS * BM / TM;
    p.tiles_r = (p.R + TM - 1) / TM;
    p.tiles_c = (p.C + BN - 1) / BN;
    p.k_blocks = (p.D + BK - 1) / BK;
    p.band_rows = p.tiles_r > BAND ? BAND : p.tiles_r;
    const long long tiles = (long long)p.tiles_r * p.tiles_c;
    if (tiles == 0) return EL_OK;
    if (p.k_blocks == 0) return EL_ERR_UNSUPPORTED_SHAPE;
    cudaLaunchConfig_t cfg = {};
    // a programmatic dependent launch, as in gemm_wt.cu: the warps that touch global memory wait (griddep_wait)
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.blockDim = dim3(num_threads(EPI), 1, 1);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = st;
    int ctas = max_ctas[dev].load(std::memory_order_acquire);
    if (ctas == 0) {       // host threads may race here: both then query and store the same number
        EL_CUDA_TRY(cudaFuncSetAttribute(gemm_dw_kernel<PAIR, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        const int rc = device_sm_count(&ctas);
        if (rc != EL_OK) return rc;
        if (PAIR) {
            int clusters = 0;
            cfg.attrs = attr + 1;          // the occupancy query knows clusters only
            cfg.numAttrs = 1;
            cfg.gridDim = dim3((unsigned)(ctas & ~1), 1, 1);
            EL_CUDA_TRY(cudaOccupancyMaxActiveClusters(&clusters, gemm_dw_kernel<PAIR, EPI>, &cfg));
            if (clusters < 1) return EL_ERR_DEVICE;
            ctas = 2 * clusters < ctas ? 2 * clusters : ctas & ~1;
        }
        max_ctas[dev].store(ctas, std::memory_order_release);
    }
    cfg.attrs = attr;
    cfg.numAttrs = PAIR ? 2 : 1;
    const long long want = PAIR ? 2 * tiles : tiles;
    cfg.gridDim = dim3((unsigned)(want < ctas ? want : ctas), 1, 1);
    EL_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_dw_kernel<PAIR, EPI>, tmA, tmB, p));
    return check_launch();
}

}  // namespace tc

namespace tc {
int make_map(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch, uint32_t box_cols,
             uint32_t box_rows, int swizzle_bytes);
}
int gemm_tc_eligible(int mode, const void* A, const void* B, int R, int C, int D);

// 128-column tiles where 256-column ones would leave half of the SMs without a tile.  Fused weight gradient, 256- / 128-column
// tiles: 1024 tokens 1536 -> 1536 16.9 / 10.8 us, 4096 tokens 4096 -> 512 23.9 / 17.5.
static bool narrow_tiles(int R, int C) {
    int sms = 0;
    if (device_sm_count(&sms) != EL_OK) return false;
    return 2LL * ((R + tc::BM - 1) / tc::BM) * ((C + 255) / 256) <= sms;
}

int launch_gemm_dw(const int8_t* Gq, const int8_t* Xq, int R, int C, int D, const EpiParams& epi, int32_t* status, cudaStream_t st) {
    int rc = gemm_tc_eligible(MODE_DW, Gq, Xq, R, C, D);
    if (rc != EL_OK) return rc;
    rc = require_sm100();
    if (rc != EL_OK) return rc;
    tc::Params p{};
    p.R = R; p.C = C; p.D = D;
    p.epi = epi;
    p.status = status;
    const int esz = (epi.out_dtype == EL_BF16 || epi.out_dtype == EL_F16) ? 2 : 4;
    p.vec_ok = ((reinterpret_cast<uintptr_t>(epi.out) & 15) == 0) && ((epi.ldo * esz) % 16 == 0);
    CUtensorMap tmA, tmB;
    if ((rc = tc::make_map(&tmA, Gq, R, D, R, 128, 128, 128)) != EL_OK) return rc;
    if ((rc = tc::make_map(&tmB, Xq, C, D, C, 128, 128, 128)) != EL_OK) return rc;
    return narrow_tiles(R, C) ? tc::launch_t<false, EPI_SCALE>(tmA, tmB, p, st) : tc::launch_t<true, EPI_SCALE>(tmA, tmB, p, st);
}

int launch_dw_hysteresis_tc(const int8_t* Gq, const int8_t* Xq, const float* g_absmax, uint8_t* Wp, uint8_t* Hp,
                            const HystParams& hp, uint32_t idx_base, int M, int N, int K, int32_t* status, cudaStream_t st) {
    int rc = gemm_tc_eligible(MODE_DW, Gq, Xq, N, K, M);
    if (rc != EL_OK) return rc;
    if (K % 32 != 0) return EL_ERR_UNSUPPORTED_SHAPE;
    if ((reinterpret_cast<uintptr_t>(Wp) & 7) || (reinterpret_cast<uintptr_t>(Hp) & 15)) return EL_ERR_ALIGNMENT;
    rc = require_sm100();
    if (rc != EL_OK) return rc;
    tc::Params p{};
    p.R = N; p.C = K; p.D = M;
    p.epi = EpiParams{nullptr, 0, EL_F32, g_absmax, 0, 1.0f};
    p.status = status;
    p.Wp = Wp; p.Hp = Hp; p.pK = K / 4; p.pH = K / 2;
    p.hp = hp; p.idx_base = idx_base;
    CUtensorMap tmA, tmB;
    if ((rc = tc::make_map(&tmA, Gq, N, M, N, 128, 128, 128)) != EL_OK) return rc;
    if ((rc = tc::make_map(&tmB, Xq, K, M, K, 128, 128, 128)) != EL_OK) return rc;
    return narrow_tiles(N, K) ? tc::launch_t<false, EPI_HYST>(tmA, tmB, p, st) : tc::launch_t<true, EPI_HYST>(tmA, tmB, p, st);
}

}  // namespace el
