// Forward and dX of layers with 16, 32 or 48 inputs (the Mamba step-size projection has 16): pitches that the tensor maps
// of the large GEMMs cannot take, and a shape whose time is the traffic of its one wide matrix.
//
//   FWD  Y [R,C] = Xq [R,D] . Wq[C,D]^T, D in {16,32,48}: the time to write Y
//   DX   dX[R,C] = dYq[R,D] . Wq[D,C],   C in {16,32,48}: the time to read dYq
//
// Both feed the warp-level int8 MMA: the reduction (FWD) or the output (DX) is narrower than any tcgen05 tile, so a tile
// there would be mostly padding, and the products are few.  The weights are expanded once per CTA - into registers (FWD)
// or shared memory (DX) - and serve all rows that the CTA walks over.
// bf16, 2048 tokens, 16 inputs, 8192 outputs: FWD 8.5 us, DX 8.6 us; the 64x64 CUDA-core kernel (gemm_simple.cu), which took
// these shapes before, runs 57.7 us (a fifth of the threads' time in byte-wise staging) and 459 us (32 CTAs, each walking all
// 8192 reduction indices).
#include "common.cuh"
#include "epilogue.cuh"

namespace el {

enum { MODE_FWD = 0, MODE_DX = 1 };

namespace {

__device__ __forceinline__ void mma_s8_k16(int d[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ void mma_s8_k32(int d[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the four codes of one packed byte as four int8 (code 0 lowest)
__device__ __forceinline__ uint32_t decode4(uint32_t b) {
    const uint32_t sel = (b & 0x3u) | ((b & 0xCu) << 2) | ((b & 0x30u) << 4) | ((b & 0xC0u) << 6);
    return __byte_perm(0x000100FFu, 0, sel);
}

// ---- forward ------------------------------------------------------------------------------------------------------------
// A warp keeps the expanded weights of 64 output columns in registers and walks over row tiles of 16; the eight warps of a
// CTA cover 512 columns.  Column c of MMA j stands for output column (c>>1)*V + 2j + (c&1) of its group, V = 16 bytes of
// outputs, so a lane ends up with V consecutive outputs of a row and four lanes store 64 consecutive bytes: whole
// 32-byte sectors with every store.  KS: reduction steps of 16.
constexpr int SF_WARPS = 8, SF_COLS = 64;

template <int KS, int DT>
__global__ void __launch_bounds__(SF_WARPS * 32)
skinny_fwd_kernel(const int8_t* __restrict__ Xq, const uint8_t* __restrict__ Wp, EpiParams epi, int R, int C) {
    constexpr bool TWO = (DT == EL_BF16 || DT == EL_F16);
    constexpr int V = TWO ? 8 : 4;                  // outputs per 16-byte store
    constexpr int J = V / 2;                        // MMAs per group of 4*V columns
    constexpr int G = SF_COLS / (4 * V);            // groups per warp
    constexpr int D = KS * 16, PD = KS * 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r8 = lane >> 2, q = lane & 3;
    const int n0 = (blockIdx.x * SF_WARPS + warp) * SF_COLS;
    if (n0 >= C) return;
    uint32_t b[G][J][KS];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int n = n0 + g * 4 * V + (r8 >> 1) * V + 2 * j + (r8 & 1);      // lane>>2 is the MMA's column here
#pragma unroll
            for (int s = 0; s < KS; ++s) b[g][j][s] = n < C ? decode4(__ldg(Wp + (size_t)n * PD + s * 4 + q)) : 0u;
        }
    const int tiles = (R + 15) >> 4;
    for (int t = blockIdx.y; t < tiles; t += gridDim.y) {
        const int row0 = t * 16 + r8, row1 = row0 + 8;
        uint32_t a0[KS], a1[KS];
#pragma unroll
        for (int s = 0; s < KS; ++s) {
            a0[s] = row0 < R ? __ldg(reinterpret_cast<const uint32_t*>(Xq + (size_t)row0 * D + s * 16) + q) : 0u;
            a1[s] = row1 < R ? __ldg(reinterpret_cast<const uint32_t*>(Xq + (size_t)row1 * D + s * 16) + q) : 0u;
        }
        const float sc0 = row0 < R ? epi_row_scale(epi, row0) : 0.0f, sc1 = row1 < R ? epi_row_scale(epi, row1) : 0.0f;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            int d[J][4];
#pragma unroll
            for (int j = 0; j < J; ++j) {
                d[j][0] = d[j][1] = d[j][2] = d[j][3] = 0;
#pragma unroll
                for (int s = 0; s < KS; ++s) mma_s8_k16(d[j], a0[s], a1[s], b[g][j][s]);
            }
            const int col = n0 + g * 4 * V + q * V;
            if (col >= C) continue;                  // C is a multiple of V: a lane's V outputs are inside or outside together
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = h ? row1 : row0;
                const float sc = h ? sc1 : sc0;
                if (row >= R) continue;
                uint32_t w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (TWO) {
                        const float lo = __fmul_rn((float)d[i % J][2 * h], sc), hi = __fmul_rn((float)d[i % J][2 * h + 1], sc);
                        w[i] = DT == EL_BF16 ? pack_bf16x2(lo, hi) : pack_f16x2(lo, hi);
                    } else {
                        const int v = d[i >> 1][2 * h + (i & 1)];
                        w[i] = DT == EL_F32 ? __float_as_uint(__fmul_rn((float)v, sc)) : (uint32_t)v;
                    }
                }
                char* out = static_cast<char*>(epi.out) + ((size_t)row * epi.ldo + col) * (TWO ? 2 : 4);
                *reinterpret_cast<uint4*>(out) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
    }
}

// ---- dX -----------------------------------------------------------------------------------------------------------------
// One CTA per SM.  The weights of up to `chunk` reduction rows lie expanded and transposed in shared memory: for every block
// of 64 rows and output column k, sixteen words of four consecutive rows each, in the order the lanes read them (a lane's 16
// bytes are its B fragments of two MMAs; 32 lanes read 512 consecutive bytes).  The reduction index inside a block is permuted
// the same way for dYq, so that a lane loads 16 consecutive bytes of a row.  The sixteen warps share the reduction of a
// 16-row tile and meet in shared memory.  CG: groups of 8 output columns.
constexpr int SX_THREADS = 512, SX_WARPS = SX_THREADS / 32, SX_BATCH = 4;
constexpr int SX_SMEM_W = 128 * 1024;

template <int CG>
__global__ void __launch_bounds__(SX_THREADS, 1)
skinny_dx_kernel(const int8_t* __restrict__ dYq, const uint8_t* __restrict__ Wp, EpiParams epi, int R, int D, int chunk) {
    constexpr int C = CG * 8, W32 = C / 16;          // words of 16 codes per packed row
    extern __shared__ uint4 sx_smem[];
    uint32_t* wt = reinterpret_cast<uint32_t*>(sx_smem);
    __shared__ int acc_sm[16 * C];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r8 = lane >> 2, q = lane & 3;
    const int tiles = (R + 15) >> 4;
    const int n_chunks = (D + chunk - 1) / chunk;
    for (int i = tid; i < 16 * C; i += SX_THREADS) acc_sm[i] = 0;

    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int row0 = t * 16 + r8, row1 = row0 + 8;
        const int8_t* y0 = dYq + (size_t)row0 * D;
        const int8_t* y1 = dYq + (size_t)row1 * D;
        int d[CG][4];
#pragma unroll
        for (int c = 0; c < CG; ++c) d[c][0] = d[c][1] = d[c][2] = d[c][3] = 0;
        for (int ch = 0; ch < n_chunks; ++ch) {
            const int base = ch * chunk;
            const int len = min(chunk, D - base), blocks = (len + 63) >> 6;
            uint4 a[SX_BATCH][2];
            auto load_batch = [&](int blk0) {
#pragma unroll
                for (int i = 0; i < SX_BATCH; ++i) {
                    const int off = (blk0 + i * SX_WARPS) * 64 + q * 16;         // D % 16 == 0: 16 bytes inside or outside together
                    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
                    a[i][0] = (off < len && row0 < R) ? __ldg(reinterpret_cast<const uint4*>(y0 + base + off)) : zero;
                    a[i][1] = (off < len && row1 < R) ? __ldg(reinterpret_cast<const uint4*>(y1 + base + off)) : zero;
                }
            };
            load_batch(warp);                        // in flight while the weights are expanded
            if (n_chunks > 1 || t == (int)blockIdx.x) {
                __syncthreads();                     // nobody still reads the previous chunk
                for (int i = tid; i < blocks * 16 * W32; i += SX_THREADS) {
                    const int g = i / W32, kw = i - g * W32;          // four reduction rows, one word of 16 output columns
                    uint32_t e[4][4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int n = g * 4 + r;
                        const uint32_t code = n < len ? __ldg(reinterpret_cast<const uint32_t*>(Wp) + (size_t)(base + n) * W32 + kw) : 0x55555555u;
                        decode16(code, e[r]);
                    }
                    uint32_t* dst = wt + ((size_t)(g >> 4) * C + kw * 16) * 16 + (g & 15);
#pragma unroll
                    for (int w = 0; w < 4; ++w) {                      // 4x4 byte transpose: columns 4w..4w+3
                        const uint32_t p0 = __byte_perm(e[0][w], e[1][w], 0x5140), p1 = __byte_perm(e[2][w], e[3][w], 0x5140);
                        const uint32_t p2 = __byte_perm(e[0][w], e[1][w], 0x7362), p3 = __byte_perm(e[2][w], e[3][w], 0x7362);
                        dst[(4 * w + 0) * 16] = __byte_perm(p0, p1, 0x5410);
                        dst[(4 * w + 1) * 16] = __byte_perm(p0, p1, 0x7632);
                        dst[(4 * w + 2) * 16] = __byte_perm(p2, p3, 0x5410);
                        dst[(4 * w + 3) * 16] = __byte_perm(p2, p3, 0x7632);
                    }
                }
                __syncthreads();
            }
            for (int blk0 = warp; blk0 < blocks; blk0 += SX_BATCH * SX_WARPS) {
#pragma unroll
                for (int i = 0; i < SX_BATCH; ++i) {
                    const int blk = blk0 + i * SX_WARPS;
                    if (blk < blocks) {
                        const uint4 u = a[i][0], v = a[i][1];
#pragma unroll
                        for (int c = 0; c < CG; ++c) {
                            const uint4 b = sx_smem[((size_t)blk * C + c * 8 + r8) * 4 + q];
                            mma_s8_k32(d[c], u.x, v.x, u.y, v.y, b.x, b.y);
                            mma_s8_k32(d[c], u.z, v.z, u.w, v.w, b.z, b.w);
                        }
                    }
                }
                if (blk0 + SX_BATCH * SX_WARPS < blocks) load_batch(blk0 + SX_BATCH * SX_WARPS);
            }
        }
#pragma unroll
        for (int c = 0; c < CG; ++c) {
            atomicAdd(&acc_sm[r8 * C + c * 8 + 2 * q], d[c][0]);
            atomicAdd(&acc_sm[r8 * C + c * 8 + 2 * q + 1], d[c][1]);
            atomicAdd(&acc_sm[(r8 + 8) * C + c * 8 + 2 * q], d[c][2]);
            atomicAdd(&acc_sm[(r8 + 8) * C + c * 8 + 2 * q + 1], d[c][3]);
        }
        __syncthreads();
        for (int i = tid; i < 16 * C; i += SX_THREADS) {
            const int r = i / C, c = i - r * C, row = t * 16 + r;
            const int v = acc_sm[i];
            acc_sm[i] = 0;
            if (row < R) epi_store_one(epi, row, c, v, epi_row_scale(epi, row));
        }
        __syncthreads();
    }
}

template <int KS>
int launch_skinny_fwd(const int8_t* A, const uint8_t* B, int R, int C, const EpiParams& epi, int sms, cudaStream_t st) {
    const int gx = (C + SF_WARPS * SF_COLS - 1) / (SF_WARPS * SF_COLS), tiles = (R + 15) / 16;
    int gy = (sms * 8 + gx - 1) / gx;                // about eight CTAs of 256 threads per SM in one wave
    gy = gy < tiles ? gy : tiles;
    if (gy > 65535) gy = 65535;
    const dim3 grid(gx, gy);
    switch (epi.out_dtype) {
        case EL_BF16: skinny_fwd_kernel<KS, EL_BF16><<<grid, SF_WARPS * 32, 0, st>>>(A, B, epi, R, C); break;
        case EL_F16: skinny_fwd_kernel<KS, EL_F16><<<grid, SF_WARPS * 32, 0, st>>>(A, B, epi, R, C); break;
        case EL_F32: skinny_fwd_kernel<KS, EL_F32><<<grid, SF_WARPS * 32, 0, st>>>(A, B, epi, R, C); break;
        default: skinny_fwd_kernel<KS, EL_I32><<<grid, SF_WARPS * 32, 0, st>>>(A, B, epi, R, C); break;
    }
    return check_launch();
}

template <int CG>
int launch_skinny_dx(const int8_t* A, const uint8_t* B, int R, int D, const EpiParams& epi, int sms, cudaStream_t st) {
    static DeviceOnce attr_once;
    int dev = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    if (!attr_once.is_done(dev)) {
        EL_CUDA_TRY(cudaFuncSetAttribute(skinny_dx_kernel<CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, SX_SMEM_W));
        attr_once.mark(dev);
    }
    constexpr int C = CG * 8;
    const int most = (SX_SMEM_W / C) & ~63;          // reduction rows whose expanded weights fit
    const int padded = (D + 63) & ~63;
    const int chunk = padded < most ? padded : most;
    const int tiles = (R + 15) / 16;
    skinny_dx_kernel<CG><<<tiles < sms ? tiles : sms, SX_THREADS, (size_t)chunk * C, st>>>(A, B, epi, R, D, chunk);
    return check_launch();
}

}  // namespace

// Whether the kernels above take the problem: the narrow side is 16, 32 or 48 wide, everything they read or write in
// 16-byte (weights: 4-byte) pieces is aligned.  From 64 on, multiples of 64 go to tensor-core tiles; 80, 96, 112 and other widths that are
// no multiple of 64 have no kernel of their own and stay with the CUDA-core kernel.
bool gemm_skinny_fits(int mode, const void* A, const void* B, int R, int C, int D, const EpiParams& epi) {
    if (R <= 0 || C <= 0 || D <= 0) return false;
    if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 3)) return false;
    if (mode == MODE_FWD) {
        const int esz = (epi.out_dtype == EL_BF16 || epi.out_dtype == EL_F16) ? 2 : 4;
        return D % 16 == 0 && D < 64 && C % (16 / esz) == 0 && (reinterpret_cast<uintptr_t>(epi.out) & 15) == 0 &&
               (epi.ldo * esz) % 16 == 0;
    }
    return mode == MODE_DX && C % 16 == 0 && C < 64 && D % 16 == 0;
}

int launch_gemm_skinny(int mode, const int8_t* A, const void* B, int R, int C, int D, const EpiParams& epi, cudaStream_t st) {
    if (!gemm_skinny_fits(mode, A, B, R, C, D, epi)) return EL_ERR_UNSUPPORTED_SHAPE;
    int sms = 0;
    const int rc = device_sm_count(&sms);
    if (rc != EL_OK) return rc;
    const uint8_t* W = static_cast<const uint8_t*>(B);
    if (mode == MODE_FWD) {
        if (D == 16) return launch_skinny_fwd<1>(A, W, R, C, epi, sms, st);
        if (D == 32) return launch_skinny_fwd<2>(A, W, R, C, epi, sms, st);
        return launch_skinny_fwd<3>(A, W, R, C, epi, sms, st);
    }
    if (C == 16) return launch_skinny_dx<2>(A, W, R, D, epi, sms, st);
    if (C == 32) return launch_skinny_dx<4>(A, W, R, D, epi, sms, st);
    return launch_skinny_dx<6>(A, W, R, D, epi, sms, st);
}

}  // namespace el
