// Forward and dX GEMMs with the weights in tensor memory, on CTA pairs (tcgen05 cta_group::2) for sm_100a.
//
// The product is formed transposed: the MMA's A operand (256 rows, 128 per CTA) are output features and comes from tensor memory,
// its B operand (NT columns) are tokens and comes from shared memory.  The 2-bit weights are expanded by warps whose lanes write
// straight into the tensor memory of their own 32 lanes (tcgen05.st), so the expanded tile never touches shared memory, whose
// bandwidth the MMAs' operand reads need (the kernel this one replaced expanded into shared memory, as the MMA's second operand).
// us per launch, bf16 out, forward / dX, of that kernel (for few tiles: its single-CTA companion) and of this one, in a CUDA graph over
// several weight matrices: 4096 tokens 4096 -> 11008 116.6 / 118.7 and 112.6 / 114.9, 4096 tokens 4096 -> 512 18.5 / 24.2 and
// 14.5 / 21.9, 1024 tokens 1536 -> 1536 11.0 / 11.0 and 9.6 / 9.7, 512 tokens 4096 -> 4096 17.6 / 17.6 and 14.3 / 13.7, 128 tokens
// 4096 -> 11008 18.7 / 36.6 and 14.9 / 21.7.  What is left at large sizes, by leaving parts out (4096 tokens, 4096 -> 11008, forward, 116 us
// with events and a cold L2): 106 without the expansion and the epilogue, 99 without the token loads too, 83 for the MMAs at full clock.
//
// Per CTA and 128-deep reduction block:
//   T   NT/2 x 128 bytes   activations, TMA, 128-byte swizzle, K-major     (bytes counted on the leader's "full" barrier)
//   P   128 x 32 bytes     packed weights, TMA, 32-byte swizzle               ("pfull" / "pempty", local)
//   A   128 lanes x 32 columns of tensor memory: 128 expanded weights per output feature (four arrivals per CTA on "full")
//
// Which lane holds which output feature:
//   FWD  lane l of warp s = feature 32 s + l: a lane reads its feature's 32 packed bytes and expands them in order.
//   DX   a packed byte holds four output features of ONE reduction index, so the tile has to be transposed.  ldmatrix (16 x 16
//        bytes, transposed) gives a thread four reduction indices of one byte column; masks and the table of decode16 turn these
//        into four consecutive reduction indices of each of the four features, words of the operand, and tcgen05.st 16x128b puts
//        them where they belong: lane 8 c + i of warp s holds feature 32 s + 4 i + c.
// The epilogue reads the sums as 16 lanes x 256 bits: a thread then holds features i, i + 8, i + 16, i + 24 (FWD) or 4 i to 4 i + 3 (DX)
// of two tokens, and the rows of the output, which run along the features, leave as stmatrix transposes (FWD) or 8-byte words (DX).
//
// Tensor memory (512 columns): two accumulators and four A slots of 32 columns.  With NT = 256 the accumulators overlap in
// 128 columns ([0, 256) and [128, 384)); the epilogue takes the shared half into registers first, at once, and the next tile's
// MMAs start.  With smaller NT they are apart.
#include <cuda.h>

#include <atomic>

#include "common.cuh"
#include "epilogue.cuh"
#include "tc_ptx.cuh"

namespace el {

enum { MODE_FWD = 0, MODE_DX = 1, MODE_DW = 2, MODE_FWD_PERM = 3 };      // FWD_PERM: tokens quantised in the order of decode16_deint

namespace wt {

using namespace tc;

constexpr int BF = 128;            // output features per CTA (the pair covers 256)
constexpr int BK = 128;            // reduction block
constexpr int DA = 4;              // A slots in tensor memory
constexpr int P_BYTES = BF * BK / 4;      // packed weights of one block
constexpr int NUM_EPI_WARPS = 8;
constexpr int WARP_TMA = 0, WARP_MMA = 1, WARP_EPI0 = 2, WARP_XF0 = 10;      // a warp reaches the tensor-memory lanes of quarter warp % 4
constexpr int STAGE_BYTES = 4096;  // epilogue staging of one warp: 32 tokens x 32 features of four bytes, or two of two bytes
constexpr uint32_t TMEM_COLS = 512;

// What depends on the token tile.  LEAN (256 tokens only): at most 80 registers per thread, see the kernel.
template <int NT, bool LEAN = false> struct Geo {
    // Blocks per step of the pipeline (a stage of the rings, an A slot, one set of arrivals and one commit).  Small tiles are bound by
    // the transform warps' instructions, half of which are the handshakes of a step.
    static constexpr int SB = NT == 256 ? 1 : 2;
    static constexpr int DT = NT == 128 ? 4 : 8;                             // stages of the token ring and of the packed ring
    static constexpr int TOK = NT / 2 * BK;                                  // tokens of one block
    static constexpr uint32_t A_COLS = SB * 32;                              // tensor-memory columns of an A slot: 32 per block
    static constexpr uint32_t A_COL0 = TMEM_COLS - DA * A_COLS;
    static constexpr bool OVERLAP = 2 * NT > (int)A_COL0;                    // the two accumulators share columns
    static constexpr int ACC1 = OVERLAP ? (int)A_COL0 - NT : NT;             // first column of the second accumulator
    static constexpr int SETS = NT == 256 ? 2 : 4;                            // sets of four transform warps
    static constexpr int THREADS = (WARP_XF0 + SETS * 4) * 32;
    static constexpr int WCOLS = NT / 2 < 32 ? 32 : NT / 2;                  // accumulator columns of one epilogue warp
    static constexpr int GCOLS = OVERLAP && !LEAN ? 64 : 32;                 // of these taken into registers at a time
    static constexpr int FIRST = OVERLAP ? (NT - ACC1) / 2 : WCOLS;          // columns a warp has to take before the next tile may write
    static constexpr int REGS = SETS == 4 ? 72 : LEAN ? 80 : 96;             // what the block's warps leave each thread
    static_assert(FIRST % GCOLS == 0 && (!OVERLAP || 2 * ACC1 == NT), "the shared columns are one half of each accumulator");
    // shared memory
    static constexpr int P = DT * SB * TOK;                                  // packed ring
    static constexpr int STAGE = P + DT * SB * P_BYTES;                      // epilogue staging
    static constexpr int SCALE = STAGE + NUM_EPI_WARPS * STAGE_BYTES;                    // token scales, a copy per epilogue warp
    static constexpr int BARS = SCALE + NUM_EPI_WARPS * WCOLS * 4;
    static constexpr int BYTES = BARS + 512 + 1024;
    static_assert(DT % DA == 0 && DT % SETS == 0 && BYTES <= 227 * 1024, "");
};

constexpr int MAX_DST = 8;         // output destinations of one launch (the ranks of an N-sharded layer)
struct OutMaps {
    CUtensorMap m[MAX_DST];
};

struct Params {
    int R, C, D;                        // tokens, output features, reduction
    int tiles_r, tiles_c, k_blocks;     // tiles_r counts NT-token tiles, tiles_c 256-feature tiles
    int k_split, kbp, steps;            // reduction split: k_split work items of kbp blocks (in `steps` steps) per output tile (1, k_blocks = none)
    int group_rows;                     // token tiles per band of the tile order (see tile_coords)
    EpiParams epi;
    int small_sums;                     // every sum is below 2^22 in magnitude
    int tma_store;                      // the output takes TMA stores (16-byte aligned base and pitch)
    int n_dst;                          // destinations that receive every output block (1 unless gathered over ranks)
    int rows_per_dst;                   // > 0: scatter instead - rows [d*rows_per_dst, (d+1)*rows_per_dst) go to destination d only
    int row_rotate;                     // scatter: token tiles are taken starting from this one (see tile_coords)
    int weights_first;                  // the launch before this one does not write the weights: load them without waiting for it
    int32_t* status;
};

// Tile order: bands of `group_rows` token tiles; inside a band the feature tiles follow one another and the band's token tiles
// run fastest.  The pairs of one wave then share a few weight tiles while the band's activation rows (sized by the host
// to stay in L2) are read from HBM once instead of once per feature tile.
__device__ __forceinline__ void tile_coords(int t, const Params& p, int& tr, int& tc) {
    const int per_band = p.group_rows * p.tiles_c;
    const int band = t / per_band, in = t - band * per_band;
    const int first = band * p.group_rows;
    const int rows_here = min(p.group_rows, p.tiles_r - first);
    tc = in / rows_here;
    tr = first + (in - tc * rows_here);
    // Scatter over ranks: every rank walks the token tiles in the same cyclic order but starts at its own rows, so that at any
    // time the ranks store into different owners (one sender per receiving link) instead of all into the same one.
    tr += p.row_rotate;
    if (tr >= p.tiles_r) tr -= p.tiles_r;
}

// Work item w -> output tile and the first reduction block of its part.  With a split reduction the parts of one tile
// are num_tiles items apart, so they run on different pairs at the same time; part q writes its int32 partial sums
// to output q, and a second pass adds the parts and scales.
__device__ __forceinline__ void item_coords(int w, int num_tiles, const Params& p, int& tr, int& tc, int& part, int& kb0) {
    part = w / num_tiles;
    tile_coords(w - part * num_tiles, p, tr, tc);
    kb0 = part * p.kbp;
}

__device__ __forceinline__ void umma_i8_pair_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], [%1], %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(z)
        : "memory");
}
// 32 words per lane into the warp's 32 lanes of tensor memory: word i in column i.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
          "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
          "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
          "r"(v[31]), "r"(taddr)
        : "memory");
}
// 16 lanes x 32 columns: v[2i] of thread t goes to lane t / 4, column 4 i + t % 4, v[2i + 1] eight lanes further.
__device__ __forceinline__ void tmem_st16x128(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x8.b32 [%16], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
          "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Two 16 x 16 byte matrices, transposed: thread t gets byte column t / 4 (r0) and t / 4 + 8 (r1) of the first, rows 4 (t % 4) to
// 4 (t % 4) + 3 as the four bytes of a word; r2, r3 are the second.  Lanes 0-15 give the rows of the first, 16-31 of the second.
__device__ __forceinline__ void ldmatrix_t16x16(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m16n16.x2.trans.shared.b8 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr)
                 : "memory");
}

// A word of four packed bytes -> the codes of each position as four int8, by the table of decode16.
__device__ __forceinline__ void expand4x4(uint32_t w, uint32_t& c0, uint32_t& c1, uint32_t& c2, uint32_t& c3) {
    const uint32_t lut = 0x000100FFu, te = w & 0x33333333u, to = (w >> 2) & 0x33333333u;
    const uint32_t e0 = __byte_perm(lut, 0, te), e1 = __byte_perm(lut, 0, te >> 16);       // first and third codes of bytes 0, 1 and 2, 3
    const uint32_t o0 = __byte_perm(lut, 0, to), o1 = __byte_perm(lut, 0, to >> 16);       // second and fourth
    c0 = __byte_perm(e0, e1, 0x6420);
    c1 = __byte_perm(o0, o1, 0x6420);
    c2 = __byte_perm(e0, e1, 0x7531);
    c3 = __byte_perm(o0, o1, 0x7531);
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

// 16 lanes x 32 columns: v[4c] and v[4c + 1] of thread t are lane t / 4, columns 8 c + 2 (t % 4) and the next; v[4c + 2], v[4c + 3] the
// same eight lanes further.
__device__ __forceinline__ void tmem_ld16x256(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// four 8 x 8 matrices of 16-bit values, each transposed on its way: lanes 8 m to 8 m + 7 give the rows of matrix m
__device__ __forceinline__ void stmatrix_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
template <int OUT> __device__ __forceinline__ uint32_t pack_out(uint32_t lo, uint32_t hi) {
    return OUT == EL_BF16 ? pack_bf16x2(__uint_as_float(lo), __uint_as_float(hi)) : pack_f16x2(__uint_as_float(lo), __uint_as_float(hi));
}

// A warp's chunk of 32 tokens x 32 features as it comes from tensor memory: v[h][4c + r] with the layout of tmem_ld16x256, h the
// upper 16 lanes.  This is the sums' way to scaled float32, in place.  Sums below 2^22 in magnitude (reductions up to 32767: weights are
// at most 1, tokens at most 128) are exact in float32 and come from adding 1.5 * 2^23 as an integer and taking it away as a float,
// two values per instruction; the conversion unit takes eight cycles per instruction.  `scale`: the thread's first token's (shared).
__device__ __forceinline__ void scale_chunk(uint32_t (&v)[2][16], uint32_t scale, bool small) {
    if (!small) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 16; ++i) v[h][i] = __float_as_uint((float)(int)v[h][i]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        uint64_t sc;
        asm volatile("ld.shared.u64 %0, [%1];" : "=l"(sc) : "r"(scale + c * 32) : "memory");
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int r = 4 * c; r < 4 * c + 4; r += 2) {
                uint64_t x;
                if (small) {
                    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "r"(v[h][r] + 0x4B400000u), "r"(v[h][r + 1] + 0x4B400000u));
                    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(x) : "l"(x), "l"(0xCB400000CB400000ull));
                } else {
                    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "r"(v[h][r]), "r"(v[h][r + 1]));
                }
                asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(x) : "l"(x), "l"(sc));
                asm("mov.b64 {%0, %1}, %2;" : "=r"(v[h][r]), "=r"(v[h][r + 1]) : "l"(x));
            }
    }
}
// ... and to the staging area in the output map's swizzle: 32 rows (tokens) of 64 bytes, 16-byte chunk k of row t at k ^ (t / 2 % 4), for
// two-byte outputs; of 128 bytes, chunk k at k ^ (t % 8), for four-byte ones.  No two lanes of a wavefront meet in a bank, but
// for the two-byte words of DX (two-way).
template <int MODE, int OUT>
__device__ __forceinline__ void stage_chunk(const uint32_t (&v)[2][16], uint32_t dst, int lane) {
    const int i = lane >> 2, q = lane & 3;
    if (MODE != MODE_DX && (OUT == EL_BF16 || OUT == EL_F16)) {
        // matrix m = features 8 m to 8 m + 7; its row is token 8 c + lane % 8
        const uint32_t at = dst + (lane & 7) * 64 + (((lane >> 3) ^ ((lane >> 1) & 3)) << 4);
#pragma unroll
        for (int c = 0; c < 4; ++c)
            stmatrix_t(at + c * 512, pack_out<OUT>(v[0][4 * c], v[0][4 * c + 1]), pack_out<OUT>(v[0][4 * c + 2], v[0][4 * c + 3]),
                       pack_out<OUT>(v[1][4 * c], v[1][4 * c + 1]), pack_out<OUT>(v[1][4 * c + 2], v[1][4 * c + 3]));
    } else if (OUT == EL_BF16 || OUT == EL_F16) {
        const uint32_t at = dst + q * 128 + (((i >> 1) ^ q) << 4) + (i & 1) * 8;             // tokens 2 q and 2 q + 1: the same swizzle
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                sts64(at + c * 512 + e * 64, pack_out<OUT>(v[0][4 * c + e], v[0][4 * c + 2 + e]), pack_out<OUT>(v[1][4 * c + e], v[1][4 * c + 2 + e]));
    } else {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t row = dst + (2 * q + e) * 128, x = (uint32_t)(2 * q + e) & 7;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (MODE == MODE_DX) {
                    sts128(row + c * 1024 + ((i ^ x) << 4), v[0][4 * c + e], v[0][4 * c + 2 + e], v[1][4 * c + e], v[1][4 * c + 2 + e]);
                } else {
#pragma unroll
                    for (int m = 0; m < 4; ++m)       // feature i + 8 m
                        sts32(row + c * 1024 + ((((i >> 2) + 2 * m) ^ x) << 4) + (i & 3) * 4, v[m >> 1][4 * c + 2 * (m & 1) + e]);
                }
            }
        }
    }
}

// Staged rows (tokens) of `feats` features to an output that no TMA store takes; `out` is the first token's first feature.
__device__ __noinline__ void store_plain(void* out, long long ldo, uint32_t stage, int tokens, int feats, bool two_byte) {
    const int lane = threadIdx.x & 31;
    if (lane >= feats) return;
    for (int t = 0; t < tokens; ++t) {
        if (two_byte) {
            uint16_t x;
            const uint32_t at = stage + t * 64 + (((lane >> 3) ^ ((t >> 1) & 3)) << 4) + (lane & 7) * 2;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(x) : "r"(at) : "memory");
            static_cast<uint16_t*>(out)[t * ldo + lane] = x;
        } else {
            uint32_t x;
            const uint32_t at = stage + t * 128 + (((lane >> 2) ^ (t & 7)) << 4) + (lane & 3) * 4;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(at) : "memory");
            static_cast<uint32_t*>(out)[t * ldo + lane] = x;
        }
    }
}

// LEAN leaves a quarter of the register file free, so that a kernel that needs no shared memory (the peer pushes of a multi-GPU
// step, on a side stream) can run beside this persistent one.
template <int MODE, int NT, bool LEAN>
__global__ void __maxnreg__((Geo<NT, LEAN>::REGS))
gemm_wt_kernel(const __grid_constant__ CUtensorMap tmT, const __grid_constant__ CUtensorMap tmP, const __grid_constant__ OutMaps outs,
               const Params p) {
    using G = Geo<NT, LEAN>;
    constexpr int DT = G::DT, SB = G::SB, T_BYTES = SB * G::TOK, PS_BYTES = SB * P_BYTES;       // of one stage
    constexpr int WCOLS = G::WCOLS, GCOLS = G::GCOLS;
    constexpr bool OVERLAP = G::OVERLAP, FWD = MODE != MODE_DX;
    constexpr int ACC1 = G::ACC1;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bars = smem_base + G::BARS;
    //   full   (leader's copy is used) both CTAs' tokens landed + both CTAs' four transform warps have written their lanes + the
    //          leader producer's expect-arrival
    //   empty  (local) the MMAs of the block are done: its token stage and its A slot are free
    //   pfull / pempty (local) the packed tile has landed / has been read by the four warps of its block
    auto bar_full = [&](int s) { return bars + 8u * s; };
    auto bar_empty = [&](int s) { return bars + 8u * (DT + s); };
    auto bar_pfull = [&](int s) { return bars + 8u * (2 * DT + s); };
    auto bar_pempty = [&](int s) { return bars + 8u * (3 * DT + s); };
    auto bar_tfull = [&](int a) { return bars + 8u * (4 * DT + a); };        // local: accumulator complete
    auto bar_tempty = [&](int a) { return bars + 8u * (4 * DT + 2 + a); };   // leader: both epilogues hold the columns the next tile needs
    volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem_gen + G::BARS + 8 * (4 * DT + 4));

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();            // 0 = leader
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
    const int num_tiles = p.tiles_r * p.tiles_c;
    const int num_items = num_tiles * p.k_split;

    if (threadIdx.x == 0) {
        for (int s = 0; s < DT; ++s) {
            mbar_init(bar_full(s), 1 + 2 * 4);
            mbar_init(bar_empty(s), 1);
            mbar_init(bar_pfull(s), 1);
            mbar_init(bar_pempty(s), 4);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(bar_tfull(a), 1);
            mbar_init(bar_tempty(a), 2 * NUM_EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == WARP_MMA) {     // both CTAs of the pair take part in the allocation
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_holder)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();          // the peer's barriers are initialised before anything signals them
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    bool failed = false;

    if (warp == WARP_TMA) {
        // ================= producer: this CTA's tokens and packed weights of every reduction block =================
        // The whole warp waits (a warp whose lanes all wait on the barrier is woken sooner than a single waiting lane);
        // lane 0 issues the copies.
        auto load_packed = [&](int s, int kb, int f0) {
            if (elect_one()) {
                mbar_expect_tx(bar_pfull(s), PS_BYTES);
                const uint32_t dst = smem_base + G::P + s * PS_BYTES;
                if (FWD) {
#pragma unroll
                    for (int b = 0; b < SB; ++b) tma_load_2d(dst + b * P_BYTES, &tmP, bar_pfull(s), (kb + b) * (BK / 4), f0);
                } else {
                    tma_load_2d(dst, &tmP, bar_pfull(s), f0 / 4, kb * BK);            // a box of SB * 128 reduction rows
                }
            }
            __syncwarp();
        };
        // Weights that the launch before this one does not write are on their way, a whole ring of them, before that launch has ended.
        int ahead = 0;
        if (p.weights_first && pair < num_items) {
            int trow, tcol, part, kb0;
            item_coords(pair, num_tiles, p, trow, tcol, part, kb0);
            for (; ahead < DT && ahead < p.steps; ++ahead) load_packed(ahead, kb0 + ahead * SB, tcol * (2 * BF) + (int)rank * BF);
        }
        griddep_wait();
        int s = 0;
        uint32_t ph = 0;
        for (int w = pair; w < num_items && !failed; w += num_pairs) {
            int trow, tcol, part, kb0;
            item_coords(w, num_tiles, p, trow, tcol, part, kb0);
            const int t0 = trow * NT + (int)rank * (NT / 2), f0 = tcol * (2 * BF) + (int)rank * BF;
            for (int st = 0, kb = kb0; st < p.steps; ++st, kb += SB) {
                if (ahead > 0) {
                    --ahead;
                } else {
                    // the packed slot is free long before the token slot (its blocks have been expanded before its MMAs run)
                    if (!mbar_wait_warp(bar_pempty(s), ph ^ 1u, p.status, 24)) { failed = true; break; }
                    load_packed(s, kb, f0);
                }
                if (!mbar_wait_cluster_warp(bar_empty(s), ph ^ 1u, p.status, 21)) { failed = true; break; }
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(bar_full(s), 2 * T_BYTES);
                    const uint32_t bar = mapa_u32(bar_full(s), 0);
#pragma unroll
                    for (int b = 0; b < SB; ++b) tma_load_2d_pair(smem_base + s * T_BYTES + b * G::TOK, &tmT, bar, (kb + b) * BK, t0);
                }
                __syncwarp();
                if (++s == DT) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp == WARP_MMA) {
        // ================= MMA issuer (leader CTA only): the whole warp waits, lane 0 issues =================
        if (rank == 0) {
            constexpr uint32_t idesc = make_idesc(0, 0, NT, 2 * BF);
            int s = 0, it = 0;
            uint32_t ph = 0;
            for (int w = pair; w < num_items && !failed; w += num_pairs, ++it) {
                // accumulators apart: the tile before last has left this one.  Overlapping: the last tile's shared half has left.
                if (OVERLAP) {
                    if (it > 0 && !mbar_wait_cluster_warp(bar_tempty((it - 1) & 1), (uint32_t)((it - 1) >> 1) & 1u, p.status, 22)) { failed = true; break; }
                } else {
                    if (it > 1 && !mbar_wait_cluster_warp(bar_tempty(it & 1), (uint32_t)((it - 2) >> 1) & 1u, p.status, 22)) { failed = true; break; }
                }
                tcgen05_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)((it & 1) * ACC1);
                for (int st = 0; st < p.steps; ++st) {        // the item's own blocks: the first one starts the sums
                    if (!mbar_wait_cluster_warp(bar_full(s), ph, p.status, 23)) { failed = true; break; }
                    tcgen05_fence_after();
                    if (elect_one()) {
                        const uint32_t t_addr = smem_base + s * T_BYTES, a_tmem = tmem_base + G::A_COL0 + (uint32_t)(s % DA) * G::A_COLS;
#pragma unroll
                        for (int k = 0; k < SB * BK / 32; ++k)
                            umma_i8_pair_ts(d_tmem, a_tmem + k * 8, make_desc(t_addr + (k / 4) * G::TOK + (k % 4) * 32, 16), idesc, (st | k) != 0);
                        umma_commit_pair(bar_empty(s));
                    }
                    __syncwarp();
                    if (++s == DT) { s = 0; ph ^= 1u; }
                }
                if (!failed && elect_one()) umma_commit_pair(bar_tfull(it & 1));
                __syncwarp();
            }
        }
    } else if (warp >= WARP_EPI0 && warp < WARP_XF0) {
        // ================= epilogue: warp (quarter, half) takes 32 lanes (features) x NT/2 columns (tokens) =================
        const int quarter = warp & 3, half = (warp - WARP_EPI0) >> 2;
        const uint32_t stage = smem_base + G::STAGE + (warp - WARP_EPI0) * STAGE_BYTES;
        const uint32_t scale = smem_base + G::SCALE + (warp - WARP_EPI0) * WCOLS * 4;
        const bool two_byte = (p.epi.out_dtype == EL_BF16 || p.epi.out_dtype == EL_F16);
        // Columns in the order they are taken: with overlapping accumulators each warp's first FIRST columns lie in the half that the
        // next tile needs.
        constexpr int PER = G::FIRST / GCOLS;
        auto group_col = [&](int g, int acc) {
            const int first = (OVERLAP && acc == 0) ? ACC1 : 0;
            return (OVERLAP ? (g < PER ? first : NT / 2 - first) : 0) + half * G::FIRST + (g % PER) * GCOLS;
        };
        // The item's coordinates and its tokens' maxima (32 per register) are fetched one item ahead: the divisions and the trip to memory
        // would take a quarter of a short tile's time.
        int trow = 0, tcol = 0, part = 0, kb0;
        float amax[WCOLS / 32];
        auto fetch = [&](int w, int acc) {
            if (w >= num_items) return;
            item_coords(w, num_tiles, p, trow, tcol, part, kb0);
#pragma unroll
            for (int i = 0; i < WCOLS / 32; ++i) {
                const int row = trow * NT + group_col(i * 32 / GCOLS, acc) + i * 32 % GCOLS + lane;
                amax[i] = (p.epi.absmax != nullptr && row < p.R) ? p.epi.absmax[(size_t)row * p.epi.absmax_stride] : 0.0f;
            }
        };
        griddep_wait();
        fetch(pair, 0);
        int it = 0;
        for (int w = pair; w < num_items && !failed; w += num_pairs, ++it) {
            const int f0 = tcol * (2 * BF) + (int)rank * BF + quarter * 32, row0 = trow * NT, out = part;       // the warp's first feature
            const int acc = it & 1;
            __syncwarp();
#pragma unroll
            for (int i = 0; i < WCOLS / 32; ++i) sts32(scale + i * 128 + lane * 4, __float_as_uint(epi_scale(p.epi, amax[i])));
            __syncwarp();
            if (!mbar_wait_warp(bar_tfull(acc), (uint32_t)(it >> 1) & 1u, p.status, 25)) { failed = true; break; }
            tcgen05_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * ACC1);
#pragma unroll 1
            for (int g = 0; g < WCOLS / GCOLS; ++g) {
                const int col = group_col(g, acc);
                uint32_t v[GCOLS / 32][2][16];
#pragma unroll
                for (int c = 0; c < GCOLS / 32; ++c)
                    if (col < NT) {
                        tmem_ld16x256(taddr + col + c * 32, v[c][0]);
                        tmem_ld16x256(taddr + col + c * 32 + (16u << 16), v[c][1]);
                    }
                tmem_ld_wait();
                if (g == PER - 1) {      // what the next tile of this accumulator's columns needs is out
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster_relaxed(mapa_u32(bar_tempty(acc), 0));
                    fetch(w + num_pairs, acc ^ 1);
                }
                if (col >= NT || f0 >= p.C) continue;
                // The chunks of 32 tokens go to shared memory and out with a TMA store each, clipped at the matrix edges: those of a group
                // together where the staging area holds them (two-byte outputs), one after the other where not.
                constexpr int CHUNKS = GCOLS / 32;
                if (p.epi.out_dtype != EL_I32) {
#pragma unroll
                    for (int c = 0; c < CHUNKS; ++c) scale_chunk(v[c], scale + (g * GCOLS + c * 32) * 4 + (lane & 3) * 8, p.small_sums != 0);
                }
#pragma unroll
                for (int c = 0; c < CHUNKS; ++c) {
                    if (c == 0 || !two_byte) {
                        if (p.tma_store && elect_one()) bulk_wait_read<0>();         // the last stores have read the area
                        __syncwarp();
                    }
                    switch (p.epi.out_dtype) {
                        case EL_BF16: stage_chunk<MODE, EL_BF16>(v[c], stage + c * 2048, lane); break;
                        case EL_F16: stage_chunk<MODE, EL_F16>(v[c], stage + c * 2048, lane); break;
                        default: stage_chunk<MODE, EL_F32>(v[c], stage, lane); break;
                    }
                    if (two_byte && c < CHUNKS - 1) continue;
                    const int first_chunk = two_byte ? 0 : c;
                    if (!p.tma_store) {                                     // unaligned output: plain stores (rare)
                        __syncwarp();
                        const int tok0 = row0 + col + first_chunk * 32;
                        store_plain(static_cast<char*>(p.epi.out) + ((long long)tok0 * p.epi.ldo + f0) * (two_byte ? 2 : 4), p.epi.ldo, stage,
                                    min((c + 1 - first_chunk) * 32, p.R - tok0), p.C - f0, two_byte);
                        __syncwarp();
                        continue;
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (elect_one()) {
                        for (int k = first_chunk; k <= c; ++k) {
                            const int tok0 = row0 + col + k * 32;
                            const uint32_t src = stage + (two_byte ? k * 2048 : 0);
                            if (tok0 >= p.R) break;
                            if (p.k_split > 1) {                       // split reduction: part q's sums go to partial output q
                                tma_store_2d(&outs.m[out], src, f0, tok0);
                            } else if (p.rows_per_dst > 0) {           // scatter: this 32-token block belongs to one owner
                                const int d = tok0 / p.rows_per_dst;
                                if (d < p.n_dst) tma_store_2d(&outs.m[d], src, f0, tok0 - d * p.rows_per_dst);
                            } else {                                   // own buffer and, when gathering, every peer's
                                tma_store_2d(&outs.m[0], src, f0, tok0);
                                for (int d = 1; d < p.n_dst; ++d) tma_store_2d(&outs.m[d], src, f0, tok0);
                            }
                        }
                        bulk_commit();
                    }
                }
            }
        }
        if (elect_one()) bulk_wait_all();      // this warp's TMA stores have left shared memory and reached global memory
    } else if (warp >= WARP_XF0) {
        // ================= transform: the sets of four warps take the steps in turn =================
        const int quarter = warp & 3, set = (warp - WARP_XF0) >> 2;
        const int my_items = (num_items > pair) ? (num_items - pair + num_pairs - 1) / num_pairs : 0;
        const int total = my_items * p.steps;
        const uint32_t a_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + G::A_COL0;
        const uint32_t full0 = mapa_u32(bar_full(0), 0);
        // FWD: this lane's row of the packed tile; DX: this lane's row address for ldmatrix (lanes 0-15 give the first matrix)
        const int row = FWD ? quarter * 32 + lane : lane;
        const int sw = (row >> 2) & 1;                          // the 32-byte swizzle exchanges the halves of a row
        const uint32_t src0 = smem_base + G::P + row * 32 + (FWD ? 0 : (((quarter >> 1) ^ sw) << 4));
        uint32_t ph = 0;
        for (int g = set; g < total && !failed; ph ^= 1u) {
#pragma unroll
            for (int i = 0; i < DT / G::SETS; ++i, g += G::SETS) {
                if (g >= total || failed) break;
                const int s = G::SETS * i + set;
                if (!mbar_wait_warp(bar_pfull(s), ph, p.status, 26)) { failed = true; break; }
                const uint32_t a_tmem = a_base + (uint32_t)((G::SETS * i) % DA + set) * G::A_COLS;
#pragma unroll
                for (int b = 0; b < SB; ++b) {
                    const uint32_t src = src0 + s * PS_BYTES + b * P_BYTES;
                    uint32_t o[32];
                    if (FWD) {
                        const uint4 lo = lds128(src + sw * 16), hi = lds128(src + (sw ^ 1) * 16);
                        const uint32_t px[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            uint32_t(&d)[4] = *reinterpret_cast<uint32_t(*)[4]>(&o[4 * j]);
                            if (MODE == MODE_FWD_PERM) decode16_deint(px[j], d);
                            else decode16(px[j], d);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; j += 2) {       // two groups of 16 reduction indices; the warp's byte columns are one half of the 16
                            uint32_t r[4];
                            ldmatrix_t16x16(src + j * 512, r[0], r[1], r[2], r[3]);
#pragma unroll
                            for (int m = 0; m < 2; ++m) {
                                const int n = 2 * (j + m);
                                expand4x4((quarter & 1) ? r[2 * m + 1] : r[2 * m], o[n], o[n + 1], o[16 + n], o[17 + n]);
                            }
                        }
                    }
                    if (b == 0) {
                        // The A slot was last read by the MMAs of step g - 4, whose commit is on the "empty" barrier of that step's stage.
                        if (g >= DA && !mbar_wait_cluster_warp(bar_empty((s + DT - DA) % DT), G::SETS * i >= DA ? ph : (ph ^ 1u), p.status, 28)) { failed = true; break; }
                        tcgen05_fence_after();
                    }
                    if (FWD) {
                        tmem_st32(a_tmem + b * 32, o);
                    } else {
                        tmem_st16x128(a_tmem + b * 32, *reinterpret_cast<uint32_t(*)[16]>(&o[0]));
                        tmem_st16x128(a_tmem + b * 32 + (16u << 16), *reinterpret_cast<uint32_t(*)[16]>(&o[16]));
                    }
                }
                if (failed) break;
                __syncwarp();                               // all lanes have read the packed tile
                tmem_st_wait();
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster_relaxed(full0 + 8u * s);
                    mbar_arrive(bar_pempty(s));
                }
            }
        }
    }

    // ---- teardown: both CTAs are done with each other's shared and tensor memory before either frees anything ------
    if (p.status != nullptr && *reinterpret_cast<volatile int32_t*>(p.status) != 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == WARP_MMA) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

template <int MODE, int NT, bool LEAN = false>
static int launch_t(const CUtensorMap& tmT, const CUtensorMap& tmP, const OutMaps& outs, Params& p, cudaStream_t st) {
    constexpr int smem = Geo<NT>::BYTES;
    static std::atomic<int> max_pairs[64];      // co-resident CTA pairs per device; 0 = not yet queried
    int dev = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return EL_ERR_DEVICE;
    cudaLaunchConfig_t cfg = {};
    // A programmatic dependent launch: the set-up of its CTAs runs under the end of the launch before it; the warps that touch
    // global memory wait for that launch to complete first (griddep_wait).
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.blockDim = dim3(Geo<NT>::THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;                    // the occupancy query below knows clusters only
    int dev_pairs = max_pairs[dev].load(std::memory_order_acquire);
    if (dev_pairs == 0) {       // host threads may race here: both then query and store the same number
        EL_CUDA_TRY(cudaFuncSetAttribute(gemm_wt_kernel<MODE, NT, LEAN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        int sms = 0;
        const int rc = device_sm_count(&sms);
        if (rc != EL_OK) return rc;
        cfg.gridDim = dim3((unsigned)(sms & ~1), 1, 1);
        int clusters = 0;
        EL_CUDA_TRY(cudaOccupancyMaxActiveClusters(&clusters, gemm_wt_kernel<MODE, NT, LEAN>, &cfg));
        if (clusters < 1) return EL_ERR_DEVICE;
        dev_pairs = clusters < sms / 2 ? clusters : sms / 2;
        max_pairs[dev].store(dev_pairs, std::memory_order_release);
    }
    p.tiles_r = (p.R + NT - 1) / NT;
    p.tiles_c = (p.C + 2 * BF - 1) / (2 * BF);
    p.k_blocks = (p.D + BK - 1) / BK;
    // a band's activation rows (NT rows x D bytes per token tile) should fit in a third of the 126 MB L2
    const long long row_tile_bytes = (long long)NT * p.k_blocks * BK;
    long long group = (40LL << 20) / (row_tile_bytes > 0 ? row_tile_bytes : 1);
    p.group_rows = (int)(group < 1 ? 1 : (group > p.tiles_r ? p.tiles_r : group));
    const long long tiles = (long long)p.tiles_r * p.tiles_c;
    if (tiles == 0) return EL_OK;
    if (p.k_blocks == 0) return EL_ERR_UNSUPPORTED_SHAPE;
    if (p.k_split < 1 || p.k_blocks % p.k_split != 0) p.k_split = 1;
    p.kbp = p.k_blocks / p.k_split;
    if (p.k_split > 1 && p.kbp % Geo<NT>::SB != 0) return EL_ERR_UNSUPPORTED_SHAPE;
    p.steps = (p.kbp + Geo<NT>::SB - 1) / Geo<NT>::SB;
    const long long items = tiles * p.k_split;
    const int pairs = (int)(items < dev_pairs ? items : dev_pairs);
    cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
    cfg.numAttrs = 2;
    EL_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_wt_kernel<MODE, NT, LEAN>, tmT, tmP, outs, p));
    return check_launch();
}

// Token tile and reduction split of a problem: the pair with the least estimated time, in SM cycles.
//   * A 128-deep block costs a pair about 700 cycles at 256 tokens (the MMAs, 512), 460 at 128, 370 at 64 and 350 at 32 (the
//     transform warps, however few tokens there are).  With many tiles the large tile wins; with few, small tiles put more pairs to
//     work.  us per launch at tile 256 / 128 / 64 / 32: 1024 tokens 1536 -> 1536 12.5 / 9.7 / 11.0 / 12.8, 4096 tokens 4096 -> 512
//     20.0 / 14.5 / - / -, 64 tokens 4096 -> 11008 17.4 / 14.6 / 12.7 / 17.9, 256 tokens 4096 -> 4096 18.0 / 13.1 / 12.2 / 17.1, 2048
//     tokens 2048 -> 2048 14.3 / 14.4 / 18.6 / 26.6, 4096 tokens 4096 -> 11008 112.6 / 135.7 / - / -.
//   * The reduction may be cut into q <= q_max parts of at least 16 blocks that run on different pairs at the same time; each part
//     stores its int32 sums and a second pass adds them (exact) and applies the epilogue: a launch (about 6000 cycles) and the
//     round trip of the sums.
struct Plan {
    int nt, q;
};
static Plan make_plan(int R, int C, int D, bool lean, int q_max) {
    int sms = 0;
    if (device_sm_count(&sms) != EL_OK || sms < 2) sms = 148;
    const long long pairs = sms / 2, k_blocks = (D + BK - 1) / BK;
    Plan best{256, 1};
    long long best_time = -1;
    constexpr int nts[4] = {256, 128, 64, 32}, cost[4] = {700, 460, 370, 350};
    for (int i = 0; i < (lean ? 1 : 4); ++i) {
        const long long tiles = ((R + nts[i] - 1LL) / nts[i]) * ((C + 2 * BF - 1LL) / (2 * BF)), sb = i == 0 ? 1 : 2;
        for (int q = 1; q <= q_max; ++q) {
            if (q > 1 && (k_blocks % (q * sb) != 0 || k_blocks / q < 16 || tiles * q > pairs)) continue;
            const long long rounds = (tiles * q + pairs - 1) / pairs, blocks = (k_blocks / q + sb - 1) / sb * sb;
            const long long time = rounds * blocks * cost[i] + (q > 1 ? 6000 + (long long)q * R * C * 4 / 2000 : 0);
            if (best_time < 0 || time < best_time) best = Plan{nts[i], q}, best_time = time;
        }
    }
    return best;
}

}  // namespace wt

namespace tc {
int make_map(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch, uint32_t box_cols,
             uint32_t box_rows, int swizzle_bytes);
int make_map_out(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch_bytes, int esz, int box_cols);
}
int gemm_tc_eligible(int mode, const void* A, const void* B, int R, int C, int D);
int launch_reduce_scale_gather(const int* parts, int n_parts, void* const* out_all, int n_ranks, long long row_offset,
                               long long rows_total, const EpiParams& epi, int Mr, int C, cudaStream_t st);

// The largest number of parts that a reduction is cut into, and what the workspace of such a call is sized for: parts of 256 x 256
// tiles that fill at most one wave of pairs, for reductions of at least 48 blocks, at least 16 blocks per part, at most 8 parts.
// (Shorter reductions gain nothing: at 4096 -> 512 and 32 blocks the second pass and its int32 round trip cost what the shorter
// main loop saves, measured.)
int gemm_wt_split_max(int R, int C, int D) {
    int sms = 0;
    if (device_sm_count(&sms) != EL_OK || sms < 2) return 1;
    const long long pairs = sms / 2;
    const long long tiles = (long long)((R + 255) / 256) * ((C + 2 * wt::BF - 1) / (2 * wt::BF));
    const int k_blocks = (D + wt::BK - 1) / wt::BK;
    int best = 1;
    for (int q = 2; q <= 8; ++q)
        if (tiles * q <= pairs && k_blocks >= 48 && k_blocks % q == 0 && k_blocks / q >= 16) best = q;
    return best;
}

// Forward (mode 0) and dX (mode 1).
// `dst` (optional): n_dst base pointers of [R, ld_total] output matrices that all receive this launch's [R, C] result
// at column `col_offset` (the own buffer and the peers' buffers of an N-sharded layer: the all-gather of the output
// happens as TMA stores from the epilogue).  With dst == nullptr the result goes to epi.out alone.
// `rows_per_dst` > 0 selects the scatter form instead: dst[d] is a dense [rows_per_dst, C] matrix that receives the
// rows [d*rows_per_dst, (d+1)*rows_per_dst) of the result (the reduce-scatter half of a cross-rank reduction of dX).
int launch_gemm_wt(int mode, const int8_t* A, const void* B, int R, int C, int D, const EpiParams& epi, int32_t* status,
                   cudaStream_t st, void* const* dst, int n_dst, long long ld_total, long long col_offset, int rows_per_dst,
                   int first_dst, void* workspace, size_t workspace_bytes, bool lean) {
    if (mode != MODE_FWD && mode != MODE_DX) return EL_ERR_INVALID_ARG;
    int rc = gemm_tc_eligible(mode, A, B, R, C, D);
    if (rc != EL_OK) return rc;
    rc = require_sm100();
    if (rc != EL_OK) return rc;
    wt::Params p{};
    p.R = R; p.C = C; p.D = D;
    p.epi = epi;
    p.status = status;
    p.k_split = 1;
    p.small_sums = D <= 32767;
    const int esz = (epi.out_dtype == EL_BF16 || epi.out_dtype == EL_F16) ? 2 : 4;
    wt::OutMaps outs{};
    CUtensorMap tmT, tmP;
    // split reduction: needs the caller's workspace, a dense scaled output and 8-column vectors in the second pass
    p.tma_store = dst != nullptr || (((reinterpret_cast<uintptr_t>(epi.out) & 15) == 0) && ((epi.ldo * esz) % 16 == 0));
    const bool may_split = dst == nullptr && workspace != nullptr && epi.out_dtype != EL_I32 && p.tma_store && epi.ldo == C && C % 8 == 0 &&
                           (reinterpret_cast<uintptr_t>(workspace) & 15) == 0;
    int q_max = may_split ? gemm_wt_split_max(R, C, D) : 1;
    while (q_max > 1 && (size_t)q_max * R * C * sizeof(int) > workspace_bytes) --q_max;
    const wt::Plan plan = wt::make_plan(R, C, D, lean, q_max);
    const int nt = plan.nt;
    if (dst != nullptr && rows_per_dst > 0) {
        if (n_dst < 1 || n_dst > wt::MAX_DST || rows_per_dst % 32 != 0 || (long long)rows_per_dst * n_dst < R) return EL_ERR_INVALID_ARG;
        for (int d = 0; d < n_dst; ++d) {
            if (dst[d] == nullptr) return EL_ERR_NULL_PTR;
            if ((rc = tc::make_map_out(&outs.m[d], dst[d], C, rows_per_dst, (uint64_t)C * esz, esz, 32)) != EL_OK) return rc;
        }
        p.n_dst = n_dst;
        p.rows_per_dst = rows_per_dst;
        if (first_dst < 0 || first_dst >= n_dst) return EL_ERR_INVALID_ARG;
        const int row_tiles = (R + nt - 1) / nt;
        p.row_rotate = (int)(((long long)first_dst * rows_per_dst / nt) % row_tiles);
    } else if (dst != nullptr) {
        if (n_dst < 1 || n_dst > wt::MAX_DST || ld_total < col_offset + C || col_offset < 0) return EL_ERR_INVALID_ARG;
        if (C % 32 != 0) return EL_ERR_UNSUPPORTED_SHAPE;      // 32-column store boxes must not reach into a neighbour's window
        for (int d = 0; d < n_dst; ++d) {
            if (dst[d] == nullptr) return EL_ERR_NULL_PTR;
            const char* base = static_cast<const char*>(dst[d]) + col_offset * esz;
            if ((rc = tc::make_map_out(&outs.m[d], base, C, R, (uint64_t)ld_total * esz, esz, 32)) != EL_OK) return rc;
        }
        p.n_dst = n_dst;
    } else {
        p.n_dst = 1;
        if (plan.q > 1) {
            p.k_split = plan.q;
            p.epi.out_dtype = EL_I32;                   // the parts are raw int32 sums; the second pass scales
            p.epi.absmax = nullptr;
            for (int part = 0; part < plan.q; ++part) {
                char* base = static_cast<char*>(workspace) + (size_t)part * R * C * sizeof(int);
                if ((rc = tc::make_map_out(&outs.m[part], base, C, R, (uint64_t)C * 4, 4, 32)) != EL_OK) return rc;
            }
        } else if (p.tma_store && (rc = tc::make_map_out(&outs.m[0], epi.out, C, R, (uint64_t)epi.ldo * esz, esz, 32)) != EL_OK) {
            return rc;
        }
    }
    if ((rc = tc::make_map(&tmT, A, D, R, D, wt::BK, nt / 2, 128)) != EL_OK) return rc;
    const bool fwd = mode == MODE_FWD;
    if (fwd) rc = tc::make_map(&tmP, B, D / 4, C, D / 4, wt::BK / 4, wt::BF, 32);                              // [C output features, D/4 bytes]
    else rc = tc::make_map(&tmP, B, C / 4, D, C / 4, wt::BF / 4, nt == 256 ? wt::BK : 2 * wt::BK, 32);        // [D reduction rows, C/4 bytes]
    if (rc != EL_OK) return rc;
    switch (nt) {
        case 256:
            if (lean) rc = fwd ? wt::launch_t<MODE_FWD, 256, true>(tmT, tmP, outs, p, st) : wt::launch_t<MODE_DX, 256, true>(tmT, tmP, outs, p, st);
            else rc = fwd ? wt::launch_t<MODE_FWD, 256>(tmT, tmP, outs, p, st) : wt::launch_t<MODE_DX, 256>(tmT, tmP, outs, p, st);
            break;
        case 128: rc = fwd ? wt::launch_t<MODE_FWD, 128>(tmT, tmP, outs, p, st) : wt::launch_t<MODE_DX, 128>(tmT, tmP, outs, p, st); break;
        case 64: rc = fwd ? wt::launch_t<MODE_FWD, 64>(tmT, tmP, outs, p, st) : wt::launch_t<MODE_DX, 64>(tmT, tmP, outs, p, st); break;
        default: rc = fwd ? wt::launch_t<MODE_FWD, 32>(tmT, tmP, outs, p, st) : wt::launch_t<MODE_DX, 32>(tmT, tmP, outs, p, st); break;
    }
    if (rc != EL_OK || p.k_split == 1) return rc;
    void* out_one[1] = {epi.out};
    return launch_reduce_scale_gather(static_cast<const int*>(workspace), p.k_split, out_one, 1, 0, R, epi, R, C, st);
}

// Up to 64 tokens quantised by launch_quantize_rows_perm or launch_prelinear_quantize_perm, the launch right before this one.  No other
// may come in between, and that one has to be an ordinary launch (see there): the first packed weights are loaded while it runs
// (weights_first), which races with a weight update queued earlier unless that has completed before the quantiser began.
int launch_gemm_wt_decode(const int8_t* xq, const float* absmax, const uint8_t* Wp, const EpiParams& epi, int M, int N, int K, int32_t* status,
                          cudaStream_t st) {
    if (M < 1 || M > 64) return EL_ERR_UNSUPPORTED_SHAPE;
    int rc = gemm_tc_eligible(MODE_FWD, xq, Wp, M, N, K);
    if (rc != EL_OK) return rc;
    rc = require_sm100();
    if (rc != EL_OK) return rc;
    wt::Params p{};
    p.R = M; p.C = N; p.D = K;
    p.epi = epi;
    p.epi.absmax = absmax;
    p.epi.absmax_stride = 1;
    p.status = status;
    p.k_split = 1;
    p.n_dst = 1;
    p.small_sums = K <= 32767;
    p.weights_first = 1;
    const int esz = (epi.out_dtype == EL_BF16 || epi.out_dtype == EL_F16) ? 2 : 4, nt = M <= 32 ? 32 : 64;
    p.tma_store = ((reinterpret_cast<uintptr_t>(epi.out) & 15) == 0) && ((epi.ldo * esz) % 16 == 0);
    wt::OutMaps outs{};
    CUtensorMap tmT, tmP;
    if (p.tma_store && (rc = tc::make_map_out(&outs.m[0], epi.out, N, M, (uint64_t)epi.ldo * esz, esz, 32)) != EL_OK) return rc;
    if ((rc = tc::make_map(&tmT, xq, K, M, K, wt::BK, nt / 2, 128)) != EL_OK) return rc;
    if ((rc = tc::make_map(&tmP, Wp, K / 4, N, K / 4, wt::BK / 4, wt::BF, 32)) != EL_OK) return rc;
    return nt == 32 ? wt::launch_t<MODE_FWD_PERM, 32>(tmT, tmP, outs, p, st) : wt::launch_t<MODE_FWD_PERM, 64>(tmT, tmP, outs, p, st);
}

}  // namespace el
