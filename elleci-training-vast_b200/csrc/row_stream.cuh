// Building blocks of the row kernels that stream: a CTA walks over token rows, and every thread owns the same vectors of 8
// columns in every row.  What a thread will read of a later row it copies itself into its own shared-memory slots with
// asynchronous 16-byte copies, so the rows ahead cost neither registers nor barriers: the thread that waits is the thread
// that issued, and no other thread reads its slots.
#pragma once
#include "row_io.cuh"

namespace el {
namespace rowio {

__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits until at most N of this thread's latest groups are still in flight.
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 16-byte pieces of 8 elements of T
template <typename T> constexpr int PIECES = (int)sizeof(T) / 2;

// A thread's slots: piece p of vector c of stage s lies at ((s*VECS + c)*PIECES + p)*blockDim.x + threadIdx.x, so the lanes of
// a warp touch consecutive 16-byte words.
template <typename T, int VECS>
struct Slots {
    uint4* base;
    __device__ __forceinline__ uint4* at(int s, int c, int p) const {
        return base + ((size_t)(s * VECS + c) * PIECES<T> + p) * blockDim.x + threadIdx.x;
    }
    __device__ __forceinline__ void fetch(int s, int c, const T* src) const {
#pragma unroll
        for (int p = 0; p < PIECES<T>; ++p) cp_async16(at(s, c, p), reinterpret_cast<const uint4*>(src) + p);
    }
    __device__ __forceinline__ typename Io<T>::Raw read(int s, int c) const {
        typename Io<T>::Raw r;
        uint4* d = reinterpret_cast<uint4*>(&r);
#pragma unroll
        for (int p = 0; p < PIECES<T>; ++p) d[p] = *at(s, c, p);
        return r;
    }
};
template <typename T> __device__ __forceinline__ typename Io<T>::Raw raw_zero() {
    float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    return Io<T>::pack(z);
}

// io(a*b) for 8 elements of the I/O type.  The product of two 16-bit values is exact in float32, so one packed multiply with
// a single rounding gives what a float32 product rounded to the I/O type gives, in a quarter of the instructions.
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t mul_f16x2(uint32_t a, uint32_t b) {
    const __half2 r = __hmul2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ Io<__nv_bfloat16>::Raw mul_raw(const Io<__nv_bfloat16>::Raw& a, const Io<__nv_bfloat16>::Raw& b) {
    return {make_uint4(mul_bf16x2(a.a.x, b.a.x), mul_bf16x2(a.a.y, b.a.y), mul_bf16x2(a.a.z, b.a.z), mul_bf16x2(a.a.w, b.a.w))};
}
__device__ __forceinline__ Io<__half>::Raw mul_raw(const Io<__half>::Raw& a, const Io<__half>::Raw& b) {
    return {make_uint4(mul_f16x2(a.a.x, b.a.x), mul_f16x2(a.a.y, b.a.y), mul_f16x2(a.a.z, b.a.z), mul_f16x2(a.a.w, b.a.w))};
}
__device__ __forceinline__ Io<float>::Raw mul_raw(const Io<float>::Raw& a, const Io<float>::Raw& b) {
    Io<float>::Raw r;
    r.a = make_float4(__fmul_rn(a.a.x, b.a.x), __fmul_rn(a.a.y, b.a.y), __fmul_rn(a.a.z, b.a.z), __fmul_rn(a.a.w, b.a.w));
    r.b = make_float4(__fmul_rn(a.b.x, b.b.x), __fmul_rn(a.b.y, b.b.y), __fmul_rn(a.b.z, b.b.z), __fmul_rn(a.b.w, b.b.w));
    return r;
}

// Running maximum of |value| on bit patterns: the order of finite values is the order of their bits, and infinities and NaN
// come out on top.  For 16-bit types both halves of a word carry a maximum until magnitude_bits joins them.
__device__ __forceinline__ uint32_t max_bits(uint32_t m, const Io<__nv_bfloat16>::Raw& r) {
    m = __vmaxu2(m, __vmaxu2(r.a.x & 0x7fff7fffu, r.a.y & 0x7fff7fffu));
    return __vmaxu2(m, __vmaxu2(r.a.z & 0x7fff7fffu, r.a.w & 0x7fff7fffu));
}
__device__ __forceinline__ uint32_t max_bits(uint32_t m, const Io<__half>::Raw& r) {
    return max_bits(m, Io<__nv_bfloat16>::Raw{r.a});
}
__device__ __forceinline__ uint32_t max_bits(uint32_t m, const Io<float>::Raw& r) {
    const float v[8] = {r.a.x, r.a.y, r.a.z, r.a.w, r.b.x, r.b.y, r.b.z, r.b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) m = max(m, __float_as_uint(v[i]) & 0x7fffffffu);
    return m;
}
template <typename T> __device__ __forceinline__ uint32_t magnitude_bits(uint32_t m) { return max(m & 0xffffu, m >> 16); }
template <> __device__ __forceinline__ uint32_t magnitude_bits<float>(uint32_t m) { return m; }
template <typename T> __device__ __forceinline__ float magnitude(uint32_t bits);
template <> __device__ __forceinline__ float magnitude<__nv_bfloat16>(uint32_t bits) { return __uint_as_float(bits << 16); }
template <> __device__ __forceinline__ float magnitude<__half>(uint32_t bits) { return __half2float(__ushort_as_half((unsigned short)bits)); }
template <> __device__ __forceinline__ float magnitude<float>(uint32_t bits) { return __uint_as_float(bits); }

// CTA-wide sum of doubles and maximum of words with one barrier each: the caller alternates between two `red` buffers of one
// entry per warp from row to row, so that a buffer is rewritten only after the barrier of the row in between.
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double sum_red(const double* red) {      // same order in every thread
    const int nw = blockDim.x >> 5;
    double t = red[0];
    for (int i = 1; i < nw; ++i) t += red[i];
    return t;
}
__device__ __forceinline__ uint32_t max_red(const uint32_t* red) {
    const int nw = blockDim.x >> 5;
    uint32_t t = red[0];
    for (int i = 1; i < nw; ++i) t = max(t, red[i]);
    return t;
}
constexpr int MAX_RED = 32;

// Threads of a streaming CTA for rows of K elements, VECS vectors of 8 per thread: whole warps.
inline int stream_threads(int K, int vecs) { return ((K + 8 * vecs - 1) / (8 * vecs) + 31) & ~31; }


}  // namespace rowio

// Tokens' int8 rows: shared by the streaming norm and gate kernels.  y*s for a row whose largest magnitude gives
// s = 127/absmax: adding 1.5*2^23 rounds |y*s| <= 127 to the nearest even integer and leaves it in the low mantissa bits (no
// trip through the conversion unit); rows with a non-finite value take the saturating conversion, NaN -> 0.
template <bool FAST>
__device__ __forceinline__ uint2 quantise8(const float y[8], float s) {
    int qi[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        qi[i] = FAST ? __float_as_int(__fadd_rn(__fmul_rn(y[i], s), 12582912.0f)) : q8_sat(__fmul_rn(finite_or_nan(y[i]), s));
    return make_uint2(pack4_s8(qi[0], qi[1], qi[2], qi[3]), pack4_s8(qi[4], qi[5], qi[6], qi[7]));
}

}  // namespace el
