// Building blocks of the row kernels that stream: a CTA walks over token rows, and every thread owns the same vectors of 8
// columns in every row.  What a thread will read of a later row it copies itself into its own shared-memory slots with
// asynchronous 16-byte copies, so the rows ahead cost neither registers nor barriers: the thread that waits is the thread
// that issued, and no other thread reads its slots.
#pragma once
#include <type_traits>

#include "row_io.cuh"

namespace el {

int device_sm_count(int* out);

namespace rowio {

__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits until at most N of this thread's latest groups are still in flight.
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 16-byte pieces of 8 elements of T
template <typename T> constexpr int PIECES = (int)sizeof(T) / 2;

// Thread t of a CTA owns, with V vectors per thread, the vectors (t/32)*32*V + t%32 + 32*c (c < V) of every row: a warp reads
// and writes runs of 512 bytes, and from one vector to the next all offsets, in memory and in the slots, are constants.
template <int V> __device__ __forceinline__ int column_of(int c) {
    return (((int)threadIdx.x >> 5) * 32 * V + ((int)threadIdx.x & 31) + 32 * c) * 8;
}

// A thread's slots: each warp has its own region of STAGES x VECS x PIECES runs of 32 16-byte words, one word per lane.
template <typename T, int STAGES, int VECS>
struct Slots {
    uint4* base;
    __device__ __forceinline__ explicit Slots(uint4* ring)
        : base(ring + (threadIdx.x >> 5) * (STAGES * VECS * PIECES<T> * 32) + (threadIdx.x & 31)) {}
    __device__ __forceinline__ uint4* at(int s, int c, int p) const { return base + ((s * VECS + c) * PIECES<T> + p) * 32; }
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
    __device__ __forceinline__ void write(int s, int c, const typename Io<T>::Raw& r) const {
        const uint4* d = reinterpret_cast<const uint4*>(&r);
#pragma unroll
        for (int p = 0; p < PIECES<T>; ++p) *at(s, c, p) = d[p];
    }
};

// Two float32 values as one operand: sm_100 multiplies and adds such pairs in one instruction, each value rounded on its own, so
// the results are those of the two scalar instructions at half the issue slots (which is what bounds these kernels).
// A product whose result is added or subtracted next goes through mul2_exact: the assembler contracts mul.rn.f32x2 and
// add.rn.f32x2 into one fused operation (seen as int8 values that differ at ties), which a product formed as a*b + nz, nz = -0
// unknown at compile time, does not allow; adding -0 changes no value and no sign.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo_of(f32x2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a;
}
__device__ __forceinline__ float hi_of(f32x2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return b;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 negative_zeros() {      // grids of these kernels are one-dimensional: blockIdx.z is 0
    const float z = __uint_as_float(0x80000000u + blockIdx.z);
    return pair(z, z);
}
__device__ __forceinline__ f32x2 mul2_exact(f32x2 a, f32x2 b, f32x2 nz) { return fma2(a, b, nz); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
template <typename T> __device__ __forceinline__ void unpack2(const typename Io<T>::Raw& r, f32x2 v[4]) {
    float f[8];
    Io<T>::unpack(r, f);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = pair(f[2 * i], f[2 * i + 1]);
}
template <typename T> __device__ __forceinline__ typename Io<T>::Raw pack2(const f32x2 v[4]) {       // rounds to the I/O type
    const float f[8] = {lo_of(v[0]), hi_of(v[0]), lo_of(v[1]), hi_of(v[1]), lo_of(v[2]), hi_of(v[2]), lo_of(v[3]), hi_of(v[3])};
    return Io<T>::pack(f);
}
// sum of the 8 float32 products a*b as float64 terms
__device__ __forceinline__ double dot8(const f32x2 a[4], const f32x2 b[4]) {
    double s = 0.0, t = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const f32x2 p = mul2(a[i], b[i]);
        s += (double)lo_of(p);
        t += (double)hi_of(p);
    }
    return s + t;
}
template <typename T> __device__ __forceinline__ typename Io<T>::Raw raw_zero() {
    float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    return Io<T>::pack(z);
}

// io(a*b) for 8 elements of the I/O type.  The product of two 16-bit values is exact in float32, so one packed multiply with
// a single rounding gives what a float32 product rounded to the I/O type gives, in a quarter of the instructions.  A bfloat16
// product (16 significant bits) with a bit below float32's last place, 2^-149, is no exception: it is below 2^-134, half of the
// smallest bfloat16, and both ways give a zero of its sign.
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

// Half of such a vector: 4 elements, for loops that would not fit in the registers eight at a time.
template <typename T> struct Quad { uint2 a; };
template <> struct Quad<float> { float4 a; };
template <typename T> __device__ __forceinline__ Quad<T> quad_of(const typename Io<T>::Raw& r, int half) {
    Quad<T> q;
    if constexpr (sizeof(T) == 2) q.a = half ? make_uint2(r.a.z, r.a.w) : make_uint2(r.a.x, r.a.y);
    else q.a = half ? r.b : r.a;
    return q;
}
template <typename T> __device__ __forceinline__ void unpack2(const Quad<T>& q, f32x2 v[2]) {
    if constexpr (std::is_same<T, float>::value) {
        v[0] = pair(q.a.x, q.a.y);
        v[1] = pair(q.a.z, q.a.w);
    } else if constexpr (std::is_same<T, __half>::value) {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&q.a.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&q.a.y));
        v[0] = pair(a.x, a.y);
        v[1] = pair(b.x, b.y);
    } else {
        v[0] = pair(__uint_as_float(q.a.x << 16), __uint_as_float(q.a.x & 0xFFFF0000u));
        v[1] = pair(__uint_as_float(q.a.y << 16), __uint_as_float(q.a.y & 0xFFFF0000u));
    }
}
template <typename T> __device__ __forceinline__ Quad<T> pack2(f32x2 v0, f32x2 v1) {       // rounds to the I/O type
    Quad<T> q;
    if constexpr (std::is_same<T, float>::value) q.a = make_float4(lo_of(v0), hi_of(v0), lo_of(v1), hi_of(v1));
    else if constexpr (std::is_same<T, __half>::value) q.a = make_uint2(pack_f16x2(lo_of(v0), hi_of(v0)), pack_f16x2(lo_of(v1), hi_of(v1)));
    else q.a = make_uint2(pack_bf16x2(lo_of(v0), hi_of(v0)), pack_bf16x2(lo_of(v1), hi_of(v1)));
    return q;
}
template <typename T> __device__ __forceinline__ Quad<T> mul_quad(const Quad<T>& a, const Quad<T>& b) {       // io(a*b)
    Quad<T> q;
    if constexpr (std::is_same<T, float>::value)
        q.a = make_float4(__fmul_rn(a.a.x, b.a.x), __fmul_rn(a.a.y, b.a.y), __fmul_rn(a.a.z, b.a.z), __fmul_rn(a.a.w, b.a.w));
    else if constexpr (std::is_same<T, __half>::value) q.a = make_uint2(mul_f16x2(a.a.x, b.a.x), mul_f16x2(a.a.y, b.a.y));
    else q.a = make_uint2(mul_bf16x2(a.a.x, b.a.x), mul_bf16x2(a.a.y, b.a.y));
    return q;
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

// CTA-wide sum of doubles and maximum of words with one barrier between the two halves: one entry of `red` per warp, then every
// warp joins the entries itself (the same operations in every warp, so all threads hold the same bits).  The caller alternates
// between two `red` buffers from row to row, so that a buffer is rewritten only after the barrier of the row in between.
constexpr int MAX_RED = 32;
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double sum_red(const double* red) {
    const int lane = threadIdx.x & 31;
    return warp_sum(lane < (int)(blockDim.x >> 5) ? red[lane] : 0.0);
}
__device__ __forceinline__ uint32_t max_red(const uint32_t* red) {
    const int lane = threadIdx.x & 31;
    return __reduce_max_sync(0xffffffffu, lane < (int)(blockDim.x >> 5) ? red[lane] : 0u);
}

// Threads that an SM holds at `regs` registers each: 16384 registers in each of its four parts.
constexpr int resident_threads(int regs) { return 512 / regs * 128; }

// Threads of a streaming CTA for rows of K elements, VECS vectors of 8 per thread: whole warps.
inline int stream_threads(int K, int vecs) { return ((K + 8 * vecs - 1) / (8 * vecs) + 31) & ~31; }

}  // namespace rowio

// The int8 row of a token, 8 elements.  FAST, for a row whose largest magnitude gives s = 127/absmax: adding 1.5*2^23 rounds
// |y*s| <= 127 to the nearest even integer and leaves it in the low mantissa bits (no trip through the conversion unit); a row
// with a non-finite value takes the saturating conversion, NaN -> 0.
template <typename T, bool FAST>
__device__ __forceinline__ uint2 quantise8(const typename rowio::Io<T>::Raw& raw, float s, rowio::f32x2 nz) {
    using namespace rowio;
    int qi[8];
    if (FAST) {
        f32x2 y[4];
        unpack2<T>(raw, y);
        const f32x2 ss = pair(s, s), magic = pair(12582912.0f, 12582912.0f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const f32x2 r = add2(mul2_exact(y[i], ss, nz), magic);
            qi[2 * i] = __float_as_int(lo_of(r));
            qi[2 * i + 1] = __float_as_int(hi_of(r));
        }
    } else {
        float y[8];
        Io<T>::unpack(raw, y);
#pragma unroll
        for (int i = 0; i < 8; ++i) qi[i] = q8_sat(__fmul_rn(finite_or_nan(y[i]), s));
    }
    return make_uint2(pack4_s8(qi[0], qi[1], qi[2], qi[3]), pack4_s8(qi[4], qi[5], qi[6], qi[7]));
}

// dweight[k] = float(sum of the CTAs' partial sums).  A CTA covers 32 columns (one per lane); its W warps (8 or 32) each add
// every W-th partial in order, and warp 0 adds their results in order: a fixed order of additions for a given width.
// Few columns take 32 warps: 592 partials of 16 columns on 8 warps are a chain of dependent loads (10.9 us, 3.8 us with 32); where
// the columns fill the SMs, 8 warps per CTA are enough and start sooner.
static __global__ void __launch_bounds__(1024)
dweight_kernel(const double* __restrict__ partial, int n_parts, float* __restrict__ dweight, int K) {
    __shared__ double part[32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int k = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (k < K) {
#pragma unroll 8
        for (int p = warp; p < n_parts; p += warps) s += partial[(size_t)p * K + k];
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && k < K) {
        double t = 0.0;
        for (int w = 0; w < warps; ++w) t += part[w][lane];
        dweight[k] = (float)t;
    }
}

static int launch_dweight(const double* partial, int n_parts, float* dweight, int K, cudaStream_t st) {
    int sms = 148;
    device_sm_count(&sms);
    dweight_kernel<<<(K + 31) / 32, (K + 31) / 32 <= sms ? 1024 : 256, 0, st>>>(partial, n_parts, dweight, K);
    return check_launch();
}

}  // namespace el
