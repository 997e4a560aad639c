// SwiGLU gate fused with the pre-linear RMSNorm and the per-token int8 quantiser of the down projection, and the
// backward pass of the three.
//
// The reference's feed-forward block is  w3( silu(w1 x) * w2 x )  (model/model.py:86-108), and its INT2 linear layer
// normalises and quantises whatever it is given (core/bitnet/bitnet_int2_optimized.py:72-86,201-210).  Between the
// gate/up GEMMs and the down GEMM lie, as tensor operations: silu, the product, the float32 norm, two casts, the
// weight product and the quantiser - about thirteen bytes of memory traffic per hidden element.  Here one kernel reads
// the gate and up rows and writes the int8 row of the down projection (five bytes per element); the backward kernel
// reads the gradient of the normalised product and the gate and up rows and writes both gradients.
//
// Every float32 step is a single correctly rounded operation in a fixed order (the exponential is a fixed polynomial
// evaluated with fused multiply-adds, row sums are accumulated in float64), so the CPU oracle reproduces the kernels
// bit for bit.
#include "row_stream.cuh"

namespace el {

int device_sm_count(int* out);
size_t rmsnorm_backward_workspace_bytes(int K);

namespace {

using namespace rowio;

// e^t in float32 for the sigmoid: t clamped to [-87, 87] (beyond it 1 + e^t no longer changes, or the sigmoid is below
// 2e-38), n = round-half-even(t*log2(e)) taken by adding and subtracting 1.5*2^23 (its low mantissa bits are n as an
// integer), r = t - n*ln2 in two fused steps (ln2 in the two parts that
// Moshier's Cephes library uses), degree-7 Taylor polynomial in Horner form with fused multiply-adds, times
// 2^n built in the exponent field.  About 1 ulp.  A NaN argument is clamped away (fmaxf returns the other operand); the
// callers multiply by the argument afterwards, which brings the NaN back.
__device__ __forceinline__ float exp_fixed(float t) {
    t = fminf(fmaxf(t, -87.0f), 87.0f);
    const float magic = 12582912.0f;
    const float nm = __fadd_rn(__fmul_rn(t, 1.44269504088896341f), magic);
    const float n = __fsub_rn(nm, magic);
    float r = __fmaf_rn(n, -0.693145751953125f, t);
    r = __fmaf_rn(n, -1.42860682030941723e-6f, r);
    float p = 1.0f / 5040.0f;
    p = __fmaf_rn(p, r, 1.0f / 720.0f);
    p = __fmaf_rn(p, r, 1.0f / 120.0f);
    p = __fmaf_rn(p, r, 1.0f / 24.0f);
    p = __fmaf_rn(p, r, 1.0f / 6.0f);
    p = __fmaf_rn(p, r, 0.5f);
    p = __fmaf_rn(p, r, 1.0f);
    p = __fmaf_rn(p, r, 1.0f);
    const float scale = __int_as_float((__float_as_int(nm) + 127) << 23);       // 2^n, n in [-126, 127]
    return __fmul_rn(p, scale);
}

// 1/d correctly rounded for d in [1, 2^126] (here d = 1 + e^t): with r0 the hardware approximation and e = 1 - d*r0 (exact
// in one fused multiply-add up to the last place), 1/d = r0/(1 - e) = r0*(1 + e + e^2 + ...), the geometric series; its
// first three terms leave an error of e^3 < 2^-66.  Compared with __frcp_rn over every mantissa and every exponent of that range.
__device__ __forceinline__ float rcp_series(float d) {
    float r0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d));
    const float e = __fmaf_rn(-d, r0, 1.0f);
    return __fmaf_rn(r0, __fmaf_rn(e, e, e), r0);
}

// sigmoid(g) = 1 / (1 + e^-g)
__device__ __forceinline__ float sigmoid_fixed(float g) { return rcp_series(__fadd_rn(1.0f, exp_fixed(-g))); }

// The same for two values at once (paired instructions: the same operations on each value in the same order).  1/d is formed
// from nd = -d, so that e = 1 - d*r0 = fma(nd, r0, 1).
__device__ __forceinline__ f32x2 both(float v) { return pair(v, v); }
__device__ __forceinline__ f32x2 sigmoid_fixed2(f32x2 g, f32x2 nz) {
    const f32x2 t = pair(fminf(fmaxf(-lo_of(g), -87.0f), 87.0f), fminf(fmaxf(-hi_of(g), -87.0f), 87.0f));
    const f32x2 nm = add2(mul2_exact(t, both(1.44269504088896341f), nz), both(12582912.0f));
    const f32x2 n = sub2(nm, both(12582912.0f));
    f32x2 r = fma2(n, both(-0.693145751953125f), t);
    r = fma2(n, both(-1.42860682030941723e-6f), r);
    f32x2 p = both(1.0f / 5040.0f);
    p = fma2(p, r, both(1.0f / 720.0f));
    p = fma2(p, r, both(1.0f / 120.0f));
    p = fma2(p, r, both(1.0f / 24.0f));
    p = fma2(p, r, both(1.0f / 6.0f));
    p = fma2(p, r, both(0.5f));
    p = fma2(p, r, both(1.0f));
    p = fma2(p, r, both(1.0f));
    const f32x2 scale = pair(__int_as_float((__float_as_int(lo_of(nm)) + 127) << 23), __int_as_float((__float_as_int(hi_of(nm)) + 127) << 23));
    const f32x2 nd = sub2(both(-1.0f), mul2_exact(p, scale, nz));          // -(1 + e^t)
    float r0, r1;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(-lo_of(nd)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(-hi_of(nd)));
    const f32x2 q = pair(r0, r1);
    const f32x2 e = fma2(nd, q, both(1.0f));
    return fma2(q, fma2(e, e, e), q);
}

// Eight elements of the gate: sig = sigmoid(g), s = io(g * sig), h = io(s * u) - silu rounded to the I/O type, then the
// product rounded to the I/O type, as the two tensor operations of the reference round them.
template <typename T>
__device__ __forceinline__ void gated8(const float g[8], const float u[8], float sig[8], float s[8], float h[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        sig[i] = sigmoid_fixed(g[i]);
        s[i] = __fmul_rn(g[i], sig[i]);
    }
    Io<T>::round8(s);
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = __fmul_rn(s[i], u[i]);
    Io<T>::round8(h);
}

// One CTA per token.  H % 8 == 0, rows 16-byte aligned.  `weight` null: no normalisation (y = h, rstd is not written).
// ROW_CACHE: vectors of 8 hidden values a thread keeps in registers between the passes (2 for float32 rows up to 4096: fewer
// registers, more CTAs per SM; 6 for the others, whose elements beyond 12288 are formed again by every pass).
template <typename T, int ROW_CACHE>
__global__ void __launch_bounds__(RN_THREADS, ROW_CACHE == 2 ? 4 : (sizeof(T) == 4 ? 2 : 3))
swiglu_quantize_rows_kernel(const T* __restrict__ gate, const T* __restrict__ up, long long ld, const float* __restrict__ weight,
                            int8_t* __restrict__ q, float* __restrict__ row_absmax, float* __restrict__ rstd_out, int H,
                            float norm_eps, float quant_eps) {
    __shared__ double red_d[RN_THREADS / 32];
    __shared__ float red_f[RN_THREADS / 32];
    const int m = blockIdx.x;
    const T* gr = gate + (size_t)m * ld;
    const T* ur = up + (size_t)m * ld;
    int8_t* qr = q + (size_t)m * H;
    const bool has_norm = weight != nullptr;

    auto hidden = [&](int k, float h[8]) {
        float g[8], u[8], sig[8], s[8];
        Io<T>::load8(gr + k, g);
        Io<T>::load8(ur + k, u);
        gated8<T>(g, u, sig, s, h);
    };

    typename Io<T>::Raw cache[ROW_CACHE];
    const int k_tail = (threadIdx.x + ROW_CACHE * RN_THREADS) * 8;

    // ---- h, and its mean of squares -> rstd ------------------------------------------------------------------------------
    double ss = 0.0;
#pragma unroll
    for (int c = 0; c < ROW_CACHE; ++c) {
        const int k = (threadIdx.x + c * RN_THREADS) * 8;
        if (k < H) {
            float h[8];
            hidden(k, h);
            cache[c] = Io<T>::pack(h);
            if (has_norm) {
#pragma unroll
                for (int i = 0; i < 8; ++i) ss += (double)__fmul_rn(h[i], h[i]);
            }
        }
    }
    float r = 1.0f;
    if (has_norm) {
        for (int k = k_tail; k < H; k += RN_THREADS * 8) {
            float h[8];
            hidden(k, h);
#pragma unroll
            for (int i = 0; i < 8; ++i) ss += (double)__fmul_rn(h[i], h[i]);
        }
        ss = block_sum(ss, red_d);
        const float ms = __fdiv_rn((float)ss, (float)H);
        r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(ms, norm_eps)));
    }

    // y = io(io(h*r) * io(w)), or h itself
    auto normed = [&](const float h[8], int k, float y[8]) {
        if (has_norm) {
            float w[8];
            Io<float>::load8(weight + k, w);
            Io<T>::round8(w);
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = __fmul_rn(h[i], r);
            Io<T>::round8(y);
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = __fmul_rn(y[i], w[i]);
            Io<T>::round8(y);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = h[i];
        }
    };

    // ---- absmax of the row that is quantised ---------------------------------------------------------------------------
    // Taken on the bit patterns of |y| as integers: the order of the finite values is the same, and an infinity or a NaN
    // comes out on top, so one comparison at the end tells whether the row needs the checked passes.
    int amax_bits = 0;
#pragma unroll
    for (int c = 0; c < ROW_CACHE; ++c) {
        const int k = (threadIdx.x + c * RN_THREADS) * 8;
        if (k < H) {
            float h[8], y[8];
            Io<T>::unpack(cache[c], h);
            normed(h, k, y);
            cache[c] = Io<T>::pack(y);
#pragma unroll
            for (int i = 0; i < 8; ++i) amax_bits = max(amax_bits, __float_as_int(y[i]) & 0x7fffffff);
        }
    }
    for (int k = k_tail; k < H; k += RN_THREADS * 8) {
        float h[8], y[8];
        hidden(k, h);
        normed(h, k, y);
#pragma unroll
        for (int i = 0; i < 8; ++i) amax_bits = max(amax_bits, __float_as_int(y[i]) & 0x7fffffff);
    }
    const bool row_finite = !__syncthreads_or(amax_bits >= 0x7f800000);     // same answer in every thread of the CTA
    float amax = block_max_f(__int_as_float(amax_bits), red_f);              // used only when every thread's value is finite
    if (!row_finite) {        // the row holds an infinity or a NaN: the maximum over its finite values only
        amax = 0.0f;
        for (int k = threadIdx.x * 8; k < H; k += RN_THREADS * 8) {
            float h[8], y[8];
            hidden(k, h);
            normed(h, k, y);
#pragma unroll
            for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(finite_or_zero(y[i])));
        }
        amax = block_max_f(amax, red_f);
    }
    const float a = fmaxf(amax, quant_eps);
    const float s = __fdiv_rn(127.0f, a);
    if (threadIdx.x == 0) {
        row_absmax[m] = a;
        if (has_norm) rstd_out[m] = r;
    }

    // ---- quantise --------------------------------------------------------------------------------------------------------
    auto quantise_y = [&](const float y[8], int k) {
        int qi[8];
        if (row_finite) {
            // |y*s| <= 127: adding 1.5*2^23 rounds to the nearest even integer and leaves it in the low mantissa bits
#pragma unroll
            for (int i = 0; i < 8; ++i) qi[i] = __float_as_int(__fadd_rn(__fmul_rn(y[i], s), 12582912.0f));
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) qi[i] = q8_sat(__fmul_rn(finite_or_nan(y[i]), s));
        }
        *reinterpret_cast<uint2*>(qr + k) = make_uint2(pack4_s8(qi[0], qi[1], qi[2], qi[3]), pack4_s8(qi[4], qi[5], qi[6], qi[7]));
    };
#pragma unroll
    for (int c = 0; c < ROW_CACHE; ++c) {
        const int k = (threadIdx.x + c * RN_THREADS) * 8;
        if (k < H) {
            float y[8];
            Io<T>::unpack(cache[c], y);
            quantise_y(y, k);
        }
    }
    for (int k = k_tail; k < H; k += RN_THREADS * 8) {
        float h[8], y[8];
        hidden(k, h);
        normed(h, k, y);
        quantise_y(y, k);
    }
}

// Streaming form (see rmsnorm_quantize_stream_kernel): two rows of gate and up ahead in thread-owned slots, the weight rounded
// once, packed products.  What bounds it: about 36 instructions per element, 22 of them the fixed sigmoid; memory 5 bytes.
// 4096 tokens x 11008, bf16: 111 us in the one-CTA-per-row form, 80 us in this one (L2 flushed).
constexpr int SF_STAGES = 2;
constexpr int SF_VECS = 4;                            // vectors of 8 per thread

template <typename T, bool NORM>
__global__ void __maxnreg__(80)
swiglu_quantize_stream_kernel(const T* __restrict__ gate, const T* __restrict__ up, long long ld, const float* __restrict__ weight,
                              int8_t* __restrict__ q, float* __restrict__ row_absmax, float* __restrict__ rstd_out, int M, int H,
                              float norm_eps, float quant_eps) {
    constexpr int V = SF_VECS;
    constexpr uint32_t INF_BITS = sizeof(T) == 4 ? 0x7f800000u : (std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u);
    extern __shared__ uint4 ring[];
    __shared__ double red_d[2][MAX_RED];
    __shared__ uint32_t red_u[2][MAX_RED];
    __shared__ uint32_t red_f[2][MAX_RED];
    const Slots<T, SF_STAGES, 2 * V> slots(ring);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const f32x2 nz = negative_zeros();
    typename Io<T>::Raw w[V];
    if (NORM) {
#pragma unroll
        for (int c = 0; c < V; ++c) {
            const int k = column_of<V>(c);
            float wv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (k < H) load8_w(weight + k, wv);
            w[c] = Io<T>::pack(wv);                  // rounds to the I/O type
        }
    }
    auto fetch = [&](int stage, int m) {
        if (m < M) {
#pragma unroll
            for (int c = 0; c < V; ++c) {
                const int k = column_of<V>(c);
                if (k < H) {
                    slots.fetch(stage, 2 * c, gate + (size_t)m * ld + k);
                    slots.fetch(stage, 2 * c + 1, up + (size_t)m * ld + k);
                }
            }
        }
        cp_async_commit();
    };
    const int G = gridDim.x;
#pragma unroll
    for (int s = 0; s < SF_STAGES; ++s) fetch(s, blockIdx.x + s * G);
    int stage = 0;
    for (int m = blockIdx.x; m < M; m += G, stage ^= 1) {
        static_assert(SF_STAGES == 2, "stage doubles as the parity of the reduction buffers");
        cp_async_wait<SF_STAGES - 1>();
        // ---- h = io(io(g*sig(g))*u), and its mean of squares -> rstd -----------------------------------------------------------
        typename Io<T>::Raw row[V];
        double ss = 0.0;
#pragma unroll
        for (int c = 0; c < V; ++c) {
            row[c] = raw_zero<T>();
            if (column_of<V>(c) < H) {
                f32x2 g[4];
                unpack2<T>(slots.read(stage, 2 * c), g);
#pragma unroll
                for (int i = 0; i < 4; ++i) g[i] = mul2(g[i], sigmoid_fixed2(g[i], nz));
                row[c] = mul_raw(pack2<T>(g), slots.read(stage, 2 * c + 1));
                if (NORM) {
                    unpack2<T>(row[c], g);
                    ss += dot8(g, g);
                }
            }
        }
        fetch(stage, m + SF_STAGES * G);             // into the slots just read, by the thread that read them
        float r = 1.0f;
        if (NORM) {
            ss = warp_sum(ss);
            if (lane == 0) red_d[stage][warp] = ss;
            __syncthreads();
            ss = sum_red(red_d[stage]);
            const float ms = __fdiv_rn((float)ss, (float)H);
            r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(ms, norm_eps)));
        }
        // ---- y = io(io(h*r) * io(w)), or h itself, and its largest magnitude -----------------------------------------------------
        uint32_t top = 0u;
#pragma unroll
        for (int c = 0; c < V; ++c) {
            if (column_of<V>(c) < H) {
                if (NORM) {
                    f32x2 v[4];
                    unpack2<T>(row[c], v);
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] = mul2(v[i], both(r));
                    row[c] = mul_raw(pack2<T>(v), w[c]);
                }
                top = max_bits(top, row[c]);
            }
        }
        top = __reduce_max_sync(0xffffffffu, magnitude_bits<T>(top));
        if (lane == 0) red_u[stage][warp] = top;
        __syncthreads();
        top = max_red(red_u[stage]);
        float amax = magnitude<T>(top);
        const bool row_finite = top < INF_BITS;      // same answer in every thread of the CTA
        if (!row_finite) {        // the row holds an infinity or a NaN: the maximum over its finite values only
            amax = 0.0f;
#pragma unroll
            for (int c = 0; c < V; ++c) {
                float y[8];
                Io<T>::unpack(row[c], y);
                if (column_of<V>(c) < H) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(finite_or_zero(y[i])));
                }
            }
            const uint32_t b = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
            if (lane == 0) red_f[stage][warp] = b;
            __syncthreads();
            amax = __uint_as_float(max_red(red_f[stage]));
        }
        const float a = fmaxf(amax, quant_eps);
        const float s = __fdiv_rn(127.0f, a);
        if (tid == 0) {
            row_absmax[m] = a;
            if (NORM) rstd_out[m] = r;
        }
        // ---- quantise ---------------------------------------------------------------------------------------------------------------
        const bool fast = row_finite && s <= 3.402823466e38f;
#pragma unroll
        for (int c = 0; c < V; ++c) {
            const int k = column_of<V>(c);
            if (k < H) {
                *reinterpret_cast<uint2*>(q + (size_t)m * H + k) = fast ? quantise8<T, true>(row[c], s, nz) : quantise8<T, false>(row[c], s, nz);
            }
        }
    }
}

// Backward.  Upstream gradient gy [M,H] with respect to the normalised product y (or to h itself when `weight` is
// null).  Follows autograd through the reference's tensor operations, each intermediate rounded where a tensor of the
// I/O type would hold it:
//   s = io(g*sig(g));  h = io(s*u)
//   with the norm:  gn = io(gy*io(w));  c = sum_k gn*h;  dh = io(gn*rstd - h*(rstd^3*c/H));  dweight[k] += gy*io(h*rstd)
//   ds = io(dh*u);  d_up = io(dh*s);  d_gate = io((ds*sig) * (1 + g*(1 - sig)))
// CTA b takes the tokens b, b + gridDim.x, ...; a thread owns the same columns in every token, so the per-column sums of
// dweight live in shared memory without any exchange, and the CTA writes its [H] partial sums to partial[b] at the end.
// SIG_CACHE (with the norm only): vectors of 8 sigmoids a thread keeps in registers from the first pass (the row sum c) to
// the second, so that the exponential is evaluated once per element for rows up to SIG_CACHE*2048 elements.
template <typename T, bool NORM, int SIG_CACHE>
__global__ void __launch_bounds__(RN_THREADS)
swiglu_backward_kernel(const T* __restrict__ gy, const T* __restrict__ gate, const T* __restrict__ up, long long ld,
                       const float* __restrict__ weight, const float* __restrict__ rstd, T* __restrict__ d_gate,
                       T* __restrict__ d_up, long long ld_d, double* __restrict__ partial, int M, int H) {
    extern __shared__ double col_sum[];          // [H] when NORM
    __shared__ double red_d[RN_THREADS / 32];
    if (NORM) {
        for (int k = threadIdx.x * 8; k < H; k += RN_THREADS * 8) {
#pragma unroll
            for (int i = 0; i < 8; ++i) col_sum[k + i] = 0.0;
        }
    }
    const int k_tail = (threadIdx.x + SIG_CACHE * RN_THREADS) * 8;
    for (int m = blockIdx.x; m < M; m += gridDim.x) {
        const T* yr = gy + (size_t)m * H;
        const T* gr = gate + (size_t)m * ld;
        const T* ur = up + (size_t)m * ld;
        T* dgr = d_gate + (size_t)m * ld_d;
        T* dur = d_up + (size_t)m * ld_d;
        float r = 1.0f, coef = 0.0f;
        float sig_c[SIG_CACHE > 0 ? SIG_CACHE : 1][8];

        // c += sum over the 8 elements at k of gn * h; hands back the sigmoids
        auto row_dot = [&](int k, float sig[8]) -> double {
            float yv[8], g[8], u[8], w[8];
            Io<T>::load8(yr + k, yv);
            Io<T>::load8(gr + k, g);
            Io<T>::load8(ur + k, u);
            Io<float>::load8(weight + k, w);
            float sv[8], h[8];
            gated8<T>(g, u, sig, sv, h);
            Io<T>::round8(w);
#pragma unroll
            for (int i = 0; i < 8; ++i) yv[i] = __fmul_rn(yv[i], w[i]);
            Io<T>::round8(yv);
            double c = 0.0;
#pragma unroll
            for (int i = 0; i < 8; ++i) c += (double)__fmul_rn(yv[i], h[i]);
            return c;
        };
        // the gradients of the 8 elements at k, given their sigmoids
        auto row_grad = [&](int k, const float sig[8]) {
            float yv[8], g[8], u[8], w[8], og[8], ou[8];
            Io<T>::load8(yr + k, yv);
            Io<T>::load8(gr + k, g);
            Io<T>::load8(ur + k, u);
            float sv[8], dh[8], ds[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) sv[i] = __fmul_rn(g[i], sig[i]);
            Io<T>::round8(sv);
            if (NORM) {
                float h[8], gn[8], hn[8];
                Io<float>::load8(weight + k, w);
                Io<T>::round8(w);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    h[i] = __fmul_rn(sv[i], u[i]);
                    gn[i] = __fmul_rn(yv[i], w[i]);
                }
                Io<T>::round8(h);
                Io<T>::round8(gn);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    dh[i] = __fsub_rn(__fmul_rn(gn[i], r), __fmul_rn(h[i], coef));
                    hn[i] = __fmul_rn(h[i], r);
                }
                Io<T>::round8(dh);
                Io<T>::round8(hn);
#pragma unroll
                for (int i = 0; i < 8; ++i) col_sum[k + i] += (double)__fmul_rn(yv[i], hn[i]);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) dh[i] = yv[i];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) ds[i] = __fmul_rn(dh[i], u[i]);
            Io<T>::round8(ds);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                ou[i] = __fmul_rn(dh[i], sv[i]);
                og[i] = __fmul_rn(__fmul_rn(ds[i], sig[i]), __fadd_rn(1.0f, __fmul_rn(g[i], __fsub_rn(1.0f, sig[i]))));
            }
            Io<T>::store8(dgr + k, og);
            Io<T>::store8(dur + k, ou);
        };

        if (NORM) {
            r = rstd[m];
            double c = 0.0;
#pragma unroll
            for (int cv = 0; cv < SIG_CACHE; ++cv) {
                const int k = (threadIdx.x + cv * RN_THREADS) * 8;
                if (k < H) c += row_dot(k, sig_c[cv]);
            }
            for (int k = k_tail; k < H; k += RN_THREADS * 8) {
                float sig[8];
                c += row_dot(k, sig);
            }
            c = block_sum(c, red_d);
            const float r3 = __fmul_rn(__fmul_rn(r, r), r);
            coef = __fdiv_rn(__fmul_rn(r3, (float)c), (float)H);
#pragma unroll
            for (int cv = 0; cv < SIG_CACHE; ++cv) {
                const int k = (threadIdx.x + cv * RN_THREADS) * 8;
                if (k < H) row_grad(k, sig_c[cv]);
            }
        }
        for (int k = NORM ? k_tail : threadIdx.x * 8; k < H; k += RN_THREADS * 8) {
            float g[8], sig[8];
            Io<T>::load8(gr + k, g);
#pragma unroll
            for (int i = 0; i < 8; ++i) sig[i] = sigmoid_fixed(g[i]);
            row_grad(k, sig);
        }
    }
    if (NORM) {
        double* out = partial + (size_t)blockIdx.x * H;
        for (int k = threadIdx.x * 8; k < H; k += RN_THREADS * 8) {
#pragma unroll
            for (int i = 0; i < 8; ++i) out[k + i] = col_sum[k + i];
        }
    }
}

// Streaming form, with the norm: one CTA walks over the tokens with up to two rows of gy, gate and up ahead in thread-owned
// slots (row_stream.cuh), the column sums of dweight and the row's sigmoids in registers, products of two 16-bit values
// packed.  What bounds it: about 55 instructions per element, 22 of them the fixed sigmoid, and two float64 conversions;
// memory 10 bytes.  (The one barrier of a token is a tenth of its time, so the next token's row sum is not pulled ahead as
// in rmsnorm_backward_stream_kernel; its sigmoids would not fit in the registers either.)
// 4096 tokens x 11008, bf16: 228 us with column sums in shared memory at a 64-byte stride (four-way bank conflicts) and
// every row read twice from memory; 138 us in this form (L2 flushed, the dweight kernel included).
// Two stages, not three: a row takes 5 us, five times the memory latency, and what shared memory does not take stays L1 for the
// 32 bytes per thread that spill.  The rounded weights lie in slots of their own instead of registers (150 bytes would spill).
constexpr int SB_STAGES = 2;
template <typename T, int V, int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
swiglu_backward_stream_kernel(const T* __restrict__ gy, const T* __restrict__ gate, const T* __restrict__ up, long long ld,
                              const float* __restrict__ weight, const float* __restrict__ rstd, T* __restrict__ d_gate,
                              T* __restrict__ d_up, long long ld_d, double* __restrict__ partial, int M, int H) {
    extern __shared__ uint4 ring[];
    __shared__ double red[2][MAX_RED];
    const Slots<T, SB_STAGES, 3 * V> slots(ring);
    const Slots<T, 1, V> w_slots(ring + SB_STAGES * 3 * V * PIECES<T> * blockDim.x);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const f32x2 nz = negative_zeros();
    double col[V][8];
#pragma unroll
    for (int c = 0; c < V; ++c) {
        const int k = column_of<V>(c);
        float wv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (k < H) load8_w(weight + k, wv);
        w_slots.write(0, c, Io<T>::pack(wv));        // rounds to the I/O type
#pragma unroll
        for (int i = 0; i < 8; ++i) col[c][i] = 0.0;
    }
    auto fetch = [&](int stage, int m) {
        if (m < M) {
#pragma unroll
            for (int c = 0; c < V; ++c) {
                const int k = column_of<V>(c);
                if (k < H) {
                    slots.fetch(stage, 3 * c, gy + (size_t)m * H + k);
                    slots.fetch(stage, 3 * c + 1, gate + (size_t)m * ld + k);
                    slots.fetch(stage, 3 * c + 2, up + (size_t)m * ld + k);
                }
            }
        }
        cp_async_commit();
    };
    const int G = gridDim.x;
#pragma unroll
    for (int s = 0; s < SB_STAGES; ++s) fetch(s, blockIdx.x + s * G);
    int stage = 0, par = 0;
    for (int m = blockIdx.x; m < M; m += G, par ^= 1) {
        cp_async_wait<SB_STAGES - 1>();
        const float r = rstd[m];
        // ---- c = sum of io(gy*io(w)) * h; the sigmoids stay in registers ------------------------------------------------------------
        f32x2 sig[V][4];
        double dot = 0.0;
#pragma unroll
        for (int c = 0; c < V; ++c) {
            if (column_of<V>(c) < H) {
                f32x2 g[4], gn[4];
                unpack2<T>(slots.read(stage, 3 * c + 1), g);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    sig[c][i] = sigmoid_fixed2(g[i], nz);
                    g[i] = mul2(g[i], sig[c][i]);
                }
                unpack2<T>(mul_raw(pack2<T>(g), slots.read(stage, 3 * c + 2)), g);           // h
                unpack2<T>(mul_raw(slots.read(stage, 3 * c), w_slots.read(0, c)), gn);
                dot += dot8(gn, g);
            }
        }
        dot = warp_sum(dot);
        if (lane == 0) red[par][warp] = dot;
        __syncthreads();
        dot = sum_red(red[par]);
        const float r3 = __fmul_rn(__fmul_rn(r, r), r);
        const float coef = __fdiv_rn(__fmul_rn(r3, (float)dot), (float)H);
        // ---- the gradients --------------------------------------------------------------------------------------------------------------
#pragma unroll
        for (int c = 0; c < V; ++c) {
            const int k = column_of<V>(c);
            if (k < H) {
                const typename Io<T>::Raw yr = slots.read(stage, 3 * c), gr = slots.read(stage, 3 * c + 1), ur = slots.read(stage, 3 * c + 2);
                const typename Io<T>::Raw wr = w_slots.read(0, c);
#pragma unroll
                for (int half = 0; half < 2; ++half) {       // four elements at a time: eight spill
                    const Quad<T> yq = quad_of<T>(yr, half), uq = quad_of<T>(ur, half);
                    f32x2 g[2], h[2], t[2];
                    unpack2<T>(quad_of<T>(gr, half), g);
                    const f32x2 s0 = sig[c][2 * half], s1 = sig[c][2 * half + 1];
                    const Quad<T> sq = pack2<T>(mul2(g[0], s0), mul2(g[1], s1));             // s = io(g*sig)
                    unpack2<T>(mul_quad<T>(sq, uq), h);                                      // h = io(s*u)
                    f32x2 yv[2];
                    unpack2<T>(yq, yv);
                    unpack2<T>(pack2<T>(mul2(h[0], both(r)), mul2(h[1], both(r))), t);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const f32x2 d = mul2(yv[i], t[i]);
                        col[c][4 * half + 2 * i] += (double)lo_of(d);
                        col[c][4 * half + 2 * i + 1] += (double)hi_of(d);
                    }
                    unpack2<T>(mul_quad<T>(yq, quad_of<T>(wr, half)), t);                    // gn = io(gy*io(w))
#pragma unroll
                    for (int i = 0; i < 2; ++i) t[i] = sub2(mul2_exact(t[i], both(r), nz), mul2_exact(h[i], both(coef), nz));
                    const Quad<T> dh = pack2<T>(t[0], t[1]);
                    *reinterpret_cast<Quad<T>*>(d_up + (size_t)m * ld_d + k + 4 * half) = mul_quad<T>(dh, sq);
                    unpack2<T>(mul_quad<T>(dh, uq), t);                                      // ds = io(dh*u)
                    t[0] = mul2(mul2(t[0], s0), add2(both(1.0f), mul2_exact(g[0], sub2(both(1.0f), s0), nz)));
                    t[1] = mul2(mul2(t[1], s1), add2(both(1.0f), mul2_exact(g[1], sub2(both(1.0f), s1), nz)));
                    *reinterpret_cast<Quad<T>*>(d_gate + (size_t)m * ld_d + k + 4 * half) = pack2<T>(t[0], t[1]);
                    asm volatile("" ::: "memory");
                }
            }
        }
        fetch(stage, m + SB_STAGES * G);             // into the slots just read, by the thread that read them
        stage = stage + 1 == SB_STAGES ? 0 : stage + 1;
    }
    double* out = partial + (size_t)blockIdx.x * H;
#pragma unroll
    for (int c = 0; c < V; ++c) {
        const int k = column_of<V>(c);
        if (k < H) {
#pragma unroll
            for (int i = 0; i < 8; i += 2) *reinterpret_cast<double2*>(out + k + i) = make_double2(col[c][i], col[c][i + 1]);
        }
    }
}

int backward_grid(int M, int H, bool norm) {
    int sms = 148;
    device_sm_count(&sms);
    int per_sm = 4;
    if (norm) {
        const size_t smem = (size_t)H * sizeof(double);
        per_sm = (int)((200u * 1024u) / (smem ? smem : 1));
        if (per_sm < 1) per_sm = 1;
        if (per_sm > 4) per_sm = 4;
    }
    const int grid = sms * per_sm;
    return M < grid ? (M < 1 ? 1 : M) : grid;
}

// The layer's input as the fused training kernels form it, written out in the I/O type instead of being quantised: for
// the small-M decode call, whose kernels quantise their few tokens themselves.  x is the layer input, or the gate when
// `up` is given (h = io(io(x*sig(x))*up)); with `weight` the row is normalised (y = io(io(h*rstd)*io(w))).  One CTA per
// token, same order of operations as swiglu_quantize_rows_kernel / rmsnorm_quantize_rows_kernel, so quantising y gives the
// int8 row those kernels give.
template <typename T>
__global__ void __launch_bounds__(RN_THREADS)
prelinear_rows_kernel(const T* __restrict__ x, const T* __restrict__ up, long long ld, const float* __restrict__ weight,
                      T* __restrict__ y, int K, float norm_eps) {
    __shared__ double red_d[RN_THREADS / 32];
    const int m = blockIdx.x;
    const T* xr = x + (size_t)m * ld;
    const T* ur = up ? up + (size_t)m * ld : nullptr;
    T* yr = y + (size_t)m * K;
    auto hidden = [&](int k, float h[8]) {
        Io<T>::load8(xr + k, h);
        if (ur) {
            float g[8], u[8], sig[8], s[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) g[i] = h[i];
            Io<T>::load8(ur + k, u);
            gated8<T>(g, u, sig, s, h);
        }
    };
    float r = 1.0f;
    if (weight) {
        double ss = 0.0;
        for (int k = threadIdx.x * 8; k < K; k += RN_THREADS * 8) {
            float h[8];
            hidden(k, h);
#pragma unroll
            for (int i = 0; i < 8; ++i) ss += (double)__fmul_rn(h[i], h[i]);
        }
        ss = block_sum(ss, red_d);
        const float ms = __fdiv_rn((float)ss, (float)K);
        r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(ms, norm_eps)));
    }
    for (int k = threadIdx.x * 8; k < K; k += RN_THREADS * 8) {
        float h[8];
        hidden(k, h);
        if (weight) {
            float w[8];
            Io<float>::load8(weight + k, w);
            Io<T>::round8(w);
#pragma unroll
            for (int i = 0; i < 8; ++i) h[i] = __fmul_rn(h[i], r);
            Io<T>::round8(h);
#pragma unroll
            for (int i = 0; i < 8; ++i) h[i] = __fmul_rn(h[i], w[i]);
            Io<T>::round8(h);
        }
        Io<T>::store8(yr + k, h);
    }
}

// prelinear_rows_kernel continued through the quantiser, for the decode kernels that take quantised tokens: the layer input is
// formed, quantised per token and written as int8 permuted inside groups of 16 (the layout of decode16_deint), with its
// absmax; y itself never reaches memory.  One CTA per token; a thread keeps one group of 16 elements (K <= 16384).
// At a few tokens the time is the chain of latencies (load, sum, maximum, store), so a row gets as many threads as it has
// groups.  Whole call (this kernel and the GEMV on quantised tokens) against prelinear_rows_kernel and el_linear_decode, CUDA graph,
// us: 4096 -> 11008 with norm, 1 token 9.8 -> 8.7, 8 tokens 12.8 -> 9.1, 64 tokens 26.1 -> 24.4; 11008 -> 4096, 8 tokens 21.2 -> 12.2, with a
// gate 25.3 -> 13.6: all 148 CTAs of the one-launch GEMV quantise all tokens, which from 3 tokens on was most of the call.
template <typename T>
__global__ void __launch_bounds__(1024)
prelinear_quantize_perm_kernel(const T* __restrict__ x, const T* __restrict__ up, long long ld, const float* __restrict__ weight,
                               int8_t* __restrict__ q, float* __restrict__ row_absmax, int K, float norm_eps, float quant_eps) {
    __shared__ double red_d[MAX_RED];
    __shared__ float red_f[MAX_RED];
    // the GEMV behind this launch requests its first weights now and waits for this grid before it reads q
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int m = blockIdx.x, k = threadIdx.x * 16, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool own = k < K;
    const T* xr = x + (size_t)m * ld + k;
    float y[2][8];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int i = 0; i < 8; ++i) y[c][i] = 0.0f;
        if (own) {
            Io<T>::load8(xr + 8 * c, y[c]);
            if (up) {
                float u[8];
                Io<T>::load8(up + (size_t)m * ld + k + 8 * c, u);
#pragma unroll
                for (int i = 0; i < 8; ++i) y[c][i] = __fmul_rn(y[c][i], sigmoid_fixed(y[c][i]));
                Io<T>::round8(y[c]);
#pragma unroll
                for (int i = 0; i < 8; ++i) y[c][i] = __fmul_rn(y[c][i], u[i]);
                Io<T>::round8(y[c]);
            }
        }
    }
    if (weight) {
        float w[2][8];
#pragma unroll
        for (int c = 0; c < 2; ++c)
            if (own) {
                Io<float>::load8(weight + k + 8 * c, w[c]);
                Io<T>::round8(w[c]);
            }
        double ss = 0.0;
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) ss += (double)__fmul_rn(y[c][i], y[c][i]);
        ss = warp_sum(ss);
        if (lane == 0) red_d[warp] = ss;
        __syncthreads();
        ss = sum_red(red_d);
        const float ms = __fdiv_rn((float)ss, (float)K);
        const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(ms, norm_eps)));
#pragma unroll
        for (int c = 0; c < 2; ++c)
            if (own) {
#pragma unroll
                for (int i = 0; i < 8; ++i) y[c][i] = __fmul_rn(y[c][i], r);
                Io<T>::round8(y[c]);
#pragma unroll
                for (int i = 0; i < 8; ++i) y[c][i] = __fmul_rn(y[c][i], w[c][i]);
                Io<T>::round8(y[c]);
            }
    }
    float amax = 0.0f;                  // over the finite values; the conversion below turns the others into 0
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(finite_or_zero(y[c][i])));
    amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
    if (lane == 0) red_f[warp] = amax;
    __syncthreads();
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) amax = fmaxf(amax, red_f[i]);
    const float a = fmaxf(amax, quant_eps);
    const float s = __fdiv_rn(127.0f, a);
    if (threadIdx.x == 0) row_absmax[m] = a;
    if (own) {
        int qi[16];
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) qi[8 * c + i] = q8_sat(__fmul_rn(finite_or_nan(y[c][i]), s));
        *reinterpret_cast<uint4*>(q + (size_t)m * K + k) =
            make_uint4(pack4_s8(qi[0], qi[2], qi[4], qi[6]), pack4_s8(qi[8], qi[10], qi[12], qi[14]),
                       pack4_s8(qi[1], qi[3], qi[5], qi[7]), pack4_s8(qi[9], qi[11], qi[13], qi[15]));
    }
}

// sig[i] = sigmoid(g[i]) as the fused kernels compute it (a check of the fixed arithmetic against a CPU restatement).
__global__ void __launch_bounds__(256) sigmoid_fixed_kernel(const float* __restrict__ g, float* __restrict__ sig, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        sig[i] = sigmoid_fixed(g[i]);
}

}  // namespace

size_t swiglu_backward_workspace_bytes(int H) { return rmsnorm_backward_workspace_bytes(H); }

int launch_prelinear_rows(const void* x, const void* up, int dt, long long ld, const float* weight, float norm_eps, void* y, int M,
                          int K, cudaStream_t st) {
    if (M == 0) return EL_OK;
    if (K <= 0 || K % 8 != 0) return EL_ERR_UNSUPPORTED_SHAPE;
    const size_t esz = (dt == EL_F32) ? 4 : 2;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(up) & 15) || (reinterpret_cast<uintptr_t>(y) & 15) ||
        ((size_t)ld * esz) % 16 != 0 || (reinterpret_cast<uintptr_t>(weight) & 15))
        return EL_ERR_ALIGNMENT;
    switch (dt) {
        case EL_BF16:
            prelinear_rows_kernel<__nv_bfloat16><<<M, RN_THREADS, 0, st>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)up, ld, weight,
                                                                           (__nv_bfloat16*)y, K, norm_eps);
            break;
        case EL_F16:
            prelinear_rows_kernel<__half><<<M, RN_THREADS, 0, st>>>((const __half*)x, (const __half*)up, ld, weight, (__half*)y, K, norm_eps);
            break;
        case EL_F32:
            prelinear_rows_kernel<float><<<M, RN_THREADS, 0, st>>>((const float*)x, (const float*)up, ld, weight, (float*)y, K, norm_eps);
            break;
        default: return EL_ERR_INVALID_ARG;
    }
    return check_launch();
}

// K % 16 == 0, K <= 16384; x, up and weight rows 16-byte aligned.  At least one of `up` and `weight`.  Has to stay an ordinary launch,
// for the reason given at launch_quantize_rows_perm: the kernels behind it read packed weights before they wait for it.
int launch_prelinear_quantize_perm(const void* x, const void* up, int dt, long long ld, const float* weight, float norm_eps, int8_t* q,
                                   float* row_absmax, int M, int K, float quant_eps, cudaStream_t st) {
    if (M == 0) return EL_OK;
    if (K <= 0 || K % 16 != 0 || K > 16384) return EL_ERR_UNSUPPORTED_SHAPE;
    const size_t esz = (dt == EL_F32) ? 4 : 2;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(up) & 15) || (reinterpret_cast<uintptr_t>(q) & 15) ||
        ((size_t)ld * esz) % 16 != 0 || (reinterpret_cast<uintptr_t>(weight) & 15))
        return EL_ERR_ALIGNMENT;
    const int threads = stream_threads(K, 2);
    switch (dt) {
        case EL_BF16:
            prelinear_quantize_perm_kernel<__nv_bfloat16><<<M, threads, 0, st>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)up, ld, weight, q,
                                                                                row_absmax, K, norm_eps, quant_eps);
            break;
        case EL_F16:
            prelinear_quantize_perm_kernel<__half><<<M, threads, 0, st>>>((const __half*)x, (const __half*)up, ld, weight, q, row_absmax, K,
                                                                         norm_eps, quant_eps);
            break;
        case EL_F32:
            prelinear_quantize_perm_kernel<float><<<M, threads, 0, st>>>((const float*)x, (const float*)up, ld, weight, q, row_absmax, K,
                                                                        norm_eps, quant_eps);
            break;
        default: return EL_ERR_INVALID_ARG;
    }
    return check_launch();
}

int launch_sigmoid_fixed(const float* g, float* sig, long long n, cudaStream_t st) {
    if (n == 0) return EL_OK;
    int sms = 148;
    device_sm_count(&sms);
    sigmoid_fixed_kernel<<<sms * 8, 256, 0, st>>>(g, sig, n);
    return check_launch();
}

template <typename T, bool NORM>
static int launch_quantize_stream(const T* gate, const T* up, long long ld, const float* weight, float norm_eps, int8_t* q,
                                  float* row_absmax, float* rstd, int M, int H, float quant_eps, cudaStream_t st) {
    static DeviceOnce attr_once;
    int dev = 0, sms = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    const int rc = device_sm_count(&sms);
    if (rc != EL_OK) return rc;
    if (!attr_once.is_done(dev)) {
        EL_CUDA_TRY(cudaFuncSetAttribute(swiglu_quantize_stream_kernel<T, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr_once.mark(dev);
    }
    const int threads = stream_threads(H, SF_VECS);
    const size_t smem = (size_t)SF_STAGES * 2 * 64 * threads;
    int per_sm = 768 / threads;                      // 80 registers per thread
    const int by_smem = (int)((200u * 1024u) / (smem + 1024));
    per_sm = per_sm < by_smem ? per_sm : by_smem;
    per_sm = per_sm < 1 ? 1 : (per_sm > 24 ? 24 : per_sm);
    const int grid = M < sms * per_sm ? M : sms * per_sm;
    swiglu_quantize_stream_kernel<T, NORM><<<grid, threads, smem, st>>>(gate, up, ld, weight, q, row_absmax, rstd, M, H, norm_eps, quant_eps);
    return check_launch();
}

// 16-bit rows of up to 16384 elements (two stages of gate and up then fit in shared memory) stream; longer ones and float32,
// whose row takes twice the slots for the same arithmetic, run the one-CTA-per-row kernel (float32, 1000 tokens x 4096: 18.4 us there,
// 22.6 us streaming).
template <typename T>
static int launch_quantize_t(const T* gate, const T* up, long long ld, const float* weight, float norm_eps, int8_t* q, float* row_absmax,
                             float* rstd, int M, int H, float quant_eps, cudaStream_t st) {
    if constexpr (sizeof(T) == 2) {
        if (H <= 16384) {
            if (weight) return launch_quantize_stream<T, true>(gate, up, ld, weight, norm_eps, q, row_absmax, rstd, M, H, quant_eps, st);
            return launch_quantize_stream<T, false>(gate, up, ld, weight, norm_eps, q, row_absmax, rstd, M, H, quant_eps, st);
        }
    }
    if constexpr (sizeof(T) == 4) {
        if (H <= 4096) {
            swiglu_quantize_rows_kernel<T, 2><<<M, RN_THREADS, 0, st>>>(gate, up, ld, weight, q, row_absmax, rstd, H, norm_eps, quant_eps);
            return check_launch();
        }
    }
    swiglu_quantize_rows_kernel<T, 6><<<M, RN_THREADS, 0, st>>>(gate, up, ld, weight, q, row_absmax, rstd, H, norm_eps, quant_eps);
    return check_launch();
}

int launch_swiglu_quantize_rows(const void* gate, const void* up, int dt, long long ld, const float* weight, float norm_eps,
                                int8_t* q, float* row_absmax, float* rstd, int M, int H, float quant_eps, cudaStream_t st) {
    if (M == 0) return EL_OK;
    if (H <= 0 || H % 8 != 0) return EL_ERR_UNSUPPORTED_SHAPE;
    const size_t esz = (dt == EL_F32) ? 4 : 2;
    if ((reinterpret_cast<uintptr_t>(gate) & 15) || (reinterpret_cast<uintptr_t>(up) & 15) || ((size_t)ld * esz) % 16 != 0 ||
        (reinterpret_cast<uintptr_t>(weight) & 15) || (reinterpret_cast<uintptr_t>(q) & 7))
        return EL_ERR_ALIGNMENT;
    switch (dt) {
        case EL_BF16: return launch_quantize_t((const __nv_bfloat16*)gate, (const __nv_bfloat16*)up, ld, weight, norm_eps, q, row_absmax, rstd, M, H, quant_eps, st);
        case EL_F16: return launch_quantize_t((const __half*)gate, (const __half*)up, ld, weight, norm_eps, q, row_absmax, rstd, M, H, quant_eps, st);
        case EL_F32: return launch_quantize_t((const float*)gate, (const float*)up, ld, weight, norm_eps, q, row_absmax, rstd, M, H, quant_eps, st);
        default: return EL_ERR_INVALID_ARG;
    }
}

template <typename T, int SIG_CACHE>
static int launch_swiglu_backward_norm(const T* gy, const T* gate, const T* up, long long ld, const float* weight, const float* rstd,
                                       T* d_gate, T* d_up, long long ld_d, float* dweight, double* partial, int M, int H,
                                       cudaStream_t st) {
    const int grid = backward_grid(M, H, true);
    const size_t smem = (size_t)H * sizeof(double);
    static DeviceOnce attr_once;
    int dev = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    if (!attr_once.is_done(dev)) {
        EL_CUDA_TRY(cudaFuncSetAttribute(swiglu_backward_kernel<T, true, SIG_CACHE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         200 * 1024));
        attr_once.mark(dev);
    }
    swiglu_backward_kernel<T, true, SIG_CACHE><<<grid, RN_THREADS, smem, st>>>(gy, gate, up, ld, weight, rstd, d_gate, d_up, ld_d,
                                                                               partial, M, H);
    int rc = check_launch();
    if (rc != EL_OK) return rc;
    return launch_dweight(partial, grid, dweight, H, st);
}

template <typename T, int THREADS>
static int launch_backward_stream(const T* gy, const T* gate, const T* up, long long ld, const float* weight, const float* rstd,
                                  T* d_gate, T* d_up, long long ld_d, float* dweight, double* partial, int M, int H, cudaStream_t st) {
    static DeviceOnce attr_once;
    int dev = 0, sms = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    int rc = device_sm_count(&sms);
    if (rc != EL_OK) return rc;
    if (!attr_once.is_done(dev)) {
        EL_CUDA_TRY(cudaFuncSetAttribute(swiglu_backward_stream_kernel<T, 2, THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         226 * 1024));
        attr_once.mark(dev);
    }
    const int threads = stream_threads(H, 2);
    const size_t smem = (size_t)(SB_STAGES * 3 + 1) * 2 * PIECES<T> * sizeof(uint4) * threads;
    // resident CTAs per SM by registers and shared memory, at most the four per SM that the workspace holds partials for
    int per_sm = THREADS / threads;
    const int by_smem = (int)((226u * 1024u) / smem);
    per_sm = per_sm < by_smem ? per_sm : by_smem;
    per_sm = per_sm < 1 ? 1 : (per_sm > 4 ? 4 : per_sm);
    const int grid = M < sms * per_sm ? M : sms * per_sm;
    swiglu_backward_stream_kernel<T, 2, THREADS><<<grid, threads, smem, st>>>(gy, gate, up, ld, weight, rstd, d_gate, d_up, ld_d, partial, M, H);
    rc = check_launch();
    if (rc != EL_OK) return rc;
    return launch_dweight(partial, grid, dweight, H, st);
}

template <typename T>
static int launch_swiglu_backward_t(const T* gy, const T* gate, const T* up, long long ld, const float* weight, const float* rstd,
                                    T* d_gate, T* d_up, long long ld_d, float* dweight, double* partial, int M, int H,
                                    cudaStream_t st) {
    if (!weight) {
        const int grid = backward_grid(M, H, false);
        swiglu_backward_kernel<T, false, 0><<<grid, RN_THREADS, 0, st>>>(gy, gate, up, ld, nullptr, nullptr, d_gate, d_up, ld_d,
                                                                         nullptr, M, H);
        return check_launch();
    }
    // Rows of up to 12288 16-bit or 8192 float32 elements stream: two vectors per thread, 80 registers at 768 threads (float32: 120
    // at 512, where two stages fill the shared memory).
    constexpr int MAX_T = sizeof(T) == 2 ? 768 : 512;
    if (stream_threads(H, 2) <= MAX_T)
        return launch_backward_stream<T, MAX_T>(gy, gate, up, ld, weight, rstd, d_gate, d_up, ld_d, dweight, partial, M, H, st);
    return launch_swiglu_backward_norm<T, 6>(gy, gate, up, ld, weight, rstd, d_gate, d_up, ld_d, dweight, partial, M, H, st);
}

int launch_swiglu_backward(const void* gy, const void* gate, const void* up, int dt, long long ld, const float* weight,
                           const float* rstd, void* d_gate, void* d_up, long long ld_d, float* dweight, void* workspace,
                           size_t workspace_bytes, int M, int H, cudaStream_t st) {
    if (H <= 0 || H % 8 != 0 || (weight && (size_t)H * sizeof(double) > 200u * 1024u)) return EL_ERR_UNSUPPORTED_SHAPE;
    if (weight && workspace_bytes < swiglu_backward_workspace_bytes(H)) return EL_ERR_INVALID_ARG;
    const size_t esz = (dt == EL_F32) ? 4 : 2;
    if ((reinterpret_cast<uintptr_t>(gy) & 15) || (reinterpret_cast<uintptr_t>(gate) & 15) || (reinterpret_cast<uintptr_t>(up) & 15) ||
        (reinterpret_cast<uintptr_t>(d_gate) & 15) || (reinterpret_cast<uintptr_t>(d_up) & 15) || ((size_t)ld * esz) % 16 != 0 ||
        ((size_t)ld_d * esz) % 16 != 0 || (reinterpret_cast<uintptr_t>(weight) & 15) || (reinterpret_cast<uintptr_t>(workspace) & 15))
        return EL_ERR_ALIGNMENT;
    if (M == 0) {
        if (weight) EL_CUDA_TRY(cudaMemsetAsync(dweight, 0, (size_t)H * sizeof(float), st));
        return EL_OK;
    }
    double* partial = static_cast<double*>(workspace);
    switch (dt) {
        case EL_BF16:
            return launch_swiglu_backward_t((const __nv_bfloat16*)gy, (const __nv_bfloat16*)gate, (const __nv_bfloat16*)up, ld, weight,
                                            rstd, (__nv_bfloat16*)d_gate, (__nv_bfloat16*)d_up, ld_d, dweight, partial, M, H, st);
        case EL_F16:
            return launch_swiglu_backward_t((const __half*)gy, (const __half*)gate, (const __half*)up, ld, weight, rstd,
                                            (__half*)d_gate, (__half*)d_up, ld_d, dweight, partial, M, H, st);
        case EL_F32:
            return launch_swiglu_backward_t((const float*)gy, (const float*)gate, (const float*)up, ld, weight, rstd, (float*)d_gate,
                                            (float*)d_up, ld_d, dweight, partial, M, H, st);
        default: return EL_ERR_INVALID_ARG;
    }
}

}  // namespace el
