// Pre-linear RMSNorm fused with the per-token int8 quantiser, and its backward pass.
//
// The reference normalises the activations right before every INT2 linear call
// (core/bitnet/bitnet_int2_optimized.py:72-86, model/common/bitnet_legacy.py:10-25):
//     norm = x_f32 * rsqrt(mean(x_f32^2) + eps);  y = norm.type_as(x) * weight.type_as(x)
// and then quantises y per token.  Done as separate tensor operations this reads and writes the [M, K] activation
// about eight times; here one kernel reads the row and writes the int8 row, its absmax and its rstd.
//
// Row sums (of squares, and in the backward pass) are accumulated in float64, so that their float32 value does not
// depend on the order of the additions: the result is the one the CPU oracle defines, bit for bit.
#include "row_stream.cuh"

namespace el {

namespace {

using namespace rowio;

// One CTA per token, for rows beyond the streaming form's 16384 elements.  K % 8 == 0; x rows, weight and q rows 16-byte (q:
// 8-byte) aligned.  A thread keeps ROW_CACHE vectors of 8 elements, the row's first 12288, in registers between the passes;
// the rest of the row is read again by every pass.
constexpr int ROW_CACHE = 6;
template <typename T>
__global__ void __launch_bounds__(RN_THREADS, 3)
rmsnorm_quantize_rows_kernel(const T* __restrict__ x, long long ldx, const float* __restrict__ weight, int8_t* __restrict__ q,
                             float* __restrict__ row_absmax, float* __restrict__ rstd_out, int K, float norm_eps,
                             float quant_eps) {
    __shared__ double red_d[RN_THREADS / 32];
    __shared__ float red_f[RN_THREADS / 32];
    const int m = blockIdx.x;
    const T* xr = x + (size_t)m * ldx;
    int8_t* qr = q + (size_t)m * K;

    typename Io<T>::Raw cache[ROW_CACHE];
    const int k_tail = (threadIdx.x + ROW_CACHE * RN_THREADS) * 8;

    // ---- mean of squares -> rstd -------------------------------------------------------------------------------------
    double ss = 0.0;
#pragma unroll
    for (int c = 0; c < ROW_CACHE; ++c) {
        const int k = (threadIdx.x + c * RN_THREADS) * 8;
        if (k < K) {
            cache[c] = Io<T>::load_raw(xr + k);
            float v[8];
            Io<T>::unpack(cache[c], v);
#pragma unroll
            for (int i = 0; i < 8; ++i) ss += (double)__fmul_rn(v[i], v[i]);
        }
    }
    for (int k = k_tail; k < K; k += RN_THREADS * 8) {
        float v[8];
        Io<T>::load8(xr + k, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += (double)__fmul_rn(v[i], v[i]);
    }
    ss = block_sum(ss, red_d);
    const float ms = __fdiv_rn((float)ss, (float)K);
    const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(ms, norm_eps)));

    // y = io(io(x*r) * io(w))
    auto normed = [&](const float v[8], const float w[8], float y[8]) {
        float wr[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            y[i] = __fmul_rn(v[i], r);
            wr[i] = w[i];
        }
        Io<T>::round8(y);
        Io<T>::round8(wr);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = __fmul_rn(y[i], wr[i]);
        Io<T>::round8(y);
    };

    // ---- absmax of the normalised row ----------------------------------------------------------------------------------
    // fmaxf drops NaN and keeps infinities: the checked pass runs only for a row that needs it
    float amax = 0.0f;
#pragma unroll
    for (int c = 0; c < ROW_CACHE; ++c) {
        const int k = (threadIdx.x + c * RN_THREADS) * 8;
        if (k < K) {
            float v[8], w[8], y[8];
            Io<T>::unpack(cache[c], v);
            load8_w(weight + k, w);
            normed(v, w, y);
            cache[c] = Io<T>::pack(y);          // from here on the cache holds the normalised row (exact: y is of type T)
#pragma unroll
            for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(y[i]));
        }
    }
    for (int k = k_tail; k < K; k += RN_THREADS * 8) {
        float v[8], w[8], y[8];
        Io<T>::load8(xr + k, v);
        load8_w(weight + k, w);
        normed(v, w, y);
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(y[i]));
    }
    amax = block_max_f(amax, red_f);
    const bool row_finite = amax <= 3.402823466e38f;
    if (!row_finite) {
        amax = 0.0f;
        for (int k = threadIdx.x * 8; k < K; k += RN_THREADS * 8) {
            float v[8], w[8], y[8];
            Io<T>::load8(xr + k, v);
            load8_w(weight + k, w);
            normed(v, w, y);
#pragma unroll
            for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(finite_or_zero(y[i])));
        }
        amax = block_max_f(amax, red_f);
    }
    const float a = fmaxf(amax, quant_eps);
    const float s = __fdiv_rn(127.0f, a);
    if (threadIdx.x == 0) {
        row_absmax[m] = a;
        rstd_out[m] = r;
    }

    // ---- quantise --------------------------------------------------------------------------------------------------------
    auto quantise_y = [&](const float y[8], int k) {
        int qi[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) qi[i] = q8_sat(__fmul_rn(row_finite ? y[i] : finite_or_nan(y[i]), s));
        *reinterpret_cast<uint2*>(qr + k) = make_uint2(pack4_s8(qi[0], qi[1], qi[2], qi[3]), pack4_s8(qi[4], qi[5], qi[6], qi[7]));
    };
#pragma unroll
    for (int c = 0; c < ROW_CACHE; ++c) {
        const int k = (threadIdx.x + c * RN_THREADS) * 8;
        if (k < K) {
            float y[8];
            Io<T>::unpack(cache[c], y);
            quantise_y(y, k);
        }
    }
    for (int k = k_tail; k < K; k += RN_THREADS * 8) {
        float v[8], w[8], y[8];
        Io<T>::load8(xr + k, v);
        load8_w(weight + k, w);
        normed(v, w, y);
        quantise_y(y, k);
    }
}

// Streaming form: CTAs of one to sixteen warps walk over the tokens, two rows ahead in thread-owned slots (row_stream.cuh), the
// weight rounded once and kept in registers.  A thread owns 64 bytes of every row, so that the warp reductions and the scalar
// arithmetic of a row are spread over many elements, and several CTAs share an SM, so that one's barriers hide behind the
// others' work.  Products of two values of a 16-bit I/O type are taken packed (one rounding, the same result), and the
// quantiser rounds by adding 1.5*2^23 instead of converting.  What bounds it: about 20 instructions per element and one
// float64 conversion; memory 3 bytes per element (bf16).
// 4096 tokens x 11008, bf16: 76 us in the one-CTA-per-row form, 47 us in this one at 64 registers a thread; x 4096: 27 -> 20.5 us (events
// around the call, L2 flushed).  At 80 registers (in a CUDA graph): 44.2 -> 38.8 and 17.0 -> 15.8 us, 16384 x 2048 30.0 -> 27.2; 8192 x
// 16384, where an SM then holds one CTA instead of two, 104.6 -> 110.6.  (Tried: the next row's squares before this row's maximum, so that
// a row has one barrier: 41.0 us at 11008, the reads of the row from its slots cost more than the barrier.)
constexpr int FW_STAGES = 2;
template <typename T> constexpr int FW_VECS = 8 / (int)sizeof(T);        // vectors of 8 per thread: 4, float32: 2

template <typename T, int REGS>
__global__ void __maxnreg__(REGS)
rmsnorm_quantize_stream_kernel(const T* __restrict__ x, long long ldx, const float* __restrict__ weight, int8_t* __restrict__ q,
                               float* __restrict__ row_absmax, float* __restrict__ rstd_out, int M, int K, float norm_eps,
                               float quant_eps) {
    constexpr int V = FW_VECS<T>;
    constexpr uint32_t INF_BITS = sizeof(T) == 4 ? 0x7f800000u : (std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u);
    extern __shared__ uint4 ring[];
    __shared__ double red_d[2][MAX_RED];
    __shared__ uint32_t red_u[2][MAX_RED];
    __shared__ uint32_t red_f[2][MAX_RED];
    const Slots<T, FW_STAGES, V> slots(ring);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const f32x2 nz = negative_zeros();
    typename Io<T>::Raw w[V];
#pragma unroll
    for (int c = 0; c < V; ++c) {
        const int k = column_of<V>(c);
        float wv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (k < K) load8_w(weight + k, wv);
        w[c] = Io<T>::pack(wv);                      // rounds to the I/O type
    }
    auto fetch = [&](int stage, int m) {
        if (m < M) {
#pragma unroll
            for (int c = 0; c < V; ++c) {
                const int k = column_of<V>(c);
                if (k < K) slots.fetch(stage, c, x + (size_t)m * ldx + k);
            }
        }
        cp_async_commit();
    };
    const int G = gridDim.x;
#pragma unroll
    for (int s = 0; s < FW_STAGES; ++s) fetch(s, blockIdx.x + s * G);
    int stage = 0;
    for (int m = blockIdx.x; m < M; m += G, stage ^= 1) {
        static_assert(FW_STAGES == 2, "stage doubles as the parity of the reduction buffers");
        cp_async_wait<FW_STAGES - 1>();
        // ---- mean of squares -> rstd ---------------------------------------------------------------------------------
        typename Io<T>::Raw row[V];
        double ss = 0.0;
#pragma unroll
        for (int c = 0; c < V; ++c) {
            row[c] = column_of<V>(c) < K ? slots.read(stage, c) : raw_zero<T>();
            f32x2 v[4];
            unpack2<T>(row[c], v);
            ss += dot8(v, v);
        }
        ss = warp_sum(ss);
        if (lane == 0) red_d[stage][warp] = ss;
        fetch(stage, m + FW_STAGES * G);             // into the slots just read, by the thread that read them
        __syncthreads();
        ss = sum_red(red_d[stage]);
        const float ms = __fdiv_rn((float)ss, (float)K);
        const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(ms, norm_eps)));
        // ---- y = io(io(x*r) * io(w)) and its largest magnitude ------------------------------------------------------------
        uint32_t top = 0u;
        const f32x2 r2 = pair(r, r);
#pragma unroll
        for (int c = 0; c < V; ++c) {
            f32x2 v[4];
            unpack2<T>(row[c], v);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = mul2(v[i], r2);
            row[c] = mul_raw(pack2<T>(v), w[c]);
            if (column_of<V>(c) < K) top = max_bits(top, row[c]);
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
                if (column_of<V>(c) < K) {
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
            rstd_out[m] = r;
        }
        // ---- quantise ---------------------------------------------------------------------------------------------------------
        const bool fast = row_finite && s <= 3.402823466e38f;
#pragma unroll
        for (int c = 0; c < V; ++c) {
            const int k = column_of<V>(c);
            if (k < K) {
                *reinterpret_cast<uint2*>(q + (size_t)m * K + k) = fast ? quantise8<T, true>(row[c], s, nz) : quantise8<T, false>(row[c], s, nz);
            }
        }
    }
}

// Backward.  CTA b takes the tokens b, b + gridDim.x, ...; thread t owns the same columns in every token, so the
// per-column sums of dweight live in shared memory (one double per column) without any exchange between threads.
// At the end the CTA writes its [K] partial sums to `partial[b]`.
template <typename T>
__global__ void __launch_bounds__(RN_THREADS)
rmsnorm_backward_kernel(const T* __restrict__ g, const T* __restrict__ x, const float* __restrict__ weight,
                        const float* __restrict__ rstd, T* __restrict__ dx, double* __restrict__ partial, int M, int K) {
    extern __shared__ double col_sum[];          // [K]
    __shared__ double red_d[RN_THREADS / 32];
    for (int k = threadIdx.x * 8; k < K; k += RN_THREADS * 8) {
#pragma unroll
        for (int i = 0; i < 8; ++i) col_sum[k + i] = 0.0;
    }
    for (int m = blockIdx.x; m < M; m += gridDim.x) {
        const T* gr = g + (size_t)m * K;
        const T* xr = x + (size_t)m * K;
        T* dr = dx + (size_t)m * K;
        const float r = rstd[m];
        // c = sum_k io(g*io(w)) * x
        double c = 0.0;
        for (int k = threadIdx.x * 8; k < K; k += RN_THREADS * 8) {
            float gv[8], xv[8], w[8];
            Io<T>::load8(gr + k, gv);
            Io<T>::load8(xr + k, xv);
            load8_w(weight + k, w);
            Io<T>::round8(w);
#pragma unroll
            for (int i = 0; i < 8; ++i) gv[i] = __fmul_rn(gv[i], w[i]);
            Io<T>::round8(gv);
#pragma unroll
            for (int i = 0; i < 8; ++i) c += (double)__fmul_rn(gv[i], xv[i]);
        }
        c = block_sum(c, red_d);
        const float r3 = __fmul_rn(__fmul_rn(r, r), r);
        const float coef = __fdiv_rn(__fmul_rn(r3, (float)c), (float)K);
        for (int k = threadIdx.x * 8; k < K; k += RN_THREADS * 8) {
            float gv[8], xv[8], w[8], o[8], gn[8], xn[8];
            Io<T>::load8(gr + k, gv);
            Io<T>::load8(xr + k, xv);
            load8_w(weight + k, w);
            Io<T>::round8(w);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                gn[i] = __fmul_rn(gv[i], w[i]);
                xn[i] = __fmul_rn(xv[i], r);
            }
            Io<T>::round8(gn);
            Io<T>::round8(xn);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                o[i] = __fsub_rn(__fmul_rn(gn[i], r), __fmul_rn(xv[i], coef));
                col_sum[k + i] += (double)__fmul_rn(gv[i], xn[i]);
            }
            Io<T>::store8(dr + k, o);
        }
    }
    double* out = partial + (size_t)blockIdx.x * K;
    for (int k = threadIdx.x * 8; k < K; k += RN_THREADS * 8) {
#pragma unroll
        for (int i = 0; i < 8; ++i) out[k + i] = col_sum[k + i];
    }
}

// Streaming form of the same: one CTA walks over the tokens with three rows per thread-owned slot set (row_stream.cuh), the
// column sums stay in registers, and the row sum of the NEXT token is formed before the gradient of the current one, so that
// its exchange between the warps hides behind the gradient and a token costs one barrier.
// What bounds it: a token is about 30 instructions and two float64 conversions per element; memory 6 bytes per element (bf16).
// 4096 tokens x 11008, bf16: 230 us with one token at a time, column sums in shared memory at a 64-byte stride (four-way bank
// conflicts) and both passes reading the rows from L2/HBM; 77 us in this form; x 4096: 83 -> 40 us (events around the call, L2 flushed, the
// dweight kernel included).
// V: vectors of 8 columns per thread; THREADS: the largest CTA (sets the register budget).
constexpr int BW_STAGES = 3;
template <typename T, int V, int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
rmsnorm_backward_stream_kernel(const T* __restrict__ g, const T* __restrict__ x, const float* __restrict__ weight,
                               const float* __restrict__ rstd, T* __restrict__ dx, double* __restrict__ partial, int M, int K) {
    extern __shared__ uint4 ring[];
    __shared__ double red[2][MAX_RED];
    const Slots<T, BW_STAGES, 2 * V> slots(ring);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const f32x2 nz = negative_zeros();
    typename Io<T>::Raw w[V];
    double col[V][8];
#pragma unroll
    for (int c = 0; c < V; ++c) {
        const int k = column_of<V>(c);
        float wv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (k < K) load8_w(weight + k, wv);
        w[c] = Io<T>::pack(wv);                      // rounds to the I/O type
#pragma unroll
        for (int i = 0; i < 8; ++i) col[c][i] = 0.0;
    }
    auto fetch = [&](int stage, int m) {
        if (m < M) {
#pragma unroll
            for (int c = 0; c < V; ++c) {
                const int k = column_of<V>(c);
                if (k < K) {
                    slots.fetch(stage, 2 * c, g + (size_t)m * K + k);
                    slots.fetch(stage, 2 * c + 1, x + (size_t)m * K + k);
                }
            }
        }
        cp_async_commit();
    };
    // this thread's share of c = sum_k io(g*io(w)) * x
    auto row_dot = [&](int stage) -> double {
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < V; ++c) {
            if (column_of<V>(c) < K) {
                f32x2 gn[4], xv[4];
                unpack2<T>(mul_raw(slots.read(stage, 2 * c), w[c]), gn);
                unpack2<T>(slots.read(stage, 2 * c + 1), xv);
                s += dot8(gn, xv);
            }
        }
        return s;
    };
    const int G = gridDim.x;
    int m = blockIdx.x, stage = 0;
#pragma unroll
    for (int s = 0; s < BW_STAGES; ++s) fetch(s, m + s * G);
    cp_async_wait<BW_STAGES - 1>();
    double csum = warp_sum(row_dot(0));
    if (lane == 0) red[0][warp] = csum;
    __syncthreads();
    csum = sum_red(red[0]);
    int par = 1;
    float r = m < M ? rstd[m] : 0.0f;
    for (; m < M; m += G, par ^= 1) {
        const int next = stage + 1 == BW_STAGES ? 0 : stage + 1;
        cp_async_wait<BW_STAGES - 2>();
        if (m + G < M) {
            const double s = warp_sum(row_dot(next));
            if (lane == 0) red[par][warp] = s;
        }
        const float r_next = m + G < M ? __ldg(rstd + m + G) : 0.0f;
        const float r3 = __fmul_rn(__fmul_rn(r, r), r);
        const float coef = __fdiv_rn(__fmul_rn(r3, (float)csum), (float)K);
        const f32x2 r2 = pair(r, r), coef2 = pair(coef, coef);
#pragma unroll
        for (int c = 0; c < V; ++c) {
            const int k = column_of<V>(c);
            if (k < K) {
                const typename Io<T>::Raw graw = slots.read(stage, 2 * c);
                f32x2 v[4], xv[4], o[4];
                unpack2<T>(mul_raw(graw, w[c]), v);                              // gn = io(g*io(w))
                unpack2<T>(slots.read(stage, 2 * c + 1), xv);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    o[i] = sub2(mul2_exact(v[i], r2, nz), mul2_exact(xv[i], coef2, nz));
                    xv[i] = mul2(xv[i], r2);
                }
                *reinterpret_cast<typename Io<T>::Raw*>(dx + (size_t)m * K + k) = pack2<T>(o);
                unpack2<T>(graw, v);
                unpack2<T>(pack2<T>(xv), xv);                                    // io(x*r)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const f32x2 t = mul2(v[i], xv[i]);
                    col[c][2 * i] += (double)lo_of(t);
                    col[c][2 * i + 1] += (double)hi_of(t);
                }
            }
        }
        fetch(stage, m + BW_STAGES * G);             // into the slots just read, by the thread that read them
        __syncthreads();
        csum = sum_red(red[par]);
        stage = next;
        r = r_next;
    }
    double* out = partial + (size_t)blockIdx.x * K;
#pragma unroll
    for (int c = 0; c < V; ++c) {
        const int k = column_of<V>(c);
        if (k < K) {
#pragma unroll
            for (int i = 0; i < 8; i += 2) *reinterpret_cast<double2*>(out + k + i) = make_double2(col[c][i], col[c][i + 1]);
        }
    }
}

int backward_grid(int M, int K) {
    int sms = 148;
    device_sm_count(&sms);
    const size_t smem = (size_t)K * sizeof(double);
    int per_sm = (int)((200u * 1024u) / (smem ? smem : 1));
    if (per_sm < 1) per_sm = 1;
    if (per_sm > 4) per_sm = 4;
    const int grid = sms * per_sm;
    return M < grid ? (M < 1 ? 1 : M) : grid;
}

}  // namespace

// Largest number of CTAs the backward kernel may use (sizes the workspace independently of M).
size_t rmsnorm_backward_workspace_bytes(int K) {
    if (K <= 0) return 0;
    int sms = 148;
    device_sm_count(&sms);
    return (size_t)sms * 4 * (size_t)K * sizeof(double);
}

template <typename T, int REGS>
static int launch_quantize_stream(const T* x, long long ldx, const float* weight, float norm_eps, int8_t* q, float* row_absmax, float* rstd,
                                  int M, int K, float quant_eps, int threads, cudaStream_t st) {
    static DeviceOnce attr_once;
    int dev = 0, sms = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    const int rc = device_sm_count(&sms);
    if (rc != EL_OK) return rc;
    if (!attr_once.is_done(dev)) {
        EL_CUDA_TRY(cudaFuncSetAttribute(rmsnorm_quantize_stream_kernel<T, REGS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr_once.mark(dev);
    }
    const size_t smem = (size_t)FW_STAGES * 64 * threads;
    int per_sm = resident_threads(REGS) / threads;
    const int by_smem = (int)((200u * 1024u) / (smem + 1024));
    per_sm = per_sm < by_smem ? per_sm : by_smem;
    per_sm = per_sm < 1 ? 1 : (per_sm > 32 ? 32 : per_sm);
    const int grid = M < sms * per_sm ? M : sms * per_sm;
    rmsnorm_quantize_stream_kernel<T, REGS><<<grid, threads, smem, st>>>(x, ldx, weight, q, row_absmax, rstd, M, K, norm_eps, quant_eps);
    return check_launch();
}

// Rows of up to 16384 elements stream (64 bytes of a row per thread, sixteen warps: 32 for float32); longer ones take the
// one-CTA-per-row kernel.
template <typename T>
static int launch_quantize_t(const T* x, long long ldx, const float* weight, float norm_eps, int8_t* q, float* row_absmax, float* rstd,
                             int M, int K, float quant_eps, cudaStream_t st) {
    if (K > 16384) {
        rmsnorm_quantize_rows_kernel<T><<<M, RN_THREADS, 0, st>>>(x, ldx, weight, q, row_absmax, rstd, K, norm_eps, quant_eps);
        return check_launch();
    }
    const int threads = stream_threads(K, FW_VECS<T>);
    // 80 registers per thread, or 64 where an SM would hold one CTA of 80 but two of 64
    const int wide = resident_threads(80) / threads, narrow = resident_threads(64) / threads;
    if (wide == 0 || (wide == 1 && narrow == 2))
        return launch_quantize_stream<T, 64>(x, ldx, weight, norm_eps, q, row_absmax, rstd, M, K, quant_eps, threads, st);
    return launch_quantize_stream<T, 80>(x, ldx, weight, norm_eps, q, row_absmax, rstd, M, K, quant_eps, threads, st);
}

int launch_rmsnorm_quantize_rows(const void* x, int dt, long long ldx, const float* weight, float norm_eps, int8_t* q,
                                 float* row_absmax, float* rstd, int M, int K, float quant_eps, cudaStream_t st) {
    if (M == 0) return EL_OK;
    if (K <= 0 || K % 8 != 0) return EL_ERR_UNSUPPORTED_SHAPE;
    const size_t esz = (dt == EL_F32) ? 4 : 2;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || ((size_t)ldx * esz) % 16 != 0 || (reinterpret_cast<uintptr_t>(weight) & 15) ||
        (reinterpret_cast<uintptr_t>(q) & 7))
        return EL_ERR_ALIGNMENT;
    switch (dt) {
        case EL_BF16: return launch_quantize_t((const __nv_bfloat16*)x, ldx, weight, norm_eps, q, row_absmax, rstd, M, K, quant_eps, st);
        case EL_F16: return launch_quantize_t((const __half*)x, ldx, weight, norm_eps, q, row_absmax, rstd, M, K, quant_eps, st);
        case EL_F32: return launch_quantize_t((const float*)x, ldx, weight, norm_eps, q, row_absmax, rstd, M, K, quant_eps, st);
        default: return EL_ERR_INVALID_ARG;
    }
}

// three stages of a row of g and a row of x, beside the reduction buffers
constexpr size_t BW_MAX_ROW_BYTES = 32 * 1024;

template <typename T, int V, int THREADS>
static int launch_backward_stream(const T* g, const T* x, const float* weight, const float* rstd, T* dx, double* partial, int M, int K,
                                  int* grid, cudaStream_t st) {
    static DeviceOnce attr_once;
    int dev = 0, sms = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    int rc = device_sm_count(&sms);
    if (rc != EL_OK) return rc;
    if (!attr_once.is_done(dev)) {
        EL_CUDA_TRY(cudaFuncSetAttribute(rmsnorm_backward_stream_kernel<T, V, THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         220 * 1024));
        attr_once.mark(dev);
    }
    const int threads = stream_threads(K, V);
    const size_t smem = (size_t)BW_STAGES * 2 * V * PIECES<T> * sizeof(uint4) * threads;
    // resident CTAs per SM by registers and shared memory, at most the four per SM that the workspace holds partials for
    int per_sm = THREADS / threads;
    const int by_smem = (int)((220u * 1024u) / smem);
    per_sm = per_sm < by_smem ? per_sm : by_smem;
    per_sm = per_sm < 1 ? 1 : (per_sm > 4 ? 4 : per_sm);
    *grid = M < sms * per_sm ? M : sms * per_sm;
    rmsnorm_backward_stream_kernel<T, V, THREADS><<<*grid, threads, smem, st>>>(g, x, weight, rstd, dx, partial, M, K);
    return check_launch();
}

template <typename T>
static int launch_rmsnorm_backward_t(const T* g, const T* x, const float* weight, const float* rstd, T* dx, float* dweight,
                                     double* partial, int M, int K, cudaStream_t st) {
    int grid = backward_grid(M, K);
    int rc = EL_OK;
    // Rows whose three stages fit in shared memory stream; the column sums decide the form: two vectors per thread while
    // the registers of one SM hold them at 768 threads, four at up to 512 threads beyond.  (float32: half the columns.)
    constexpr int MAX_V2 = sizeof(T) == 2 ? 768 : 512;
    if ((size_t)K * sizeof(T) <= BW_MAX_ROW_BYTES) {
        if (stream_threads(K, 2) <= MAX_V2) rc = launch_backward_stream<T, 2, MAX_V2>(g, x, weight, rstd, dx, partial, M, K, &grid, st);
        else if constexpr (sizeof(T) == 2) rc = launch_backward_stream<T, 4, 512>(g, x, weight, rstd, dx, partial, M, K, &grid, st);
        if (rc != EL_OK) return rc;
        return launch_dweight(partial, grid, dweight, K, st);
    }
    const size_t smem = (size_t)K * sizeof(double);
    static DeviceOnce attr_once;
    int dev = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    if (!attr_once.is_done(dev)) {
        EL_CUDA_TRY(cudaFuncSetAttribute(rmsnorm_backward_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr_once.mark(dev);
    }
    rmsnorm_backward_kernel<T><<<grid, RN_THREADS, smem, st>>>(g, x, weight, rstd, dx, partial, M, K);
    rc = check_launch();
    if (rc != EL_OK) return rc;
    return launch_dweight(partial, grid, dweight, K, st);
}

int launch_rmsnorm_backward(const void* g, const void* x, int dt, const float* weight, const float* rstd, void* dx,
                            float* dweight, void* workspace, size_t workspace_bytes, int M, int K, cudaStream_t st) {
    if (K <= 0 || K % 8 != 0 || (size_t)K * sizeof(double) > 200u * 1024u) return EL_ERR_UNSUPPORTED_SHAPE;
    if (workspace_bytes < rmsnorm_backward_workspace_bytes(K)) return EL_ERR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(g) & 15) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(dx) & 15) ||
        (reinterpret_cast<uintptr_t>(weight) & 15) || (reinterpret_cast<uintptr_t>(workspace) & 15))
        return EL_ERR_ALIGNMENT;
    if (M == 0) {
        EL_CUDA_TRY(cudaMemsetAsync(dweight, 0, (size_t)K * sizeof(float), st));
        return EL_OK;
    }
    double* partial = static_cast<double*>(workspace);
    switch (dt) {
        case EL_BF16:
            return launch_rmsnorm_backward_t((const __nv_bfloat16*)g, (const __nv_bfloat16*)x, weight, rstd, (__nv_bfloat16*)dx,
                                             dweight, partial, M, K, st);
        case EL_F16:
            return launch_rmsnorm_backward_t((const __half*)g, (const __half*)x, weight, rstd, (__half*)dx, dweight, partial, M, K, st);
        case EL_F32:
            return launch_rmsnorm_backward_t((const float*)g, (const float*)x, weight, rstd, (float*)dx, dweight, partial, M, K, st);
        default: return EL_ERR_INVALID_ARG;
    }
}

}  // namespace el
