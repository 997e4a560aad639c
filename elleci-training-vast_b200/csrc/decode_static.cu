// The decode call on a static device array.
#include <cuda_runtime.h>

#include "common.cuh"
#include "epilogue.cuh"

namespace el {

// ---- decode call that allocates nothing ------------------------------------------------------------------------------
//
// Some hosts of this library cannot hand it device memory: an inference server whose plug-ins are forbidden to call
// cudaMalloc once serving has started, a runtime that owns the whole memory pool, a process already at its memory
// budget.  el_linear_decode needs scratch buffers from its caller; this variant keeps what it uses of them in one array that
// is part of the loaded library image, so the caller passes only the input, the weights and the output.

constexpr int STATIC_MAX_TOKENS = 64;
constexpr int STATIC_MAX_N = 16384;       // largest out_features
constexpr int STATIC_MAX_K = 16384;       // largest in_features
constexpr size_t STATIC_ABSMAX_OFFSET = (size_t)STATIC_MAX_TOKENS * STATIC_MAX_K;       // behind the quantised tokens
constexpr size_t STATIC_TOTAL_BYTES = STATIC_ABSMAX_OFFSET + 256;          // one megabyte per device

// Lives in every GPU that loads the library, until the process exits.  In host code this name is only a handle for
// cudaGetSymbolAddress; it is not a device address and must never be passed to a kernel as one.
static __device__ __align__(256) unsigned char g_decode_scratch[STATIC_TOTAL_BYTES];

static std::atomic<void*> g_decode_scratch_ptr[64];    // device address of the array, per device ordinal (filled at set-up)

// Set-up for the current device: resolves the array's device address once.  Not an allocation.  Host threads that
// race through the first call each resolve the same address and store the same value.
static int decode_static_setup(unsigned char** out) {
    int dev = 0;
    EL_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return EL_ERR_DEVICE;
    void* ptr = g_decode_scratch_ptr[dev].load(std::memory_order_acquire);
    if (ptr == nullptr) {
        EL_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_decode_scratch));
        if (ptr == nullptr) return EL_ERR_DEVICE;
        g_decode_scratch_ptr[dev].store(ptr, std::memory_order_release);
    }
    *out = static_cast<unsigned char*>(ptr);
    return EL_OK;
}

int launch_quantize_rows_perm(const void* x, int dt, long long ldx, int8_t* q, float* a, int M, int K, float eps,
                              cudaStream_t st);
int launch_gemv_small(const void* x, int x_dtype, const uint8_t* Wp, const EpiParams& epi, int M, int N, int K, cudaStream_t st, bool overlap);
int launch_gemv_mma(const void* x, int x_dtype, const uint8_t* Wp, const EpiParams& epi, int M, int N, int K, cudaStream_t st,
                    bool overlap);
bool gemv_mma_fits(int M, int K);
int launch_decode_preq(const int8_t* xq, const float* absmax, const uint8_t* Wp, const EpiParams& epi, int M, int N, int K, int32_t* status,
                       cudaStream_t st);
bool decode_overlap();
int decode_gemv_max_tokens();
int decode_mma_max_tokens();

}  // namespace el

extern "C" EL_API int el_linear_decode_static(const void* x, int x_dtype, const uint8_t* W_packed, void* Y, int out_dtype,
                                              float gamma, int M, int N, int K, int32_t* dev_status, el_stream_t stream) {
    using namespace el;
    auto is_float = [](int dt) { return dt == EL_F16 || dt == EL_BF16 || dt == EL_F32; };
    if (M < 0 || N < 0 || K < 0 || !is_float(x_dtype) || !is_float(out_dtype)) return EL_ERR_INVALID_ARG;
    if (M > STATIC_MAX_TOKENS || N > STATIC_MAX_N || K > STATIC_MAX_K) return EL_ERR_TOO_LARGE;
    if (M == 0 || N == 0) return EL_OK;
    if (K == 0 || K % 64 != 0) return EL_ERR_UNSUPPORTED_SHAPE;
    if (!x || !W_packed || !Y) return EL_ERR_NULL_PTR;
    cudaStream_t st = (cudaStream_t)stream;
    // Set-up comes first, whichever kernel this call ends up on: the first call on a device resolves the array's
    // address even when it is a one-token warm-up, so no later call has to do it (inside a stream capture, say).
    unsigned char* base = nullptr;
    int rc = decode_static_setup(&base);
    if (rc != EL_OK) return rc;
    if (M <= decode_gemv_max_tokens()) {      // the few-token kernel needs no scratch at all
        const EpiParams gepi{Y, (long long)N, out_dtype, nullptr, 0, gamma};
        return launch_gemv_small(x, x_dtype, W_packed, gepi, M, N, K, st, decode_overlap());
    }
    if (M <= DECODE_MMA_SINGLE_MAX && M <= decode_mma_max_tokens() && gemv_mma_fits(M, K)) {      // neither does the warp-MMA kernel
        const EpiParams gepi{Y, (long long)N, out_dtype, nullptr, 0, gamma};
        return launch_gemv_mma(x, x_dtype, W_packed, gepi, M, N, K, st, decode_overlap());
    }
    int8_t* xq = reinterpret_cast<int8_t*>(base);
    float* absmax = reinterpret_cast<float*>(base + STATIC_ABSMAX_OFFSET);
    rc = launch_quantize_rows_perm(x, x_dtype, K, xq, absmax, M, K, 1e-5f, st);
    if (rc != EL_OK) return rc;
    const EpiParams epi{Y, (long long)N, out_dtype, nullptr, 0, gamma};
    return launch_decode_preq(xq, absmax, W_packed, epi, M, N, K, dev_status, st);
}
