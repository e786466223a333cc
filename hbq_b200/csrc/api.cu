// C ABI of the library (declared in include/hbq_b200.h).
#include "common.cuh"
#include <atomic>
#include <mutex>
#include <cstring>
#include <cstdio>

namespace hbq {

static std::atomic<long long> g_launches{0};
static thread_local char g_last_cuda_error[256] = "";

void note_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

int set_cuda_error(cudaError_t e, const char* where)
{
    snprintf(g_last_cuda_error, sizeof(g_last_cuda_error), "%s: %s", where, cudaGetErrorString(e));
    return HBQ_ERR_CUDA;
}

// (kernel, device) -> largest dynamic shared-memory size already granted
struct SmemGrant { const void* kernel; int dev; size_t bytes; };
static SmemGrant g_grants[256];
static int g_ngrants = 0;
static std::mutex g_grant_mutex;

int ensure_dynamic_smem_impl(const void* kernel, size_t bytes)
{
    int dev = 0;
    HBQ_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_grant_mutex);
    SmemGrant* slot = nullptr;
    for (int i = 0; i < g_ngrants; ++i)
        if (g_grants[i].kernel == kernel && g_grants[i].dev == dev) { slot = &g_grants[i]; break; }
    if (slot && slot->bytes >= bytes) return HBQ_OK;
    HBQ_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    if (!slot && g_ngrants < 256) slot = &g_grants[g_ngrants++];
    if (slot) *slot = {kernel, dev, bytes};
    return HBQ_OK;
}

// (kernel, device, threads, smem) -> resident CTAs per SM
struct Occupancy { const void* kernel; int dev, threads; size_t smem; int ctas; };
static Occupancy g_occ[256];
static int g_nocc = 0;

int resident_ctas_impl(const void* kernel, int threads, size_t smem, int* ctas)
{
    int dev = 0;
    HBQ_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_grant_mutex);
    for (int i = 0; i < g_nocc; ++i)
        if (g_occ[i].kernel == kernel && g_occ[i].dev == dev && g_occ[i].threads == threads && g_occ[i].smem == smem) {
            *ctas = g_occ[i].ctas;
            return HBQ_OK;
        }
    int n = 0;
    HBQ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem));
    if (n < 1) n = 1;
    if (g_nocc < 256) g_occ[g_nocc++] = {kernel, dev, threads, smem, n};
    *ctas = n;
    return HBQ_OK;
}

// implemented in quantize.cu / gemm_simt.cu / gemm_tc.cu
int quantize_launch(const void*, int, int64_t, int64_t, const hbq_format*, void*, int, const hbq_packed_out*,
                    const float*, cudaStream_t, const KvWriteOpts*);
int dequantize_launch(const hbq_packed_out*, int64_t, int64_t, const hbq_format*, void*, int, cudaStream_t);   // dequantize.cu
int rmsnorm_quantize_launch(const void*, const void*, const void*, float, int64_t, int64_t, const hbq_format*, void*, void*,
                            cudaStream_t);
int softmax_quantize_launch(const void*, int64_t, int64_t, int64_t, int64_t, float, int, const void*, int64_t,
                            const hbq_format*, void*, cudaStream_t);
int fp_quant_launch(const void*, int64_t, int, int, int, int, int, void*, cudaStream_t);
int64_t absmax_scratch_bytes();
int absmax_launch(const void*, int, int64_t, float*, void*, cudaStream_t);
int gemm_simt_launch(const void*, const void*, void*, int64_t, int64_t, int64_t, int, int, int, int,
                     const void*, cudaStream_t);
bool gemm_tc_eligible(int64_t, int64_t, int64_t, int, int, int);
int gemm_tc_launch(const void*, const void*, void*, int64_t, int64_t, int64_t, int, int, int, const void*,
                   cudaStream_t);
int gemm_tc_launch_ex(const void*, const void*, void*, int64_t, int64_t, int64_t, int, int, int, const void*,
                      cudaStream_t, uint32_t, int);
int transpose_launch(const void*, void*, int64_t, int64_t, cudaStream_t);
int gemm_tc_status(int*);
int gemm_tc_status_reset();
int gemm_tc_reserve_sms(int n);
int gemm_tc_usable_sms(int*);
int gemm_tc_tile_width(int64_t, int64_t, int, int);
int gemm_tc_grouped_launch(const void*, int64_t, const int*, int, const void* const*, void* const*, const int*, int64_t, int64_t, int,
                           int, int, cudaStream_t);
int moe_route_launch(const int64_t*, int64_t, int, int, int*, int64_t*, int*, cudaStream_t);                      // moe.cu
int moe_combine_launch(const void*, const void*, const int*, int64_t, int, int64_t, void*, cudaStream_t);
int rope_heads_launch(const void*, int64_t, int64_t, int64_t, int64_t, const void*, const void*, int64_t, void*, cudaStream_t);   // rope.cu
int64_t gemm_w4_prepacked_bytes(int64_t, int64_t, int);
int gemm_w4_prepack(const hbq_packed_out*, int64_t, int64_t, const hbq_format*, int, void*, cudaStream_t);
int64_t gemm_w4_workspace_bytes(int64_t, int64_t, int64_t);
int gemm_w4_launch(const void*, const void*, void*, int64_t, int64_t, int64_t, const hbq_format*, int, const void*, void*,
                   cudaStream_t, uint32_t);
bool gemm_w16_eligible(int64_t, int64_t, int64_t);
int gemm_w16_launch(const void*, const void*, void*, int64_t, int64_t, int64_t, const void*, void*, cudaStream_t);

}  // namespace hbq

using namespace hbq;

extern "C" {

int hbq_quantize(const void* x, int dtype, int64_t rows, int64_t K, const hbq_format* fmt, void* deq,
                 int deq_dtype, const hbq_packed_out* out, const float* tensor_amax, void* stream)
{
    return quantize_launch(x, dtype, rows, K, fmt, deq, deq_dtype, out, tensor_amax, (cudaStream_t)stream, nullptr);
}

int hbq_kv_write_k(const void* k, int dtype, int64_t B, int64_t T, int64_t H, int64_t D, const void* cos,
                   const void* sin, int64_t rope_rows, const void* center, const hbq_format* fmt, void* out,
                   int out_dtype, void* stream)
{
    if (!fmt || B < 0 || T < 0 || H < 0 || D <= 0 || (cos != nullptr) != (sin != nullptr)) return HBQ_ERR_ARG;
    if (B * T * H == 0) return HBQ_OK;
    if (!out) return HBQ_ERR_ARG;
    if (fmt->kind == HBQ_KIND_MXFP && fmt->per_tensor_scale) return HBQ_ERR_UNSUPPORTED;   // needs max|x| of the rotated tensor first
    KvWriteOpts kv = {cos, sin, rope_rows, B, T, H, D, 0, center, 0, nullptr};
    return quantize_launch(k, dtype, B * T * H, D, fmt, out, out_dtype, nullptr, nullptr, (cudaStream_t)stream, &kv);
}

int hbq_rope_heads(const void* x, int64_t B, int64_t T, int64_t H, int64_t D, const void* cos, const void* sin, int64_t rope_rows,
                   void* out, void* stream)
{
    return rope_heads_launch(x, B, T, H, D, cos, sin, rope_rows, out, (cudaStream_t)stream);
}

int hbq_quantize_q_runs(const void* q, int64_t B, int64_t T, int64_t H, int64_t D, int64_t run, int64_t group, const void* cos,
                        const void* sin, int64_t rope_rows, const hbq_format* fmt, void* out, void* stream)
{
    if (!fmt || B < 0 || T < 0 || H <= 0 || D <= 0 || run <= 0 || group <= 0 || T % run || H % group || !cos || !sin) return HBQ_ERR_ARG;
    if (B * T == 0) return HBQ_OK;
    if (!out) return HBQ_ERR_ARG;
    if (fmt->kind == HBQ_KIND_MXFP && fmt->per_tensor_scale) return HBQ_ERR_UNSUPPORTED;
    KvWriteOpts kv = {cos, sin, rope_rows, B, T, H, D, 0, nullptr, 0, nullptr};
    kv.run = run; kv.group = group;
    return quantize_launch(q, HBQ_DTYPE_F16, B * T * H, D, fmt, out, HBQ_DTYPE_F16, nullptr, nullptr, (cudaStream_t)stream, &kv);
}

int hbq_quantize_head_rows(const void* x, int64_t B, int64_t H, int64_t run, int64_t D, int64_t T0, int64_t T,
                           const hbq_format* fmt, void* out, void* stream)
{
    if (!fmt || B < 0 || H <= 0 || run < 0 || D <= 0 || T0 < 0 || T0 + run > T || T > 0x7FFFFFFF) return HBQ_ERR_ARG;
    if (B * run == 0) return HBQ_OK;
    if (!out) return HBQ_ERR_ARG;
    if (fmt->kind == HBQ_KIND_MXFP && fmt->per_tensor_scale) return HBQ_ERR_UNSUPPORTED;
    KvWriteOpts kv = {nullptr, nullptr, 0, B, run, H, D, 0, nullptr, 0, nullptr};
    kv.from_runs = 1; kv.T0 = T0; kv.Tall = T;
    return quantize_launch(x, HBQ_DTYPE_F16, B * H * run, D, fmt, out, HBQ_DTYPE_F16, nullptr, nullptr, (cudaStream_t)stream, &kv);
}

int hbq_kv_write_v(const void* v, int dtype, int64_t B, int64_t T, int64_t H, int64_t D, const hbq_format* fmt,
                   void* out, int out_dtype, int out_token_major, void* stream)
{
    if (!fmt || B < 0 || T < 0 || H < 0 || D <= 0) return HBQ_ERR_ARG;
    if (B * T * H == 0) return HBQ_OK;
    if (!out) return HBQ_ERR_ARG;
    KvWriteOpts kv = {nullptr, nullptr, 0, B, T, H, D, 1, nullptr, out_token_major, nullptr};
    // rows / K only size the format checks here; the token-axis kernel takes its shape from kv
    return quantize_launch(v, dtype, B * H * D, fmt->block_size, fmt, out, out_dtype, nullptr, nullptr,
                           (cudaStream_t)stream, &kv);
}

int hbq_swiglu_quantize(const void* gate, const void* up, int64_t rows, int64_t K, const hbq_format* fmt, void* out,
                        void* stream)
{
    if (!fmt || rows < 0 || K <= 0) return HBQ_ERR_ARG;
    if (rows == 0) return HBQ_OK;
    if (!gate || !up || !out) return HBQ_ERR_ARG;
    KvWriteOpts o = {nullptr, nullptr, 0, 0, 0, 0, 0, 0, nullptr, 0, gate};
    return quantize_launch(up, HBQ_DTYPE_F16, rows, K, fmt, out, HBQ_DTYPE_F16, nullptr, nullptr, (cudaStream_t)stream, &o);
}

int hbq_rmsnorm_quantize(const void* x, const void* residual, const void* weight, float eps, int64_t rows, int64_t K,
                         const hbq_format* fmt, void* x_out, void* out, void* stream)
{
    return rmsnorm_quantize_launch(x, residual, weight, eps, rows, K, fmt, x_out, out, (cudaStream_t)stream);
}

int hbq_softmax_quantize(const void* scores, int64_t rows, int64_t S, int64_t L, int64_t heads, float scale, int causal,
                         const void* mask, int64_t mask_batches, const hbq_format* fmt, void* out, void* stream)
{
    return softmax_quantize_launch(scores, rows, S, L, heads, scale, causal, mask, mask_batches, fmt, out, (cudaStream_t)stream);
}

int hbq_absmax(const void* x, int dtype, int64_t n, float* amax, void* scratch, void* stream)
{
    return absmax_launch(x, dtype, n, amax, scratch, (cudaStream_t)stream);
}
int64_t hbq_absmax_scratch_bytes(void) { return absmax_scratch_bytes(); }

int hbq_dequantize(const hbq_packed_out* in, int64_t rows, int64_t K, const hbq_format* fmt, void* deq,
                   int dtype, void* stream)
{
    return dequantize_launch(in, rows, K, fmt, deq, dtype, (cudaStream_t)stream);
}

int hbq_fp_quant(const void* x, int64_t n, int ebit, int mbit, int allow_subnormal, int use_ceil,
                 int elem_variant, void* out, void* stream)
{
    return fp_quant_launch(x, n, ebit, mbit, allow_subnormal, use_ceil, elem_variant, out, (cudaStream_t)stream);
}

constexpr int64_t kMaxGemmDim = 0x7FFFFFFF;

static int check_gemm_args(const void* A, const void* B, void* C, int64_t M, int64_t N, int64_t K, int mode,
                           int group_k, int group_n)
{
    if (!A || !B || !C || M < 0 || N < 0 || K < 0) return HBQ_ERR_ARG;
    // every kernel indexes with 32-bit dimensions; this also keeps M*N, N*K and their byte counts inside int64
    if (M > kMaxGemmDim || N > kMaxGemmDim || K > kMaxGemmDim) return HBQ_ERR_UNSUPPORTED;
    if (mode < HBQ_ACC_FP32 || mode > HBQ_ACC_PSUM_E3M4) return HBQ_ERR_ARG;
    if (mode >= HBQ_ACC_GROUPED && group_k <= 0) return HBQ_ERR_ARG;
    if (mode >= HBQ_ACC_PSUM_INT8 && (group_n <= 0 || 64 % group_n != 0)) return HBQ_ERR_ARG;
    return HBQ_OK;
}

int hbq_gemm_uses_tensor_cores(int64_t M, int64_t N, int64_t K, int b_is_nk, int mode, int group_k, int group_n)
{
    (void)b_is_nk;
    return gemm_tc_eligible(M, N, K, mode, group_k, group_n) ? 1 : 0;
}

// Decode-sized fp32-accumulation products whose 128-column tiles would not fill the SMs run the pipeline of
// gemm_packed.cu with fp16 weight tiles (a tile's K split over a thread-block cluster, or equal runs of K blocks per
// SM) when the caller hands over its workspace; without one they take the tile-per-CTA kernel.
// Measured on B200 (16 tokens): [4096, 14336] 28 us against 63 us, [4096, 4096] 15 against 23, [12288, 4096] 25 against
// 32, one token x [14336, 4096] 27 against 39; beyond 128 MB of weight ([14336, 8192]: 51 against 47 us) or 32 tokens
// the tile-per-CTA kernel is the faster one.
static bool decode_stream_k(int64_t M, int64_t N, int64_t K, int mode)
{
    int sms = 0;
    return mode == HBQ_ACC_FP32 && M <= 32 && gemm_w16_eligible(M, N, K) && device_sms(&sms) == HBQ_OK &&
           ((N / 128) * 2 <= sms || (N / 128 <= sms && N * K * 2 <= (128ll << 20)));
}

int64_t hbq_gemm_workspace_bytes(int64_t M, int64_t N, int64_t K, int b_is_nk, int mode, int group_k, int group_n)
{
    if (!gemm_tc_eligible(M, N, K, mode, group_k, group_n)) return 0;
    const int64_t sk = decode_stream_k(M, N, K, mode) ? gemm_w4_workspace_bytes(M, N, K) : 0;
    const int64_t tr = b_is_nk ? 0 : N * K * 2;      // eligible operands have N, K <= 2^30: the product fits
    return (tr + 15) / 16 * 16 + (sk > 0 ? sk : 0);
}

int hbq_gemm(const void* A, const void* B, void* C, int64_t M, int64_t N, int64_t K, int b_is_nk, int mode,
             int group_k, int group_n, const void* bias, void* workspace, int64_t workspace_bytes, void* stream)
{
    int rc = check_gemm_args(A, B, C, M, N, K, mode, group_k, group_n);
    if (rc) return rc;
    if (M == 0 || N == 0) return HBQ_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const bool aligned = (((uintptr_t)A | (uintptr_t)B | (uintptr_t)C | (uintptr_t)bias) & 15) == 0;
    if (K > 0 && aligned && gemm_tc_eligible(M, N, K, mode, group_k, group_n)) {
        const void* W = B;
        int64_t used = 0;
        if (!b_is_nk) {
            if (!workspace || workspace_bytes < N * K * 2 || ((uintptr_t)workspace & 15)) return HBQ_ERR_WORKSPACE;
            rc = transpose_launch(B, workspace, K, N, st);
            if (rc) return rc;
            W = workspace;
            used = (N * K * 2 + 15) / 16 * 16;
        }
        if (decode_stream_k(M, N, K, mode) && workspace && !((uintptr_t)workspace & 15)) {
            const int64_t sk = gemm_w4_workspace_bytes(M, N, K);
            if (sk > 0 && workspace_bytes >= used + sk)
                return gemm_w16_launch(A, W, C, M, N, K, bias, (uint8_t*)workspace + used, st);
        }
        return gemm_tc_launch(A, W, C, M, N, K, mode, group_k, group_n, bias, st);
    }
    return gemm_simt_launch(A, B, C, M, N, K, b_is_nk, mode, group_k, group_n, bias, st);
}

int hbq_gemm_simt(const void* A, const void* B, void* C, int64_t M, int64_t N, int64_t K, int b_is_nk, int mode,
                  int group_k, int group_n, const void* bias, void* stream)
{
    int rc = check_gemm_args(A, B, C, M, N, K, mode, group_k, group_n);
    if (rc) return rc;
    if (M == 0 || N == 0) return HBQ_OK;
    return gemm_simt_launch(A, B, C, M, N, K, b_is_nk, mode, group_k, group_n, bias, (cudaStream_t)stream);
}

int hbq_gemm_wait_selftest(const void* A, const void* W, void* C, int64_t M, int64_t N, int64_t K, int mode, int group_k,
                           int group_n, uint32_t poll_limit, void* stream)
{
    int rc = check_gemm_args(A, W, C, M, N, K, mode, group_k, group_n);
    if (rc) return rc;
    if (poll_limit == 0 || poll_limit > (1u << 23)) return HBQ_ERR_ARG;
    if (M == 0 || N == 0 || K == 0) return HBQ_ERR_ARG;
    if ((((uintptr_t)A | (uintptr_t)W | (uintptr_t)C) & 15) || !gemm_tc_eligible(M, N, K, mode, group_k, group_n))
        return HBQ_ERR_UNSUPPORTED;
    return gemm_tc_launch_ex(A, W, C, M, N, K, mode, group_k, group_n, nullptr, (cudaStream_t)stream, poll_limit, 1);
}

int hbq_moe_route(const int64_t* ids, int64_t tokens, int top_k, int experts, int32_t* offsets, int64_t* src_rows,
                  int32_t* pos, void* stream)
{
    return moe_route_launch(ids, tokens, top_k, experts, offsets, src_rows, pos, (cudaStream_t)stream);
}

int hbq_gemm_grouped(const void* A, int64_t rows, const int32_t* offsets, int entries, const void* const* W_host,
                     void* const* C_host, const int32_t* expert_host, int64_t N, int64_t K, int mode, int group_k,
                     int group_n, void* stream)
{
    if (rows < 0 || N < 0 || K < 0 || entries < 0) return HBQ_ERR_ARG;
    if (rows == 0 || N == 0 || entries == 0) return HBQ_OK;
    if (!offsets || !W_host || !C_host || !expert_host) return HBQ_ERR_ARG;
    for (int i = 0; i < entries; ++i) {
        const int rc = check_gemm_args(A, W_host[i], C_host[i], rows, N, K, mode, group_k, group_n);
        if (rc) return rc;
        if (expert_host[i] < 0) return HBQ_ERR_ARG;
    }
    return gemm_tc_grouped_launch(A, rows, offsets, entries, W_host, C_host, expert_host, N, K, mode, group_k, group_n,
                                  (cudaStream_t)stream);
}

int hbq_moe_combine(const void* y_rows, const void* weights, const int32_t* pos, int64_t tokens, int top_k, int64_t hidden,
                    void* out, void* stream)
{
    return moe_combine_launch(y_rows, weights, pos, tokens, top_k, hidden, out, (cudaStream_t)stream);
}

int64_t hbq_gemm_w4_prepacked_bytes(int64_t N, int64_t K, int container_bits)
{
    return gemm_w4_prepacked_bytes(N, K, container_bits);
}

int hbq_gemm_w4_prepack(const hbq_packed_out* in, int64_t N, int64_t K, const hbq_format* fmt, int container_bits,
                        void* out, void* stream)
{
    if (N <= 0 || K <= 0) return HBQ_ERR_ARG;
    return gemm_w4_prepack(in, N, K, fmt, container_bits, out, (cudaStream_t)stream);
}

int64_t hbq_gemm_w4_workspace_bytes(int64_t M, int64_t N, int64_t K) { return gemm_w4_workspace_bytes(M, N, K); }

int hbq_gemm_w4(const void* X, const void* Wp, void* C, int64_t M, int64_t N, int64_t K, const hbq_format* fmt,
                int container_bits, const void* bias, void* workspace, int64_t workspace_bytes, void* stream)
{
    if (M < 0 || N < 0 || K < 0) return HBQ_ERR_ARG;
    if (M == 0 || N == 0) return HBQ_OK;
    const int64_t need = gemm_w4_workspace_bytes(M, N, K);
    if (need < 0) return HBQ_ERR_UNSUPPORTED;
    if (!workspace || workspace_bytes < need) return HBQ_ERR_WORKSPACE;
    return gemm_w4_launch(X, Wp, C, M, N, K, fmt, container_bits, bias, workspace, (cudaStream_t)stream, 0);
}

int hbq_gemm_status(int* status_host)
{
    if (!status_host) return HBQ_ERR_ARG;
    return gemm_tc_status(status_host);
}
int hbq_gemm_status_reset(void) { return gemm_tc_status_reset(); }
int hbq_gemm_reserve_sms(int n) { return gemm_tc_reserve_sms(n); }
int hbq_gemm_tile_columns(int64_t M, int64_t N, int mode, int sms)
{
    if (M <= 0 || N <= 0) return HBQ_ERR_ARG;
    if (sms <= 0) { const int rc = gemm_tc_usable_sms(&sms); if (rc) return rc; }
    return gemm_tc_tile_width((M + 127) / 128, N, sms, mode);
}

const char* hbq_error_string(int code)
{
    switch (code) {
        case HBQ_OK: return "ok";
        case HBQ_ERR_ARG: return "invalid argument";
        case HBQ_ERR_UNSUPPORTED: return "format or shape not supported by the CUDA kernels";
        case HBQ_ERR_CUDA: return "CUDA call failed (see hbq_last_cuda_error)";
        case HBQ_ERR_ALIGN: return "pointer not 16-byte aligned";
        case HBQ_ERR_WORKSPACE: return "workspace missing, too small or misaligned";
        case HBQ_ERR_DEVICE: return "device error reported by a kernel";
        case HBQ_ERR_TOO_LARGE: return "operand larger than the fixed scratch of the no-allocation entry point "
                                       "(N*K > HBQ_GEMM_NOALLOC_MAX_ELEMS)";
    }
    return "unknown error";
}
const char* hbq_last_cuda_error(void) { return g_last_cuda_error; }
int hbq_version(void) { return 100; }
int64_t hbq_launch_count(void) { return (int64_t)g_launches.load(); }

}  // extern "C"
