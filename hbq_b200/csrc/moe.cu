// Routing and combination of a sparse MoE block whose experts are all on this GPU: the token copies sorted by expert
// with their row offsets left on the device (the grouped GEMM reads them there, so the block needs no host read), and
// the weighted sum of the experts' rows per token.
#include "common.cuh"

namespace hbq {

constexpr int ROUTE_WARPS = 32;
constexpr int ROUTE_MAX_EXPERTS = 256;

// A stable counting sort of n expert ids by ONE CTA: warp w owns a contiguous run of the copies, counts them per expert
// (lanes with the same id find each other with match.any), the counts become start positions in (expert, warp) order,
// and the second sweep hands them out.  An id outside [0, experts) counts as one of a further, last bucket: its copies
// lie behind every expert's rows and have no position (pos -1).  2000 copies of 8 experts: 4.0 us (the radix sort
// alone took 25, before its histogram, division and a host synchronisation).
__global__ void __launch_bounds__(ROUTE_WARPS * 32) moe_route_kernel(const int64_t* ids, int n, int top_k, int experts,
                                                                      int* offsets, int64_t* src_rows, int* pos)
{
    __shared__ int s_cnt[ROUTE_MAX_EXPERTS + 1][ROUTE_WARPS + 1];
    __shared__ int s_off[ROUTE_MAX_EXPERTS + 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, buckets = experts + 1;
    for (int i = threadIdx.x; i < buckets * (ROUTE_WARPS + 1); i += ROUTE_WARPS * 32) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    const int run = (n + ROUTE_WARPS * 32 - 1) / (ROUTE_WARPS * 32) * 32;
    const int c0 = warp * run, c1 = min(c0 + run, n);
    auto bucket = [&](int c) -> int {                            // -1: no copy; compared in 64 bits, before it is narrowed
        if (c >= c1) return -1;
        const int64_t id = ids[c];
        return id >= 0 && id < experts ? (int)id : experts;
    };
    for (int c = c0; c < c1; c += 32) {
        const int e = bucket(c + lane);
        const uint32_t same = __match_any_sync(0xFFFFFFFFu, e);
        if (e >= 0 && lane == __ffs(same) - 1) s_cnt[e][warp] += __popc(same);
        __syncwarp();
    }
    __syncthreads();
    for (int e = warp; e < buckets; e += ROUTE_WARPS) {          // a warp per bucket: prefix sum over the warps' counts
        const int v = s_cnt[e][lane];
        int inc = v;
        #pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_up_sync(0xFFFFFFFFu, inc, off);
            if (lane >= off) inc += o;
        }
        s_cnt[e][lane] = inc - v;
        if (lane == 31) s_off[e + 1] = inc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        s_off[0] = 0;
        for (int e = 0; e < buckets; ++e) s_off[e + 1] += s_off[e];
    }
    __syncthreads();
    for (int e = threadIdx.x; e <= experts; e += ROUTE_WARPS * 32) offsets[e] = s_off[e];
    for (int c = c0; c < c1; c += 32) {
        const int e = bucket(c + lane);
        const uint32_t same = __match_any_sync(0xFFFFFFFFu, e);
        int base = 0;
        if (e >= 0) base = s_cnt[e][warp];
        __syncwarp();
        if (e >= 0) {
            const int p = s_off[e] + base + __popc(same & ((1u << lane) - 1u));
            src_rows[p] = (c + lane) / top_k;
            pos[c + lane] = e < experts ? p : -1;
            if (lane == __ffs(same) - 1) s_cnt[e][warp] = base + __popc(same);
        }
        __syncwarp();
    }
}

// out[t] = sum over the token's choices of fp16(row * weight): each product rounded to fp16 as the separate
// multiplication rounds it, the sum kept in fp32 and rounded once (two choices: the same value as an fp16 addition).
// Bound by the rows' memory traffic: 1000 tokens x 4096, two choices, 4.6 us (multiplication and index_add: 67 us).
__global__ void __launch_bounds__(256) moe_combine_kernel(const uint4* __restrict__ rows, const __half* __restrict__ w,
                                                          const int* __restrict__ pos, int64_t tokens, int top_k, int cpr, uint4* __restrict__ out)
{
    const int64_t total = tokens * cpr;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
        const int64_t t = i / cpr;
        const int c = (int)(i - t * cpr);
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int j = 0; j < top_k; ++j) {
            const int64_t k = t * top_k + j;
            const int p0 = __ldg(pos + k);
            if (p0 < 0) continue;                                // a copy without an expert
            const uint4 v = __ldg(rows + (int64_t)p0 * cpr + c);
            const __half2 wv = __half2half2(w[k]);
            const uint32_t r[4] = {v.x, v.y, v.z, v.w};
            #pragma unroll
            for (int p = 0; p < 4; ++p) {
                const float2 f = __half22float2(__hmul2_rn(bits_h2(r[p]), wv));
                acc[2 * p] += f.x;
                acc[2 * p + 1] += f.y;
            }
        }
        uint32_t o[4];
        #pragma unroll
        for (int p = 0; p < 4; ++p) o[p] = h2_bits(__floats2half2_rn(acc[2 * p], acc[2 * p + 1]));
        out[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

int moe_route_launch(const int64_t* ids, int64_t tokens, int top_k, int experts, int* offsets, int64_t* src_rows, int* pos,
                     cudaStream_t stream)
{
    if (tokens < 0 || top_k <= 0 || experts <= 0 || !offsets) return HBQ_ERR_ARG;
    const int64_t n = tokens * top_k;
    if (experts > ROUTE_MAX_EXPERTS || n > (1 << 30)) return HBQ_ERR_UNSUPPORTED;
    if (n > 0 && (!ids || !src_rows || !pos)) return HBQ_ERR_ARG;
    moe_route_kernel<<<1, ROUTE_WARPS * 32, 0, stream>>>(ids, (int)n, top_k, experts, offsets, src_rows, pos);
    HBQ_LAUNCH_CHECK("moe_route_kernel");
    return HBQ_OK;
}

int moe_combine_launch(const void* rows, const void* w, const int* pos, int64_t tokens, int top_k, int64_t hidden, void* out,
                       cudaStream_t stream)
{
    if (tokens < 0 || top_k <= 0 || hidden < 0) return HBQ_ERR_ARG;
    if (tokens == 0 || hidden == 0) return HBQ_OK;
    if (!rows || !w || !pos || !out) return HBQ_ERR_ARG;
    if ((hidden % 8) != 0 || hidden > (1 << 30)) return HBQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(out)) & 15) return HBQ_ERR_ALIGN;
    int sms = 0;
    { const int rc = device_sms(&sms); if (rc) return rc; }
    const int64_t need = (tokens * (hidden / 8) + 255) / 256, cap = (int64_t)sms * 8;
    moe_combine_kernel<<<(int)(need < cap ? need : cap), 256, 0, stream>>>((const uint4*)rows, (const __half*)w, pos, tokens, top_k,
                                                                            (int)(hidden / 8), (uint4*)out);
    HBQ_LAUNCH_CHECK("moe_combine_kernel");
    return HBQ_OK;
}

}  // namespace hbq
