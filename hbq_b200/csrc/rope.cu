// Rotary embedding of projected queries or keys without a quantizer, stored by head: what the K-cache write does for the
// configurations that quantise neither (apply_rotary_pos_emb on the transposed projection, src/module.py:147-157).
#include "common.cuh"

namespace hbq {

// A thread takes 8 elements of each half of a head, d and d + D / 2: the rotation's partners.  Every product and the sum
// are rounded to fp16 as the separate tensor ops round them.  Bound by memory, and
// for a prompt's tokens by its launch: the transpose, negation, concatenation, two products and sum as tensor ops took
// 106 us for q and k of 1000 tokens (32 and 8 heads of 128); prefill of a one-layer Mixtral-8x7B 1640 -> 1608 us.
__global__ void __launch_bounds__(256) rope_heads_kernel(const uint4* x, const uint4* cos, const uint4* sin, uint4* out, int64_t total,
                                                         uint32_t T, uint32_t H, uint32_t hc, uint32_t rope_rows)
{
    grid_dependency_wait();
    dependents_may_start();
    const uint4 *xi = behind_wait(x), *ci = behind_wait(cos), *si = behind_wait(sin);
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
        const uint32_t row = (uint32_t)(i / hc), c = (uint32_t)(i - (int64_t)row * hc);         // (b, t, h), chunk of the half head
        const uint32_t bt = row / H, h = row - bt * H, b = bt / T, t = bt - b * T;
        const int64_t in = (int64_t)row * 2 * hc + c, rr = (int64_t)(rope_rows == T ? t : bt % rope_rows) * 2 * hc + c;
        const int64_t o = (((int64_t)b * H + h) * T + t) * 2 * hc + c;
        const uint4 lo = __ldg(xi + in), hi = __ldg(xi + in + hc);
        const uint4 c0 = __ldg(ci + rr), c1 = __ldg(ci + rr + hc), s0 = __ldg(si + rr), s1 = __ldg(si + rr + hc);
        const uint32_t l[4] = {lo.x, lo.y, lo.z, lo.w}, u[4] = {hi.x, hi.y, hi.z, hi.w};
        const uint32_t cl[4] = {c0.x, c0.y, c0.z, c0.w}, cu[4] = {c1.x, c1.y, c1.z, c1.w};
        const uint32_t sl[4] = {s0.x, s0.y, s0.z, s0.w}, su[4] = {s1.x, s1.y, s1.z, s1.w};
        uint32_t rl[4], ru[4];
        #pragma unroll
        for (int p = 0; p < 4; ++p) {
            rl[p] = h2_bits(__hadd2_rn(__hmul2_rn(bits_h2(l[p]), bits_h2(cl[p])), __hmul2_rn(bits_h2(u[p] ^ 0x80008000u), bits_h2(sl[p]))));
            ru[p] = h2_bits(__hadd2_rn(__hmul2_rn(bits_h2(u[p]), bits_h2(cu[p])), __hmul2_rn(bits_h2(l[p]), bits_h2(su[p]))));
        }
        out[o] = make_uint4(rl[0], rl[1], rl[2], rl[3]);
        out[o + hc] = make_uint4(ru[0], ru[1], ru[2], ru[3]);
    }
}

int rope_heads_launch(const void* x, int64_t B, int64_t T, int64_t H, int64_t D, const void* cos, const void* sin, int64_t rope_rows,
                      void* out, cudaStream_t stream)
{
    if (B < 0 || T < 0 || H < 0 || D <= 0) return HBQ_ERR_ARG;
    if (B * T * H == 0) return HBQ_OK;
    if (!x || !cos || !sin || !out || rope_rows <= 0) return HBQ_ERR_ARG;
    if ((D % 16) != 0 || D > (1 << 20) || B * T * H > 0x7FFFFFFFll || rope_rows > 0x7FFFFFFFll) return HBQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(cos) | reinterpret_cast<uintptr_t>(sin) | reinterpret_cast<uintptr_t>(out)) & 15)
        return HBQ_ERR_ALIGN;
    int sms = 0;
    { const int rc = device_sms(&sms); if (rc) return rc; }
    const int64_t total = B * T * H * (D / 16), need = (total + 255) / 256, cap = (int64_t)sms * 8;
    HBQ_CUDA_TRY(launch_dependent(rope_heads_kernel, (unsigned)(need < cap ? need : cap), 256, 0, stream, (const uint4*)x, (const uint4*)cos,
                                  (const uint4*)sin, (uint4*)out, total, (uint32_t)T, (uint32_t)H, (uint32_t)(D / 16), (uint32_t)rope_rows));
    HBQ_LAUNCH_CHECK("rope_heads_kernel");
    return HBQ_OK;
}

}  // namespace hbq
