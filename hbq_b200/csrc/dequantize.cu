// Packed codes and scales -> fake-quantised fp16 / bf16 tensor (hbq_dequantize).
//
// Bound: issue slots (67 % used) and the half-rate ALU pipe (63 %): two bit fields and a candidate select per pair (codes
// and scales in, 2 bytes per element out would take HBM 23 us).  A thread owns DQ_UNROLL chunks of 8 elements, one
// CTA-width apart, so that its code words and scales are all in flight before the first is used and every warp
// access is contiguous.  All planes are rows of whole blocks, so a chunk's block is its flat index shifted; only
// the output address of a tensor with a padded last block needs the row.
//
// Element values without tables: exponent and mantissa of a code, put at the top of the mantissa and the bottom of
// the exponent field of an fp16 pattern, are the value times 2^(bias - 15) -- subnormal codes included -- so one
// exact multiply by 2^(15 - bias) decodes any format of up to five exponent bits; integers go through the pattern
// of 1024 + v.  With five exponent bits the top field stands for 2^16 and more, beyond fp16: infinity whatever the
// mantissa says, so the mantissa is cleared there (its pattern would be a NaN's).
// HBQ weight [14336, 4096] (150 MB moved): 37-39 us = 4.0 TB/s; one chunk per thread with scalar ldexpf decoding and a
// 64-bit division each took 301 us.
#include "quantize_dev.cuh"
#include <string.h>

namespace hbq {

int packed_form_supported(const hbq_format*);               // quantize.cu
int l2_tables(int scheme, int bits, float tab[2][16]);

constexpr int DQ_THREADS = 256;
constexpr int DQ_UNROLL = 4;

struct DqArgs {
    hbq_packed_out in;
    void* deq;
    int64_t K, total_chunks, cpr;
    int flat;                 // no padded last block: output chunk = flat chunk
    int aligned;              // 128-bit stores are legal
    int out_bf16;
    int log2cpb;              // log2(chunks per block)
    uint32_t magmask2;        // FP codes: magnitude bits, in both halves
    int mshift, sshift;       // magnitude / sign -> their place in an fp16 pattern
    uint32_t unbias2;         // 2^(15 - bias) as an fp16 pair
    int e5;                   // five exponent bits
    int log2L, l2_bits, l2_bytes, l2_aligned;
    uint32_t tab2[2][16];     // HBQ candidates as fp16 pairs
};

// Two elements of a chunk as an fp16 pair.  b: their codes, one per 16-bit half; ss: their signs in bits 15 and 31
// (5-bit codes, whose signs are a plane of their own).
template <int BITS, bool INT>
__device__ __forceinline__ __half2 decode_pair(const DqArgs& a, uint32_t b, uint32_t ss)
{
    if (INT) {
        // two's complement v, its sign bit flipped, is v + 2^(BITS-1): the mantissa of 1024 + that
        constexpr uint32_t FLIP = BITS == 8 ? 0x00800080u : 0x00080008u;
        return __hsub2(bits_h2((b ^ FLIP) | 0x64006400u), bits_h2(0x64006400u | FLIP));
    }
    const uint32_t s = BITS == 5 ? ss : (b << a.sshift) & 0x80008000u;
    uint32_t v = (b & a.magmask2) << a.mshift;
    if (BITS == 8 && a.e5) v = __vminu2(v, 0x7C007C00u);
    return __hmul2(bits_h2(v | s), bits_h2(a.unbias2));
}

template <int BITS, bool INT, bool HBQ>
__global__ void __launch_bounds__(DQ_THREADS) dequantize_kernel(const DqArgs a)
{
    __shared__ uint32_t s_tab[32];
    if (HBQ) {
        if (threadIdx.x < 32) s_tab[threadIdx.x] = a.tab2[threadIdx.x >> 4][threadIdx.x & 15];
        __syncthreads();
    }
    const int64_t c0 = (int64_t)blockIdx.x * (DQ_THREADS * DQ_UNROLL) + threadIdx.x;
    uint2 w[DQ_UNROLL];
    uint32_t sg[DQ_UNROLL], sc[DQ_UNROLL], l2[DQ_UNROLL], sch[DQ_UNROLL];
    #pragma unroll
    for (int u = 0; u < DQ_UNROLL; ++u) {
        const int64_t ci = c0 + u * DQ_THREADS;
        w[u] = make_uint2(0u, 0u);
        sg[u] = sc[u] = l2[u] = sch[u] = 0u;
        if (ci >= a.total_chunks) continue;
        if (BITS == 8) w[u] = __ldg(reinterpret_cast<const uint2*>(a.in.codes) + ci);
        else w[u].x = __ldg(reinterpret_cast<const uint32_t*>(a.in.codes) + ci);
        if (BITS == 5) sg[u] = __ldg(a.in.sign + ci);
        const int64_t blk = ci >> a.log2cpb;
        sc[u] = __ldg(a.in.scale_u8 + blk);
        if (HBQ) {
            if (!a.l2_aligned) {
                for (int b = 0; b < a.l2_bytes; ++b) l2[u] |= (uint32_t)__ldg(a.in.l2_packed + blk * a.l2_bytes + b) << (8 * b);
            } else if (a.l2_bytes == 4) l2[u] = __ldg(reinterpret_cast<const uint32_t*>(a.in.l2_packed) + blk);
            else if (a.l2_bytes == 2) l2[u] = __ldg(reinterpret_cast<const uint16_t*>(a.in.l2_packed) + blk);
            else l2[u] = __ldg(a.in.l2_packed + blk);
            if (a.in.scheme) sch[u] = __ldg(a.in.scheme + blk);
        }
    }
    #pragma unroll
    for (int u = 0; u < DQ_UNROLL; ++u) {
        const int64_t ci = c0 + u * DQ_THREADS;
        if (ci >= a.total_chunks) break;
        const __half2 s2 = bits_h2((sc[u] << 7) * 0x00010001u);
        __half2 t[2] = {s2, s2};                            // HBQ: candidates of the chunk's two halves
        if (HBQ) {
            const int kin = ((int)ci & ((1 << a.log2cpb) - 1)) * 8;
            const uint32_t im = (1u << a.l2_bits) - 1u, row = (sch[u] & 1u) * 16u;
            t[0] = bits_h2(s_tab[row + ((l2[u] >> ((kin >> a.log2L) * a.l2_bits)) & im)]);
            t[1] = bits_h2(s_tab[row + ((l2[u] >> (((kin + 4) >> a.log2L) * a.l2_bits)) & im)]);
        }
        uint32_t o[4];
        #pragma unroll
        for (int p = 0; p < 4; ++p) {
            uint32_t b, ss = 0u;
            if (BITS == 8) b = __byte_perm(p < 2 ? w[u].x : w[u].y, 0u, (p & 1) ? 0x4342u : 0x4140u);
            else b = ((w[u].x >> (8 * p)) & 0xFu) | (((w[u].x >> (8 * p + 4)) & 0xFu) << 16);
            if (BITS == 5) ss = ((sg[u] << (15 - 2 * p)) & 0x8000u) | ((sg[u] << (30 - 2 * p)) & 0x80000000u);
            __half2 d = decode_pair<BITS, INT>(a, b, ss);
            if (HBQ) d = __hmul2(d, t[p >> 1]);
            d = __hmul2(d, s2);
            if (a.out_bf16) {
                const float2 f = __half22float2(d);
                const __nv_bfloat162 bb = __floats2bfloat162_rn(f.x, f.y);
                o[p] = *reinterpret_cast<const uint32_t*>(&bb);
            } else o[p] = h2_bits(d);
        }
        if (a.flat) {
            if (a.aligned) { reinterpret_cast<uint4*>(a.deq)[ci] = make_uint4(o[0], o[1], o[2], o[3]); continue; }
        }
        const int64_t row = ci / a.cpr, k0 = (ci - row * a.cpr) * 8;
        uint16_t* dp = reinterpret_cast<uint16_t*>(a.deq) + row * a.K + k0;
        if (a.aligned && k0 + 8 <= a.K) { *reinterpret_cast<uint4*>(dp) = make_uint4(o[0], o[1], o[2], o[3]); continue; }
        #pragma unroll
        for (int j = 0; j < 8; ++j)
            if (k0 + j < a.K) dp[j] = (uint16_t)(o[j >> 1] >> (16 * (j & 1)));
    }
}

int dequantize_launch(const hbq_packed_out* in, int64_t rows, int64_t K, const hbq_format* f, void* deq, int dtype,
                      cudaStream_t stream)
{
    if (!in || !f || !deq || !in->codes || !in->scale_u8) return HBQ_ERR_ARG;
    { const int rc = packed_form_supported(f); if (rc) return rc; }
    if (rows == 0 || K == 0) return HBQ_OK;
    const int B = f->block_size;
    if (B < 8 || (B & (B - 1))) return HBQ_ERR_UNSUPPORTED;          // what hbq_quantize packs
    DqArgs a;
    memset(&a, 0, sizeof(a));
    a.in = *in; a.deq = deq; a.K = K;
    const int64_t nblk = (K + B - 1) / B;
    a.cpr = nblk * (B / 8);
    a.total_chunks = rows * a.cpr;
    a.flat = K == nblk * B;
    a.aligned = (K % 8) == 0 && (reinterpret_cast<uintptr_t>(deq) & 15) == 0;
    a.out_bf16 = dtype == HBQ_DTYPE_BF16;
    while ((8 << a.log2cpb) < B) ++a.log2cpb;
    const bool is_int = f->kind == HBQ_KIND_MXINT;
    int code_bits;
    if (is_int) {
        if (f->mbit != 4 && f->mbit != 8) return HBQ_ERR_UNSUPPORTED;
        code_bits = f->mbit;
    } else {
        if (f->ebit < 1 || f->ebit > 5 || f->mbit < 0 || f->ebit + f->mbit > 7) return HBQ_ERR_UNSUPPORTED;
        code_bits = 1 + f->ebit + f->mbit;
        if (code_bits < 4) code_bits = 4;
        if (code_bits > 5) code_bits = 8;
        const int mag_bits = f->ebit + f->mbit;
        a.e5 = f->ebit == 5;
        a.magmask2 = ((1u << mag_bits) - 1u) * 0x00010001u;
        a.mshift = 10 - f->mbit;
        a.sshift = 15 - (code_bits == 4 ? 3 : mag_bits);
        a.unbias2 = (uint32_t)(15 + 15 - ((1 << (f->ebit - 1)) - 1)) * (1u << 10) * 0x00010001u;
    }
    if (code_bits == 5 && !in->sign) return HBQ_ERR_ARG;
    // the planes are read in words of a chunk's codes
    if (reinterpret_cast<uintptr_t>(in->codes) & (code_bits == 8 ? 7 : 3)) return HBQ_ERR_ALIGN;
    const bool hbq = f->kind == HBQ_KIND_HBQ;
    if (hbq) {
        const int L = f->l2_block_size;
        if (L < 4 || (L & (L - 1)) || L > B || f->l2_sc_bit < 0 || f->l2_sc_bit > 4) return HBQ_ERR_UNSUPPORTED;
        while ((1 << a.log2L) < L) ++a.log2L;
        a.l2_bits = f->l2_sc_bit;
        const int tb = (B / L) * a.l2_bits;
        if (tb != 8 && tb != 16 && tb != 32) return HBQ_ERR_UNSUPPORTED;
        if (!in->l2_packed || (f->l2_scheme == HBQ_L2_MIX && !in->scheme)) return HBQ_ERR_ARG;
        a.l2_bytes = tb / 8;
        a.l2_aligned = (reinterpret_cast<uintptr_t>(in->l2_packed) & (a.l2_bytes - 1)) == 0;
        if (f->l2_scheme != HBQ_L2_MIX) a.in.scheme = nullptr;
        float tab[2][16] = {};
        if (l2_tables(f->l2_scheme, f->l2_sc_bit, tab) < 0) return HBQ_ERR_ARG;
        for (int s = 0; s < 2; ++s)
            for (int i = 0; i < 16; ++i) a.tab2[s][i] = (uint32_t)__half_as_ushort(__float2half_rn(tab[s][i])) * 0x00010001u;
    }
    const int64_t per_cta = DQ_THREADS * DQ_UNROLL, grid = (a.total_chunks + per_cta - 1) / per_cta;
    if (grid > 0x7FFFFFFF) return HBQ_ERR_UNSUPPORTED;
    const unsigned g = (unsigned)grid;
    if (hbq) {
        if (code_bits == 4) dequantize_kernel<4, false, true><<<g, DQ_THREADS, 0, stream>>>(a);
        else if (code_bits == 5) dequantize_kernel<5, false, true><<<g, DQ_THREADS, 0, stream>>>(a);
        else dequantize_kernel<8, false, true><<<g, DQ_THREADS, 0, stream>>>(a);
    } else if (is_int) {
        if (code_bits == 4) dequantize_kernel<4, true, false><<<g, DQ_THREADS, 0, stream>>>(a);
        else dequantize_kernel<8, true, false><<<g, DQ_THREADS, 0, stream>>>(a);
    } else {
        if (code_bits == 4) dequantize_kernel<4, false, false><<<g, DQ_THREADS, 0, stream>>>(a);
        else if (code_bits == 5) dequantize_kernel<5, false, false><<<g, DQ_THREADS, 0, stream>>>(a);
        else dequantize_kernel<8, false, false><<<g, DQ_THREADS, 0, stream>>>(a);
    }
    HBQ_LAUNCH_CHECK("dequantize_kernel");
    return HBQ_OK;
}

}  // namespace hbq
