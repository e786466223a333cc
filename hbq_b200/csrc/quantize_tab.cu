// HBQ quantize, byte-table kernels: the per-step activation quantizer (one candidate table, E2M1 / E2M2
// elements, up to 4 micro-scale candidates; src/quantizer.py:741-859).
//
// What HBQ asks per element is 2^l2_sc_bit quantise-dequantise-error evaluations with an fp16 rounding
// after every op.  As in quantize_lut.cu the element quantizer is a table lookup keyed by the fp16
// pattern of |a| = |x / l1|, but here
//   * an entry is 4 BYTES: for each candidate the top byte of the fp16 pattern of the element value
//     c_i = Q(fp16(a / t_i)) (E2M1 / E2M2 values have at most two mantissa bits).  Half the shared-memory
//     traffic and bank passes of the 8-byte entries, and a 29 KB table, so that two CTAs fit an SM;
//   * the table is built once per format on the host, kept in a device array of the library image, and
//     each CTA stages it into shared memory with ONE bulk async copy (cp.async.bulk + mbarrier) instead
//     of rebuilding it from thresholds;
//   * the two halves of a half2 are two ELEMENTS, not two candidates: one PRMT builds (c_i(x0), c_i(x1))
//     from the two elements' entries, the candidate's -t_i*l1 is a per-block constant, and
//       r = fma(c, -t*l1, |x|)   e = r*r (fp16)   acc_i += e (fp32)
//     need no broadcast of |x|;
//   * a thread owns C chunks (8 elements each) of ONE block, chunk g + k*Gt for lane g of the block's Gt
//     lanes: the block maximum, the E5M3 scale and the division constants are computed once per C chunks,
//     and every warp load / store still covers whole 32-byte sectors.
// Results are bit-identical to the reference's eager fp16 quantizer (golden vectors + oracle tests) for finite inputs.  An
// infinite or NaN quotient takes the smallest level in the one-table kernels (their clamp's maximum, which drops a NaN, is
// the inner one), so such an input becomes a zero; hbq_tab_mix_kernel keeps both.
#include "quantize_tab.cuh"
#include "vcache_dev.cuh"
#include <mutex>
#include <string.h>

namespace hbq {

constexpr int TAB_THREADS = 512;
constexpr int MIX_THREADS = 384;            // 80 registers a thread at two CTAs per SM
constexpr int TAB_SLOTS = 32;               // formats that can have a device table at the same time
constexpr int TAB_MAX_ENTRIES = 8192;       // 32 KB per table

// The staged tables.  In host code this name is only a handle for cudaGetSymbolAddress.
static __device__ __align__(128) uint32_t g_tab_slots[TAB_SLOTS][TAB_MAX_ENTRIES];

// The second candidate table of the two-table ("Mix") weight formats, as TabArgs describes the first.
struct TabSecond {
    const uint32_t* table;
    int entries;
    uint32_t base2, hi2, big_l1;
    float inv_ele_max;
    uint32_t nt2[4];
    float tabf[4];
};

struct TabArgs {
    const uint4* x;
    const uint4* gate;        // GLU: the tensor to quantise is silu(gate) * x
    uint4* deq;
    hbq_packed_out out;       // SIDE
    const uint32_t* table;    // device address of the format's byte table
    int64_t total_units;      // thread-units of C chunks
    int entries;              // table entries (a multiple of 4)
    uint32_t entry_bytes;     // 4
    uint32_t base2, hi2;      // first / last covered |a| pattern, in both halves
    uint32_t big_l1;
    float inv_ele_max;
    uint32_t nt2[4];          // (-t_i, -t_i) as fp16 pairs
    float tabf[4];            // t_i, for the rare exact sign-of-zero check
    uint16_t rm[8];           // fp16(1 / m) for the eight E5M3 mantissas
    int in_bf16, out_bf16;
    int log2Gt;               // log2(lanes per block)
    int m_lanes, log2m;       // chunks (= lanes) per micro-block
    int l2_sc_bit, nl2, l2_bytes;
    // KV: the K / post-RoPE Q cache write; a row (b, t, h) is one block, stored at (b, h, t)
    const uint4* rope_cos;    // fp16 [rope_rows, block] or NULL (no rotation)
    const uint4* rope_sin;
    const uint4* center;      // fp16 [B, H, block] or NULL: subtracted after the rotation
    uint32_t kv_T, kv_H, rope_rows;
    uint32_t kv_B, run, group;    // run > 0: stored run by run of `run` tokens, the `group` heads of a key-value head together
    uint32_t from_runs, T0;   // from_runs: the rows are (b, h, t), t the kv_T tokens of a run that starts at token T0,
    uint32_t Tall;            // and stored at (b, T0 + t, h) of Tall tokens
    TabSecond b;              // hbq_tab_mix_kernel
};
static_assert(sizeof(TabArgs) <= 4000, "kernel parameters are limited to 4 KB");

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// acc += lo(e); acc += hi(e): fp32 accumulation of two fp16 values, in that order (one rounding each)
__device__ __forceinline__ void acc_pair(float& acc, uint32_t e)
{
    asm("{ .reg .b16 lo, hi;\n mov.b32 {lo, hi}, %1;\n"
        " add.rn.f32.f16 %0, lo, %0;\n add.rn.f32.f16 %0, hi, %0; }"
        : "+f"(acc) : "r"(e));
}
// acc = lo(e) + hi(e), the start of such a sum (lo(e) + 0 is exact)
__device__ __forceinline__ void acc_pair_first(float& acc, uint32_t e)
{
    asm("{ .reg .b16 lo, hi;\n mov.b32 {lo, hi}, %1;\n"
        " add.rn.f32.f16 %0, lo, 0f00000000;\n add.rn.f32.f16 %0, hi, %0; }"
        : "=f"(acc) : "r"(e));
}

// Byte i of both entries as the high bytes of an fp16 pair: (c_i(element 0), c_i(element 1)).  The low
// bytes are filled by sign replication of the (non-negative) value bytes, i.e. with zeros.
__device__ __forceinline__ uint32_t cand_pair(uint32_t e0, uint32_t e1, int i)
{
    return prmt(e0, e1, ((4u + i) << 12) | ((0xCu + i) << 8) | ((uint32_t)i << 4) | (8u + i));
}

// One 8-element chunk (x: its values as fp16 pairs; only |x| is used): every candidate's squared-error sum.
// SMALL: value * t * l1 cannot overflow fp16 for this block, so fma(c, -t*l1, |x|) equals the reference's
// fp16(|x| - fp16(fp16(c*t)*l1)) (both products are exact).  Otherwise the product keeps its own rounding.
template <bool SMALL>
__device__ __forceinline__ void chunk_errors(const uint32_t* ent, const uint32_t* x, const uint32_t* tl, const uint32_t* nt2,
                                             uint32_t l1u, float* acc)
{
    #pragma unroll
    for (int p = 0; p < 4; ++p) {
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __half2 c = bits_h2(cand_pair(ent[2 * p], ent[2 * p + 1], i));
            __half2 r;
            if (SMALL) r = __hfma2(c, bits_h2(tl[i]), __habs2(bits_h2(x[p])));
            else r = __hadd2(__habs2(bits_h2(x[p])), __hmul2(__hmul2(c, bits_h2(nt2[i])), bits_h2(l1u)));
            if (p == 0) acc_pair_first(acc[i], h2_bits(__hmul2(r, r)));
            else acc_pair(acc[i], h2_bits(__hmul2(r, r)));
        }
    }
}

// First minimum among four non-negative fp16 values given as fp32 sums: the sums are rounded to fp16 (as the
// reference rounds them), and since non-negative fp16 patterns order like integers, pattern * 4 + index is a
// key whose minimum is the first minimum.
__device__ __forceinline__ int first_min4(const float* acc)
{
    const uint32_t E01 = h2_bits(__floats2half2_rn(acc[0], acc[1])), E23 = h2_bits(__floats2half2_rn(acc[2], acc[3]));
    const uint32_t k0 = (E01 & 0xFFFFu) * 4u, k1 = (E01 >> 16) * 4u + 1u;
    const uint32_t k2 = (E23 & 0xFFFFu) * 4u + 2u, k3 = (E23 >> 16) * 4u + 3u;
    return (int)(min(min(k0, k1), min(k2, k3)) & 3u);
}

// The eight element codes of a chunk: cw = its element values as fp16 pairs (non-negative), sg = words whose bits 15
// and 31 are the elements' signs.  A value times 2^-14 is, as an fp16 pattern, the code shifted left by 10 - MB (the
// code's exponent and mantissa fields ARE the pattern's low exponent bits and top mantissa bits, subnormal codes
// included), so one multiply per pair replaces the field extraction (HBQ-A activations [8192, 8192] bf16 to packed
// planes and the bf16 tensor: 113 -> 95 us).  E2M1: nibbles with the sign on top, E2M2:
// magnitude nibbles and the signs in `sbits`.
template <int MB>
__device__ __forceinline__ uint32_t pack_codes(const uint32_t* cw, const uint32_t* sg, uint32_t& sbits)
{
    uint32_t v[4];
    #pragma unroll
    for (int p = 0; p < 4; ++p)
        v[p] = h2_bits(__hmul2(bits_h2(cw[p]), bits_h2(0x04000400u))) | (sg[p] & 0x80008000u);
    // the high bytes of the elements: {sign, -, -, -, code} (E2M2), {sign, -, -, -, code, -} (E2M1)
    const uint32_t t0 = prmt(v[0], v[1], 0x7531u), t1 = prmt(v[2], v[3], 0x7531u);
    const uint32_t ev = prmt(t0, t1, 0x6420u), od = prmt(t0, t1, 0x7531u);
    if (MB == 1) {
        const uint32_t e = ((ev >> 1) & 0x07070707u) | ((ev >> 4) & 0x08080808u);
        return e | ((od << 3) & 0x70707070u) | (od & 0x80808080u);
    }
    // bit 7 of byte j -> bit 2j of the top byte
    const uint32_t se = (((ev >> 7) & 0x01010101u) * 0x01041040u) >> 24, so = (((od >> 7) & 0x01010101u) * 0x01041040u) >> 24;
    sbits = (se & 0x55u) | ((so & 0x55u) << 1);
    return (ev & 0x0F0F0F0Fu) | ((od & 0x0F0F0F0Fu) << 4);
}

// The C chunks of one thread-unit, after the block scale is known.  SMALL: see chunk_errors (warp-uniform).
// On return xb[k] holds chunk k's fake-quantised values (fp16 pairs with the inputs' signs), `bests` the chosen
// candidate of every chunk (2 bits each) and the return value is the packed minimum of all quotients a.
// The reference returns +0 (not -0) when fp16(a / t) is exactly zero; only quotients a below 2^-19 can do
// that, and deciding it needs the exact a (the scaled division may be off down there), so it is a rare slow
// path.  TINY = 0: the caller runs it (from the returned minimum, re-reading its inputs); 1: it runs here, per
// chunk, before the inputs are overwritten; 2: the inputs are non-negative, the rule cannot apply.
template <int MB, int C, int ML, bool SMALL, bool SIDE, int TINY>
__device__ __forceinline__ uint32_t unit_chunks(const TabArgs& a, const uint32_t tab_addr, const uint32_t* s_nt2,
                                                 const float* s_tabf, uint32_t (*xb)[4], uint32_t l1b, const uint4 cst,
                                                 int m_lanes, uint32_t& bests, uint32_t* codes, uint32_t* sbits)
{
    const __half2 pre2 = bits_h2(cst.x), post2 = bits_h2(cst.y), nm2 = bits_h2(cst.z), rm2 = bits_h2(cst.w);
    const uint32_t l1u = l1b * 0x00010001u;
    uint32_t tl[4];                                         // (-t_i * l1) pairs; exact products (SMALL only)
    #pragma unroll
    for (int i = 0; i < 4; ++i) tl[i] = h2_bits(__hmul2(bits_h2(l1u), bits_h2(a.nt2[i])));
    uint32_t amin = 0x7C007C00u;
    bests = 0u;
    // byte address of entry (pattern): tab_addr + 4 * (pattern - base)
    const uint32_t addr0 = tab_addr - 4u * (a.base2 & 0xFFFFu);
    #pragma unroll
    for (int k = 0; k < C; ++k) {
        uint32_t ent[8], av[TINY == 1 ? 4 : 1];
        #pragma unroll
        for (int p = 0; p < 4; ++p) {
            // a = fp16(|x| / l1) by the pre-scaled Markstein division (exact for every quotient >= 2^-14)
            const __half2 axs = __hmul2(__habs2(bits_h2(xb[k][p])), pre2);
            const __half2 q0 = __hmul2(axs, rm2);
            const __half2 r = __hfma2(q0, nm2, axs);
            const __half2 q1 = __hfma2(r, rm2, q0);
            const __half2 aa = __hmul2(q1, post2);
            if (TINY == 0) amin = h2_bits(__hmin2(bits_h2(amin), aa));
            if (TINY == 1) av[p] = h2_bits(aa);
            const uint32_t w = h2_bits(__hmin2(__hmax2(aa, bits_h2(a.base2)), bits_h2(a.hi2)));
            uint32_t e0, e1;
            // entry address = pattern * 4 + addr0; the 4 is a kernel argument so that the scaling stays one
            // multiply-add on the (full-rate) FMA pipe instead of shifts on the half-rate ALU pipe
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(e0) : "r"((w & 0xFFFFu) * a.entry_bytes + addr0));
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(e1) : "r"((w >> 16) * a.entry_bytes + addr0));
            ent[2 * p] = e0; ent[2 * p + 1] = e1;
        }
        float acc[4];
        chunk_errors<SMALL>(ent, xb[k], tl, a.nt2, l1u, acc);
        if (ML > 0) {
            #pragma unroll
            for (int off = ML >> 1; off >= 1; off >>= 1) {
                #pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] += __shfl_xor_sync(0xFFFFFFFFu, acc[i], off);
            }
        } else {
            for (int off = m_lanes >> 1; off >= 1; off >>= 1) {
                #pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] += __shfl_xor_sync(0xFFFFFFFFu, acc[i], off);
            }
        }
        const int best = first_min4(acc);
        bests |= (uint32_t)best << (2 * k);
        // the winner's values with the inputs' signs
        const uint32_t wsel = 0x4C08u + (uint32_t)best * 0x1111u;
        const uint32_t ntb = s_nt2[best];
        const __half2 tlb = __hmul2(bits_h2(l1u), bits_h2(ntb));
        uint32_t dq[4], cwv[SIDE ? 4 : 1];
        #pragma unroll
        for (int p = 0; p < 4; ++p) {
            const uint32_t cw = prmt(ent[2 * p], ent[2 * p + 1], wsel);
            if (SIDE) cwv[p] = cw;
            const __half2 dneg = SMALL ? __hmul2(bits_h2(cw), tlb)
                                       : __hmul2(__hmul2(bits_h2(cw), bits_h2(ntb)), bits_h2(l1u));
            dq[p] = (h2_bits(dneg) & 0x7FFF7FFFu) | (xb[k][p] & 0x80008000u);
        }
        if (SIDE) codes[k] = pack_codes<MB>(cwv, xb[k], sbits[k]);
        if (TINY == 1) {
            const __half2 am = __hmin2(__hmin2(bits_h2(av[0]), bits_h2(av[1])), __hmin2(bits_h2(av[2]), bits_h2(av[3])));
            if (__hle2_mask(am, bits_h2(0x00200020u)) != 0u) {
                const float l1f = __half2float(bits_h((uint16_t)l1b)), tc = s_tabf[best];
                #pragma unroll
                for (int p = 0; p < 4; ++p)
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t xbits = (xb[k][p] >> (16 * h)) & 0xFFFFu;
                        if ((xbits & 0x8000u) && ((av[p] >> (16 * h)) & 0xFFFFu) <= 0x0020u) {
                            const float xf = __half2float(bits_h((uint16_t)(xbits & 0x7FFFu)));
                            if (rh(__fdiv_rn(rh(__fdiv_rn(xf, l1f)), tc)) == 0.f) dq[p] &= ~(0x8000u << (16 * h));
                        }
                    }
            }
        }
        #pragma unroll
        for (int p = 0; p < 4; ++p) xb[k][p] = dq[p];
    }
    return amin;
}

// Stage a format's tables into shared memory; every thread of the CTA calls it.  The candidate table comes
// by ONE bulk async copy whose completion is counted on an mbarrier, with a bounded wait: if the copy has not
// landed by then, every thread loads the table with plain loads (the same values, so a late completion of the
// copy is harmless).  MIX: the second table follows the first.  Returns the shared-memory address of the first table.
template <bool MIX = false>
__device__ __forceinline__ uint32_t stage_table(const TabArgs& a, uint32_t* s_tab, uint4* s_l1c, unsigned long long* s_bar,
                                                 uint32_t* s_nt2, float* s_tabf, int nthreads)
{
    const int tid = threadIdx.x;
    if (tid < 4) { s_nt2[tid] = a.nt2[tid]; s_tabf[tid] = a.tabf[tid]; }
    if (MIX && tid >= 4 && tid < 8) { s_nt2[tid] = a.b.nt2[tid - 4]; s_tabf[tid] = a.b.tabf[tid - 4]; }
    const uint32_t bar = smem_addr(s_bar), dst = smem_addr(s_tab);
    const uint32_t bytes = (uint32_t)a.entries * 4u, bytes1 = MIX ? (uint32_t)a.b.entries * 4u : 0u;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tid == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes + bytes1) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(dst), "l"(a.table), "r"(bytes), "r"(bar) : "memory");
        if (MIX)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(dst + bytes), "l"(a.b.table), "r"(bytes1), "r"(bar) : "memory");
    }
    if (tid < 256) {
        const uint32_t l1b = (uint32_t)tid << 7;
        const int e5 = (int)(l1b >> 10) - 15;
        const int s1 = min(15, 8 - e5);
        uint4 c;
        c.x = ((uint32_t)(s1 + 15) << 10) * 0x00010001u;
        c.y = ((uint32_t)(15 - (s1 + e5)) << 10) * 0x00010001u;
        c.z = (0xBC00u | (l1b & 0x03FFu)) * 0x00010001u;
        c.w = (uint32_t)a.rm[(l1b >> 7) & 7u] * 0x00010001u;
        s_l1c[tid] = c;
    }
    bool landed = false;
    #pragma unroll 1
    for (int it = 0; it < (1 << 20) && !landed; ++it) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], 0;\n selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok) : "r"(bar) : "memory");
        landed = ok != 0;
    }
    if (!__syncthreads_and(landed ? 1 : 0)) {
        const uint4* src = reinterpret_cast<const uint4*>(a.table);
        uint4* d4 = reinterpret_cast<uint4*>(s_tab);
        for (int i = tid; i < a.entries / 4; i += nthreads) d4[i] = __ldg(src + i);
        if (MIX) {
            const uint4* src1 = reinterpret_cast<const uint4*>(a.b.table);
            for (int i = tid; i < a.b.entries / 4; i += nthreads) d4[a.entries / 4 + i] = __ldg(src1 + i);
        }
        __syncthreads();
    }
    return dst;
}

// The block scale of a thread-unit whose C chunks are in xb: the maximum over the block's GT lanes, then the
// E5M3 scale (round-half-up of the 3-bit mantissa).  Returns the scale's fp16 pattern.
template <int C>
__device__ __forceinline__ uint32_t unit_scale(const uint32_t (*xb)[4], int Gt, float inv_ele_max)
{
    uint32_t mx = 0u;
    #pragma unroll
    for (int k = 0; k < C; ++k)
        #pragma unroll
        for (int p = 0; p < 4; ++p) mx = h2_bits(__hmax2(bits_h2(mx), __habs2(bits_h2(xb[k][p]))));
    for (int off = Gt >> 1; off >= 1; off >>= 1)
        mx = h2_bits(__hmax2(bits_h2(mx), bits_h2(__shfl_xor_sync(0xFFFFFFFFu, mx, off))));
    const uint32_t am16 = max(mx & 0xFFFFu, mx >> 16);
    const float sf = __half2float(bits_h((uint16_t)am16)) * inv_ele_max;
    uint32_t sb = (uint32_t)h_bits(__float2half_rn(sf));
    sb = min(max(sb, 0x0400u), 0x7B80u);
    return (sb + 0x40u) & 0xFF80u;
}

// The E5M3 scale's fp16 pattern for a block whose maximum divided by the largest element value is `sf`.
__device__ __forceinline__ uint32_t e5m3_scale(float sf)
{
    const uint32_t sb = min(max((uint32_t)h_bits(__float2half_rn(sf)), 0x0400u), 0x7B80u);
    return (sb + 0x40u) & 0xFF80u;
}

// A block's error total from its chunks' sums (chunk g + k * Gt of lane g): the tree of an exchange between lanes
// that hold one chunk each, distances 8, 4, 2, 1 (16 chunks), with the distances of Gt and more inside the thread.
template <int C>
__device__ __forceinline__ float block_error(const float* e, int Gt)
{
    float t = C == 4 ? (e[0] + e[2]) + (e[1] + e[3]) : e[0] + e[1];
    for (int off = Gt >> 1; off >= 1; off >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, off);
    return t;
}

// The per-block side outputs, by the block's first lane (`store`); l2word: this lane's share of the micro-scale indices.
__device__ __forceinline__ void store_block_side(const TabArgs& a, int64_t bi, int Gt, bool store, uint32_t l1b, uint32_t scheme,
                                                 uint32_t l2word)
{
    if (a.out.l2_packed) l2word = group_or(l2word, Gt);
    if (!store) return;
    if (a.out.scale_h) a.out.scale_h[bi] = (uint16_t)l1b;
    if (a.out.scale_u8) a.out.scale_u8[bi] = (uint8_t)(l1b >> 7);
    if (a.out.scheme) a.out.scheme[bi] = (uint8_t)scheme;
    if (a.out.l2_packed) {
        uint8_t* lp = a.out.l2_packed + bi * a.l2_bytes;
        if (a.l2_bytes == 4) *reinterpret_cast<uint32_t*>(lp) = l2word;
        else if (a.l2_bytes == 2) *reinterpret_cast<uint16_t*>(lp) = (uint16_t)l2word;
        else *lp = (uint8_t)l2word;
    }
}

// Rotary embedding and centring of the K / post-RoPE Q cache write on a thread-unit's fp16 chunks: a row is one block,
// so chunk k's rotation partner (d +- D/2) is chunk k +- C/2 of the same thread.  Every product, the sum and the
// difference are rounded to fp16 like the reference's tensor ops (the _rn forms keep ptxas from contracting them).
template <int C>
__device__ __forceinline__ void kv_rows(const TabArgs& a, const uint4* rope_cos, const uint4* rope_sin, const uint4* center, uint32_t (*xb)[4], uint32_t bt, uint32_t b, uint32_t t, uint32_t h,
                                        int Gt, int g)
{
    const int cpr = C * Gt;
    if (rope_cos) {
        const int64_t r0 = (int64_t)(a.rope_rows == a.kv_T ? t : bt % a.rope_rows) * cpr + g;
        #pragma unroll
        for (int k = 0; k < C / 2; ++k) {
            const uint4 c0 = __ldg(rope_cos + r0 + k * Gt), s0 = __ldg(rope_sin + r0 + k * Gt);
            const uint4 c1 = __ldg(rope_cos + r0 + (k + C / 2) * Gt), s1 = __ldg(rope_sin + r0 + (k + C / 2) * Gt);
            const uint32_t cl[4] = {c0.x, c0.y, c0.z, c0.w}, sl[4] = {s0.x, s0.y, s0.z, s0.w};
            const uint32_t ch[4] = {c1.x, c1.y, c1.z, c1.w}, sh[4] = {s1.x, s1.y, s1.z, s1.w};
            #pragma unroll
            for (int p = 0; p < 4; ++p) {
                const uint32_t lo = xb[k][p], hi = xb[k + C / 2][p];
                xb[k][p] = h2_bits(__hadd2_rn(__hmul2_rn(bits_h2(lo), bits_h2(cl[p])), __hmul2_rn(bits_h2(hi ^ 0x80008000u), bits_h2(sl[p]))));
                xb[k + C / 2][p] = h2_bits(__hadd2_rn(__hmul2_rn(bits_h2(hi), bits_h2(ch[p])), __hmul2_rn(bits_h2(lo), bits_h2(sh[p]))));
            }
        }
    }
    if (center) {
        const int64_t r0 = ((int64_t)b * a.kv_H + h) * cpr + g;
        #pragma unroll
        for (int k = 0; k < C; ++k) {
            const uint4 cv = __ldg(center + r0 + k * Gt);
            const uint32_t c[4] = {cv.x, cv.y, cv.z, cv.w};
            #pragma unroll
            for (int p = 0; p < 4; ++p) xb[k][p] = h2_bits(__hsub2_rn(bits_h2(xb[k][p]), bits_h2(c[p])));
        }
    }
}

// GT / ML: lanes per block / per micro-block as compile-time constants (0: read from the arguments).
// KV: the K / post-RoPE Q cache write (TabArgs).  K of [4, 1999, 8 x 128] fp16: 22.0 us with the 8-byte
// tables of quantize_lut.cu, 11.8 us here (2.8 TB/s of input and output; instruction issue bounds it).
template <int MB, int C, int GT, int ML, bool SIDE, bool GLU, bool KV = false>
__global__ void __launch_bounds__(TAB_THREADS, 2) hbq_tab_kernel(const TabArgs a)
{
    extern __shared__ __align__(128) uint32_t s_tab[];
    __shared__ uint4 s_l1c[256];             // per E5M3 scale (pattern >> 7): {2^s1, 2^-(s1+e), -m, fp16(1/m)} as fp16 pairs
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ uint32_t s_nt2[4];            // the candidates, where a run-time index can reach them
    __shared__ float s_tabf[4];
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t dst = stage_table(a, s_tab, s_l1c, &s_bar, s_nt2, s_tabf, TAB_THREADS);
    grid_dependency_wait();
    dependents_may_start();
    const uint4* const xin = behind_wait(a.x);
    const uint4* const gin = GLU ? behind_wait(a.gate) : nullptr;
    const uint4* const rope_cos = KV ? behind_wait(a.rope_cos) : nullptr;
    const uint4* const rope_sin = KV ? behind_wait(a.rope_sin) : nullptr;
    const uint4* const center = KV ? behind_wait(a.center) : nullptr;

    const int log2Gt = GT > 0 ? (GT == 1 ? 0 : GT == 2 ? 1 : GT == 4 ? 2 : GT == 8 ? 3 : GT == 16 ? 4 : 5) : a.log2Gt;
    const int Gt = 1 << log2Gt;
    // warps take turns over the CTAs (not a CTA's 16 warps over consecutive units), so that a work total that is not a
    // whole number of rounds leaves every SM the same number of warps' work
    const int64_t stride = (int64_t)gridDim.x * TAB_THREADS;
    const int64_t u0 = ((int64_t)(tid >> 5) * gridDim.x + blockIdx.x) * 32 + lane;

    // raw loads of a thread-unit (zeros beyond the end)
    auto load_unit = [&](int64_t uu, uint4* rx, uint4* rg) {
        const bool ok = uu < a.total_units;
        const int64_t cc = (uu >> log2Gt) * (int64_t)(C * Gt) + ((int)uu & (Gt - 1));
        #pragma unroll
        for (int k = 0; k < C; ++k) {
            rx[k] = make_uint4(0u, 0u, 0u, 0u);
            if (ok) rx[k] = __ldg(xin + cc + k * Gt);
            if (GLU) {
                rg[k] = make_uint4(0u, 0u, 0u, 0u);
                if (ok) rg[k] = __ldg(gin + cc + k * Gt);
            }
        }
    };
    #pragma unroll 1
    for (int64_t u = u0; u - lane < a.total_units; u += stride) {
        const bool valid = u < a.total_units;
        const int64_t bi = u >> log2Gt;                         // block index (flat over rows)
        const int g = (int)u & (Gt - 1);                        // lane of the block
        const int64_t c0 = bi * (int64_t)(C * Gt) + g;          // chunk k of this thread: c0 + k * Gt

        // ---- the thread's C chunks ----
        uint4 rx[C], rg[GLU ? C : 1];
        load_unit(u, rx, rg);
        uint32_t xb[C][4];
        #pragma unroll
        for (int k = 0; k < C; ++k) {
            xb[k][0] = rx[k].x; xb[k][1] = rx[k].y; xb[k][2] = rx[k].z; xb[k][3] = rx[k].w;
            if (GLU) {
                const uint32_t gb[4] = {rg[k].x, rg[k].y, rg[k].z, rg[k].w};
                #pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const float2 gg = __half22float2(bits_h2(gb[p])), uu = __half22float2(bits_h2(xb[k][p]));
                    const float s0 = rh(__fdiv_rn(gg.x, 1.f + expf(-gg.x))), s1 = rh(__fdiv_rn(gg.y, 1.f + expf(-gg.y)));
                    xb[k][p] = h2_bits(__floats2half2_rn(s0 * uu.x, s1 * uu.y));      // fp16 x fp16 is exact in fp32
                }
            }
        }
        if (a.in_bf16) {
            #pragma unroll
            for (int k = 0; k < C; ++k)
                #pragma unroll
                for (int p = 0; p < 4; ++p)
                    xb[k][p] = h2_bits(__floats2half2_rn(__uint_as_float(xb[k][p] << 16), __uint_as_float(xb[k][p] & 0xFFFF0000u)));
        }

        int64_t o0 = c0;                                        // where chunk 0 is stored
        if (KV) {
            const uint32_t row = valid ? (uint32_t)bi : 0u;
            int64_t orow;
            if (a.from_runs) {
                const uint32_t bh = row / a.kv_T, t = row - bh * a.kv_T, b = bh / a.kv_H, h = bh - b * a.kv_H;
                orow = ((int64_t)b * a.Tall + a.T0 + t) * a.kv_H + h;
            } else {
                const uint32_t bt = row / a.kv_H, h = row - bt * a.kv_H, b = bt / a.kv_T, t = bt - b * a.kv_T;
                kv_rows<C>(a, rope_cos, rope_sin, center, xb, bt, b, t, h, Gt, g);
                if (a.run) {
                    const uint32_t hk = h / a.group, hg = h - hk * a.group, c = t / a.run, tc = t - c * a.run;
                    orow = ((((int64_t)c * a.kv_B + b) * (a.kv_H / a.group) + hk) * a.group + hg) * a.run + tc;
                } else orow = ((int64_t)b * a.kv_H + h) * a.kv_T + t;
            }
            o0 = orow * (C * Gt) + g;
        }

        // ---- block maximum and the E5M3 shared scale (round-half-up of the 3-bit mantissa) ----
        uint32_t mx = 0u;
        #pragma unroll
        for (int k = 0; k < C; ++k)
            #pragma unroll
            for (int p = 0; p < 4; ++p) mx = h2_bits(__hmax2(bits_h2(mx), __habs2(bits_h2(xb[k][p]))));
        if (GT > 0) {
            #pragma unroll
            for (int off = GT >> 1; off >= 1; off >>= 1)
                mx = h2_bits(__hmax2(bits_h2(mx), bits_h2(__shfl_xor_sync(0xFFFFFFFFu, mx, off))));
        } else {
            for (int off = Gt >> 1; off >= 1; off >>= 1)
                mx = h2_bits(__hmax2(bits_h2(mx), bits_h2(__shfl_xor_sync(0xFFFFFFFFu, mx, off))));
        }
        const uint32_t am16 = max(mx & 0xFFFFu, mx >> 16);
        const float sf = __half2float(bits_h((uint16_t)am16)) * a.inv_ele_max;
        uint32_t sb = (uint32_t)h_bits(__float2half_rn(sf));
        sb = min(max(sb, 0x0400u), 0x7B80u);
        const uint32_t l1b = (sb + 0x40u) & 0xFF80u;
        const uint4 cst = s_l1c[l1b >> 7];

        // ---- the chunks: candidates' errors, choice, values ----
        uint32_t bests, amin;
        uint32_t codes[SIDE ? C : 1], sbits[SIDE ? C : 1];
        // value * t * l1 overflows fp16 only for blocks whose maximum is within 1 % of fp16's own: one
        // warp-uniform branch between the fused form and the form that keeps each product's rounding
        constexpr int TINY = KV ? 1 : 0;                        // a second read of the inputs would rotate them again
        if (__all_sync(0xFFFFFFFFu, l1b < a.big_l1)) amin = unit_chunks<MB, C, ML, true, SIDE, TINY>(a, dst, s_nt2, s_tabf, xb, l1b, cst, a.m_lanes, bests, codes, sbits);
        else amin = unit_chunks<MB, C, ML, false, SIDE, TINY>(a, dst, s_nt2, s_tabf, xb, l1b, cst, a.m_lanes, bests, codes, sbits);

        // The reference returns +0 (not -0) when fp16(a / t) is exactly zero.  Only quotients a below 2^-19
        // can do that; deciding it needs the exact a, where the scaled division may be off: rare, so the
        // inputs are read again and the quotients redone with true divisions.
        if (!KV && __hle2_mask(bits_h2(amin), bits_h2(0x00200020u)) != 0u && valid) {
            const float l1f = __half2float(bits_h((uint16_t)l1b));
            #pragma unroll
            for (int k = 0; k < C; ++k) {                  // unrolled: xb must stay in registers
                const float tc = s_tabf[(bests >> (2 * k)) & 3u];
                uint4 raw = __ldg(xin + c0 + k * Gt);
                uint32_t xr[4] = {raw.x, raw.y, raw.z, raw.w};
                if (GLU) {
                    const uint4 graw = __ldg(gin + c0 + k * Gt);
                    const uint32_t gb[4] = {graw.x, graw.y, graw.z, graw.w};
                    for (int p = 0; p < 4; ++p) {
                        const float2 gg = __half22float2(bits_h2(gb[p])), uu = __half22float2(bits_h2(xr[p]));
                        const float s0 = rh(__fdiv_rn(gg.x, 1.f + expf(-gg.x))), s1 = rh(__fdiv_rn(gg.y, 1.f + expf(-gg.y)));
                        xr[p] = h2_bits(__floats2half2_rn(s0 * uu.x, s1 * uu.y));
                    }
                }
                if (a.in_bf16)
                    for (int p = 0; p < 4; ++p)
                        xr[p] = h2_bits(__floats2half2_rn(__uint_as_float(xr[p] << 16), __uint_as_float(xr[p] & 0xFFFF0000u)));
                #pragma unroll
                for (int p = 0; p < 4; ++p)
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t xbits = (xr[p] >> (16 * h)) & 0xFFFFu;
                        if (xbits & 0x8000u) {
                            const float xf = __half2float(bits_h((uint16_t)(xbits & 0x7FFFu)));
                            if (rh(__fdiv_rn(rh(__fdiv_rn(xf, l1f)), tc)) == 0.f) {
                                xb[k][p] &= ~(0x8000u << (16 * h));
                                if (SIDE && MB == 1) codes[k] &= ~(8u << (4 * (2 * p + h)));
                                if (SIDE && MB == 2) sbits[k] &= ~(1u << (2 * p + h));
                            }
                        }
                    }
            }
        }

        // ---- stores ----
        uint32_t l2word = 0u;
        #pragma unroll
        for (int k = 0; k < C; ++k) {
            const int64_t ci = c0 + k * Gt;
            if (SIDE) {
                const int best = (int)((bests >> (2 * k)) & 3u);
                const int cib = g + k * Gt;                      // chunk index inside the block
                const int mbi = cib >> a.log2m;                  // its micro-block
                const bool leader = (g & (a.m_lanes - 1)) == 0;
                if (valid && a.out.codes) {
                    reinterpret_cast<uint32_t*>(a.out.codes)[ci] = codes[k];
                    if (MB == 2 && a.out.sign) a.out.sign[ci] = (uint8_t)sbits[k];
                }
                if (leader) {
                    if (a.out.l2_packed) l2word |= (uint32_t)best << (mbi * a.l2_sc_bit);
                    if (valid && a.out.l2_idx) a.out.l2_idx[bi * a.nl2 + mbi] = (uint8_t)best;
                }
            }
            if (valid && (!SIDE || a.deq)) {
                uint32_t dq[4] = {xb[k][0], xb[k][1], xb[k][2], xb[k][3]};
                if (a.out_bf16) {
                    #pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const float2 f = __half22float2(bits_h2(dq[p]));
                        __nv_bfloat162 bb = __floats2bfloat162_rn(f.x, f.y);
                        dq[p] = *reinterpret_cast<uint32_t*>(&bb);
                    }
                }
                a.deq[o0 + k * Gt] = make_uint4(dq[0], dq[1], dq[2], dq[3]);
            }
        }
        if (SIDE) store_block_side(a, bi, Gt, valid && g == 0, l1b, 0u, l2word);
    }
}


// ---- the two-table ("Mix") weight formats ----------------------------------------------------------------------
// Both candidate tables are evaluated, each with its own block scale; the one with the smaller fp16 total of the chosen
// candidates' squared errors over the block wins, the first on ties (src/quantizer.py:806-840).  Per scheme a chunk
// leaves its chosen candidate (2 bits), its eight winning value bytes (two registers) and its error sum, so that after
// the comparison only the values are formed: the division, the lookups and the candidates' errors are paid twice,
// everything else once.  The totals are added in the order of the tree over the block's chunks that the other kernels
// use (chunk distance 8, 4, 2, 1), so a sum that the fp32 additions round is the same number in all of them.
// Bound: instruction issue (about twice hbq_tab_kernel's work per element).  Weight [14336, 4096] to packed planes:
// 139 us; the arithmetic kernel of quantize.cu, which alone had these outputs, took 507 us.  The tensor alone: 118 us with
// micro-blocks of 8, 130 with 32 (NaNs put over the stored values; patched before the store: 122 and 127; infinities and
// NaNs read as zeros: 114 and 128).
// An infinite |x|, whose quotient comes out of the division as NaN, takes the largest level: the minimum, which drops
// the NaN, is the inner one.
template <int MB, int C, int ML, bool SMALL>
__device__ __forceinline__ void scheme_chunks(const uint32_t tab_addr, uint32_t base2, uint32_t hi2, uint32_t entry_bytes,
                                              const uint32_t* nt2, const uint32_t (*xb)[4], uint32_t l1b, const uint4 cst,
                                              int m_lanes, uint32_t& bests, uint32_t (*win)[2], float* err, uint32_t& amin)
{
    const __half2 pre2 = bits_h2(cst.x), post2 = bits_h2(cst.y), nm2 = bits_h2(cst.z), rm2 = bits_h2(cst.w);
    const uint32_t l1u = l1b * 0x00010001u;
    uint32_t tl[4];
    #pragma unroll
    for (int i = 0; i < 4; ++i) tl[i] = h2_bits(__hmul2(bits_h2(l1u), bits_h2(nt2[i])));
    bests = 0u;
    amin = 0x7C007C00u;
    const uint32_t addr0 = tab_addr - 4u * (base2 & 0xFFFFu);
    #pragma unroll
    for (int k = 0; k < C; ++k) {
        uint32_t ent[8];
        #pragma unroll
        for (int p = 0; p < 4; ++p) {
            const __half2 axs = __hmul2(__habs2(bits_h2(xb[k][p])), pre2);
            const __half2 q0 = __hmul2(axs, rm2);
            const __half2 r = __hfma2(q0, nm2, axs);
            const __half2 aa = __hmul2(__hfma2(r, rm2, q0), post2);
            amin = h2_bits(__hmin2(bits_h2(amin), aa));
            const uint32_t w = h2_bits(__hmax2(__hmin2(aa, bits_h2(hi2)), bits_h2(base2)));
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(ent[2 * p]) : "r"((w & 0xFFFFu) * entry_bytes + addr0));
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(ent[2 * p + 1]) : "r"((w >> 16) * entry_bytes + addr0));
        }
        float own[4], acc[4];
        chunk_errors<SMALL>(ent, xb[k], tl, nt2, l1u, own);
        #pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = own[i];
        if (ML > 0) {
            #pragma unroll
            for (int off = ML >> 1; off >= 1; off >>= 1) {
                #pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] += __shfl_xor_sync(0xFFFFFFFFu, acc[i], off);
            }
        } else {
            for (int off = m_lanes >> 1; off >= 1; off >>= 1) {
                #pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] += __shfl_xor_sync(0xFFFFFFFFu, acc[i], off);
            }
        }
        const uint32_t best = (uint32_t)first_min4(acc);
        bests |= best << (2 * k);
        const float e01 = (best & 1u) ? own[1] : own[0], e23 = (best & 1u) ? own[3] : own[2];
        err[k] = (best & 2u) ? e23 : e01;
        const uint32_t sel = best * 0x11u + 0x40u;              // byte `best` of both operands
        win[k][0] = prmt(prmt(ent[0], ent[1], sel), prmt(ent[2], ent[3], sel), 0x5410u);
        win[k][1] = prmt(prmt(ent[4], ent[5], sel), prmt(ent[6], ent[7], sel), 0x5410u);
    }
}

template <int MB, int GT, int ML, bool SIDE>
__global__ void __launch_bounds__(MIX_THREADS, 2) hbq_tab_mix_kernel(const TabArgs a)
{
    constexpr int C = 4;
    extern __shared__ __align__(128) uint32_t s_tab[];
    __shared__ uint4 s_l1c[256];
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ uint32_t s_nt2[8];
    __shared__ float s_tabf[8];
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t dst = stage_table<true>(a, s_tab, s_l1c, &s_bar, s_nt2, s_tabf, MIX_THREADS);
    grid_dependency_wait();
    dependents_may_start();
    const uint4* const xin = behind_wait(a.x);
    const int log2Gt = GT == 4 ? 2 : a.log2Gt;
    const int Gt = 1 << log2Gt;
    const int64_t stride = (int64_t)gridDim.x * MIX_THREADS;
    const int64_t u0 = ((int64_t)(tid >> 5) * gridDim.x + blockIdx.x) * 32 + lane;    // as in hbq_tab_kernel

    #pragma unroll 1
    for (int64_t u = u0; u - lane < a.total_units; u += stride) {
        const bool valid = u < a.total_units;
        const int64_t bi = u >> log2Gt;
        const int g = (int)u & (Gt - 1);
        const int64_t c0 = bi * (int64_t)(C * Gt) + g;
        uint32_t xb[C][4];
        #pragma unroll
        for (int k = 0; k < C; ++k) {
            const uint4 r = valid ? __ldg(xin + c0 + k * Gt) : make_uint4(0u, 0u, 0u, 0u);
            xb[k][0] = r.x; xb[k][1] = r.y; xb[k][2] = r.z; xb[k][3] = r.w;
        }
        if (a.in_bf16) {
            #pragma unroll
            for (int k = 0; k < C; ++k)
                #pragma unroll
                for (int p = 0; p < 4; ++p)
                    xb[k][p] = h2_bits(__floats2half2_rn(__uint_as_float(xb[k][p] << 16), __uint_as_float(xb[k][p] & 0xFFFF0000u)));
        }
        // The block maximum serves both schemes; their scales differ by the largest candidate.  It is taken with the
        // maximum that keeps a NaN (the same cost), so that blocks with one are known; a NaN does not count for the scale.
        uint32_t mx = 0u;
        #pragma unroll
        for (int k = 0; k < C; ++k)
            #pragma unroll
            for (int p = 0; p < 4; ++p) mx = h2_bits(__hmax2_nan(bits_h2(mx), __habs2(bits_h2(xb[k][p]))));
        for (int off = Gt >> 1; off >= 1; off >>= 1)
            mx = h2_bits(__hmax2_nan(bits_h2(mx), bits_h2(__shfl_xor_sync(0xFFFFFFFFu, mx, off))));
        const bool nans = max(mx & 0x7FFFu, (mx >> 16) & 0x7FFFu) > 0x7C00u;
        uint32_t nan_elems = 0u;                                 // tensor alone: element j of chunk k at bit 8 k + j
        if (__any_sync(0xFFFFFFFFu, nans)) {
            if (!SIDE) {
                #pragma unroll
                for (int k = 0; k < C; ++k)
                    #pragma unroll
                    for (int p = 0; p < 4; ++p)
                        nan_elems |= (((xb[k][p] & 0x7FFFu) > 0x7C00u ? 1u : 0u) | (((xb[k][p] >> 16) & 0x7FFFu) > 0x7C00u ? 2u : 0u)) << (8 * k + 2 * p);
            }
            mx = 0u;
            #pragma unroll
            for (int k = 0; k < C; ++k)
                #pragma unroll
                for (int p = 0; p < 4; ++p) mx = h2_bits(__hmax2(bits_h2(mx), __habs2(bits_h2(xb[k][p]))));
            for (int off = Gt >> 1; off >= 1; off >>= 1)
                mx = h2_bits(__hmax2(bits_h2(mx), bits_h2(__shfl_xor_sync(0xFFFFFFFFu, mx, off))));
        }
        const float amax = __half2float(bits_h((uint16_t)max(mx & 0xFFFFu, mx >> 16)));
        const uint32_t l1a = e5m3_scale(amax * a.inv_ele_max), l1c = e5m3_scale(amax * a.b.inv_ele_max);

        uint32_t bests, bests1, win[C][2], win1[C][2], amin, amin1;
        float err[C], err1[C];
        const bool small = __all_sync(0xFFFFFFFFu, l1a < a.big_l1 && l1c < a.b.big_l1);
        if (small) scheme_chunks<MB, C, ML, true>(dst, a.base2, a.hi2, a.entry_bytes, a.nt2, xb, l1a, s_l1c[l1a >> 7], a.m_lanes, bests, win, err, amin);
        else scheme_chunks<MB, C, ML, false>(dst, a.base2, a.hi2, a.entry_bytes, a.nt2, xb, l1a, s_l1c[l1a >> 7], a.m_lanes, bests, win, err, amin);
        const float tot = block_error<C>(err, Gt);
        const uint32_t dst1 = dst + (uint32_t)a.entries * 4u;
        if (small) scheme_chunks<MB, C, ML, true>(dst1, a.b.base2, a.b.hi2, a.entry_bytes, a.b.nt2, xb, l1c, s_l1c[l1c >> 7], a.m_lanes, bests1, win1, err1, amin1);
        else scheme_chunks<MB, C, ML, false>(dst1, a.b.base2, a.b.hi2, a.entry_bytes, a.b.nt2, xb, l1c, s_l1c[l1c >> 7], a.m_lanes, bests1, win1, err1, amin1);
        const float tot1 = block_error<C>(err1, Gt);
        const bool second = rh(tot1) < rh(tot);                  // the same in every lane of the block
        if (second) {
            bests = bests1; amin = amin1;
            #pragma unroll
            for (int k = 0; k < C; ++k) { win[k][0] = win1[k][0]; win[k][1] = win1[k][1]; }
        }
        const uint32_t l1b = second ? l1c : l1a, sidx = second ? 4u : 0u;
        const uint32_t l1u = l1b * 0x00010001u;
        const float l1f = __half2float(bits_h((uint16_t)l1b));
        const bool tiny = __hle2_mask(bits_h2(amin), bits_h2(0x00200020u)) != 0u;

        uint32_t l2word = 0u;
        #pragma unroll
        for (int k = 0; k < C; ++k) {
            const int64_t ci = c0 + k * Gt;
            const uint32_t best = (bests >> (2 * k)) & 3u;
            const uint32_t nt = s_nt2[sidx + best];
            const __half2 tlb = __hmul2(bits_h2(l1u), bits_h2(nt));
            uint32_t cw[4], sg[4], dq[4];
            #pragma unroll
            for (int p = 0; p < 4; ++p) {
                cw[p] = prmt(win[k][p >> 1], 0u, (p & 1) ? 0x3424u : 0x1404u);       // value bytes -> fp16 pair
                sg[p] = xb[k][p] & 0x80008000u;
            }
            if (tiny) {                                          // the reference's +0 where fp16(a / t) is zero (see unit_chunks)
                const float tc = s_tabf[sidx + best];
                #pragma unroll
                for (int p = 0; p < 4; ++p)
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t xbits = (xb[k][p] >> (16 * h)) & 0xFFFFu;
                        if (xbits & 0x8000u) {
                            const float xf = __half2float(bits_h((uint16_t)(xbits & 0x7FFFu)));
                            if (rh(__fdiv_rn(rh(__fdiv_rn(xf, l1f)), tc)) == 0.f) sg[p] &= ~(0x8000u << (16 * h));
                        }
                    }
            }
            #pragma unroll
            for (int p = 0; p < 4; ++p) {
                const __half2 dneg = small ? __hmul2(bits_h2(cw[p]), tlb) : __hmul2(__hmul2(bits_h2(cw[p]), bits_h2(nt)), bits_h2(l1u));
                dq[p] = (h2_bits(dneg) & 0x7FFF7FFFu) | sg[p];
            }
            if (SIDE && nans) {                                  // a NaN stays one in the tensor; its code has all bits set (E2M2: no sign)
                #pragma unroll
                for (int p = 0; p < 4; ++p)
                    #pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (((xb[k][p] >> (16 * h)) & 0x7FFFu) > 0x7C00u) {
                            dq[p] = (dq[p] & ~(0xFFFFu << (16 * h))) | (0x7FFFu << (16 * h));
                            sg[p] = MB == 1 ? sg[p] | (0x8000u << (16 * h)) : sg[p] & ~(0x8000u << (16 * h));
                        }
            }
            if (SIDE) {
                const int mbi = (g + k * Gt) >> a.log2m;
                const bool leader = (g & (a.m_lanes - 1)) == 0;
                if (valid && a.out.codes) {
                    uint32_t sb = 0u;
                    reinterpret_cast<uint32_t*>(a.out.codes)[ci] = pack_codes<MB>(cw, sg, sb);
                    if (MB == 2 && a.out.sign) a.out.sign[ci] = (uint8_t)sb;
                }
                if (leader) {
                    if (a.out.l2_packed) l2word |= best << (mbi * a.l2_sc_bit);
                    if (valid && a.out.l2_idx) a.out.l2_idx[bi * a.nl2 + mbi] = (uint8_t)best;
                }
            }
            if (valid && a.deq) {
                if (a.out_bf16) {
                    #pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const float2 f = __half22float2(bits_h2(dq[p]));
                        const __nv_bfloat162 bb = __floats2bfloat162_rn(f.x, f.y);
                        dq[p] = *reinterpret_cast<const uint32_t*>(&bb);
                    }
                }
                a.deq[ci] = make_uint4(dq[0], dq[1], dq[2], dq[3]);
            }
        }
        if (SIDE) store_block_side(a, bi, Gt, valid && g == 0, l1b, second ? 1u : 0u, l2word);
        else if (nan_elems != 0u && valid)                       // NaNs over what the chunks stored for them
            for (uint32_t m = nan_elems; m != 0u; m &= m - 1u) {
                const int i = __ffs(m) - 1;
                reinterpret_cast<uint16_t*>(a.deq + c0 + (i >> 3) * Gt)[i & 7] = 0x7FFFu;
            }
    }
}


// ---- V-cache write: blocks of 128 consecutive TOKENS per (batch, head, channel) --------------------------------
// A CTA of 256 threads takes a tile of 128 tokens x 64 channels of [B, T, H, D], turns it through shared memory and
// hands every channel's block to the table quantizer with the geometry of the activation kernel (four lanes a block,
// four chunks a lane).  The tile is kept as one row of 64 token-PAIR words per channel, so that a chunk is one 16-byte
// word: a thread of the load and store phases holds two tokens x 8 channels and regroups them with byte permutes.
// 16-byte granules of a row are XOR-swizzled by the channel: the load phase's 8 segments x 4 words and a quarter
// warp's 2 channels x 4 chunks each cover all 32 banks.  Tokens beyond T are the reference's zero padding.
// Bound: instruction issue, as hbq_tab_kernel.  V of [4, 1999, 8 x 128] fp16: 28.0 us with the
// 8-byte tables and one chunk a lane, 17.0 us here.
constexpr int TABV_THREADS = 256, TABV_D = 64, TABV_T = 128;
constexpr int TABV_TILE_WORDS = TABV_D * TABV_T / 2;

__device__ __forceinline__ int tabv_word(int d, int tp)
{
    return d * (TABV_T / 2) + ((((tp >> 2) ^ ((d >> 3) & 7) ^ ((d & 1) << 2)) << 2) | (tp & 3));
}

template <int MB, int ML>
__global__ void __launch_bounds__(TABV_THREADS, 4) hbq_tab_v_kernel(const TabArgs a, const VArgs v)
{
    extern __shared__ __align__(128) uint32_t s_tab[];
    __shared__ __align__(16) uint32_t tile[TABV_TILE_WORDS];
    __shared__ uint4 s_l1c[256];
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ uint32_t s_nt2[4];
    __shared__ float s_tabf[4];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t dst = stage_table(a, s_tab, s_l1c, &s_bar, s_nt2, s_tabf, TABV_THREADS);
    grid_dependency_wait();
    dependents_may_start();
    const uint16_t* const vin = behind_wait(v.in);
    const int seg = tid & 7;                                     // load / store phases: 8 channels
    #pragma unroll 1
    for (int64_t tl = blockIdx.x; tl < v.tiles; tl += gridDim.x) {
        const int ds = (int)(tl % v.dslabs);
        const int64_t rest = tl / v.dslabs;
        const int tb = (int)(rest % v.tblocks);
        const int64_t bh = rest / v.tblocks;
        const int64_t b = bh / v.H, h = bh - b * v.H;
        const int64_t t0 = (int64_t)tb * TABV_T;
        const int d0 = ds * TABV_D + seg * 8;
        const uint16_t* src = vin + ((b * v.T * v.H + h) * v.D + d0);

        uint4 ld[4];
        #pragma unroll
        for (int r = 0; r < 4; ++r) {                            // tokens 2 tp, 2 tp + 1 of tp = tid / 8 and tid / 8 + 32
            const int64_t t = t0 + 2 * ((tid >> 3) + 32 * (r >> 1)) + (r & 1);
            ld[r] = make_uint4(0u, 0u, 0u, 0u);
            if (t < v.T) ld[r] = __ldg(reinterpret_cast<const uint4*>(src + t * v.H * v.D));
        }
        #pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int tp = (tid >> 3) + 32 * r;
            uint32_t e[4] = {ld[2 * r].x, ld[2 * r].y, ld[2 * r].z, ld[2 * r].w};
            uint32_t o[4] = {ld[2 * r + 1].x, ld[2 * r + 1].y, ld[2 * r + 1].z, ld[2 * r + 1].w};
            #pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (v.in_bf16) {
                    e[i] = h2_bits(__floats2half2_rn(__uint_as_float(e[i] << 16), __uint_as_float(e[i] & 0xFFFF0000u)));
                    o[i] = h2_bits(__floats2half2_rn(__uint_as_float(o[i] << 16), __uint_as_float(o[i] & 0xFFFF0000u)));
                }
                tile[tabv_word(seg * 8 + 2 * i, tp)] = prmt(e[i], o[i], 0x5410u);
                tile[tabv_word(seg * 8 + 2 * i + 1, tp)] = prmt(e[i], o[i], 0x7632u);
            }
        }
        __syncthreads();
        {
            const int d = warp * 8 + (lane >> 2), g = lane & 3;
            uint32_t xb[4][4];
            #pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint4 c = *reinterpret_cast<const uint4*>(tile + tabv_word(d, (g + 4 * k) * 4));
                xb[k][0] = c.x; xb[k][1] = c.y; xb[k][2] = c.z; xb[k][3] = c.w;
            }
            const uint32_t l1b = unit_scale<4>(xb, 4, a.inv_ele_max);
            const uint4 cst = s_l1c[l1b >> 7];
            uint32_t bests, nocodes[1], nosigns[1];
            if (__all_sync(0xFFFFFFFFu, l1b < a.big_l1)) unit_chunks<MB, 4, ML, true, false, 1>(a, dst, s_nt2, s_tabf, xb, l1b, cst, ML, bests, nocodes, nosigns);
            else unit_chunks<MB, 4, ML, false, false, 1>(a, dst, s_nt2, s_tabf, xb, l1b, cst, ML, bests, nocodes, nosigns);
            #pragma unroll
            for (int k = 0; k < 4; ++k)
                *reinterpret_cast<uint4*>(tile + tabv_word(d, (g + 4 * k) * 4)) = make_uint4(xb[k][0], xb[k][1], xb[k][2], xb[k][3]);
        }
        __syncthreads();
        #pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int tp = (tid >> 3) + 32 * r;
            uint32_t w[2][4];
            #pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t c0 = tile[tabv_word(seg * 8 + 2 * i, tp)], c1 = tile[tabv_word(seg * 8 + 2 * i + 1, tp)];
                w[0][i] = prmt(c0, c1, 0x5410u);
                w[1][i] = prmt(c0, c1, 0x7632u);
            }
            #pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int64_t t = t0 + 2 * tp + j;
                if (t >= v.T) continue;
                if (v.out_bf16) {
                    #pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __half22float2(bits_h2(w[j][i]));
                        const __nv_bfloat162 bb = __floats2bfloat162_rn(f.x, f.y);
                        w[j][i] = *reinterpret_cast<const uint32_t*>(&bb);
                    }
                }
                const int64_t orow = v.out_token_major ? (b * v.T + t) * v.H + h : (b * v.H + h) * v.T + t;
                *reinterpret_cast<uint4*>(v.out + (orow * v.D + d0)) = make_uint4(w[j][0], w[j][1], w[j][2], w[j][3]);
            }
        }
        __syncthreads();
    }
}

// ---- row kernels: a per-row prologue fused in front of the quantizer --------------------------------
// Two activation quantizers of the attention / MLP blocks consume a tensor that only exists to be quantised
// and whose producer needs a whole-row reduction first:
//   RMSNORM  the input of q/k/v_proj and gate/up_proj: aq(weight * rmsnorm(x [+ residual])) (the decoder
//            layer's input_layernorm / post_attention_layernorm followed by _QBaseLinear.forward's
//            self.aq(x), src/module.py:45); the sum x + residual is also written (the new residual stream);
//   SOFTMAX  the attention probabilities: attn_wgt_quantizer.q(softmax(q k^T * scale + bias)) along the key
//            axis (manual_sdpa, src/module.py:108-115).
// One warp owns a row.  It sweeps the row for the reduction (sum of squares; maximum, then sum of exponentials),
// then sweeps it again (from L1 / L2) to form the fp16 values with the reference's per-op roundings and hands
// each 128-element block straight to the table quantizer above -- the normalised tensor / the probabilities
// never go to HBM unquantised.  Geometry: blocks of 128, four lanes per block, four chunks per lane.
enum { ROW_RMSNORM = 0, ROW_SOFTMAX = 1 };
constexpr int ROW_THREADS = 512;
constexpr int ROW_WARPS = ROW_THREADS / 32;

struct RowArgs {
    TabArgs t;                // the quantizer's format (table, candidates); t.x / t.deq unused
    const uint4* in;          // [rows, K] fp16: x (RMSNORM) or the raw scores q k^T (SOFTMAX)
    uint4* out;               // [rows, K] fp16
    int64_t rows;
    int K, nblk;              // row length, 128-element blocks per row
    // RMSNORM
    const uint4* res;         // residual to add first, or NULL
    uint4* x_out;             // where x + residual goes (required with res)
    const uint4* w;           // weight [K] fp16
    float eps;
    // SOFTMAX
    float scale;              // the score scale (a Python float in the reference: applied in fp32)
    int causal;               // key j of query row r is masked when j > (r % L) + key_offset
    int64_t L, HL, key_offset;
    const uint4* mask;        // additive fp16 mask [mask_batches, L, K] or NULL (row r uses batch r / HL, query r % L)
    int64_t mask_batches;
};
static_assert(sizeof(RowArgs) <= 4000, "kernel parameters are limited to 4 KB");

// Reductions over the W lanes that share a row (a whole warp, or one of its halves).
template <int W>
__device__ __forceinline__ float lanes_sum(float v)
{
    #pragma unroll
    for (int off = W / 2; off >= 1; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
    return v;
}
template <int W>
__device__ __forceinline__ float lanes_max(float v)
{
    #pragma unroll
    for (int off = W / 2; off >= 1; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, off));
    return v;
}

// -inf into the halves of a packed pair whose key index (j0, j0 + 1) lies beyond the causal limit.
__device__ __forceinline__ uint32_t mask_beyond(uint32_t b, int64_t j0, int64_t limit)
{
    if (j0 > limit) b = (b & 0xFFFF0000u) | 0x0000FC00u;
    if (j0 + 1 > limit) b = (b & 0x0000FFFFu) | 0xFC000000u;
    return b;
}

// The pre-softmax score chunk as the reference's fp16 ops leave it: fp16(fp16(s * scale) + bias), bias = the
// additive mask and / or -inf beyond the causal limit.  cir: chunk index in the row.
__device__ __forceinline__ void score_chunk(const RowArgs& a, const uint4* rin, const uint4* rmask, int cir, int64_t limit,
                                            uint32_t* sv)
{
    const uint4 raw = __ldg(rin + cir);
    const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
    uint32_t m[4] = {0u, 0u, 0u, 0u};
    if (rmask) { const uint4 mv = __ldg(rmask + cir); m[0] = mv.x; m[1] = mv.y; m[2] = mv.z; m[3] = mv.w; }
    #pragma unroll
    for (int p = 0; p < 4; ++p) {
        // tensor * Python scalar: torch multiplies in fp32 with the scalar as fp32 and rounds the product to fp16
        const float2 sf = __half22float2(bits_h2(r[p]));
        __half2 v = __floats2half2_rn(sf.x * a.scale, sf.y * a.scale);
        if (rmask) v = __hadd2(v, bits_h2(m[p]));
        sv[p] = h2_bits(v);
    }
    if ((int64_t)cir * 8 + 7 > limit) {                      // the chunk that holds the causal limit (or lies beyond it)
        #pragma unroll
        for (int p = 0; p < 4; ++p) sv[p] = mask_beyond(sv[p], (int64_t)cir * 8 + 2 * p, limit);
    }
}

// fp32 quotient a / b, correctly rounded, from r = RN(1 / b): first guess, its exact residual, one correction
// (Markstein's sequence).  b is a softmax row sum (>= 1 when finite); NaN and Inf operands end in NaN like a / b.
__device__ __forceinline__ float div_by_sum(float a, float b, float r)
{
    const float q0 = a * r;
    const float rem = fmaf(-q0, b, a);
    return fmaf(rem, r, q0);
}

template <int MB, int ML, int PRO, bool QUANT>
__global__ void __launch_bounds__(ROW_THREADS, 2) hbq_row_kernel(const RowArgs a)
{
    extern __shared__ __align__(128) uint32_t s_tab[];
    __shared__ uint4 s_l1c[256];
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ uint32_t s_nt2[4];
    __shared__ float s_tabf[4];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t dst = 0u;
    if (QUANT) dst = stage_table(a.t, s_tab, s_l1c, &s_bar, s_nt2, s_tabf, ROW_THREADS);
    grid_dependency_wait();
    dependents_may_start();
    const uint4* const ain = behind_wait(a.in);
    const uint4* const ares = PRO == ROW_RMSNORM ? behind_wait(a.res) : nullptr;
    const uint4* const aw = PRO == ROW_RMSNORM ? behind_wait(a.w) : nullptr;
    const uint4* const amask = PRO == ROW_SOFTMAX ? behind_wait(a.mask) : nullptr;
    // RMSNorm: one row per warp, 8 blocks (1024 elements) per iteration.  Softmax: one row per half-warp, 4 blocks
    // per iteration -- a causal row ends anywhere, and the masked blocks of its last iteration are lanes without
    // work (1.5 blocks on average instead of 3.5).
    constexpr int RPW = PRO == ROW_SOFTMAX ? 2 : 1;          // rows per warp
    constexpr int BPI = 8 / RPW;                             // blocks of a row per iteration
    constexpr int RL = 32 / RPW;                             // lanes of a row
    const int sub = lane / RL;
    const int bl = (lane >> 2) & (BPI - 1), g = lane & 3;    // block of the iteration, lane of the block
    const int cpr = a.K >> 3;                                // chunks per row
    const int iters_all = (a.nblk + BPI - 1) / BPI;

    #pragma unroll 1
    // warps take turns over the CTAs: the rows of one CTA then lie far apart, so that causal rows of every length and the
    // rows of a last partial round are spread over the SMs
    for (int64_t rb = ((int64_t)warp * gridDim.x + blockIdx.x) * RPW; rb < a.rows; rb += (int64_t)gridDim.x * ROW_WARPS * RPW) {
        int64_t row = rb + sub;
        const bool live = row < a.rows;                      // odd row count: the idle half repeats the last row, stores nothing
        if (!live) row = a.rows - 1;
        const uint4* rin = ain + row * cpr;
        uint4* rout = a.out + row * cpr;
        float stat0 = 0.f, stat1 = 0.f;                      // RMSNORM: rstd; SOFTMAX: max, sum
        int iters = iters_all;
        int64_t limit = (int64_t)a.K;                        // SOFTMAX: last unmasked key
        const uint4* rmask = nullptr;
        const uint4* rsrc = rin;                             // what the second sweep reads

        if (PRO == ROW_RMSNORM) {
            float ss = 0.f;
            uint4* rx = a.x_out ? a.x_out + row * cpr : nullptr;
            const uint4* rres = ares ? ares + row * cpr : nullptr;
            if (rres) rsrc = rx;
            for (int it = 0; it < iters; ++it) {
                const int blk = it * BPI + bl;
                if (blk < a.nblk) {
                    #pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int ci = blk * 16 + g + 4 * k;
                        if (ci >= cpr) continue;                 // ragged last block (unquantised form only)
                        uint4 v = __ldg(rin + ci);
                        if (rres) {
                            const uint4 rv = __ldg(rres + ci);
                            v.x = h2_bits(__hadd2(bits_h2(v.x), bits_h2(rv.x))); v.y = h2_bits(__hadd2(bits_h2(v.y), bits_h2(rv.y)));
                            v.z = h2_bits(__hadd2(bits_h2(v.z), bits_h2(rv.z))); v.w = h2_bits(__hadd2(bits_h2(v.w), bits_h2(rv.w)));
                            rx[ci] = v;
                        }
                        const uint32_t q[4] = {v.x, v.y, v.z, v.w};
                        #pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            const float2 f = __half22float2(bits_h2(q[p]));
                            ss = fmaf(f.x, f.x, ss); ss = fmaf(f.y, f.y, ss);
                        }
                    }
                }
            }
            ss = lanes_sum<32>(ss);
            stat0 = rsqrtf(ss / (float)a.K + a.eps);
        } else {
            const int64_t qpos = row % a.L;
            if (a.causal) limit = qpos + a.key_offset;
            if (limit > (int64_t)a.K - 1) limit = (int64_t)a.K - 1;
            if (amask) rmask = amask + ((a.mask_batches > 1 ? row / a.HL : 0) * a.L + qpos) * cpr;
            // whole iterations beyond the causal limit hold only masked keys: probabilities 0
            iters = min(iters_all, (int)(limit / (128 * BPI)) + 1);
            float mx = -INFINITY;
            if (!rmask && a.scale > 0.f) {
                // rounding is monotonic, so the largest scaled score is the scaled largest score: one max per pair
                __half2 m2 = bits_h2(0xFC00FC00u);
                for (int it = 0; it < iters; ++it) {
                    const int blk = it * BPI + bl;
                    #pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int ci = blk * 16 + g + 4 * k;
                        const int64_t j0 = (int64_t)ci * 8;
                        if (ci >= cpr || j0 > limit) continue;
                        const uint4 raw = __ldg(rin + ci);
                        uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
                        if (j0 + 7 > limit) {
                            #pragma unroll
                            for (int p = 0; p < 4; ++p) r[p] = mask_beyond(r[p], j0 + 2 * p, limit);
                        }
                        m2 = __hmax2(m2, __hmax2(__hmax2(bits_h2(r[0]), bits_h2(r[1])), __hmax2(bits_h2(r[2]), bits_h2(r[3]))));
                    }
                }
                mx = lanes_max<RL>(fmaxf(__low2float(m2), __high2float(m2)));
                mx = __half2float(__float2half_rn(mx * a.scale));
            } else {
                for (int it = 0; it < iters; ++it) {
                    const int blk = it * BPI + bl;
                    #pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        uint32_t sv[4];
                        const int ci = blk * 16 + g + 4 * k;
                        if (ci >= cpr) continue;
                        score_chunk(a, rin, rmask, ci, limit, sv);
                        const __half2 m2 = __hmax2(__hmax2(bits_h2(sv[0]), bits_h2(sv[1])), __hmax2(bits_h2(sv[2]), bits_h2(sv[3])));
                        mx = fmaxf(mx, fmaxf(__low2float(m2), __high2float(m2)));
                    }
                }
                mx = lanes_max<RL>(mx);
            }
            float sum = 0.f;
            for (int it = 0; it < iters; ++it) {
                const int blk = it * BPI + bl;
                #pragma unroll
                for (int k = 0; k < 4; ++k) {
                    uint32_t sv[4];
                    const int ci = blk * 16 + g + 4 * k;
                    if (ci >= cpr || (int64_t)ci * 8 > limit) continue;      // masked keys add exp(-inf) = 0
                    score_chunk(a, rin, rmask, ci, limit, sv);
                    #pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const float2 f = __half22float2(bits_h2(sv[p]));
                        sum += expf(f.x - mx); sum += expf(f.y - mx);
                    }
                }
            }
            __syncwarp();
            stat0 = mx;
            stat1 = lanes_sum<RL>(sum);
        }

        // ---- second sweep: the fp16 values, block by block into the quantizer ----
        int iters_w = iters;                                 // the quantizer's shuffles need the whole warp in every iteration
        float rsum = 0.f;
        if (PRO == ROW_SOFTMAX) {
            iters_w = max(iters, __shfl_xor_sync(0xFFFFFFFFu, iters, 16));
            rsum = __frcp_rn(stat1);
        }
        for (int it = 0; it < iters_all; ++it) {
            const int blk = it * BPI + bl;
            const bool valid = blk < a.nblk && live;
            if (PRO == ROW_SOFTMAX && it >= iters_w) {       // only masked keys: zeros (warp-uniform branch)
                if (valid) {
                    #pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (blk * 16 + g + 4 * k < cpr) rout[blk * 16 + g + 4 * k] = make_uint4(0u, 0u, 0u, 0u);
                }
                continue;
            }
            uint32_t xb[4][4];
            #pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int ci = blk * 16 + g + 4 * k;
                #pragma unroll
                for (int p = 0; p < 4; ++p) xb[k][p] = 0u;
                if (blk >= a.nblk || ci >= cpr) continue;
                if (PRO == ROW_RMSNORM) {
                    // weight * fp16(x_f32 * rstd): the rounding points of transformers' LlamaRMSNorm on an fp16 tensor
                    const uint4 v = ares ? rsrc[ci] : __ldg(rsrc + ci), wv = __ldg(aw + ci);
                    const uint32_t q[4] = {v.x, v.y, v.z, v.w}, ww[4] = {wv.x, wv.y, wv.z, wv.w};
                    #pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const float2 f = __half22float2(bits_h2(q[p]));
                        xb[k][p] = h2_bits(__hmul2(bits_h2(ww[p]), __floats2half2_rn(f.x * stat0, f.y * stat0)));
                    }
                } else {
                    if ((int64_t)ci * 8 > limit) continue;   // masked keys: exp(-inf) / sum = 0
                    uint32_t sv[4];
                    score_chunk(a, rin, rmask, ci, limit, sv);
                    #pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const float2 f = __half22float2(bits_h2(sv[p]));
                        xb[k][p] = h2_bits(__floats2half2_rn(div_by_sum(expf(f.x - stat0), stat1, rsum),
                                                             div_by_sum(expf(f.y - stat0), stat1, rsum)));
                    }
                }
            }
            if (QUANT) {
                const uint32_t l1b = unit_scale<4>(xb, 4, a.t.inv_ele_max);
                const uint4 cst = s_l1c[l1b >> 7];
                uint32_t bests;
                uint32_t nocodes[1], nosigns[1];
                constexpr int TINY = PRO == ROW_SOFTMAX ? 2 : 1;
                if (__all_sync(0xFFFFFFFFu, l1b < a.t.big_l1)) unit_chunks<MB, 4, ML, true, false, TINY>(a.t, dst, s_nt2, s_tabf, xb, l1b, cst, ML, bests, nocodes, nosigns);
                else unit_chunks<MB, 4, ML, false, false, TINY>(a.t, dst, s_nt2, s_tabf, xb, l1b, cst, ML, bests, nocodes, nosigns);
            }
            if (valid) {
                #pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (blk * 16 + g + 4 * k < cpr) rout[blk * 16 + g + 4 * k] = make_uint4(xb[k][0], xb[k][1], xb[k][2], xb[k][3]);
            }
        }
    }
}

// ---- host side ------------------------------------------------------------------------------------
static std::mutex g_tab_mutex;
static uint32_t* g_tab_dev[kMaxDevices];                 // device address of g_tab_slots, per device
static bool g_tab_ready[kMaxDevices][TAB_SLOTS];         // the slot holds its format's table on that device

// Device address of the format's table on the current device, uploading it at the first use there.  The
// upload is followed by a stream synchronisation (once per format and device), so it cannot happen while
// the stream is being captured: *addr stays NULL then and the caller takes another kernel.
static int table_on_device(const TabTable& t, cudaStream_t stream, const uint32_t** addr)
{
    *addr = nullptr;
    int dev = 0;
    HBQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return HBQ_ERR_DEVICE;
    std::lock_guard<std::mutex> lock(g_tab_mutex);
    if (!g_tab_ready[dev][t.slot]) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess) { (void)cudaGetLastError(); return HBQ_OK; }
        if (cs != cudaStreamCaptureStatusNone) return HBQ_OK;
        if (!g_tab_dev[dev]) {
            void* p = nullptr;
            HBQ_CUDA_TRY(cudaGetSymbolAddress(&p, g_tab_slots));
            g_tab_dev[dev] = (uint32_t*)p;
        }
        HBQ_CUDA_TRY(cudaMemcpyAsync(g_tab_dev[dev] + (size_t)t.slot * TAB_MAX_ENTRIES, t.host, (size_t)t.entries * 4,
                                     cudaMemcpyHostToDevice, stream));
        HBQ_CUDA_TRY(cudaStreamSynchronize(stream));
        g_tab_ready[dev][t.slot] = true;
    }
    *addr = g_tab_dev[dev] + (size_t)t.slot * TAB_MAX_ENTRIES;
    return HBQ_OK;
}

// CTAs for a number of thread-units: as many as are resident at once, each with at least four warps' work -- small
// tensors are spread over the SMs (HBQ-A activations [33, 14336]: 4.8 us with 16 warps' work a CTA, 3.4 with four, 3.8
// with two or one; [8, 4096]: 4.6, 3.1, 3.0), where staging the table costs each CTA the same.
constexpr int TAB_MIN_WARPS = 4;
static int tab_grid(int64_t total_units, int64_t cap)
{
    const int64_t need = (total_units + 32 * TAB_MIN_WARPS - 1) / (32 * TAB_MIN_WARPS);
    return (int)(need < cap ? need : cap);
}

template <int MB, int C, int GT, int ML, bool SIDE, bool GLU, bool KV = false>
static int launch_tab(const TabArgs& a, size_t smem, cudaStream_t stream)
{
    int sms = 0, per_sm = 0;
    { const int rc = device_sms(&sms); if (rc) return rc; }
    { const int rc = ensure_dynamic_smem(hbq_tab_kernel<MB, C, GT, ML, SIDE, GLU, KV>, smem); if (rc) return rc; }
    { const int rc = resident_ctas(hbq_tab_kernel<MB, C, GT, ML, SIDE, GLU, KV>, TAB_THREADS, smem, &per_sm); if (rc) return rc; }
    const int grid = tab_grid(a.total_units, (int64_t)sms * per_sm);
    HBQ_CUDA_TRY(launch_dependent(hbq_tab_kernel<MB, C, GT, ML, SIDE, GLU, KV>, grid, TAB_THREADS, smem, stream, a));
    HBQ_LAUNCH_CHECK("hbq_tab_kernel");
    return HBQ_OK;
}

template <int MB, int C, int GT, int ML>
static int launch_tab_variant(const TabArgs& a, bool side, bool glu, size_t smem, cudaStream_t stream)
{
    if (glu) return launch_tab<MB, C, GT, ML, false, true>(a, smem, stream);
    if (side) return launch_tab<MB, C, GT, ML, true, false>(a, smem, stream);
    return launch_tab<MB, C, GT, ML, false, false>(a, smem, stream);
}

template <int MB, int GT, int ML, bool SIDE>
static int launch_mix(const TabArgs& a, size_t smem, cudaStream_t stream)
{
    int sms = 0, per_sm = 0;
    { const int rc = device_sms(&sms); if (rc) return rc; }
    { const int rc = ensure_dynamic_smem(hbq_tab_mix_kernel<MB, GT, ML, SIDE>, smem); if (rc) return rc; }
    { const int rc = resident_ctas(hbq_tab_mix_kernel<MB, GT, ML, SIDE>, MIX_THREADS, smem, &per_sm); if (rc) return rc; }
    HBQ_CUDA_TRY(launch_dependent(hbq_tab_mix_kernel<MB, GT, ML, SIDE>, tab_grid(a.total_units, (int64_t)sms * per_sm), MIX_THREADS, smem, stream, a));
    HBQ_LAUNCH_CHECK("hbq_tab_mix_kernel");
    return HBQ_OK;
}

template <int MB>
static int launch_mix_geometry(const TabArgs& a, int Gt, int m, bool side, size_t smem, cudaStream_t stream)
{
    if (Gt == 4 && m == 1) return side ? launch_mix<MB, 4, 1, true>(a, smem, stream) : launch_mix<MB, 4, 1, false>(a, smem, stream);
    if (Gt == 4 && m == 4) return side ? launch_mix<MB, 4, 4, true>(a, smem, stream) : launch_mix<MB, 4, 4, false>(a, smem, stream);
    return side ? launch_mix<MB, 0, 0, true>(a, smem, stream) : launch_mix<MB, 0, 0, false>(a, smem, stream);
}

// The shipped configurations (block 128: 4 chunks per thread, 4 lanes per block; micro-block 8 or 32) have
// their lane counts compiled in; every other geometry runs the same kernel with run-time loop bounds.
template <int MB>
static int launch_tab_geometry(const TabArgs& a, int C, int Gt, int m, bool side, bool glu, size_t smem, cudaStream_t stream)
{
    if (a.kv_T) {                                            // C == 4
        if (Gt == 4 && m == 1) return launch_tab<MB, 4, 4, 1, false, false, true>(a, smem, stream);
        if (Gt == 4 && m == 4) return launch_tab<MB, 4, 4, 4, false, false, true>(a, smem, stream);
        return launch_tab<MB, 4, 0, 0, false, false, true>(a, smem, stream);
    }
    if (C == 4 && Gt == 4 && m == 1) return launch_tab_variant<MB, 4, 4, 1>(a, side, glu, smem, stream);
    if (C == 4 && Gt == 4 && m == 4) return launch_tab_variant<MB, 4, 4, 4>(a, side, glu, smem, stream);
    if (C == 4) return launch_tab_variant<MB, 4, 0, 0>(a, side, glu, smem, stream);
    return launch_tab_variant<MB, 2, 0, 0>(a, side, glu, smem, stream);
}

// Fill the format part of the arguments shared by every kernel of this file (table on the device, candidates,
// scale constants).  *ok = false when the format has no byte table or its table cannot be uploaded now.
static int fill_format(const QArgs& q, int mb, cudaStream_t stream, TabArgs* a, bool* ok)
{
    *ok = false;
    TabTable t;
    if (!hbq_tab_table(mb, q.tab[0], q.nc, &t) || t.slot >= TAB_SLOTS || t.entries > TAB_MAX_ENTRIES) return HBQ_OK;
    memset(a, 0, sizeof(*a));
    { const int rc = table_on_device(t, stream, &a->table); if (rc) return rc; }
    if (!a->table) return HBQ_OK;
    a->entries = t.entries;
    a->entry_bytes = 4u;
    a->base2 = (uint32_t)t.base * 0x00010001u;
    a->hi2 = (uint32_t)t.hi * 0x00010001u;
    a->big_l1 = t.big_l1;
    a->inv_ele_max = 1.f / q.ele_max[0];
    for (int i = 0; i < 4; ++i) {
        const float tv = q.tab[0][i < q.nc ? i : q.nc - 1];     // unused slots repeat the last candidate: they never win a tie
        a->tabf[i] = tv;
        a->nt2[i] = (uint32_t)__half_as_ushort(__float2half_rn(-tv)) * 0x00010001u;
    }
    memcpy(a->rm, t.rm, sizeof(a->rm));
    *ok = true;
    return HBQ_OK;
}

template <int MB, int ML, int PRO>
static int launch_row(const RowArgs& a, bool quant, cudaStream_t stream)
{
    int sms = 0;
    { const int rc = device_sms(&sms); if (rc) return rc; }
    const size_t smem = quant ? (size_t)a.t.entries * 4 : 0;
    constexpr int RPW = PRO == ROW_SOFTMAX ? 2 : 1;
    const int64_t need = (a.rows + RPW * TAB_MIN_WARPS - 1) / (RPW * TAB_MIN_WARPS);
    const int grid = (int)(need < 2ll * sms ? need : 2ll * sms);
    if (quant) {
        { const int rc = ensure_dynamic_smem(hbq_row_kernel<MB, ML, PRO, true>, smem); if (rc) return rc; }
        HBQ_CUDA_TRY(launch_dependent(hbq_row_kernel<MB, ML, PRO, true>, grid, ROW_THREADS, smem, stream, a));
    } else {
        HBQ_CUDA_TRY(launch_dependent(hbq_row_kernel<MB, ML, PRO, false>, grid, ROW_THREADS, 0, stream, a));
    }
    HBQ_LAUNCH_CHECK("hbq_row_kernel");
    return HBQ_OK;
}

// q: the validated HBQ format (QArgs as quantize_launch builds it), or NULL for the prologue alone.  Returns
// HBQ_ERR_UNSUPPORTED when the format does not fit the fused kernel (the caller then runs the prologue alone
// and the plain quantizer).
int hbq_row_launch(int pro, const QArgs* q, int mb, RowArgs& a, cudaStream_t stream)
{
    if (a.rows == 0 || a.K == 0) return HBQ_OK;
    if ((a.K % 8) != 0) return HBQ_ERR_UNSUPPORTED;
    a.nblk = (a.K + 127) / 128;
    bool quant = false;
    int ml = 1;
    if (q) {
        const int L = q->f.l2_block_size;
        if (mb < 1 || mb > 2 || q->nscheme != 1 || q->nc > 4 || !q->scale_fast_e5m3 || q->f.block_size != 128 ||
            (L != 8 && L != 32) || (a.K % 128) != 0)
            return HBQ_ERR_UNSUPPORTED;
        bool ok = false;
        { const int rc = fill_format(*q, mb, stream, &a.t, &ok); if (rc) return rc; }
        if (!ok) return HBQ_ERR_UNSUPPORTED;
        quant = true;
        ml = L / 8;
    }
    #define HBQ_ROW(MBV, MLV)                                                                              \
        return pro == ROW_RMSNORM ? launch_row<MBV, MLV, ROW_RMSNORM>(a, quant, stream)                   \
                                  : launch_row<MBV, MLV, ROW_SOFTMAX>(a, quant, stream);
    if (mb == 1) { if (ml == 4) { HBQ_ROW(1, 4) } else { HBQ_ROW(1, 1) } }
    if (ml == 4) { HBQ_ROW(2, 4) } else { HBQ_ROW(2, 1) }
    #undef HBQ_ROW
}

int hbq_format_qargs(const hbq_format* f, QArgs* a, int* mb);      // quantize.cu

int rmsnorm_quantize_launch(const void* x, const void* residual, const void* weight, float eps, int64_t rows, int64_t K,
                            const hbq_format* fmt, void* x_out, void* out, cudaStream_t stream)
{
    if (rows < 0 || K < 0) return HBQ_ERR_ARG;
    if (rows == 0 || K == 0) return HBQ_OK;
    if (!x || !weight || !out || (residual && !x_out) || K > (1 << 24)) return HBQ_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(weight) |
         reinterpret_cast<uintptr_t>(x_out) | reinterpret_cast<uintptr_t>(out)) & 15)
        return HBQ_ERR_ALIGN;
    RowArgs a;
    memset(&a, 0, sizeof(a));
    a.in = (const uint4*)x; a.out = (uint4*)out; a.rows = rows; a.K = (int)K;
    a.res = (const uint4*)residual; a.x_out = residual ? (uint4*)x_out : nullptr; a.w = (const uint4*)weight; a.eps = eps;
    QArgs q;
    int mb = 0;
    if (fmt) { const int rc = hbq_format_qargs(fmt, &q, &mb); if (rc) return rc; }
    return hbq_row_launch(ROW_RMSNORM, fmt ? &q : nullptr, mb ? mb : 2, a, stream);
}

int softmax_quantize_launch(const void* scores, int64_t rows, int64_t S, int64_t L, int64_t heads, float scale, int causal,
                            const void* mask, int64_t mask_batches, const hbq_format* fmt, void* out, cudaStream_t stream)
{
    if (rows < 0 || S < 0 || L <= 0 || heads <= 0) return HBQ_ERR_ARG;
    if (rows == 0 || S == 0) return HBQ_OK;
    if (!scores || !out || S > (1 << 24) || (mask && mask_batches < 1)) return HBQ_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(scores) | reinterpret_cast<uintptr_t>(mask) | reinterpret_cast<uintptr_t>(out)) & 15)
        return HBQ_ERR_ALIGN;
    RowArgs a;
    memset(&a, 0, sizeof(a));
    a.in = (const uint4*)scores; a.out = (uint4*)out; a.rows = rows; a.K = (int)S;
    a.scale = scale;
    a.causal = causal; a.L = L; a.HL = heads * L; a.key_offset = S - L;
    a.mask = (const uint4*)mask; a.mask_batches = mask_batches;
    QArgs q;
    int mb = 0;
    if (fmt) { const int rc = hbq_format_qargs(fmt, &q, &mb); if (rc) return rc; }
    return hbq_row_launch(ROW_SOFTMAX, fmt ? &q : nullptr, mb ? mb : 2, a, stream);
}

int hbq_tab_try_launch(const QArgs& q, int mb, cudaStream_t stream, bool* launched)
{
    *launched = false;
    if (mb < 1 || mb > 2 || q.nscheme > 2 || q.nc > 4 || !q.scale_fast_e5m3) return HBQ_OK;
    if (!q.aligned || q.K != q.Kp) return HBQ_OK;
    const bool kv = q.rope_cos || q.perm_T > 0 || q.k_center;
    const bool side = q.out.codes || q.out.sign || q.out.scale_u8 || q.out.scale_h || q.out.l2_packed || q.out.l2_idx ||
                      q.out.scheme;
    const bool glu = q.glu_gate != nullptr, mix = q.nscheme == 2;
    if (!side && !q.deq) return HBQ_OK;
    // the K / post-RoPE Q cache write: rows of one block each (the rotation partners share a thread), indices in 32 bits
    if (kv && (mix || side || glu || q.perm_T <= 0 || q.K != q.f.block_size || q.rows > 0x7FFFFFFFll || q.rope_rows > 0x7FFFFFFFll))
        return HBQ_OK;
    if (glu && (mix || side || q.in_bf16 || q.out_bf16)) return HBQ_OK;
    if ((reinterpret_cast<uintptr_t>(q.out.codes) & 3) || (reinterpret_cast<uintptr_t>(q.out.l2_packed) & 3) ||
        (reinterpret_cast<uintptr_t>(q.out.scale_h) & 1))
        return HBQ_OK;
    const int cpb = q.G, L = q.f.l2_block_size;              // chunks per block, elements per micro-block
    if (L < 8) return HBQ_OK;
    const int m = L / 8;
    int C = 0;
    if (cpb % 4 == 0 && m <= cpb / 4) C = 4;
    else if (cpb % 2 == 0 && m <= cpb / 2) C = 2;
    if (C == 0 || ((mix || kv) && C != 4)) return HBQ_OK;
    const int Gt = cpb / C;
    if (Gt > 32 || (Gt & (Gt - 1)) || (m & (m - 1))) return HBQ_OK;

    TabArgs a;
    bool ok = false;
    { const int rc = fill_format(q, mb, stream, &a, &ok); if (rc) return rc; }
    if (!ok) return HBQ_OK;
    if (mix) {                                               // the second table, through the same steps
        QArgs q2;
        memset(&q2, 0, sizeof(q2));
        memcpy(q2.tab[0], q.tab[1], sizeof(q2.tab[0]));
        q2.nc = q.nc;
        q2.ele_max[0] = q.ele_max[1];
        TabArgs b;
        { const int rc = fill_format(q2, mb, stream, &b, &ok); if (rc) return rc; }
        if (!ok) return HBQ_OK;
        a.b.table = b.table; a.b.entries = b.entries;
        a.b.base2 = b.base2; a.b.hi2 = b.hi2; a.b.big_l1 = b.big_l1; a.b.inv_ele_max = b.inv_ele_max;
        memcpy(a.b.nt2, b.nt2, sizeof(b.nt2));
        memcpy(a.b.tabf, b.tabf, sizeof(b.tabf));
    }

    a.x = reinterpret_cast<const uint4*>(q.x);
    a.gate = reinterpret_cast<const uint4*>(q.glu_gate);
    a.deq = reinterpret_cast<uint4*>(q.deq);
    a.out = q.out;
    a.total_units = q.total_chunks / C;
    a.in_bf16 = q.in_bf16; a.out_bf16 = q.out_bf16;
    while ((1 << a.log2Gt) < Gt) ++a.log2Gt;
    a.m_lanes = m;
    while ((1 << a.log2m) < m) ++a.log2m;
    a.l2_sc_bit = q.f.l2_sc_bit;
    a.nl2 = q.f.block_size / L;
    a.l2_bytes = (a.nl2 * a.l2_sc_bit) >> 3;
    if (kv) {
        a.rope_cos = reinterpret_cast<const uint4*>(q.rope_cos); a.rope_sin = reinterpret_cast<const uint4*>(q.rope_sin);
        a.center = reinterpret_cast<const uint4*>(q.k_center);
        a.kv_T = (uint32_t)q.perm_T; a.kv_H = (uint32_t)q.perm_H; a.rope_rows = (uint32_t)q.rope_rows;
        a.kv_B = (uint32_t)(q.rows / (q.perm_T * q.perm_H));
        a.run = (uint32_t)q.run; a.group = (uint32_t)q.group;
        a.from_runs = (uint32_t)q.from_runs; a.T0 = (uint32_t)q.T0; a.Tall = (uint32_t)q.Tall;
    }

    const size_t smem = (size_t)(a.entries + (mix ? a.b.entries : 0)) * 4;
    int rc;
    if (mix) rc = mb == 1 ? launch_mix_geometry<1>(a, Gt, m, side, smem, stream) : launch_mix_geometry<2>(a, Gt, m, side, smem, stream);
    else rc = mb == 1 ? launch_tab_geometry<1>(a, C, Gt, m, side, glu, smem, stream)
                      : launch_tab_geometry<2>(a, C, Gt, m, side, glu, smem, stream);
    if (rc == HBQ_OK) *launched = true;
    return rc;
}

template <int MB, int ML>
static int launch_tab_v(const TabArgs& a, const VArgs& v, cudaStream_t stream)
{
    const size_t smem = (size_t)a.entries * 4;
    int sms = 0, per_sm = 0;
    { const int rc = device_sms(&sms); if (rc) return rc; }
    { const int rc = ensure_dynamic_smem(hbq_tab_v_kernel<MB, ML>, smem); if (rc) return rc; }
    { const int rc = resident_ctas(hbq_tab_v_kernel<MB, ML>, TABV_THREADS, smem, &per_sm); if (rc) return rc; }
    const int64_t cap = (int64_t)sms * per_sm;
    HBQ_CUDA_TRY(launch_dependent(hbq_tab_v_kernel<MB, ML>, (unsigned)(v.tiles < cap ? v.tiles : cap), TABV_THREADS, smem, stream, a, v));
    HBQ_LAUNCH_CHECK("hbq_tab_v_kernel");
    return HBQ_OK;
}

int hbq_tab_v_try_launch(const QArgs& q, int mb, const void* in, void* out, int in_bf16, int out_bf16, int64_t B, int64_t T,
                         int64_t H, int64_t D, int out_token_major, cudaStream_t stream, bool* launched)
{
    *launched = false;
    const int L = q.f.l2_block_size;
    if (mb < 1 || mb > 2 || q.nscheme != 1 || q.nc > 4 || !q.scale_fast_e5m3) return HBQ_OK;
    if (q.f.block_size != TABV_T || (L != 8 && L != 32) || ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15))
        return HBQ_OK;
    VArgs v;
    if (!v_args_fill(&v, in, out, in_bf16, out_bf16, B, T, H, D, q.f.block_size, out_token_major) || v.tiles == 0) return HBQ_OK;
    TabArgs a;
    bool ok = false;
    { const int rc = fill_format(q, mb, stream, &a, &ok); if (rc) return rc; }
    if (!ok) return HBQ_OK;
    a.m_lanes = L / 8;
    int rc;
    if (mb == 1) rc = L == 8 ? launch_tab_v<1, 1>(a, v, stream) : launch_tab_v<1, 4>(a, v, stream);
    else rc = L == 8 ? launch_tab_v<2, 1>(a, v, stream) : launch_tab_v<2, 4>(a, v, stream);
    if (rc == HBQ_OK) *launched = true;
    return rc;
}

}  // namespace hbq
