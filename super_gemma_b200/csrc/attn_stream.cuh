// The reference's streaming-softmax statement, one key at a time in f32 (attn_decode_sliding.wgsl:84-107): row loads in every
// cache format and the per-warp state.  The scalar kernels are built from it, and the tensor-core kernels fall back to it
// for rows whose tiled result is not finite.
#pragma once

#include "sgb_common.cuh"
#include "sgb_kernels.h"

namespace sgb {

// FMT_Q8: value = f32(scale) * f32(q), unrounded (attn_decode_global_q8k.wgsl:82, and the exact product the
// int8 path of attn_prefill_global_flash_sp_iq.wgsl forms).  FMT_Q8_F16: the same product rounded to f16,
// the value attn_prefill_global_flash_sp_q8.wgsl:104 stages in shared memory (= kv_dequant_q8).
enum : int { FMT_F16 = 0, FMT_Q8 = 1, FMT_Q8_F16 = 2 };

struct KvOperand {
    const void* data;           // f16 rows, or int8 quants
    const __half* scales;       // Q8_0 scales (FMT_Q8 only)
    const uint32_t* page_table; // nullptr = linear
    uint32_t table_len;
    uint32_t page;
    size_t rows;                // rows the buffer holds (bounds checks)
};

template <int DPL>
__device__ __forceinline__ void load_f16(const __half* p, float (&out)[DPL])
{
    if constexpr (DPL % 8 == 0) {
#pragma unroll
        for (int i = 0; i < DPL / 8; i++) {
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(p) + i);
            const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __half22float2(h[j]);
                out[i * 8 + 2 * j] = f.x;
                out[i * 8 + 2 * j + 1] = f.y;
            }
        }
    } else {
        static_assert(DPL % 4 == 0, "lanes own 4 or more dims");
#pragma unroll
        for (int i = 0; i < DPL / 4; i++) {
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(p) + i);
            const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float2 f = __half22float2(h[j]);
                out[i * 4 + 2 * j] = f.x;
                out[i * 4 + 2 * j + 1] = f.y;
            }
        }
    }
}

// kk = f32(scale) * f32(q), not re-rounded (attn_decode_global_q8k.wgsl:82).  A lane's DPL dims
// (DPL <= 32, d0 a multiple of DPL) lie inside one 32-value block.
template <int DPL>
__device__ __forceinline__ void load_q8(const int8_t* q, const __half* scales, int d0, float (&out)[DPL])
{
    const float s = __half2float(__ldg(scales + d0 / 32));
#pragma unroll
    for (int i = 0; i < DPL / 4; i++) {
        const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(q) + i);
        out[4 * i] = __fmul_rn(s, (float)(int8_t)(w & 0xFF));
        out[4 * i + 1] = __fmul_rn(s, (float)(int8_t)((w >> 8) & 0xFF));
        out[4 * i + 2] = __fmul_rn(s, (float)(int8_t)((w >> 16) & 0xFF));
        out[4 * i + 3] = __fmul_rn(s, (float)(int8_t)(w >> 24));
    }
}

// One K or V row slice for this lane.  `row` is already physical.
template <int HD, int FMT, int DPL>
__device__ __forceinline__ void load_row(const KvOperand& op, size_t row, int kvh, int n_kv, int d0, float (&out)[DPL])
{
    const size_t base = (row * n_kv + kvh) * HD;
    if constexpr (FMT == FMT_F16) {
        load_f16<DPL>(reinterpret_cast<const __half*>(op.data) + base + d0, out);
    } else {
        load_q8<DPL>(reinterpret_cast<const int8_t*>(op.data) + base + d0, op.scales + (row * n_kv + kvh) * (HD / 32), d0,
                     out);
        if constexpr (FMT == FMT_Q8_F16) {
#pragma unroll
            for (int d = 0; d < DPL; d++) out[d] = __half2float(__float2half_rn(out[d]));
        }
    }
}

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int G, int DPL>
struct Stream {
    float m[G], l[G], acc[G][DPL];
    __device__ __forceinline__ void init()
    {
#pragma unroll
        for (int g = 0; g < G; g++) {
            m[g] = NEG_SENTINEL;
            l[g] = 0.0f;
#pragma unroll
            for (int d = 0; d < DPL; d++) acc[g][d] = 0.0f;
        }
    }
    // attn_decode_sliding.wgsl:92-106 for head g
    __device__ __forceinline__ void step(int g, const float (&qr)[DPL], const float (&kk)[DPL], const float (&vv)[DPL],
                                         float scale)
    {
        float dot = 0.0f;
#pragma unroll
        for (int d = 0; d < DPL; d++) dot = fmaf(qr[d], kk[d], dot);
        const float s = warp_sum(dot) * scale;
        const float m_new = fmaxf(m[g], s);
        const float corr = __expf(m[g] - m_new);
        const float w = __expf(s - m_new);
        l[g] = l[g] * corr + w;
#pragma unroll
        for (int d = 0; d < DPL; d++) acc[g][d] = acc[g][d] * corr + w * vv[d];
        m[g] = m_new;
    }
};

__device__ __forceinline__ bool resolve_row(const KvOperand& op, size_t t, size_t& row, uint32_t* status, uint32_t site)
{
    row = t;
    if (op.page_table != nullptr) {
        const size_t p = t / op.page;
        if (p >= op.table_len) {
            report_error(status, DEV_ERR_BOUNDS, site, (uint32_t)p, op.table_len);
            return false;
        }
        row = (size_t)op.page_table[p] * op.page + t % op.page;
    }
    if (row >= op.rows) {
        report_error(status, DEV_ERR_BOUNDS, site + 1, (uint32_t)row, (uint32_t)op.rows);
        return false;
    }
    return true;
}

// What load_f16 asks of the base of rows of `hd` f16 values: a lane reads hd / 32 of them with accesses of up to 16 bytes.
constexpr uint32_t row_alignment(int hd) { return hd / 32 % 8 == 0 ? 16 : 8; }

inline KvOperand linear_f16(const BufView& b, int n_kv, int hd)
{
    return KvOperand{b.ptr, nullptr, nullptr, 0, 1, b.bytes / ((size_t)n_kv * hd * 2)};
}
inline KvOperand linear_q8(const BufView& quants, const BufView& scales, int n_kv, int hd)
{
    return KvOperand{quants.ptr, (const __half*)scales.ptr, nullptr, 0, 1, quants.bytes / ((size_t)n_kv * hd)};
}

// One query row of prefill by the streaming statement, by a warp: history rows [begin, q0) or all rows [begin, qpos] of (k0, v0) at
// t % ring, then (two sources) the chunk's rows of (k1, v1).  For rows whose tiled result is not finite.
template <int HD, int G, bool QI8, bool TWO_SRC>
__device__ __forceinline__ void stream_prefill_row(const void* q, const __half* q_scales, const KvOperand& k0, const KvOperand& v0, const KvOperand& k1,
                                                   const KvOperand& v1, __half* out, uint32_t q0, uint32_t i, int head, int n_kv, uint32_t window,
                                                   uint32_t ring, float scale)
{
    constexpr int DPL = HD / 32, KFMT = QI8 ? FMT_Q8 : FMT_F16;
    const int d0 = (threadIdx.x & 31) * DPL, kvh = head / G;
    const size_t qrow = (size_t)i * (n_kv * G) + head;
    float qr[DPL], kk[DPL], vv[DPL];
    if constexpr (QI8)
        load_q8<DPL>(reinterpret_cast<const int8_t*>(q) + qrow * HD + d0, q_scales + qrow * (HD / 32), d0, qr);
    else
        load_f16<DPL>(reinterpret_cast<const __half*>(q) + qrow * HD + d0, qr);
    Stream<1, DPL> st;
    st.init();
    const uint32_t qpos = q0 + i, begin = (window != 0 && qpos + 1 > window) ? qpos + 1 - window : 0;
    const uint32_t hist_end = TWO_SRC ? min(q0, qpos + 1) : qpos + 1;
    for (uint32_t t = begin; t < hist_end; t++) {
        const size_t row = ring ? t % ring : t;
        if (row >= k0.rows || row >= v0.rows) break;  // reported where the tiles are laid out
        load_row<HD, KFMT, DPL>(k0, row, kvh, n_kv, d0, kk);
        load_row<HD, FMT_F16, DPL>(v0, row, kvh, n_kv, d0, vv);
        st.step(0, qr, kk, vv, scale);
    }
    if (TWO_SRC) {
        for (uint32_t c = begin > q0 ? begin - q0 : 0; c <= i; c++) {
            load_row<HD, FMT_F16, DPL>(k1, c, kvh, n_kv, d0, kk);
            load_row<HD, FMT_F16, DPL>(v1, c, kvh, n_kv, d0, vv);
            st.step(0, qr, kk, vv, scale);
        }
    }
#pragma unroll
    for (int d = 0; d < DPL; d++) out[qrow * HD + d0 + d] = __float2half_rn(st.acc[0][d] / st.l[0]);
}

}  // namespace sgb
