// The reference's streaming-softmax statement, one key at a time in f32 (attn_decode_sliding.wgsl:84-107): row loads in every
// cache format and the per-warp state.  The scalar kernels are built from it, and the tensor-core kernels fall back to its form of
// several keys at a time for rows whose tiled result is not finite.
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
            const uint4 u = ld_global(reinterpret_cast<const uint4*>(p) + i);
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
            const uint2 u = ld_global(reinterpret_cast<const uint2*>(p) + i);
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
    const float s = __half2float(ld_global(scales + d0 / 32));
#pragma unroll
    for (int i = 0; i < DPL / 4; i++) {
        const uint32_t w = ld_global(reinterpret_cast<const uint32_t*>(q) + i);
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

// warp_sum of N values (a power of two): the lanes share out the values while they add, about 2 N shuffles instead of 5 N.
template <int N>
__device__ __forceinline__ void warp_sums(float* v)
{
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int n = N / 2; n > 0; n >>= 1, o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const float send = upper ? v[i] : v[i + n], keep = upper ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    float total = v[0];  // of value lane / (32 / N)
#pragma unroll
    for (o = 16 / N; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = __shfl_sync(0xffffffffu, total, i * (32 / N));
}

// ---- the same by one warp, several keys at a time: for the rows whose tiled result is not finite ----------------------------
// A slice of a row as it lies in memory.
template <int FMT, int DPL>
struct RawSlice {
    uint32_t w[FMT == FMT_F16 ? DPL / 2 : DPL / 4];
    float s;
    __device__ __forceinline__ void load(const char* p)
    {
        constexpr int N = sizeof(w) / 4;
        if constexpr (FMT == FMT_F16 && N % 4 == 0) {
#pragma unroll
            for (int i = 0; i < N / 4; i++) {
                const uint4 u = ld_global(reinterpret_cast<const uint4*>(p) + i);
                w[4 * i] = u.x, w[4 * i + 1] = u.y, w[4 * i + 2] = u.z, w[4 * i + 3] = u.w;
            }
        } else if constexpr (FMT == FMT_F16) {
#pragma unroll
            for (int i = 0; i < N / 2; i++) {
                const uint2 u = ld_global(reinterpret_cast<const uint2*>(p) + i);
                w[2 * i] = u.x, w[2 * i + 1] = u.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < N; i++) w[i] = ld_global(reinterpret_cast<const uint32_t*>(p) + i);
        }
    }
    __device__ __forceinline__ float at(int d) const
    {
        if constexpr (FMT == FMT_F16) {
            const float2 f = __half22float2(reinterpret_cast<const __half2*>(w)[d / 2]);
            return (d & 1) ? f.y : f.x;
        } else {
            return __fmul_rn(s, (float)(int8_t)((w[d / 4] >> (8 * (d & 3))) & 0xFF));
        }
    }
};

// H query heads of a kv head against the keys [begin, end), key t in row t, or t % ring.  One key at a time a warp waits for memory
// at every step (490 ns a key); KEYS of them cost one wait, and share the rescale.
template <int HD, int KFMT, int H, int KEYS>
__device__ __forceinline__ void stream_keys(Stream<H, HD / 32>& st, const float (&qr)[H][HD / 32], const KvOperand& k, const KvOperand& v,
                                            uint32_t begin, uint32_t end, uint32_t ring, int kvh, int n_kv, float scale)
{
    constexpr int DPL = HD / 32;
    const int d0 = (threadIdx.x & 31) * DPL;
    const uint32_t k_pitch = (uint32_t)n_kv * HD * (KFMT == FMT_F16 ? 2 : 1), v_pitch = (uint32_t)n_kv * HD * 2, s_pitch = (uint32_t)n_kv * (HD / 32);
    const char* k_base = reinterpret_cast<const char*>(k.data) + (kvh * HD + d0) * (KFMT == FMT_F16 ? 2 : 1);
    const char* v_base = reinterpret_cast<const char*>(v.data) + (kvh * HD + d0) * 2;
    for (uint32_t t0 = begin; t0 < end; t0 += KEYS) {
        // Past the end the last key once more, with a score of -inf and zeros for its value: no branches between the keys
        RawSlice<KFMT, DPL> kk[KEYS];
        RawSlice<FMT_F16, DPL> vv[KEYS];
        const uint32_t row0 = ring ? t0 % ring : t0;
#pragma unroll
        for (int j = 0; j < KEYS; j++) {
            uint32_t row = row0 + min((uint32_t)j, end - 1 - t0);
            if (ring && row >= ring) row -= ring;
            kk[j].load(k_base + (uint64_t)row * k_pitch);
            if constexpr (KFMT != FMT_F16) kk[j].s = __half2float(ld_global(k.scales + (uint64_t)row * s_pitch + kvh * (HD / 32) + d0 / 32));
            vv[j].load(v_base + (uint64_t)row * v_pitch);
        }
        float s[KEYS][H];
#pragma unroll
        for (int j = 0; j < KEYS; j++) {
#pragma unroll
            for (int h = 0; h < H; h++) s[j][h] = 0.0f;
#pragma unroll
            for (int d = 0; d < DPL; d++) {
                const float x = kk[j].at(d);
#pragma unroll
                for (int h = 0; h < H; h++) s[j][h] = fmaf(qr[h][d], x, s[j][h]);
            }
        }
        warp_sums<KEYS * H>(&s[0][0]);
#pragma unroll
        for (int h = 0; h < H; h++) {
            float top = st.m[h];
#pragma unroll
            for (int j = 0; j < KEYS; j++) {
                s[j][h] = t0 + j < end ? s[j][h] * scale : -INFINITY;
                top = fmaxf(top, s[j][h]);
            }
            const float corr = __expf(st.m[h] - top);
            st.m[h] = top;
            st.l[h] *= corr;
#pragma unroll
            for (int d = 0; d < DPL; d++) st.acc[h][d] *= corr;
#pragma unroll
            for (int j = 0; j < KEYS; j++) {
                s[j][h] = __expf(s[j][h] - top);
                st.l[h] += s[j][h];
            }
        }
#pragma unroll
        for (int j = 0; j < KEYS; j++) {
#pragma unroll
            for (int d = 0; d < DPL; d++) {
                const float x = t0 + j < end ? vv[j].at(d) : 0.0f;
#pragma unroll
                for (int h = 0; h < H; h++) st.acc[h][d] = fmaf(s[j][h], x, st.acc[h][d]);
            }
        }
    }
}

// Two heads (head0 and the next, of one kv head) of prefill token i by a warp: history rows [begin, q0) or all rows [begin, qpos] of
// (k0, v0) at t % ring, then (two sources) the chunk's rows of (k1, v1).  Writes the heads in `which`.
template <int HD, int G, bool QI8, bool TWO_SRC>
__device__ __forceinline__ void stream_prefill_rows(const void* q, const __half* q_scales, const KvOperand& k0, const KvOperand& v0, const KvOperand& k1,
                                                    const KvOperand& v1, __half* out, uint32_t q0, uint32_t i, int head0, uint32_t which, int n_kv,
                                                    uint32_t window, uint32_t ring, float scale)
{
    constexpr int DPL = HD / 32, KFMT = QI8 ? FMT_Q8 : FMT_F16, KEYS = 4;
    static_assert(G % 2 == 0, "a pair of heads shares its kv head");
    const int d0 = (threadIdx.x & 31) * DPL, kvh = head0 / G;
    const size_t qrow = (size_t)i * (n_kv * G) + head0;
    float qr[2][DPL];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if constexpr (QI8)
            load_q8<DPL>(reinterpret_cast<const int8_t*>(q) + (qrow + h) * HD + d0, q_scales + (qrow + h) * (HD / 32), d0, qr[h]);
        else
            load_f16<DPL>(reinterpret_cast<const __half*>(q) + (qrow + h) * HD + d0, qr[h]);
    }
    Stream<2, DPL> st;
    st.init();
    const uint32_t qpos = q0 + i, begin = (window != 0 && qpos + 1 > window) ? qpos + 1 - window : 0;
    uint32_t hist_end = TWO_SRC ? min(q0, qpos + 1) : qpos + 1;
    if (ring == 0) hist_end = (uint32_t)min((size_t)hist_end, min(k0.rows, v0.rows));  // reported where the tiles are laid out
    stream_keys<HD, KFMT, 2, KEYS>(st, qr, k0, v0, begin, hist_end, ring, kvh, n_kv, scale);
    if constexpr (TWO_SRC)
        stream_keys<HD, FMT_F16, 2, KEYS>(st, qr, k1, v1, begin > q0 ? begin - q0 : 0, i + 1, 0, kvh, n_kv, scale);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if ((which >> h) & 1) {
#pragma unroll
            for (int d = 0; d < DPL; d++) out[(qrow + h) * HD + d0 + d] = __float2half_rn(st.acc[h][d] / st.l[h]);
        }
    }
}

}  // namespace sgb
