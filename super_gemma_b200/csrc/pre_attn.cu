// The steps between the QKV projections and the attention kernels: per-head RMS norm (QK-norm, weightless
// V-norm), rotate-half RoPE from a host-filled cos/sin table, and the quantise-and-append of K and V.
//
// Reference chain per layer (crates/sg-model/src/graph.rs:552-610): rmsnorm(q), rmsnorm(k), rmsnorm(v, ones),
// rope(q), rope(k), append(k), append(v) -- seven launches with an f16 round trip between every two.  Here:
//   rmsnorm_256/512[_plus1], rope_sliding_q/k, rope_global_q/k   the reference's names, bindings and grids
//       (crates/sg-gpu/shaders/rmsnorm.wgsl, rope.wgsl; build.rs:84-157)
//   attn_norm_rope_d128                       norm + rope of a [rows x 128] tensor in one pass
//   kv_norm_rope_append_paged_q8_d128         norm(k) + rope(k) + norm(v) + Q8_0 quantise + paged append
// The fused kernels round to f16 exactly where the chain stores f16 (after the norm, after the rotation), so
// they give the bits of their own unfused pieces.  All of it is HBM-bound: the head_dim-128 kernels give a row to 16
// consecutive lanes (16-byte accesses, partner dims and block maxima by shuffle), the append 8 (both partners in a lane), the
// reference-named ones a 32-value block to a thread; the row's sum of squares always goes through a fixed shuffle tree (deterministic).
//
// Arithmetic (f32): inv = 1/sqrt(sum(x^2)/n + 1e-6); y = f16(x * inv * w)  [w or 1 + w];
// rope pair i couples dims (i, i + n/2), live for i < rot_dims/2: lo' = f16(lo*c - hi*s), hi' = f16(hi*c + lo*s).
#include "sgb_common.cuh"
#include "sgb_kernels.h"

namespace sgb {

namespace {

constexpr int PRE_THREADS = 256;
constexpr float RMS_EPS = 1e-6f;

__device__ __forceinline__ void load_f16x32(const __half* p, float (&x)[32])
{
    const uint4* v = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint4 u = ld_global(v + i);
        const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(h[j]);
            x[i * 8 + j * 2] = f.x;
            x[i * 8 + j * 2 + 1] = f.y;
        }
    }
}

__device__ __forceinline__ void pack_f16x32(const float (&x)[32], uint4 (&out)[4])
{
#pragma unroll
    for (int i = 0; i < 4; i++) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const __half2 h = __floats2half2_rn(x[i * 8 + j * 2], x[i * 8 + j * 2 + 1]);
            w[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        out[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

__device__ __forceinline__ float round_f16(float v) { return __half2float(__float2half_rn(v)); }

// Sum of squares of a row spread over BPR consecutive lanes (one 32-value block each): in-thread sum in index
// order, then an xor butterfly, which gives every lane the same bits.
template <int BPR>
__device__ __forceinline__ float row_inv_rms(const float (&x)[32])
{
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; i++) ss = fmaf(x[i], x[i], ss);
#pragma unroll
    for (int d = 1; d < BPR; d <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
    return rsqrtf(ss / (float)(BPR * 32) + RMS_EPS);
}

// rmsnorm_<ROW_LEN>[_plus1]: x f16[rows x ROW_LEN], w f32[ROW_LEN], y f16.  grid [rows].  y = f16(x * inv * weight), weight = 1 + w with
// PLUS_ONE (rmsnorm.wgsl:52-58).  A few rows are one memory latency: the weights are asked for together with the values (AHEAD), 16 bytes
// at a time where the caller's array allows it (one by one and behind the sum of squares, 32 rows of 512 took 4.0 us in a recorded
// chain, with AHEAD 2.6).  That takes 75 registers, three blocks an SM; without AHEAD it is 47, five.  rmsnorm_ahead() chooses.
template <int BPR, bool PLUS_ONE, bool AHEAD>
__global__ void __launch_bounds__(PRE_THREADS) rmsnorm_kernel(const __half* x, const float* w,
                                                              __half* __restrict__ y, size_t n_blocks)
{
    pdl_wait();
    pdl_launch_dependents();
    const size_t blk = (size_t)blockIdx.x * PRE_THREADS + threadIdx.x;
    const bool live = blk < n_blocks;  // whole rows only, and BPR divides 32: a row never straddles a warp
    const float* wp = w + (blk % BPR) * 32;
    float v[32], wv[32];
    if (live) {
        load_f16x32(x + blk * 32, v);
        if constexpr (AHEAD) {
            if ((reinterpret_cast<uintptr_t>(w) & 15) == 0) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 f = ld_global(reinterpret_cast<const float4*>(wp) + i);
                    wv[4 * i] = f.x;
                    wv[4 * i + 1] = f.y;
                    wv[4 * i + 2] = f.z;
                    wv[4 * i + 3] = f.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) wv[i] = ld_global(wp + i);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; i++) v[i] = 0.0f;
    }
    const float inv = row_inv_rms<BPR>(v);
    if (!live) return;
#pragma unroll
    for (int i = 0; i < 32; i++) {
        const float weight = AHEAD ? wv[i] : ld_global(wp + i);
        v[i] = v[i] * inv * (PLUS_ONE ? 1.0f + weight : weight);
    }
    uint4 out[4];
    pack_f16x32(v, out);
    uint4* o = reinterpret_cast<uint4*>(y + blk * 32);
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = out[i];
}

// rope_*: in place over rows [token x head x head_dim], one thread per (row, live pair) (rope.wgsl:36-52).
__global__ void __launch_bounds__(PRE_THREADS) rope_kernel(__half* __restrict__ xs, const float2* cos_sin,
                                                           uint32_t head_dim, uint32_t half_rot, uint32_t n_heads, size_t pairs_total)
{
    pdl_wait();
    pdl_launch_dependents();
    const size_t g = (size_t)blockIdx.x * PRE_THREADS + threadIdx.x;
    if (g >= pairs_total) return;
    const size_t row = g / half_rot;
    const uint32_t pair = (uint32_t)(g % half_rot);
    const size_t token = row / n_heads;
    const float2 cs = ld_global(cos_sin + token * half_rot + pair);
    __half* lo = xs + row * head_dim + pair;
    __half* hi = lo + head_dim / 2;
    const float a = __half2float(*lo), b = __half2float(*hi);
    *lo = __float2half_rn(__fsub_rn(__fmul_rn(a, cs.x), __fmul_rn(b, cs.y)));
    *hi = __float2half_rn(__fadd_rn(__fmul_rn(b, cs.x), __fmul_rn(a, cs.y)));
}

// One 8-dim piece of a 128-dim row after norm and rotation, as f16-exact floats.  The 16 threads of a row are
// consecutive lanes (two rows per warp, 16-byte accesses); thread `o` owns dims [8 o, 8 o + 8) and gets its
// rotation partner's normalised values (dims +-64, lane o ^ 8) by shuffle.  Every lane of the warp must call
// it (dead lanes with live = false), and half_rot must be the same for the whole warp.
template <bool PLUS_ONE>
__device__ __forceinline__ void norm_rope_oct_d128(const __half* row_ptr, const float* w,
                                                    const float2* cs_row, uint32_t half_rot, int o, bool live,
                                                    float (&v)[8])
{
    if (live) {
        const uint4 u = ld_global(reinterpret_cast<const uint4*>(row_ptr + 8 * o));
        const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(h[j]);
            v[2 * j] = f.x;
            v[2 * j + 1] = f.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = 0.0f;
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) ss = fmaf(v[i], v[i], ss);
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);  // fixed tree: every lane gets the same bits
    const float inv = rsqrtf(ss / 128.0f + RMS_EPS);
    float wv[8];
#pragma unroll
    for (int i = 0; i < 8; i++) wv[i] = 1.0f;
    if (w != nullptr && live) {
        const float4 w0 = ld_global(reinterpret_cast<const float4*>(w + 8 * o)), w1 = ld_global(reinterpret_cast<const float4*>(w + 8 * o) + 1);
        const float t[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int i = 0; i < 8; i++) wv[i] = PLUS_ONE ? 1.0f + t[i] : t[i];
    }
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = round_f16(v[i] * inv * wv[i]);
    if (half_rot == 0) return;
    float other[8];
#pragma unroll
    for (int i = 0; i < 8; i++) other[i] = __shfl_xor_sync(0xffffffffu, v[i], 8);
    const uint32_t pair0 = (uint32_t)(o & 7) * 8;
    if (!live || pair0 >= half_rot) return;
    const float4* cp = reinterpret_cast<const float4*>(cs_row + pair0);  // (cos, sin) pairs; 16-byte aligned: half_rot % 8 == 0
#pragma unroll
    for (int j = 0; j < 4; j++) {  // half_rot is a multiple of 8 (checked on the host): all 8 pairs of a live piece rotate
        const float4 cs = ld_global(cp + j);
        const float c[2] = {cs.x, cs.z}, sn[2] = {cs.y, cs.w};
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int i = 2 * j + e;
            // low half: lo*c - hi*s with lo = own; high half: hi*c + lo*s with hi = own
            v[i] = (o < 8) ? round_f16(__fsub_rn(__fmul_rn(v[i], c[e]), __fmul_rn(other[i], sn[e])))
                           : round_f16(__fadd_rn(__fmul_rn(v[i], c[e]), __fmul_rn(other[i], sn[e])));
        }
    }
}

__device__ __forceinline__ uint4 pack_f16x8(const float (&v)[8])
{
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
        w[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// attn_norm_rope_d128: x f16[rows x 128] (rows = tokens x n_heads), w f32[128], cos_sin f32[tokens x rot/2 x 2], y f16.
template <bool PLUS_ONE>
__global__ void __launch_bounds__(PRE_THREADS) norm_rope_d128_kernel(const __half* x, const float* w,
                                                                     const float2* cos_sin, __half* __restrict__ y,
                                                                     uint32_t n_heads, uint32_t half_rot, uint32_t rows)
{
    pdl_wait();
    pdl_launch_dependents();
    // 32-bit index arithmetic (the host checks rows * 16 < 2^32): 64-bit divisions would cost more than the rest
    const uint32_t g = blockIdx.x * PRE_THREADS + threadIdx.x;
    const uint32_t row = g >> 4;
    const int o = (int)(g & 15);
    const bool live = row < rows;
    float v[8];
    norm_rope_oct_d128<PLUS_ONE>(x + (size_t)row * 128, w, cos_sin + (size_t)(row / n_heads) * half_rot, half_rot, o, live, v);
    if (live) *reinterpret_cast<uint4*>(y + (size_t)row * 128 + 8 * o) = pack_f16x8(v);
}

// Multiplies and additions of pairs, each half rounded by itself: ptxas contracts a packed multiply and add that do not say .rn.
__device__ __forceinline__ float2 mul2_rn(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 add2_rn(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 unpack_half2(uint32_t u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }

// Q8_0 of the 32-value blocks that four consecutive lanes hold (8 values each, two blocks side by side): the arithmetic of
// kv_quant_q8.wgsl:38-57 (see kv_codec.cu).  The values are f16, so the block maxima are taken of f16 pairs, both blocks' in one
// word and two shuffles; the conversion adds 1.5 * 2^23, which leaves the nearest whole number in the low bytes and costs an
// eighth of a convert instruction.  Blocks that hold an infinity or a NaN convert value by value.  All lanes of the warp call it.
__device__ __forceinline__ void quant_2x8(const uint32_t (&x)[8], __half (&scale)[2], uint2 (&packed)[2])
{
    auto habs = [](uint32_t u) { return __habs2(*reinterpret_cast<const __half2*>(&u)); };
    __half2 top[2];
#pragma unroll
    for (int e = 0; e < 2; e++) top[e] = __hmax2_nan(__hmax2_nan(habs(x[4 * e]), habs(x[4 * e + 1])), __hmax2_nan(habs(x[4 * e + 2]), habs(x[4 * e + 3])));
    __half2 both = __hmax2_nan(__lows2half2(top[0], top[1]), __highs2half2(top[0], top[1]));
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
        const uint32_t o = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const uint32_t*>(&both), d);
        both = __hmax2_nan(both, *reinterpret_cast<const __half2*>(&o));
    }
    float2 amax = __half22float2(both);
    const bool odd = __any_sync(0xffffffffu, !(fmaxf(amax.x, amax.y) <= 65504.0f) || amax.x != amax.x || amax.y != amax.y);
    if (odd) {  // the maximum of what is a number
        float m[2] = {0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float2 f = unpack_half2(x[i]);
            m[i >> 2] = max3(m[i >> 2], fabsf(f.x), fabsf(f.y));
        }
#pragma unroll
        for (int e = 0; e < 2; e++) {
            m[e] = fmaxf(m[e], __shfl_xor_sync(0xffffffffu, m[e], 1));
            m[e] = fmaxf(m[e], __shfl_xor_sync(0xffffffffu, m[e], 2));
        }
        amax = make_float2(m[0], m[1]);
    }
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const float d = __fmul_rn(e ? amax.y : amax.x, 1.0f / 127.0f);
        const float id = d > 0.0f ? __frcp_rn(d) : 0.0f;
        scale[e] = __float2half_rn(d);
        uint32_t w[4];  // two quants each, in the low bytes
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 y = mul2_rn(unpack_half2(x[4 * e + i]), make_float2(id, id));
            if (odd) {
                w[i] = __byte_perm((uint32_t)__float2int_rn(y.x), (uint32_t)__float2int_rn(y.y), 0x0040);
            } else {
                const float2 n = add2_rn(y, make_float2(12582912.0f, 12582912.0f));
                w[i] = __byte_perm(__float_as_uint(n.x), __float_as_uint(n.y), 0x0040);
            }
        }
        packed[e] = make_uint2(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410));
    }
}

// kv_norm_rope_append_paged_q8_d128: K rows (norm with k_w, rope) and V rows (weightless norm), both landing Q8_0-quantised at
// row page_table[t / page] * page + t % page with t = step[0] + token; and, for qkv_norm_rope_append_paged_q8_d128, Q rows
// (norm with q_w, rope, f16 out): the whole pre-attention step of a layer in one launch.
//
// 2^slot_bits groups of 8 lanes (and gridDim.y times as many) share the rows of a token (q heads, k heads, v heads in this order).
// A lane has the octet of dims 8 o .. and the one 64 dims further on that it turns with, so the rotation stays in the lane; it
// keeps its octets for all of its rows, so the token's cos/sin values and the page lookup are read once and stay in
// registers.  Bound by issued instructions: 16 lanes a row, which exchanged partners by shuffle and converted what they got,
// took 40.5 us for 4096 tokens of q, k and v with 16 kv heads, this form 30.9 (120 MB: 18.4 at the copy bandwidth).  What the launcher
// chooses is at append_shape.
constexpr int APPEND_THREADS = 128, APPEND_BLOCKS = 8;
constexpr int ROW_LANES = 8;
constexpr int MOST_SLOTS = 32;  // groups per token and grid row
constexpr int ROWS_EACH = 4;   // rows of a group where a launch has more than it takes to fill the GPU

template <bool PLUS_ONE, bool AHEAD>
__global__ void __launch_bounds__(APPEND_THREADS, AHEAD ? APPEND_BLOCKS / 2 : APPEND_BLOCKS)
    kv_norm_rope_append_kernel(const __half* q_raw, const float* q_w, __half* __restrict__ q_out,
                               uint32_t n_q, const __half* k_raw, const __half* v_raw, const float* k_w,
                               const float2* cos_sin, __half* __restrict__ k_scales, int8_t* __restrict__ k_quants,
                               __half* __restrict__ v_scales, int8_t* __restrict__ v_quants, const uint32_t* page_table,
                               uint32_t table_len, uint32_t page, const uint32_t* step, uint32_t n_kv, uint32_t half_rot,
                               size_t dst_rows, uint32_t tokens, uint32_t slot_bits, uint32_t* status)
{
    pdl_wait();  // the raw q, k, v rows come from earlier kernels of the stream
    pdl_launch_dependents();
    const int o = threadIdx.x & (ROW_LANES - 1);
    const uint32_t rows = n_q + 2 * n_kv, group = blockIdx.x * (APPEND_THREADS / ROW_LANES) + threadIdx.x / ROW_LANES;
    uint32_t token = group >> slot_bits, slot = group & ((1u << slot_bits) - 1);
    if (token >= tokens) {  // behind the last token: no row of the first
        token = 0;
        slot = rows;
    }
    // rotation: dims 8 o + i and 64 + 8 o + i; half_rot is a multiple of 8 (checked on the host), so a whole octet turns or none
    const bool turns = 8 * (uint32_t)o < half_rot;
    float c[8], sn[8];
    if (turns) {
        const float4* cp = reinterpret_cast<const float4*>(cos_sin + (size_t)token * half_rot + 8 * o);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float4 cs = ld_global(cp + j);
            c[2 * j] = cs.x;
            sn[2 * j] = cs.y;
            c[2 * j + 1] = cs.z;
            sn[2 * j + 1] = cs.w;
        }
    }
    size_t dst_row = 0;
    bool placed = true;
    {
        const uint32_t t = ld_global(step + STEP_POS) + token, p = t / page;
        if (p < table_len) dst_row = (size_t)ld_global(page_table + p) * page + (t - p * page);
        placed = p < table_len && dst_row < dst_rows;
        if (!placed && slot == 0 && o == 0 && blockIdx.y == 0) {
            if (p >= table_len)
                report_error(status, DEV_ERR_BOUNDS, 104, p, table_len);
            else
                report_error(status, DEV_ERR_BOUNDS, 105, (uint32_t)dst_row, (uint32_t)dst_rows);
        }
    }
    struct Octets {
        uint4 lo, hi;
    };
    auto octets = [&](uint32_t r) {
        if (r >= rows) return Octets{make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
        const __half* src = r < n_q           ? q_raw + ((size_t)token * n_q + r) * 128
                            : r < n_q + n_kv ? k_raw + ((size_t)token * n_kv + (r - n_q)) * 128
                                             : v_raw + ((size_t)token * n_kv + (r - n_q - n_kv)) * 128;
        const uint4* p = reinterpret_cast<const uint4*>(src + 8 * o);
        return Octets{ld_global(p), ld_global(p + 8)};
    };
    auto work = [&](uint32_t r0, const Octets& u) {
        const uint32_t r = r0 + slot;
        const bool live = r < rows, is_q = r < n_q, is_v = r >= n_q + n_kv;
        const uint32_t head = is_q ? r : is_v ? r - n_q - n_kv : r - n_q;
        uint32_t own[8] = {u.lo.x, u.lo.y, u.lo.z, u.lo.w, u.hi.x, u.hi.y, u.hi.z, u.hi.w};
        float4 wt[4];
        if constexpr (AHEAD) {
            if (live && !is_v) {
                const float4* w = reinterpret_cast<const float4*>((is_q ? q_w : k_w) + 8 * o);
#pragma unroll
                for (int j = 0; j < 4; j++) wt[j] = ld_global(w + (j >> 1) * 16 + (j & 1));
            }
        }
        float ss[2] = {0.0f, 0.0f};
        float2 v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            v[j] = unpack_half2(own[j]);
            ss[j >> 2] = fmaf(v[j].x, v[j].x, ss[j >> 2]);
            ss[j >> 2] = fmaf(v[j].y, v[j].y, ss[j >> 2]);
        }
        // a fixed tree, every lane gets the same bits: the sixteen octets by 1, 2, 4 and 8
#pragma unroll
        for (int d = 1; d < ROW_LANES; d <<= 1) {
            ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], d);
            ss[1] += __shfl_xor_sync(0xffffffffu, ss[1], d);
        }
        const float inv = rsqrtf((ss[0] + ss[1]) / 128.0f + RMS_EPS);
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = mul2_rn(v[j], make_float2(inv, inv));
        if (live && !is_v) {
            const float4* w = reinterpret_cast<const float4*>((is_q ? q_w : k_w) + 8 * o);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 f = AHEAD ? wt[j] : ld_global(w + (j >> 1) * 16 + (j & 1));
                const float2 one = make_float2(1.0f, 1.0f), w0 = make_float2(f.x, f.y), w1 = make_float2(f.z, f.w);
                v[2 * j] = mul2_rn(v[2 * j], PLUS_ONE ? add2_rn(one, w0) : w0);
                v[2 * j + 1] = mul2_rn(v[2 * j + 1], PLUS_ONE ? add2_rn(one, w1) : w1);
            }
        }
        // the normed octets as f16 pairs: what the chain of kernels stores between norm and rotation
#pragma unroll
        for (int j = 0; j < 8; j++) own[j] = pack_half2(v[j].x, v[j].y);
        if (turns && !is_v) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 a = unpack_half2(own[j]), b = unpack_half2(own[4 + j]);
                const float c0 = c[2 * j], c1 = c[2 * j + 1], s0 = sn[2 * j], s1 = sn[2 * j + 1];
                own[j] = pack_half2(__fsub_rn(__fmul_rn(a.x, c0), __fmul_rn(b.x, s0)), __fsub_rn(__fmul_rn(a.y, c1), __fmul_rn(b.y, s1)));
                own[4 + j] = pack_half2(__fadd_rn(__fmul_rn(b.x, c0), __fmul_rn(a.x, s0)), __fadd_rn(__fmul_rn(b.y, c1), __fmul_rn(a.y, s1)));
            }
        }
        if (is_q && live) {
            uint4* to = reinterpret_cast<uint4*>(q_out + ((size_t)token * n_q + head) * 128 + 8 * o);
            to[0] = make_uint4(own[0], own[1], own[2], own[3]);
            to[8] = make_uint4(own[4], own[5], own[6], own[7]);
        }
        if (r0 + (1u << slot_bits) <= n_q) return;  // only q rows in this pass (uniform over the block)
        __half s[2];
        uint2 packed[2];
        quant_2x8(own, s, packed);
        if (live && !is_q && placed) {
            const size_t drow = dst_row * n_kv + head;  // row of [128] quants / [4] scales
            if ((o & 3) == 0) {
                __half* to = (is_v ? v_scales : k_scales) + drow * 4 + (o >> 2);
                to[0] = s[0];
                to[2] = s[1];
            }
            uint2* to = reinterpret_cast<uint2*>((is_v ? v_quants : k_quants) + drow * 128 + 8 * o);
            to[0] = packed[0];
            to[8] = packed[1];
        }
    };
    const uint32_t stride = gridDim.y << slot_bits;
    // one row's loads under way at a time: registers for eight blocks an SM are worth more (append_shape)
    for (uint32_t base = blockIdx.y << slot_bits; base < rows; base += stride) work(base, octets(base + slot));
}

struct AppendShape {
    dim3 grid;
    uint32_t slot_bits;
    bool ahead;  // weights asked for together with the values
};
// Slots and blocks.  Few rows: one per group, which takes least time for one; beyond, two, then ROWS_EACH of them, which takes least
// instructions per row, and few rows a token (few kv heads) put several tokens into a block.  us in a recorded chain, 1 row | 2 | 4: 16 kv
// heads with q, 64 tokens 2.6 | 3.2 | 4.6, 290 tokens 4.1 | 4.1 | 5.1, 600 tokens 7.4 | 6.9 | 8.4, 1024 tokens 10.5 | 9.3 | 8.9, 4096 tokens
// 37 | 32 | 30; 4 kv heads, 1000 tokens 4.2 | 3.9 | 5.0, 2000 tokens 6.9 | 5.7 | 6.0, 8192 tokens 19.3 | 15.3 | 14.4.  Six blocks an SM and two
// rows' loads under way took 31.6 for 4096 tokens, five and four 32.6.
// Up to 48 rows an SM a launch is one memory latency, and it and the one behind it stand side by side on the GPU (three blocks each, of the six that
// 78 registers leave): the weights are asked for together with the values.  One token of 16 kv heads 1.87 us, with weights 1 + w 2.03; behind the
// sum of squares 2.00 and 2.11.  128 tokens of 16 kv heads, 56 rows an SM: 3.38 | 2.76 with eight blocks and the weights behind the sum.
inline AppendShape append_shape(const LaunchArgs& a, size_t tokens, uint32_t rows)
{
    const size_t per_sm = (tokens * rows + a.sm_count - 1) / a.sm_count;
    const uint32_t per_thread = per_sm <= 64 ? 1 : per_sm <= 384 ? 2 : ROWS_EACH;
    uint32_t bits = 0;
    while ((1u << bits) < MOST_SLOTS && (per_thread << bits) < rows) bits++;
    const size_t groups = tokens << bits;  // < 2^29: at most 2^26 rows of q and of k
    const uint32_t per_token = (rows + (1u << bits) - 1) >> bits;
    return {dim3((uint32_t)((groups * ROW_LANES + APPEND_THREADS - 1) / APPEND_THREADS), per_thread == 1 ? min(1024u, per_token) : 1), bits, per_sm <= 48};
}

inline auto append_kernel(bool plus_one, bool ahead)
{
    return plus_one ? (ahead ? kv_norm_rope_append_kernel<true, true> : kv_norm_rope_append_kernel<true, false>)
                    : (ahead ? kv_norm_rope_append_kernel<false, true> : kv_norm_rope_append_kernel<false, false>);
}

// Whether rmsnorm asks for its weights ahead: rows of 512 whose weights lie on 16 bytes always, others but where the measurements say
// otherwise, us in a recorded chain of launches, ahead | not.  Up to 3 blocks for 2 SMs a launch and the one behind it stand side by side: rows of 256, 32
// of them 2.6 | 3.1, 6000 4.6 | 4.7.  Up to 2 an SM they do so only with five blocks an SM: 8192 6.3 | 4.8; rows of 512 with weights on 4 bytes, 4096
// 9.8 | 6.9.  Up to 8: 10000 6.3 | 6.5, 16384 8.0 | 11.7, 32768 14.7 | 15.7.  Beyond, what counts is the bytes under way: 65536 27.5 | 26.6; of 512, on 4
// bytes, 82.8 | 81.4.  (Rows of 512 on 16 bytes: 4096 6.3 | 7.0, 16384 15.3 | 23.0, 65536 53.5 | 81.7.)
inline bool rmsnorm_ahead(const LaunchArgs& a, uint32_t grid, int row_len, const void* w)
{
    if (row_len == 512 && (reinterpret_cast<uintptr_t>(w) & 15) == 0) return true;
    const uint64_t halves = 2 * (uint64_t)grid, sms = a.sm_count;
    return halves <= 3 * sms || (halves > 4 * sms && halves <= 16 * sms);
}

inline uint32_t grid_for(size_t n) { return (uint32_t)((n + PRE_THREADS - 1) / PRE_THREADS); }

struct PushNormRope {
    uint32_t n_heads, rot_dims, plus_one;
};
struct PushKvNormRope {
    uint32_t row_len, page, rot_dims, plus_one;
};
struct PushQkvNormRope {
    uint32_t n_q_heads, row_len, page, rot_dims, plus_one;
};

}  // namespace

template <int ROW_LEN, int PLUS_ONE>
int launch_rmsnorm(const LaunchArgs& a)
{
    static_assert(ROW_LEN % 32 == 0 && 32 % (ROW_LEN / 32) == 0, "a row is 1..32 blocks that divide a warp");
    if (a.b[0].bytes % (ROW_LEN * 2)) return fail_validation(a, "rmsnorm: x is not whole rows");
    if (int r = need_bytes(a, 1, ROW_LEN * 4, "w")) return r;
    if (int r = need_bytes(a, 2, a.b[0].bytes, "y")) return r;
    const size_t n_blocks = a.b[0].bytes / 64;
    if (n_blocks == 0) return 0;
    if (int r = need_aligned(a, {16, 4, 16})) return r;
    const auto kernel = rmsnorm_ahead(a, grid_for(n_blocks), ROW_LEN, a.b[1].ptr) ? rmsnorm_kernel<ROW_LEN / 32, PLUS_ONE != 0, true> : rmsnorm_kernel<ROW_LEN / 32, PLUS_ONE != 0, false>;
    const cudaError_t e = launch_dependent(kernel, dim3(grid_for(n_blocks)), dim3(PRE_THREADS), 0, a.stream, (const __half*)a.b[0].ptr, (const float*)a.b[1].ptr, (__half*)a.b[2].ptr, n_blocks);
    ++*a.launches;
    return check_cuda(a, e, "rmsnorm");
}
template int launch_rmsnorm<256, 0>(const LaunchArgs&);
template int launch_rmsnorm<256, 1>(const LaunchArgs&);
template int launch_rmsnorm<512, 0>(const LaunchArgs&);
template int launch_rmsnorm<512, 1>(const LaunchArgs&);

template <int HEAD_DIM, int ROT_DIMS, int N_HEADS>
int launch_rope(const LaunchArgs& a)
{
    if (a.b[0].bytes % (HEAD_DIM * 2 * N_HEADS)) return fail_validation(a, "rope: xs is not whole tokens");
    const size_t rows = a.b[0].bytes / (HEAD_DIM * 2);
    const size_t pairs = rows * (ROT_DIMS / 2);
    if (int r = need_bytes(a, 1, rows / N_HEADS * (ROT_DIMS / 2) * 8, "cos_sin")) return r;
    if (pairs == 0) return 0;
    if (int r = need_aligned(a, {2, 8})) return r;
    const cudaError_t e = launch_dependent(rope_kernel, dim3(grid_for(pairs)), dim3(PRE_THREADS), 0, a.stream, (__half*)a.b[0].ptr, (const float2*)a.b[1].ptr, HEAD_DIM, ROT_DIMS / 2, N_HEADS, pairs);
    ++*a.launches;
    return check_cuda(a, e, "rope");
}
template int launch_rope<256, 256, 32>(const LaunchArgs&);
template int launch_rope<256, 256, 16>(const LaunchArgs&);
template int launch_rope<512, 128, 32>(const LaunchArgs&);
template int launch_rope<512, 128, 4>(const LaunchArgs&);

// attn_norm_rope_d128: x, w, cos_sin, y.  push {n_heads, rot_dims (0 = no rotation), plus_one}.
int launch_norm_rope_d128(const LaunchArgs& a)
{
    const PushNormRope p = *(const PushNormRope*)a.push;
    if (p.n_heads == 0 || p.rot_dims > 128 || p.rot_dims % 16) return fail_validation(a, "attn_norm_rope_d128: n_heads > 0, rot_dims a multiple of 16 up to 128");
    if (a.b[0].bytes % (256 * (size_t)p.n_heads)) return fail_validation(a, "attn_norm_rope_d128: x is not whole tokens of n_heads x 128");
    const size_t rows = a.b[0].bytes / 256;
    if (int r = need_bytes(a, 1, 128 * 4, "w")) return r;
    if (int r = need_bytes(a, 2, rows / p.n_heads * (p.rot_dims / 2) * 8, "cos_sin")) return r;
    if (int r = need_bytes(a, 3, a.b[0].bytes, "y")) return r;
    if (rows == 0) return 0;
    if (rows >= (1u << 27)) return fail_validation(a, "attn_norm_rope_d128: at most 2^27 rows per launch");
    if (int r = need_aligned(a, {16, 16, 16, 16})) return r;
    auto kern = p.plus_one ? norm_rope_d128_kernel<true> : norm_rope_d128_kernel<false>;
    const cudaError_t e = launch_dependent(kern, dim3(grid_for(rows * 16)), dim3(PRE_THREADS), 0, a.stream, (const __half*)a.b[0].ptr, (const float*)a.b[1].ptr, (const float2*)a.b[2].ptr, (__half*)a.b[3].ptr, p.n_heads, p.rot_dims / 2, (uint32_t)rows);
    ++*a.launches;
    return check_cuda(a, e, "attn_norm_rope_d128");
}

// kv_norm_rope_append_paged_q8_d128: k_raw, v_raw f16[n x row_len], k_w f32[128], cos_sin, k_scales, k_quants,
// v_scales, v_quants, page_table, step.  push {row_len, page, rot_dims, plus_one}.
int launch_kv_norm_rope_append_paged_q8_d128(const LaunchArgs& a)
{
    const PushKvNormRope p = *(const PushKvNormRope*)a.push;
    if (p.row_len == 0 || p.row_len % 128 || p.page == 0 || p.rot_dims > 128 || p.rot_dims % 16)
        return fail_validation(a, "kv_norm_rope_append_paged_q8_d128: row_len = n_kv_heads*128, page > 0, rot_dims a multiple of 16 up to 128");
    if (a.b[0].bytes % (p.row_len * 2) || a.b[1].bytes != a.b[0].bytes)
        return fail_validation(a, "kv_norm_rope_append_paged_q8_d128: k_raw and v_raw must be the same whole rows");
    const size_t tokens = a.b[0].bytes / (p.row_len * 2);
    if (int r = need_bytes(a, 2, 128 * 4, "k_w")) return r;
    if (int r = need_bytes(a, 3, tokens * (p.rot_dims / 2) * 8, "cos_sin")) return r;
    if (int r = need_bytes(a, 9, 16, "step")) return r;
    const size_t dst_rows = a.b[5].bytes / p.row_len;
    if (a.b[7].bytes / p.row_len != dst_rows) return fail_validation(a, "kv_norm_rope_append_paged_q8_d128: K and V pools differ in rows");
    if (a.b[4].bytes / 2 < dst_rows * (p.row_len / 32) || a.b[6].bytes / 2 < dst_rows * (p.row_len / 32))
        return fail_validation(a, "kv_norm_rope_append_paged_q8_d128: scales buffer too short for the quants buffer");
    const size_t kv_rows = a.b[0].bytes / 256;
    if (kv_rows == 0) return 0;
    if (kv_rows >= (1u << 26)) return fail_validation(a, "kv_norm_rope_append_paged_q8_d128: at most 2^26 (token, head) rows per launch");
    if (int r = need_aligned(a, {16, 16, 16, 16, 2, 8, 2, 8, 4, 4})) return r;
    const AppendShape shape = append_shape(a, tokens, 2 * (p.row_len / 128));
    const auto kern = append_kernel(p.plus_one != 0, shape.ahead);
    const cudaError_t e = launch_dependent(kern, shape.grid, dim3(APPEND_THREADS), 0, a.stream,
        nullptr, nullptr, nullptr, 0u,
        (const __half*)a.b[0].ptr, (const __half*)a.b[1].ptr, (const float*)a.b[2].ptr, (const float2*)a.b[3].ptr, (__half*)a.b[4].ptr,
        (int8_t*)a.b[5].ptr, (__half*)a.b[6].ptr, (int8_t*)a.b[7].ptr, (const uint32_t*)a.b[8].ptr, (uint32_t)(a.b[8].bytes / 4), p.page,
        (const uint32_t*)a.b[9].ptr, p.row_len / 128, p.rot_dims / 2, dst_rows, (uint32_t)tokens, shape.slot_bits, a.status);
    ++*a.launches;
    return check_cuda(a, e, "kv_norm_rope_append_paged_q8_d128");
}

// qkv_norm_rope_append_paged_q8_d128: q_raw f16[n x n_q x128], q_w f32[128], q_out f16, then the ten bindings of
// kv_norm_rope_append_paged_q8_d128.  push {n_q_heads, row_len, page, rot_dims, plus_one}.
int launch_qkv_norm_rope_append_paged_q8_d128(const LaunchArgs& a)
{
    const PushQkvNormRope p = *(const PushQkvNormRope*)a.push;
    if (p.n_q_heads == 0 || p.row_len == 0 || p.row_len % 128 || p.page == 0 || p.rot_dims > 128 || p.rot_dims % 16)
        return fail_validation(a, "qkv_norm_rope_append_paged_q8_d128: n_q_heads > 0, row_len = n_kv_heads*128, page > 0, rot_dims a multiple of 16 up to 128");
    const BufView* kv = a.b + 3;
    if (kv[0].bytes % (p.row_len * 2) || kv[1].bytes != kv[0].bytes)
        return fail_validation(a, "qkv_norm_rope_append_paged_q8_d128: k_raw and v_raw must be the same whole rows");
    const size_t tokens = kv[0].bytes / (p.row_len * 2);
    if (a.b[0].bytes != tokens * p.n_q_heads * 256) return fail_validation(a, "qkv_norm_rope_append_paged_q8_d128: q_raw must hold the same tokens");
    if (int r = need_bytes(a, 1, 128 * 4, "q_w")) return r;
    if (int r = need_bytes(a, 2, a.b[0].bytes, "q_out")) return r;
    if (int r = need_bytes(a, 5, 128 * 4, "k_w")) return r;
    if (int r = need_bytes(a, 6, tokens * (p.rot_dims / 2) * 8, "cos_sin")) return r;
    if (int r = need_bytes(a, 12, 16, "step")) return r;
    const size_t dst_rows = kv[5].bytes / p.row_len;
    if (kv[7].bytes / p.row_len != dst_rows) return fail_validation(a, "qkv_norm_rope_append_paged_q8_d128: K and V pools differ in rows");
    if (kv[4].bytes / 2 < dst_rows * (p.row_len / 32) || kv[6].bytes / 2 < dst_rows * (p.row_len / 32))
        return fail_validation(a, "qkv_norm_rope_append_paged_q8_d128: scales buffer too short for the quants buffer");
    const size_t kv_rows = kv[0].bytes / 256, q_rows = a.b[0].bytes / 256;
    if (kv_rows == 0) return 0;
    if (kv_rows >= (1u << 26) || q_rows >= (1u << 26))
        return fail_validation(a, "qkv_norm_rope_append_paged_q8_d128: at most 2^26 (token, head) rows of q and of k per launch");
    if (int r = need_aligned(a, {16, 16, 16, 16, 16, 16, 16, 2, 8, 2, 8, 4, 4})) return r;
    const AppendShape shape = append_shape(a, tokens, p.n_q_heads + 2 * (p.row_len / 128));
    const auto kern = append_kernel(p.plus_one != 0, shape.ahead);
    const cudaError_t e = launch_dependent(kern, shape.grid, dim3(APPEND_THREADS), 0, a.stream,
        (const __half*)a.b[0].ptr, (const float*)a.b[1].ptr, (__half*)a.b[2].ptr, p.n_q_heads, (const __half*)kv[0].ptr,
        (const __half*)kv[1].ptr, (const float*)kv[2].ptr, (const float2*)kv[3].ptr, (__half*)kv[4].ptr, (int8_t*)kv[5].ptr,
        (__half*)kv[6].ptr, (int8_t*)kv[7].ptr, (const uint32_t*)kv[8].ptr, (uint32_t)(kv[8].bytes / 4), p.page,
        (const uint32_t*)kv[9].ptr, p.row_len / 128, p.rot_dims / 2, dst_rows, (uint32_t)tokens, shape.slot_bits, a.status);
    ++*a.launches;
    return check_cuda(a, e, "qkv_norm_rope_append_paged_q8_d128");
}

}  // namespace sgb
