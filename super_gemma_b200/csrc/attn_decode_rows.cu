// Decode over f16 values: the reference-shaped split-K kernels (head_dim 256 over the ring, head_dim 512 over f16 or Q8_0 keys,
// head_dim 128 over the ring) and the verify step of up to four drafted tokens over the ring, head_dim 128.
//
// All of them are a few query rows (<= 8: the query heads of a kv head, times the drafted tokens) against many keys, bound by
// the bytes of K and V.  A warp takes 16 keys at a time: they arrive by TMA, 128 bytes of all 16 rows to a copy (128-byte
// swizzle), in the warp's own slots (K and V apart, so that the next K is on its way while this V is used).  S = K Q^T
// and O^T += V^T P^T are mma.sync m16n8k16 with the keys or 16 dims as M and the rows as N: tcgen05 has no tile this small.
// Warps never wait for one another before the end, where their states merge in warp order.
// Precision is that of the f32 statement (attn_decode_sliding.wgsl:84-107): Q8_0 keys enter as whole numbers and every block's
// sum is multiplied by its f32 scale; products of f16 keys are added up 16 at a time in f32, for the tensor pipe truncates what it
// adds to; P = (hi + lo) * 2^-14, both halves f16, which together miss p by at most one unit of its last f32 place (the factor keeps
// lo out of f16's subnormals; a p below 2^-39 of its row's maximum is in l but too small for lo); running maximum and sums in f32.
// Error of the verify step against 64 bits, streaming kernel | this one: 60 cached tokens 1.56e-7 | 1.49e-7 (2.2e-7 while scores were
// summed in the tensor pipe and hi went first), 700 tokens 3.0e-7 | 1.9e-7, 9000 tokens 3.5e-7 | 2.1e-7.
// Measured (us a call, streaming kernel before -> this one): head_dim 512, Q8_0 keys, 32768 tokens, 32 splits 427 -> 40.6
// (206 MB, 5.1 TB/s on the 128 SMs that 4 x 32 CTAs occupy); head_dim 256, 1024 slots, 16 splits 12.3 -> 5.7; verify of 4 tokens over
// the ring, 16 kv heads 145 -> 8.2.
// A bulk copy per row instead (48 a tile at head_dim 512) took 41.8 us.
// V rows that hold no visible key are zeroed once they have arrived, and rows that are not finite are computed again by the streaming
// statement: a tile multiplies by p = 0 what that statement skips (all of them at 32768 tokens: 427 us on the streaming kernel).
#include <mutex>
#include <string>

#include "attn_stream.cuh"
#include "sgb_common.cuh"
#include "sgb_kernels.h"

namespace sgb {

namespace {

constexpr int TILE = 16;
constexpr float P_SCALE = 16384.0f;

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a)
{
    uint32_t d;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ float key_max(float v)
{
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 4));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 8));
    return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 16));
}
__device__ __forceinline__ float key_sum(float v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
}
// Four signed bytes as two f16 pairs, exactly: 0x6400 | (q + 128) = q + 1152 as f16.
__device__ __forceinline__ void bytes_to_f16(uint32_t x, uint32_t& p01, uint32_t& p23)
{
    const uint32_t u = x ^ 0x80808080u;
    uint32_t a = __byte_perm(u, 0x64646464u, 0x4140), b = __byte_perm(u, 0x64646464u, 0x4342);
    const __half2 off = __float2half2_rn(1152.0f);
    __half2 ha = __hsub2(*reinterpret_cast<__half2*>(&a), off), hb = __hsub2(*reinterpret_cast<__half2*>(&b), off);
    p01 = *reinterpret_cast<uint32_t*>(&ha);
    p23 = *reinterpret_cast<uint32_t*>(&hb);
}

// One 16-key tile: its tensor maps and first row, which of its rows are keys, [from, to), and the position of row 0.
struct KeyTile {
    const CUtensorMap *k, *sc, *v;
    int row0, from, to;
    int64_t pos0;
};

template <int HD, bool KQ8, int ROWS>
struct RowsWarp {
    static constexpr int K_PIECES = HD * (KQ8 ? 1 : 2) / 128, V_PIECES = HD * 2 / 128;  // copies of [16 rows][128 bytes]
    static constexpr uint32_t PIECE = TILE * 128, SC_ROW = KQ8 ? HD / 16 : 0;           // bytes
    struct __align__(1024) Slots {
        uint8_t k[K_PIECES][PIECE];
        uint8_t v[V_PIECES][PIECE];  // afterwards the warp's output [ROWS][HD] f32
        __align__(128) uint8_t sc[TILE * SC_ROW + 128];
        uint64_t k_full, v_full;
        float m[8], l[8];
    };
    static_assert(sizeof(Slots::v) >= ROWS * HD * 4, "the V slot doubles as the merge buffer");

    float o[HD / 16][4];  // dims 16c + g, 16c + g + 8 x rows 2*t4, 2*t4 + 1
    float m[2], l[2];
    uint32_t odd;  // rows with an infinite Q8_0 scale among their keys, as far as this lane saw

    // All tiles of this warp.  n tiles; tile(i, KeyTile&) describes the i-th.  row_lo/row_hi: positions rows 2*t4 + e may see.
    // q_sm: [8][q_pitch] f16 query rows.
    template <typename TileFn>
    __device__ __forceinline__ void run(Slots& sl, int n, TileFn tile, const uint8_t* q_sm, int kvh, float scale, const int64_t (&row_lo)[2],
                                        const int64_t (&row_hi)[2], uint32_t* status)
    {
        constexpr int Q_PITCH = HD * 2 + (KQ8 ? 32 : 16);
        const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
        auto issue_k = [&](int i) {
            KeyTile t;
            tile(i, t);
            fence_proxy_async_smem();  // the slot was read through the generic proxy
            if (lane == 0) mbar_arrive_expect_tx(&sl.k_full, K_PIECES * PIECE + TILE * SC_ROW);
            __syncwarp();
            if (lane < K_PIECES) tma_load_3d(sl.k[lane], t.k, &sl.k_full, lane * (KQ8 ? 128 : 64), kvh, t.row0);
            if (KQ8 && lane == K_PIECES) tma_load_3d(sl.sc, t.sc, &sl.k_full, 0, kvh, t.row0);
        };
        auto issue_v = [&](int i) {
            KeyTile t;
            tile(i, t);
            fence_proxy_async_smem();
            if (lane == 0) mbar_arrive_expect_tx(&sl.v_full, V_PIECES * PIECE);
            __syncwarp();
            if (lane < V_PIECES) tma_load_3d(sl.v[lane], t.v, &sl.v_full, lane * 64, kvh, t.row0);
        };
#pragma unroll
        for (int c = 0; c < HD / 16; c++) o[c][0] = o[c][1] = o[c][2] = o[c][3] = 0.0f;
        m[0] = m[1] = NEG_SENTINEL;
        l[0] = l[1] = 0.0f;
        float most[2] = {0.0f, 0.0f};  // largest magnitude of the rows' scores, whole tiles (Q8_0 keys)
        bool failed = false;
        if (n > 0) {
            issue_k(0);
            issue_v(0);
        }
        // ldmatrix: K plain, lane -> (row (lane & 7) + 8 * bit 3, 16-byte chunk + bit 4); V transposed, the two bits swapped.  Chunk c
        // of a row lies in piece c / 8 at (c % 8) ^ (row & 7).
        const uint32_t sw = lane & 7, k_addr = smem_u32(sl.k) + (sw + 8 * ((lane >> 3) & 1)) * 128, v_addr = smem_u32(sl.v) + (sw + 8 * (lane >> 4)) * 128;
        const uint32_t k_bit = lane >> 4, v_bit = (lane >> 3) & 1;
        auto at = [&](uint32_t base, uint32_t chunk) { return base + (chunk >> 3) * PIECE + (((chunk & 7) ^ sw) << 4); };
        const uint8_t* q_row = q_sm + g * Q_PITCH + t4 * (KQ8 ? 8 : 4);
        for (int i = 0; i < n; ++i) {
            KeyTile t;
            tile(i, t);
            if (!mbar_wait_warp(&sl.k_full, i & 1, status, 601, failed)) break;
            float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // keys g (0, 1) and g + 8 (2, 3) x rows 2*t4, 2*t4 + 1
            if constexpr (KQ8) {
                uint4 sa[2], sc[2];  // 16 block scales of keys g and g + 8
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    sa[h] = *reinterpret_cast<const uint4*>(sl.sc + g * SC_ROW + 16 * h);
                    sc[h] = *reinterpret_cast<const uint4*>(sl.sc + (g + 8) * SC_ROW + 16 * h);
                }
                const __half* ha = reinterpret_cast<const __half*>(sa);
                const __half* hc = reinterpret_cast<const __half*>(sc);
#pragma unroll
                for (int b = 0; b < HD / 32; b += 2) {  // two blocks side by side: their MMAs do not wait for each other
                    float acc[2][4] = {};
                    uint32_t x[2][4];
#pragma unroll
                    for (int h = 0; h < 2; h++) ldsm_x4(at(k_addr, 2 * (b + h) + k_bit), x[h]);
#pragma unroll
                    for (int cc = 0; cc < 2; cc++) {
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            uint32_t a[4];
                            bytes_to_f16(x[h][2 * cc], a[0], a[2]);
                            bytes_to_f16(x[h][2 * cc + 1], a[1], a[3]);
                            const uint2 q = *reinterpret_cast<const uint2*>(q_row + (2 * (b + h) + cc) * 32);
                            mma16816(acc[h], a, q.x, q.y);
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float fa = __half2float(ha[b + h]), fc = __half2float(hc[b + h]);
                        s[0] = fmaf(fa, acc[h][0], s[0]);
                        s[1] = fmaf(fa, acc[h][1], s[1]);
                        s[2] = fmaf(fc, acc[h][2], s[2]);
                        s[3] = fmaf(fc, acc[h][3], s[3]);
                    }
                }
            } else {
                // every product starts from 0 and is added in f32: the tensor pipe truncates what it adds to
#pragma unroll
                for (int c = 0; c < HD / 16; c += 2) {
                    float acc[2][4] = {};
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint32_t a[4];
                        ldsm_x4(at(k_addr, 2 * (c + h) + k_bit), a);
                        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(q_row + 32 * (c + h)), b1 = *reinterpret_cast<const uint32_t*>(q_row + 32 * (c + h) + 16);
                        mma16816(acc[h], a, b0, b1);
                    }
#pragma unroll
                    for (int e = 0; e < 4; e++) s[e] += acc[0][e] + acc[1][e];
                }
            }
            __syncwarp();
            if (i + 1 < n) issue_k(i + 1);
            if (KQ8)
                for (int e = 0; e < 2; e++) most[e] = max3(most[e], fabsf(s[e]), fabsf(s[2 + e]));
#pragma unroll
            for (int e = 0; e < 4; e++) {
                s[e] *= scale;
                const int key = g + 8 * (e >> 1);
                const int64_t pos = t.pos0 + key;
                if (key < t.from || key >= t.to || pos < row_lo[e & 1] || pos > row_hi[e & 1]) s[e] = -INFINITY;
            }
            float p[4];
            const float n0 = fmaxf(m[0], key_max(fmaxf(s[0], s[2]))), n1 = fmaxf(m[1], key_max(fmaxf(s[1], s[3])));
            if (__any_sync(0xffffffffu, n0 != m[0] || n1 != m[1])) {
                const float c0 = __expf(m[0] - n0), c1 = __expf(m[1] - n1);
                l[0] *= c0;
                l[1] *= c1;
#pragma unroll
                for (int c = 0; c < HD / 16; c++) {
                    o[c][0] *= c0;
                    o[c][1] *= c1;
                    o[c][2] *= c0;
                    o[c][3] *= c1;
                }
                m[0] = n0;
                m[1] = n1;
            }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                p[e] = __expf(s[e] - m[e & 1]);
                l[e & 1] += p[e];
                p[e] *= P_SCALE;
            }
            uint32_t hi[2], lo[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t w = pack_half2(p[2 * h], p[2 * h + 1]);
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
                hi[h] = movmatrix_trans(w);
                lo[h] = movmatrix_trans(pack_half2(p[2 * h] - f.x, p[2 * h + 1] - f.y));
            }
            if (!mbar_wait_warp(&sl.v_full, i & 1, status, 602, failed)) break;
            if (t.from > 0 || t.to < TILE) {  // p = 0 in the rows that are no keys, and 0 times a stale Inf or NaN would not be
                for (int w = lane; w < V_PIECES * TILE * 8; w += 32) {
                    const int r = (w >> 3) & (TILE - 1);
                    if (r < t.from || r >= t.to) *reinterpret_cast<uint4*>(&sl.v[0][0] + 16 * w) = make_uint4(0u, 0u, 0u, 0u);
                }
                __syncwarp();
            }
#pragma unroll
            for (int c = 0; c < HD / 16; c += 4) {  // four accumulators at a time: hi and lo of one would wait for each other
                uint32_t a[4][4];
#pragma unroll
                for (int k = 0; k < 4; k++) ldsm_x4_trans(at(v_addr, 2 * (c + k) + v_bit), a[k]);
#pragma unroll
                for (int k = 0; k < 4; k++) mma16816(o[c + k], a[k], lo[0], lo[1]);  // before hi: the first tile's is then exact in o
#pragma unroll
                for (int k = 0; k < 4; k++) mma16816(o[c + k], a[k], hi[0], hi[1]);
            }
            __syncwarp();
            if (i + 1 < n) issue_v(i + 1);
        }
        if (failed) let_copies_land();  // into this warp's slots, one of which is written next
        // Finite scales cannot give an infinite score.  An infinite one times a block's whole sum could pass as a weight of 0; the statement
        // multiplies the scale with every quant, and infinities of both signs make a NaN.  (Rows that are no keys count here
        // too: the statement then only confirms the row.)
        odd = 0;
        for (int e = 0; e < 2; e++)
            if (most[e] == INFINITY) odd |= 1u << (2 * t4 + e);
        // the state for the merge: [row][HD], m, l
        l[0] = key_sum(l[0]);
        l[1] = key_sum(l[1]);
        float* dst = reinterpret_cast<float*>(sl.v);
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int r = 2 * t4 + e;
            if (r < ROWS) {
#pragma unroll
                for (int c = 0; c < HD / 16; c++) {
                    dst[r * HD + 16 * c + g] = o[c][e] * (1.0f / P_SCALE);
                    dst[r * HD + 16 * c + g + 8] = o[c][2 + e] * (1.0f / P_SCALE);
                }
                if (g == 0) {
                    sl.m[r] = m[e];
                    sl.l[r] = l[e];
                }
            }
        }
    }
};

// Query rows -> shared memory, [8][HD] f16 with the pitch the MMAs want; rows >= live are zero.
template <int HD, bool KQ8, typename RowPtr>
__device__ __forceinline__ void stage_queries(uint8_t* q_sm, int live, RowPtr row_ptr)
{
    constexpr int Q_PITCH = HD * 2 + (KQ8 ? 32 : 16);
    for (int i = threadIdx.x; i < 8 * HD / 8; i += blockDim.x) {
        const int r = i / (HD / 8), c = i % (HD / 8);
        uint4 u = make_uint4(0u, 0u, 0u, 0u);
        if (r < live) u = ld_global(reinterpret_cast<const uint4*>(row_ptr(r)) + c);
        *reinterpret_cast<uint4*>(q_sm + r * Q_PITCH + 16 * c) = u;
    }
}

template <int HD, int G, bool KQ8, int WARPS>
struct DecodeRowsSmem {
    typename RowsWarp<HD, KQ8, G>::Slots w[WARPS];
    uint8_t q[8 * (HD * 2 + (KQ8 ? 32 : 16))];
    uint32_t redo;  // rows that are not finite, a bit each
};

// Split-K partials.  Grid, split ranges and partials as decode_generic_kernel.
template <int HD, int G, bool KQ8, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, HD == 512 ? 1 : HD == 256 ? 3 : 5)  // CTAs that the slots let an SM hold, one less at 128 (6: 80 registers, slower)
    decode_rows_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_sc, const __grid_constant__ CUtensorMap tm_v,
                       const __half* q, const __grid_constant__ KvOperand kop, const __grid_constant__ KvOperand vop,
                       float* __restrict__ part, const uint32_t* step, int step_slot, uint32_t n_splits, float scale, uint32_t* status)
{
    using W = RowsWarp<HD, KQ8, G>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    DecodeRowsSmem<HD, G, KQ8, WARPS>& sm = *reinterpret_cast<DecodeRowsSmem<HD, G, KQ8, WARPS>*>(smem_raw);
    if ((smem_u32(smem_raw) & 1023u) != 0u) {  // the swizzled tiles need it; never seen, but never assumed
        if (threadIdx.x == 0) report_error(status, DEV_ERR_BOUNDS, 603, smem_u32(smem_raw), 0);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kvh = blockIdx.x, n_kv = gridDim.x, split = blockIdx.y, n_q = n_kv * G;
    const uint32_t i = blockIdx.z, m_q = gridDim.z;
    if (lane == 0) {
        mbar_init(&sm.w[warp].k_full, 1);
        mbar_init(&sm.w[warp].v_full, 1);
        mbar_fence_init();
    }
    if (threadIdx.x == 0) sm.redo = 0;
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t kv_len = ld_global(step + step_slot);
    const uint32_t chunk = (kv_len + n_splits - 1) / n_splits;
    const uint32_t t_begin = min((uint32_t)split * chunk, kv_len);
    uint32_t t_end = min(t_begin + chunk, kv_len);
    const uint32_t vis_end = kv_len + i >= m_q ? kv_len + i - m_q + 1 : 0;  // query i of m_q sees t <= kv_len - m_q + i
    t_end = min(t_end, vis_end);
    const size_t have = min(kop.rows, vop.rows);
    if (t_end > t_begin && t_end > have) {
        if (threadIdx.x == 0) report_error(status, DEV_ERR_BOUNDS, kop.rows <= vop.rows ? 202 : 204, (uint32_t)have, (uint32_t)have);
        t_end = max((uint32_t)have, t_begin);
    }
    if (t_end <= t_begin) {  // an empty split (a short sequence, many splits): nothing to wait for
        for (int idx = threadIdx.x; idx < G * (HD + 2); idx += WARPS * 32) {
            const int r = idx / (HD + 2), d = idx % (HD + 2);
            part[(((size_t)i * n_q + kvh * G + r) * n_splits + split) * (HD + 2) + d] = d == HD ? NEG_SENTINEL : 0.0f;
        }
        return;
    }
    const int tiles = (int)((t_end - t_begin + TILE - 1) / TILE);
    auto q_row = [&](int r) { return q + ((size_t)i * n_q + kvh * G + r) * HD; };
    stage_queries<HD, KQ8>(sm.q, G, q_row);
    __syncthreads();
    W w;
    const int64_t lo[2] = {0, 0}, hi[2] = {INT64_MAX, INT64_MAX};
    w.run(sm.w[warp], tiles > warp ? (tiles - warp + WARPS - 1) / WARPS : 0,
          [&](int n, KeyTile& t) {
              t.row0 = (int)(t_begin + (uint32_t)(warp + n * WARPS) * TILE);
              t.from = 0;
              t.to = min(TILE, (int)t_end - t.row0);
              t.pos0 = 0;
              t.k = &tm_k;
              t.sc = &tm_sc;
              t.v = &tm_v;
          },
          sm.q, kvh, scale, lo, hi, status);
    __syncthreads();
    uint32_t odd = KQ8 ? w.odd : 0;
    for (int idx = threadIdx.x; idx < G * HD; idx += WARPS * 32) {
        const int r = idx / HD, d = idx % HD;
        float big = sm.w[0].m[r];
#pragma unroll
        for (int k = 1; k < WARPS; k++) big = fmaxf(big, sm.w[k].m[r]);
        float acc = 0.0f, l = 0.0f;
#pragma unroll
        for (int k = 0; k < WARPS; k++) {
            const float f = __expf(sm.w[k].m[r] - big);
            acc = fmaf(f, reinterpret_cast<const float*>(sm.w[k].v)[idx], acc);
            l = fmaf(f, sm.w[k].l[r], l);
        }
        if (!(fabsf(acc) <= 3.4e38f) || !(fabsf(l) <= 3.4e38f)) odd |= 1u << r;
        float* row = part + (((size_t)i * n_q + kvh * G + r) * n_splits + split) * (HD + 2);
        row[d] = acc;
        if (d == 0) {
            row[HD] = big;
            row[HD + 1] = l;
        }
    }
    if (odd != 0) atomicOr(&sm.redo, odd);
    if (__syncthreads_or(odd)) {  // again by the streaming statement, a warp per row
        constexpr int DPL = HD / 32;
        const uint32_t redo = sm.redo;
        for (int r = warp; r < G; r += WARPS) {
            if (((redo >> r) & 1) == 0) continue;
            float qr[1][DPL];
            load_f16<DPL>(q_row(r) + lane * DPL, qr[0]);
            Stream<1, DPL> st;
            st.init();
            stream_keys<HD, KQ8 ? FMT_Q8 : FMT_F16, 1, HD == 128 ? 4 : 8>(st, qr, kop, vop, t_begin, t_end, 0, kvh, n_kv, scale);
            float* row = part + (((size_t)i * n_q + kvh * G + r) * n_splits + split) * (HD + 2);
#pragma unroll
            for (int d = 0; d < DPL; d++) row[lane * DPL + d] = st.acc[0][d];
            if (lane == 0) {
                row[HD] = st.m[0];
                row[HD + 1] = st.l[0];
            }
        }
    }
}

// ---- verify over the ring: m <= 4 tokens x 2 heads = 8 rows, a cluster of 8 CTAs per kv head ------------------------------
constexpr int V_HD = 128, V_G = 2, V_WARPS = 4, V_CTAS = 8, V_DPL = V_HD / 32;

struct VerifySmem {
    RowsWarp<V_HD, false, 8>::Slots w[V_WARPS];
    uint8_t q[8 * (V_HD * 2 + 16)];
    float acc[8][V_HD], m[8], l[8];  // this CTA's merged rows, read by the cluster
};

__device__ __forceinline__ const float* map_to_rank(const float* p, uint32_t rank)
{
    uint64_t out;
    asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<uint64_t>(p)), "r"(rank));
    return reinterpret_cast<const float*>(out);
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(V_CTAS, 1, 1) __launch_bounds__(V_WARPS * 32)
    verify_ring_kernel(const __grid_constant__ CUtensorMap tm_kr, const __grid_constant__ CUtensorMap tm_vr, const __grid_constant__ CUtensorMap tm_kn,
                       const __grid_constant__ CUtensorMap tm_vn, const __half* q, const __grid_constant__ KvOperand k_ring, const __grid_constant__ KvOperand v_ring,
                       const __grid_constant__ KvOperand k_new, const __grid_constant__ KvOperand v_new, float* __restrict__ out,
                       const uint32_t* step, uint32_t n_kv, uint32_t m_q, uint32_t window, uint32_t ring, float scale, uint32_t* status)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    VerifySmem& sm = *reinterpret_cast<VerifySmem*>(smem_raw);
    if ((smem_u32(smem_raw) & 1023u) != 0u) {  // the swizzled tiles need it; never seen, but never assumed
        if (threadIdx.x == 0) report_error(status, DEV_ERR_BOUNDS, 604, smem_u32(smem_raw), 0);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t4 = lane & 3;
    const int kvh = blockIdx.x / V_CTAS, rank = blockIdx.x % V_CTAS, n_q = (int)n_kv * V_G, rows = (int)m_q * V_G;
    if (lane == 0) {
        mbar_init(&sm.w[warp].k_full, 1);
        mbar_init(&sm.w[warp].v_full, 1);
        mbar_fence_init();
    }
    pdl_wait();
    pdl_launch_dependents();
    const int64_t q0 = ld_global(step + STEP_Q0);
    const int64_t band_lo = q0 + 1 > window ? q0 + 1 - window : 0;  // the first query's
    const int64_t first = band_lo / TILE * TILE;
    const int n_hist = q0 > band_lo ? (int)((q0 - 1) / TILE - first / TILE + 1) : 0, tiles = n_hist + 1;  // the draft is one tile
    auto q_row = [&](int r) { return q + ((size_t)(r / V_G) * n_q + kvh * V_G + r % V_G) * V_HD; };
    stage_queries<V_HD, false>(sm.q, rows, q_row);
    __syncthreads();
    int64_t lo[2], hi[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int64_t qpos = q0 + min(2 * t4 + e, rows - 1) / V_G;
        lo[e] = qpos + 1 > window ? qpos + 1 - window : 0;
        hi[e] = qpos;
    }
    const int me = rank * V_WARPS + warp;
    RowsWarp<V_HD, false, 8> w;
    w.run(sm.w[warp], tiles > me ? (tiles - me + V_CTAS * V_WARPS - 1) / (V_CTAS * V_WARPS) : 0,
          [&](int n, KeyTile& t) {
              const int it = me + n * V_CTAS * V_WARPS;
              if (it < n_hist) {
                  t.pos0 = first + (int64_t)it * TILE;
                  t.row0 = (int)(t.pos0 % ring);
                  t.from = (int)max((int64_t)0, band_lo - t.pos0);
                  t.to = (int)min((int64_t)TILE, q0 - t.pos0);
                  t.k = &tm_kr;
                  t.v = &tm_vr;
              } else {
                  t.pos0 = q0;
                  t.row0 = 0;
                  t.from = 0;
                  t.to = (int)m_q;
                  t.k = &tm_kn;
                  t.v = &tm_vn;
              }
          },
          sm.q, kvh, scale, lo, hi, status);
    __syncthreads();
    for (int idx = threadIdx.x; idx < 8 * V_HD; idx += V_WARPS * 32) {
        const int r = idx / V_HD, d = idx % V_HD;
        float big = sm.w[0].m[r];
#pragma unroll
        for (int k = 1; k < V_WARPS; k++) big = fmaxf(big, sm.w[k].m[r]);
        float acc = 0.0f, l = 0.0f;
#pragma unroll
        for (int k = 0; k < V_WARPS; k++) {
            const float f = __expf(sm.w[k].m[r] - big);
            acc = fmaf(f, reinterpret_cast<const float*>(sm.w[k].v)[idx], acc);
            l = fmaf(f, sm.w[k].l[r], l);
        }
        sm.acc[r][d] = acc;
        if (d == 0) {
            sm.m[r] = big;
            sm.l[r] = l;
        }
    }
    cluster_sync();
    bool odd = false;
    if (rank < rows) {  // CTA `rank` owns row `rank`: merge the cluster's states in rank order
        const int d = threadIdx.x;  // V_WARPS * 32 == V_HD
        float mk[V_CTAS], big = NEG_SENTINEL;
#pragma unroll
        for (int k = 0; k < V_CTAS; k++) {
            mk[k] = *map_to_rank(&sm.m[rank], k);
            big = fmaxf(big, mk[k]);
        }
        float acc = 0.0f, l = 0.0f;
#pragma unroll
        for (int k = 0; k < V_CTAS; k++) {
            const float f = __expf(mk[k] - big);
            acc = fmaf(f, *map_to_rank(&sm.acc[rank][d], k), acc);
            l = fmaf(f, *map_to_rank(&sm.l[rank], k), l);
        }
        const float y = acc / l;
        odd = !(fabsf(y) <= 3.4e38f);
        out[((size_t)(rank / V_G) * n_q + kvh * V_G + rank % V_G) * V_HD + d] = y;
    }
    cluster_sync();  // nobody leaves while its shared memory is read
    if (__syncthreads_or(odd) && warp == 0) {  // this CTA's row again, by the streaming statement
        const uint32_t i = rank / V_G, qpos = (uint32_t)q0 + i, begin = qpos + 1 > window ? qpos + 1 - window : 0;
        float qr[1][V_DPL];
        load_f16<V_DPL>(q_row(rank) + lane * V_DPL, qr[0]);
        Stream<1, V_DPL> st;
        st.init();
        stream_keys<V_HD, FMT_F16, 1, 8>(st, qr, k_ring, v_ring, begin, (uint32_t)q0, ring, kvh, (int)n_kv, scale);
        const uint32_t c0 = begin > (uint32_t)q0 ? begin - (uint32_t)q0 : 0;
        stream_keys<V_HD, FMT_F16, 1, 4>(st, qr, k_new, v_new, c0, i + 1, 0, kvh, (int)n_kv, scale);
#pragma unroll
        for (int d = 0; d < V_DPL; d++) out[((size_t)i * n_q + kvh * V_G + rank % V_G) * V_HD + lane * V_DPL + d] = st.acc[0][d] / st.l[0];
    }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// [row][head][n] tensor of `elem`-byte values, boxes of n_box x 1 x 16 rows.
int encode_tiles(const LaunchArgs& a, CUtensorMap* tm, const void* base, uint64_t rows, uint64_t heads, uint64_t n, uint32_t n_box, int elem, int swizzle)
{
    const uint64_t dims[3] = {n, heads, rows};
    const uint64_t strides[2] = {n * elem, heads * n * elem};
    const uint32_t box[3] = {n_box, 1, TILE};
    return encode_tensor_map(a, tm, elem == 2, 3, const_cast<void*>(base), dims, strides, box, swizzle);
}

template <typename Kern>
int allow_smem(const LaunchArgs& a, Kern kern, size_t smem)
{
    static std::mutex attr_mutex;
    static bool attr_set[64] = {};
    std::lock_guard<std::mutex> lock(attr_mutex);
    if (a.device < 64 && attr_set[a.device]) return 0;
    if (int r = check_cuda(a, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "cudaFuncSetAttribute(decode_rows)")) return r;
    if (a.device < 64) attr_set[a.device] = true;
    return 0;
}

}  // namespace

// The copies need 16-byte aligned bases and row numbers within an int.  What else the launcher accepts stays on the streaming kernel:
// quants and scales of any alignment, head_dim 128 rows on 8 bytes (f16 rows of 256 and 512 need 16 there too).
bool decode_rows_takes(const KvOperand& k, const KvOperand& v, const void* q)
{
    for (const KvOperand* o : {&k, &v})
        if (o->rows == 0 || o->rows >= (1u << 30)) return false;
    return aligned16(k.data) && aligned16(v.data) && aligned16(q) && (k.scales == nullptr || aligned16(k.scales));
}

template <int HD, int G, bool KQ8>
int launch_decode_rows(const LaunchArgs& a, const void* q, const KvOperand& k, const KvOperand& v, void* part, const void* step, int step_slot,
                       uint32_t n_kv, uint32_t n_splits, uint32_t m_q, float scale)
{
    // warps per CTA: what fits the shared memory at head_dim 512 (one CTA per SM), four elsewhere (three or more CTAs per SM)
    constexpr int WARPS = HD == 512 ? (KQ8 ? 8 : 6) : 4;
    constexpr size_t smem = sizeof(DecodeRowsSmem<HD, G, KQ8, WARPS>);
    static_assert(smem <= 227 * 1024, "one CTA per SM");
    auto kern = decode_rows_kernel<HD, G, KQ8, WARPS>;
    {
        static std::mutex attr_mutex;
        static bool attr_set[64] = {};
        std::lock_guard<std::mutex> lock(attr_mutex);
        if (a.device >= 64 || !attr_set[a.device]) {
            if (int r = check_cuda(a, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "cudaFuncSetAttribute(decode_rows)")) return r;
            if (a.device < 64) attr_set[a.device] = true;
        }
    }
    CUtensorMap tk, ts, tv;
    if (int r = encode_tiles(a, &tk, k.data, k.rows, n_kv, HD, KQ8 ? 128 : 64, KQ8 ? 1 : 2, 3)) return r;
    if (int r = encode_tiles(a, &tv, v.data, v.rows, n_kv, HD, 64, 2, 3)) return r;
    ts = tk;
    if (KQ8)
        if (int r = encode_tiles(a, &ts, k.scales, k.rows, n_kv, HD / 32, HD / 32, 2, 0)) return r;
    const cudaError_t e = launch_dependent(kern, dim3(n_kv, n_splits, m_q), dim3(WARPS * 32), smem, a.stream, tk, ts, tv, (const __half*)q, k, v, (float*)part,
                                           (const uint32_t*)step, step_slot, n_splits, scale, a.status);
    ++*a.launches;
    return check_cuda(a, e, "attn_decode");
}
template int launch_decode_rows<256, 2, false>(const LaunchArgs&, const void*, const KvOperand&, const KvOperand&, void*, const void*, int, uint32_t, uint32_t, uint32_t, float);
template int launch_decode_rows<512, 8, false>(const LaunchArgs&, const void*, const KvOperand&, const KvOperand&, void*, const void*, int, uint32_t, uint32_t, uint32_t, float);
template int launch_decode_rows<512, 8, true>(const LaunchArgs&, const void*, const KvOperand&, const KvOperand&, void*, const void*, int, uint32_t, uint32_t, uint32_t, float);
template int launch_decode_rows<128, 2, false>(const LaunchArgs&, const void*, const KvOperand&, const KvOperand&, void*, const void*, int, uint32_t, uint32_t, uint32_t, float);

int launch_verify_ring_d128(const LaunchArgs& a, const void* q, const KvOperand& k_ring, const KvOperand& v_ring, const KvOperand& k_new,
                            const KvOperand& v_new, void* out, const void* step, uint32_t n_kv, uint32_t m, uint32_t window, uint32_t ring, float scale)
{
    constexpr size_t smem = sizeof(VerifySmem);
    static_assert(smem <= 100 * 1024, "two or more CTAs per SM");
    if (int r = allow_smem(a, verify_ring_kernel, smem)) return r;
    CUtensorMap tm[4];
    const KvOperand* const ops[4] = {&k_ring, &v_ring, &k_new, &v_new};
    for (int i = 0; i < 4; i++)
        if (int r = encode_tiles(a, &tm[i], ops[i]->data, ops[i]->rows, n_kv, V_HD, 64, 2, 3)) return r;
    const cudaError_t e = launch_dependent(verify_ring_kernel, dim3(n_kv * V_CTAS), dim3(V_WARPS * 32), smem, a.stream, tm[0], tm[1], tm[2], tm[3], (const __half*)q, k_ring, v_ring,
                                           k_new, v_new, (float*)out, (const uint32_t*)step, n_kv, m, window, ring, scale, a.status);
    ++*a.launches;
    return check_cuda(a, e, "attn_verify_sliding_ring");
}

}  // namespace sgb
