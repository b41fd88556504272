// Prefill attention for the reference model's global layers on tcgen05: head_dim 512, int8 Q and K with f16 block scales, f16 V,
// 8 query heads per kv head (attn_prefill_global_flash_sp_iq.wgsl).
//
// A head of 512 dims fills tensor memory with a 128-row f32 output alone, so everything here is transposed: keys and output
// dims are the M = 128 side of the MMAs, and a CTA's 64 query rows (8 tokens x the 8 query heads of one kv head, which
// share every K/V tile) are the N side.  Per 128-key tile:
//   S^T[128 keys x 64 rows]  = K Q^T    thread = key, so a key's scales are that thread's registers
//   O^T[512 dims x 64 rows] += V^T P^T  V is the MN-major A operand straight from its [key][dim] tile, P^T the MN-major B
//                                       operand that each thread writes as one swizzled 128-byte row
// One kind::i8 MMA (K = 32) per scale block gives that block's whole-number dot product, exactly; the two f16 scales multiply
// it in f32 (f32(qs) * f32(ks) is exact), so the score is closer to f32(scale) * f32(q) arithmetic than an f32 dot product.
// Blocks go through four 64-column buffers, two per hand-over.
// P = hi + lo, both halves f16, two MMAs per V tile: together they miss p by at most one unit of its last f32 place.  The exponent
// carries +7, so that lo stays clear of f16's subnormals (the factor cancels in O / l); a p below 2^-32 of its row's reference
// maximum is in l but too small for lo.
// The tensor pipe truncates an accumulator each time it adds to it: in one accumulator, outputs shrank by 2e-9 of themselves per
// key (1.7e-5 at 8192 keys, 6.7e-5 at 33280, where the error against 64 bits was 2.22e-4 instead of f16's own 2.08e-4).  From the
// fifth tile on the softmax threads therefore settle one of the four dim blocks of O in every tile: the block, plus what was
// settled of it before, added in f32 with rounding, splits into its upper 16 bits, which they keep in this CTA's share of the
// output, and the exact rest, from which the tensor pipe goes on; what it adds to stays as small as the sum of four tiles.
// Another block comes first in each tile's products, so that it can be settled while the tensor pipe is at the others.  Errors since:
// 2.0762e-4 and 2.0773e-4 (streaming kernel: 2.0762e-4, 2.0774e-4), for 23 us of 533 at 8192 keys; all four blocks in every
// fourth tile, with the tensor pipe waiting, took 44.
// Roles: warps 0-7 softmax (two threads per key, 32 rows each), one MMA thread, one K and one V loader; mbarriers only.
// The row maximum over keys runs across threads; it is only computed (32 values in 31 shuffles) when some score exceeds its
// row's running maximum by 2^8, which one barrier with an OR finds out.
// Measured: 256 queries at 7936 + 256 keys 13500 us on the streaming kernel, 533 here (floor 86).  Two things bound it: V as the
// MN-major A operand costs 160 cycles per instruction (10000 of a tile's 14400), and every block's scores cross from tensor
// memory to registers (16 x 32 KB a tile, 500 cycles each).  Rows as the M side with the 512 dims and the blocks split over
// two CTAs that exchange partial scores took the first away and was slower, 787 us with 8 softmax warps and 741 with 16 (649
// without the remote stores): the second then stands in one chain with the softmax.
//
// What a tile reads beyond a query's own keys must not matter: scores are masked by selection, V rows that hold no key are
// zeroed.  A V row that is visible to some query of the tile and not finite is visible to all of them as 0 * Inf, so rows that are
// not finite are computed again by the streaming statement, which reads what each query sees (all of 256 queries at 8192
// keys: 13600 us on the streaming kernel, 12400 here).
#include <mutex>
#include <string>

#include "attn_stream.cuh"
#include "sgb_common.cuh"
#include "sgb_kernels.h"

namespace sgb {

namespace {

constexpr int HD = 512, G = 8;
constexpr int ROWS = 64;       // query rows per CTA (N)
constexpr int TILE_K = 128;    // keys per tile (M of S^T)
constexpr int SOFT_THREADS = 256;
constexpr int MMA_W = 8, K_W = 9, V_W = 10;
constexpr int INT8_THREADS = 352;
constexpr int NV = 5;                          // V units in flight
constexpr uint32_t Q_CHUNK = ROWS * 128;       // 128 bytes of every row
constexpr uint32_t K_CHUNK = TILE_K * 128;
constexpr uint32_t V_UNIT = 64 * 256;          // 64 keys x 128 dims f16, as two [64 keys][128 B] halves
constexpr uint32_t P_TILE = TILE_K * ROWS * 2; // [128 keys][64 rows] f16
constexpr float EXP_BIAS = 7.0f, GROW_T = 8.0f;

struct Int8Smem {
    uint8_t q[4][Q_CHUNK];
    uint8_t k[4][K_CHUNK];
    uint8_t p[2][P_TILE];  // hi, lo
    uint8_t v[NV][V_UNIT];
    float qs[16][ROWS];    // scales of Q, [block][row]
    float red[4][ROWS];
    float m_ref[ROWS], corr[ROWS];
    uint64_t q_bar, k_full[4], k_free[4], v_full[NV], v_free[NV], v_ok[NV], s_ready[2], s_free[2], p_ready, first_done, pv_done;
    uint32_t tmem_base, abort;
    uint32_t redo[ROWS / 32];  // rows that are not finite, a bit each
};
static_assert(sizeof(Int8Smem) + 1024 <= 227 * 1024, "one CTA per SM");

struct Int8Params {
    const uint32_t* step;
    __half* out;
    uint32_t* status;
    const __half* q_scales;
    uint32_t m_tokens, n_kv;
    float scale;
    const void* q;  // for the streaming statement
    KvOperand k0, v0;
};

// tcgen05.mma kind::i8: int8 operands, int32 accumulator, K = 32 (32 bytes, like a K = 16 step of f16).
__device__ __forceinline__ void umma_i8_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc)
        : "memory");
}
// Instruction descriptor of kind::i8: D format 2 = s32, A and B format 1 = signed 8 bit, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc_i8(uint32_t m, uint32_t n)
{
    return (2u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
// Reduce 32 values over the 32 lanes of a warp: lane c is left with the total of v[c].  Each step halves the values.
template <bool MAX>
__device__ __forceinline__ float transpose_reduce(float (&v)[32], int lane)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; i++) {
            const float send = upper ? v[i] : v[i + o], keep = upper ? v[i + o] : v[i];
            const float r = __shfl_xor_sync(0xffffffffu, send, o);
            v[i] = MAX ? fmaxf(keep, r) : keep + r;
        }
    }
    return v[0];
}

// The rows that are not finite by the streaming statement, a warp per pair of heads.
__device__ __noinline__ void stream_rows(const Int8Params& prm, const Int8Smem& sm, uint32_t m0, int kvh)
{
    const uint32_t q0 = prm.step[STEP_Q0];
    for (uint32_t r = 2 * (threadIdx.x >> 5); r < ROWS; r += 2 * (INT8_THREADS / 32)) {
        const uint32_t which = (sm.redo[r / 32] >> (r % 32)) & 3u;
        if (which != 0)
            stream_prefill_rows<HD, G, true, false>(prm.q, prm.q_scales, prm.k0, prm.v0, prm.k0, prm.v0, prm.out, q0, m0 + r / G, kvh * G + r % G, which,
                                                    (int)prm.n_kv, 0, 0, prm.scale);
    }
}

__global__ void __launch_bounds__(INT8_THREADS, 1)
    int8_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                        const __grid_constant__ Int8Params prm)
{
    constexpr int TOK = ROWS / G, DB = HD / 128, UNITS = 2 * DB;  // V units per tile: (dim block, key half)
    constexpr int GROUPS = 8;  // S hand-overs per tile
    constexpr uint32_t S_COLS = 128;  // columns of one hand-over
    constexpr uint32_t TMEM_O = 0, TMEM_S = DB * 64, TMEM_COLS = 512;
    static_assert(TMEM_S + 2 * S_COLS <= TMEM_COLS, "O and two S buffers fit");
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Int8Smem& sm = *reinterpret_cast<Int8Smem*>(smem_raw);
    if ((smem_u32(smem_raw) & 1023u) != 0u) {  // the swizzled tiles need it; never seen, but never assumed
        if (threadIdx.x == 0) report_error(prm.status, DEV_ERR_BOUNDS, 500, smem_u32(smem_raw), 0);
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_wait();  // the step words, q, K and V come from earlier kernels of the stream
    pdl_launch_dependents();
    const int kvh = blockIdx.x % prm.n_kv;
    const uint32_t n_qt = (prm.m_tokens + TOK - 1) / TOK;
    const uint32_t m0 = (n_qt - 1 - blockIdx.x / prm.n_kv) * TOK;  // latest query tile (most keys) first
    const uint32_t live_tok = min((uint32_t)TOK, prm.m_tokens - m0);
    const int64_t q0 = prm.step[STEP_Q0];
    const int64_t first_qpos = q0 + m0, last_qpos = first_qpos + live_tok - 1;
    const int64_t rows0 = (int64_t)min(prm.k0.rows, prm.v0.rows);
    int64_t end = last_qpos;  // positions that hold a visible key end here
    if (end >= rows0) {
        if (tid == 0) report_error(prm.status, DEV_ERR_BOUNDS, 211, (uint32_t)rows0, (uint32_t)rows0);
        end = rows0 - 1;
    }
    const int n_tiles = (int)(end / TILE_K + 1);
    // rows of a tile that hold a key of this problem end here; V rows behind it are zeroed
    const int64_t valid_end = min(rows0 - 1, q0 + (int64_t)prm.m_tokens - 1);

    if (tid == 0) {
        mbar_init(&sm.q_bar, 1);
        for (int i = 0; i < 4; i++) {
            mbar_init(&sm.k_full[i], 1);
            mbar_init(&sm.k_free[i], 1);
        }
        for (int i = 0; i < NV; i++) {
            mbar_init(&sm.v_full[i], 1);
            mbar_init(&sm.v_free[i], 1);
            mbar_init(&sm.v_ok[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&sm.s_ready[i], 1);
            mbar_init(&sm.s_free[i], SOFT_THREADS / 32);
        }
        mbar_init(&sm.p_ready, SOFT_THREADS / 32);
        mbar_init(&sm.first_done, 1);
        mbar_init(&sm.pv_done, 1);
        sm.abort = 0;
        sm.redo[0] = sm.redo[1] = 0;
        mbar_fence_init();
    }
    if (tid < ROWS) sm.m_ref[tid] = NEG_SENTINEL;
    {
        for (int i = tid; i < 16 * ROWS; i += INT8_THREADS) {
            const int r = i >> 4, b = i & 15;
            const uint32_t tok = m0 + r / G;
            float s = 0.0f;
            if (tok < prm.m_tokens) s = __half2float(ld_global(prm.q_scales + ((size_t)tok * (prm.n_kv * G) + kvh * G + r % G) * 16 + b));
            sm.qs[b][r] = s;
        }
    }
    if (warp == 0) {
        tmem_alloc(&sm.tmem_base, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = sm.tmem_base;
    bool failed = false;
    auto block_at = [](int j, int u) { return ((u >> 1) + j) & (DB - 1); };  // dim block of V unit u of tile j: another one first in each tile

    if (warp == K_W) {
        // ======================= Q and K loads: K(j) chunk by chunk as the MMAs of tile j - 1 let go of them ==========
        if (lane == 0) {
            constexpr int CE = 128;  // elements of a 128-byte chunk
            mbar_arrive_expect_tx(&sm.q_bar, 4 * Q_CHUNK);
            for (int c = 0; c < 4; c++) tma_load_3d(sm.q[c], &tm_q, &sm.q_bar, c * CE, kvh * G, (int)m0);
            for (int j = 0; j < n_tiles && !failed; ++j) {
                for (int c = 0; c < 4; c++) {
                    if (j > 0) mbar_wait(&sm.k_free[c], (j - 1) & 1, prm.status, 511, failed, 50);
                    if (failed) break;  // never write into a buffer that may still be read
                    mbar_arrive_expect_tx(&sm.k_full[c], K_CHUNK);
                    tma_load_3d(sm.k[c], &tm_k, &sm.k_full[c], c * CE, kvh, j * TILE_K);
                }
            }
        }
    } else if (warp == V_W) {
        // ======================= V loads in units of 64 keys x 128 dims =======================
        // It also looks at the scales of K.  An infinite one times a whole sum that is negative would pass as a weight of 0; the
        // statement multiplies it with every quant, and infinities of both signs make a NaN.  A key with such a scale sends all
        // rows to that statement.  (The softmax threads, which hold the scales anyway, took 5 us of 530 for it.)
        uint32_t sc_top = 0;  // largest magnitudes as f16 bits, two at a time: from 0x7C00 on, not finite
        int n = 0;
        for (int j = 0; j < n_tiles && !failed; ++j) {
            const int64_t pos0 = (int64_t)j * TILE_K;
            uint4 sc[8];  // used at the end of the tile
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int64_t pos = pos0 + 32 * i + lane;
                const uint4* p = reinterpret_cast<const uint4*>(prm.k0.scales + ((size_t)pos * prm.n_kv + kvh) * 16);
                const bool key = pos <= min(end, valid_end);
                sc[2 * i] = key ? ld_global(p) : make_uint4(0u, 0u, 0u, 0u);
                sc[2 * i + 1] = key ? ld_global(p + 1) : make_uint4(0u, 0u, 0u, 0u);
            }
            const bool tail = pos0 + TILE_K - 1 > valid_end;  // the MMA warp computes the same
            for (int u = 0; u < UNITS; u++, n++) {
                const int st = n % NV;
                if (n >= NV && !mbar_wait_warp(&sm.v_free[st], (n / NV - 1) & 1, prm.status, 512, failed, 50)) break;
                const int kh = u & 1, db = block_at(j, u);
                if (lane == 0) {
                    mbar_arrive_expect_tx(&sm.v_full[st], V_UNIT);
                    tma_load_3d(sm.v[st], &tm_v, &sm.v_full[st], db * 128, kvh, (int)pos0 + kh * 64);
                    tma_load_3d(sm.v[st] + V_UNIT / 2, &tm_v, &sm.v_full[st], db * 128 + 64, kvh, (int)pos0 + kh * 64);
                }
                if (tail) {
                    __syncwarp();
                    if (!mbar_wait_warp(&sm.v_full[st], (n / NV) & 1, prm.status, 513, failed)) break;
                    for (int r = lane; r < 64; r += 32) {
                        if (pos0 + kh * 64 + r <= valid_end) continue;
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            uint4* row = reinterpret_cast<uint4*>(sm.v[st] + h * (V_UNIT / 2) + r * 128);
#pragma unroll
                            for (int i = 0; i < 8; i++) row[i] = make_uint4(0u, 0u, 0u, 0u);
                        }
                    }
                    fence_proxy_async_smem();  // generic-proxy writes, read next by the tensor pipe
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sm.v_ok[st]);
                }
            }
#pragma unroll
            for (int i = 0; i < 32; i++) sc_top = __vmaxu2(sc_top, reinterpret_cast<const uint32_t*>(sc)[i] & 0x7FFF7FFFu);
        }
        if ((sc_top & 0xFFFFu) >= 0x7C00u || (sc_top >> 16) >= 0x7C00u) sm.redo[0] = sm.redo[1] = 0xFFFFFFFFu;
    } else if (warp == MMA_W) {
        // ======================= MMA issue =======================
        if (lane == 0) {
            constexpr uint32_t IDESC_QK = umma_idesc_i8(TILE_K, ROWS);
            constexpr uint32_t IDESC_PV = umma_idesc_f16(128, ROWS, 1, 1);
            const uint64_t dq = umma_desc_sw128(smem_u32(sm.q[0]), 16, 1024), dk = umma_desc_sw128(smem_u32(sm.k[0]), 16, 1024);
            const uint64_t dv = umma_desc_sw128(smem_u32(sm.v[0]), V_UNIT / 2, 1024);
            const uint64_t dp = umma_desc_sw128(smem_u32(sm.p[0]), 16, 1024);
            uint32_t ok_phase = 0;  // of v_ok, a bit per slot: only tail tiles use it up
            // S of (tile j, group g) into buffer n & 1, n = j * GROUPS + g
            auto issue_qk = [&](int j, int g) {
                const int n = j * GROUPS + g;
                if (n >= 2) mbar_wait(&sm.s_free[n & 1], ((n - 2) >> 1) & 1, prm.status, 521, failed);
                const uint32_t d = tmem + TMEM_S + (n & 1) * S_COLS;
                const int c = g >> 1;  // 128-byte chunk; the group is its lower or upper two blocks
                if ((g & 1) == 0) mbar_wait(&sm.k_full[c], j & 1, prm.status, 522, failed);
                if (failed) return;
                tc_fence_after_sync();
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const uint32_t off = 2 * (2 * (g & 1) + e);
                    umma_i8_ss(d + e * 64, dk + c * (K_CHUNK >> 4) + off, dq + c * (Q_CHUNK >> 4) + off, IDESC_QK);
                }
                if (g & 1) umma_commit(&sm.k_free[c]);
                umma_commit(&sm.s_ready[n & 1]);
            };
            // O^T += V^T P^T for one unit of tile j
            auto issue_pv = [&](int j, int u, bool tail) {
                const int n = j * UNITS + u, st = n % NV, kh = u & 1, db = block_at(j, u);
                mbar_wait(&sm.v_full[st], (n / NV) & 1, prm.status, 523, failed);
                if (tail) {
                    mbar_wait(&sm.v_ok[st], (ok_phase >> st) & 1, prm.status, 524, failed);
                    ok_phase ^= 1u << st;
                }
                if (failed) return;
                tc_fence_after_sync();
                const uint64_t v = dv + (uint64_t)st * (V_UNIT >> 4), p = dp + kh * (64 * 128 >> 4);
                const uint32_t d = tmem + TMEM_O + db * 64;
#pragma unroll
                for (int half = 0; half < 2; half++)
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)
                        umma_f16_ss(d, v + 128 * kk, p + half * (P_TILE >> 4) + 128 * kk, IDESC_PV, (j > 0 || kh || half || kk) ? 1u : 0u);
                umma_commit(&sm.v_free[st]);
            };
            mbar_wait(&sm.q_bar, 0, prm.status, 520, failed);
            if (n_tiles > 0)
                for (int g = 0; g < GROUPS; g++) issue_qk(0, g);
            for (int j = 0; j < n_tiles && !failed; ++j) {
                const bool tail = (int64_t)j * TILE_K + TILE_K - 1 > valid_end, more = j + 1 < n_tiles;
                // the next tile's scores go ahead of this tile's products, and between them
                int g = 0;
                for (; more && g < 2; g++) issue_qk(j + 1, g);
                mbar_wait(&sm.p_ready, j & 1, prm.status, 525, failed);
                if (failed) break;
                tc_fence_after_sync();
                for (int u = 0; u < UNITS; u++) {
                    issue_pv(j, u, tail);
                    if (u == 1) umma_commit(&sm.first_done);
                    if (u == UNITS - 1) umma_commit(&sm.pv_done);
                    if (more && g < GROUPS) issue_qk(j + 1, g++);
                }
            }
        }
    } else {
        // ======================= softmax: thread = (key kq * 32 + lane, rows 32 * half ..) =======================
        const int kq = warp & 3, half = warp >> 2, key = kq * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)(kq * 32) << 16);
        const float scale2 = prm.scale * 1.4426950408889634f;  // > 0 (checked on the host)
        float2 l2[16];
#pragma unroll
        for (int i = 0; i < 16; i++) l2[i] = make_float2(0.0f, 0.0f);
        uint4 ks_next[2] = {};
        auto fetch_scales = [&](int it) {
            const size_t pos = (size_t)it * TILE_K + key;
            ks_next[0] = ks_next[1] = make_uint4(0u, 0u, 0u, 0u);
            if ((int64_t)pos <= valid_end) {
                const uint4* p = reinterpret_cast<const uint4*>(prm.k0.scales + (pos * prm.n_kv + kvh) * 16);
                ks_next[0] = ld_global(p);
                ks_next[1] = ld_global(p + 1);
            }
        };
        if (n_tiles > 0) fetch_scales(0);
        // The settled part of this thread's O as 16-bit halves, in this CTA's own share of the output (64 rows x 512 dims x 2 bytes),
        // which nobody reads before the end.  A step takes 16 of the 32 values of a block; 8 values c of step h at [2 * h + c][thread].
        uint32_t settled = 0;  // a bit per block
        auto settled_at = [&](int h, int c) {
            const int e = 2 * h + c;
            return reinterpret_cast<uint4*>(prm.out + ((size_t)(m0 + e / 2) * (prm.n_kv * G) + kvh * G) * HD) + (e & 1) * SOFT_THREADS + tid;
        };
        auto o_at = [&](int h) { return lane_addr + TMEM_O + (h >> 1) * 64 + 32 * half + 16 * (h & 1); };
        auto fetch_settled = [&](int h, uint4 (&u)[2]) {
            u[0] = *settled_at(h, 0);
            u[1] = *settled_at(h, 1);
        };
        auto add_settled = [&](const uint4 (&u)[2], uint32_t (&o)[16]) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t w = reinterpret_cast<const uint32_t*>(u)[i];
                o[2 * i] = __float_as_uint(__fadd_rn(__uint_as_float(o[2 * i]), __uint_as_float(w << 16)));
                o[2 * i + 1] = __float_as_uint(__fadd_rn(__uint_as_float(o[2 * i + 1]), __uint_as_float(w & 0xFFFF0000u)));
            }
        };
        auto settle = [&](int h, uint32_t (&o)[16]) {  // o: whole values, left as the rest
#pragma unroll
            for (int c = 0; c < 2; c++) {
                uint32_t w[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    uint32_t &a = o[8 * c + 2 * k], &b = o[8 * c + 2 * k + 1];
                    w[k] = __byte_perm(a, b, 0x7632);
                    a = __float_as_uint(__uint_as_float(a) - __uint_as_float(a & 0xFFFF0000u));
                    b = __float_as_uint(__uint_as_float(b) - __uint_as_float(b & 0xFFFF0000u));
                }
                *settled_at(h, c) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        };

        for (int it = 0; it < n_tiles; ++it) {
            float s[32];
            {
                const uint4 ks4[2] = {ks_next[0], ks_next[1]};
                if (it + 1 < n_tiles) fetch_scales(it + 1);
                float2 a2[16];
#pragma unroll
                for (int i = 0; i < 16; i++) a2[i] = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int g = 0; g < 8; g++) {
                    mbar_wait(&sm.s_ready[g & 1], ((it * 8 + g) >> 1) & 1, prm.status, 531, failed);
                    tc_fence_after_sync();
                    uint32_t r0[32], r1[32];
                    tmem_ld_32x32b_x32(lane_addr + TMEM_S + (g & 1) * S_COLS + 32 * half, r0);
                    tmem_ld_32x32b_x32(lane_addr + TMEM_S + (g & 1) * S_COLS + 64 + 32 * half, r1);
                    tc_wait_ld();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sm.s_free[g & 1]);  // one arrival per warp: they serialise on the barrier's word
                    const uint32_t w = reinterpret_cast<const uint32_t*>(ks4)[g];
                    const float2 ks = __half22float2(*reinterpret_cast<const __half2*>(&w));
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const float4* qs = reinterpret_cast<const float4*>(&sm.qs[2 * g + e][32 * half]);
                        const float2 kk = e ? make_float2(ks.y, ks.y) : make_float2(ks.x, ks.x);
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const float4 f = qs[i];
                            const uint32_t* r = (e ? r1 : r0) + 4 * i;
                            a2[2 * i] = __ffma2_rn(make_float2((float)(int)r[0], (float)(int)r[1]), __fmul2_rn(kk, make_float2(f.x, f.y)), a2[2 * i]);
                            a2[2 * i + 1] = __ffma2_rn(make_float2((float)(int)r[2], (float)(int)r[3]), __fmul2_rn(kk, make_float2(f.z, f.w)), a2[2 * i + 1]);
                        }
                    }
                    if (g == 3 && it >= 4) {
                        // the last tile's products of its first block were issued ahead of these scores, and both S buffers are free: the
                        // tensor pipe goes on meanwhile
                        const int db = block_at(it - 1, 0);
                        mbar_wait(&sm.first_done, (it - 1) & 1, prm.status, 535, failed);
                        tc_fence_after_sync();
#pragma unroll 1
                        for (int h = 2 * db; h < 2 * db + 2; h++) {
                            uint32_t o[16];
                            uint4 u[2] = {};
                            if ((settled >> db) & 1) fetch_settled(h, u);
                            tmem_ld_32x32b_x16(o_at(h), o);
                            tc_wait_ld();
                            add_settled(u, o);
                            settle(h, o);
                            tmem_st_32x32b_x16(o_at(h), o);
                        }
                        tc_wait_st();
                        settled |= 1u << db;
                    }
                }
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    s[2 * i] = a2[i].x;
                    s[2 * i + 1] = a2[i].y;
                }
            }

            // masks only where the tile crosses the diagonal or the end of the cache: row r (token r / G of the tile) sees the key
            // from its own position on
            const int64_t pos0 = (int64_t)it * TILE_K;
            if (pos0 + TILE_K - 1 > min(first_qpos, rows0 - 1)) {
                const int from = pos0 + key <= rows0 - 1 ? (int)(pos0 + key - first_qpos) : TOK;
#pragma unroll
                for (int i = 0; i < 32; i++)
                    if ((32 * half + i) / G < from) s[i] = -INFINITY;
            }
            // does any score exceed its row's reference by more than 2^8?
            const float4* mr = reinterpret_cast<const float4*>(&sm.m_ref[32 * half]);
            bool over = false;
            {
                const float2 sc2 = make_float2(scale2, scale2);
                float top = -INFINITY;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 f = mr[i];
                    const float2 a = __ffma2_rn(make_float2(s[4 * i], s[4 * i + 1]), sc2, make_float2(-f.x, -f.y));
                    const float2 b = __ffma2_rn(make_float2(s[4 * i + 2], s[4 * i + 3]), sc2, make_float2(-f.z, -f.w));
                    top = max3(top, max3(a.x, a.y, b.x), b.y);
                }
                over = top > GROW_T;
            }
            const bool raise = named_barrier_or(1, SOFT_THREADS, over);
            if (raise) {
                float c[32];
#pragma unroll
                for (int i = 0; i < 32; i++) c[i] = s[i];
                sm.red[kq][32 * half + lane] = transpose_reduce<true>(c, lane);
                named_barrier_sync(2, SOFT_THREADS);
                if (tid < ROWS) {
                    const float mx = fmaxf(fmaxf(sm.red[0][tid], sm.red[1][tid]), fmaxf(sm.red[2][tid], sm.red[3][tid])) * scale2;
                    const float old = sm.m_ref[tid];
                    const float now = mx > old + GROW_T ? mx : old;
                    sm.corr[tid] = ex2(old - now);
                    sm.m_ref[tid] = now;
                }
                named_barrier_sync(2, SOFT_THREADS);
                const float4* cr = reinterpret_cast<const float4*>(&sm.corr[32 * half]);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 f = cr[i];
                    l2[2 * i] = __fmul2_rn(l2[2 * i], make_float2(f.x, f.y));
                    l2[2 * i + 1] = __fmul2_rn(l2[2 * i + 1], make_float2(f.z, f.w));
                }
            }
            if (raise && it > 0) {
                mbar_wait(&sm.pv_done, (it - 1) & 1, prm.status, 532, failed);
                tc_fence_after_sync();
#pragma unroll 1
                for (int h = 0; h < 2 * DB; h++) {
                    const bool in_parts = (settled >> (h >> 1)) & 1;
                    uint32_t o[16];
                    uint4 u[2];
                    tmem_ld_32x32b_x16(o_at(h), o);
                    if (in_parts) fetch_settled(h, u);
                    tc_wait_ld();
                    if (in_parts) add_settled(u, o);
#pragma unroll
                    for (int i = 0; i < 16; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * sm.corr[32 * half + 16 * (h & 1) + i]);
                    if (in_parts) settle(h, o);
                    tmem_st_32x32b_x16(o_at(h), o);
                }
                tc_wait_st();
            }
            // P = 2^(s * scale2 - m + 7) as f16 hi + lo; l from the unrounded values
            uint32_t hi[16], lo[16];
            {
                const float2 sc2 = make_float2(scale2, scale2);
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float2 m = reinterpret_cast<const float2*>(mr)[i];
                    const float2 x = __ffma2_rn(make_float2(s[2 * i], s[2 * i + 1]), sc2, make_float2(EXP_BIAS - m.x, EXP_BIAS - m.y));
                    const float2 p = make_float2(ex2(x.x), ex2(x.y));
                    l2[i] = __fadd2_rn(l2[i], p);
                    hi[i] = pack_half2(p.x, p.y);
                    const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi[i]));
                    lo[i] = pack_half2(p.x - h.x, p.y - h.y);
                }
            }
            if (it > 0) mbar_wait(&sm.pv_done, (it - 1) & 1, prm.status, 533, failed);  // P of the last tile has been read
            {
                uint8_t* row = sm.p[0] + key * 128;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint32_t off = ((4 * half + c) ^ (key & 7)) << 4;
                    *reinterpret_cast<uint4*>(row + off) = make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
                    *reinterpret_cast<uint4*>(row + P_TILE + off) = make_uint4(lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]);
                }
            }
            fence_proxy_async_smem();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.p_ready);
        }

        // ---- epilogue: thread = output dim db * 128 + key -----------------------------------------------
        float l[32];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            l[2 * i] = l2[i].x;
            l[2 * i + 1] = l2[i].y;
        }
        named_barrier_sync(2, SOFT_THREADS);  // every thread is done with red and corr
        sm.red[kq][32 * half + lane] = transpose_reduce<false>(l, lane);
        named_barrier_sync(2, SOFT_THREADS);
        if (tid < ROWS) sm.corr[tid] = 1.0f / ((sm.red[0][tid] + sm.red[1][tid]) + (sm.red[2][tid] + sm.red[3][tid]));
        named_barrier_sync(2, SOFT_THREADS);
        if (n_tiles > 0) mbar_wait(&sm.pv_done, (n_tiles - 1) & 1, prm.status, 534, failed);
        tc_fence_after_sync();
        if (settled != 0) {  // whole again before the first result is written over a settled part
#pragma unroll 1
            for (int h = 0; h < 2 * DB; h++) {
                if (((settled >> (h >> 1)) & 1) == 0) continue;
                uint32_t o[16];
                uint4 u[2];
                tmem_ld_32x32b_x16(o_at(h), o);
                fetch_settled(h, u);
                tc_wait_ld();
                add_settled(u, o);
                tmem_st_32x32b_x16(o_at(h), o);
            }
            tc_wait_st();
            named_barrier_sync(2, SOFT_THREADS);
        }
        uint32_t odd = 0;  // also a row with a scale of Q that is not finite (see the V loader)
        for (int b = 4 * kq; b < 4 * kq + 4; b++)
            if (!(fabsf(sm.qs[b][32 * half + lane]) <= 65504.0f)) odd |= 1u << lane;
#pragma unroll 1
        for (int db = 0; db < DB; db++) {
            uint32_t o[32];
            if (n_tiles > 0) {  // uniform over the CTA
                tmem_ld_32x32b_x32(lane_addr + TMEM_O + db * 64 + 32 * half, o);
                tc_wait_ld();
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) o[i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const int r = 32 * half + i;
                const float y = __uint_as_float(o[i]) * sm.corr[r];
                if ((uint32_t)(r / G) < live_tok) {
                    if (!(fabsf(y) <= 3.4e38f)) odd |= 1u << i;
                    prm.out[((size_t)(m0 + r / G) * (prm.n_kv * G) + kvh * G + r % G) * HD + db * 128 + key] = __float2half_rn(y);
                }
            }
        }
        odd = __reduce_or_sync(0xffffffffu, odd);
        if (odd != 0 && lane == 0) atomicOr(&sm.redo[half], odd);
    }
    // A wait that ran out leaves copies and MMAs of this CTA in flight that nobody will wait for: give them a bounded
    // time to land before the shared and tensor memory they target is handed to the next CTA.
    if (failed) sm.abort = 1;
    tc_fence_before_sync();
    __syncthreads();
    if (*(volatile uint32_t*)&sm.abort != 0u) {
        let_copies_land();
        __syncthreads();
    }
    if (warp == 0) tmem_dealloc(tmem, TMEM_COLS);
    if ((*(volatile uint32_t*)&sm.redo[0] | *(volatile uint32_t*)&sm.redo[1]) != 0) stream_rows(prm, sm, m0, kvh);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// [row][head][512] tensor of `elem`-byte values, boxes of 128 bytes x box_heads x box_rows.
int encode_rows(const LaunchArgs& a, CUtensorMap* tm, const void* base, uint64_t rows, uint64_t heads, int elem, uint32_t box_heads, uint32_t box_rows)
{
    const uint64_t dims[3] = {HD, heads, rows};
    const uint64_t strides[2] = {(uint64_t)HD * elem, heads * HD * elem};
    const uint32_t box[3] = {128u / elem, box_heads, box_rows};
    return encode_tensor_map(a, tm, elem == 2, 3, const_cast<void*>(base), dims, strides, box, 3);
}

}  // namespace

// What the tensor-core kernel takes: a positive softmax scale (the row maximum is taken before it), operands whose rows the
// copies can address (16-byte aligned bases, K and V with at least one row, row indexes within an int), an output that can be
// settled into (16-byte accesses, whole query tiles).  What else the launcher accepts stays on the streaming kernel: quants on 4
// bytes, scales and output on 2.
bool prefill_int8_takes(const KvOperand& k, const KvOperand& v, const void* q, const void* out, uint32_t m, float scale)
{
    if (!(scale > 0.0f) || !(scale < 1e30f) || !aligned16(q) || !aligned16(k.scales) || !aligned16(out) || m % (ROWS / G) != 0) return false;
    for (const KvOperand* o : {&k, &v})
        if (o->rows == 0 || o->rows >= (1u << 30) || !aligned16(o->data)) return false;
    return true;
}

int launch_prefill_int8(const LaunchArgs& a, const void* q, const __half* q_scales, const KvOperand& k, const KvOperand& v, void* out, const void* step,
                        uint32_t n_kv, uint32_t m, float scale)
{
    const Int8Params prm{(const uint32_t*)step, (__half*)out, a.status, q_scales, m, n_kv, scale, q, k, v};
    CUtensorMap tq, tk, tv;
    if (int r = encode_rows(a, &tq, q, m, n_kv * G, 1, G, ROWS / G)) return r;
    if (int r = encode_rows(a, &tk, k.data, k.rows, n_kv, 1, 1, TILE_K)) return r;
    if (int r = encode_rows(a, &tv, v.data, v.rows, n_kv, 2, 1, 64)) return r;
    {
        static std::mutex attr_mutex;
        static bool attr_set[64] = {};
        std::lock_guard<std::mutex> lock(attr_mutex);
        if (a.device >= 64 || !attr_set[a.device]) {
            if (int r = check_cuda(a, cudaFuncSetAttribute(int8_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Int8Smem)),
                                   "cudaFuncSetAttribute(int8_prefill)"))
                return r;
            if (a.device < 64) attr_set[a.device] = true;
        }
    }
    const uint32_t q_tiles = (m + ROWS / G - 1) / (ROWS / G);
    const cudaError_t err = launch_dependent(int8_prefill_kernel, dim3(q_tiles * n_kv), dim3(INT8_THREADS), sizeof(Int8Smem), a.stream, tq, tk, tv, prm);
    ++*a.launches;
    return check_cuda(a, err, "attn_prefill_global_flash_sp_iq");
}

}  // namespace sgb
