// Prefill attention for the reference model's sliding layers on tcgen05: head_dim 256, f16 K/V, 2 query heads per kv head,
// 1024-token window over a linear cache or ring history + chunk.  Semantics: attn_prefill_sliding.wgsl:53-125,
// attn_prefill_sliding_ring.wgsl:88-140.
//
// A CTA owns 128 query rows (64 tokens x the 2 query heads of one kv head, which share every K/V tile).  Per 64-key tile
// S[128 x 64] = Q K^T, softmax with two threads per row (32 keys each), O[128 x 256] += P V with P as the tensor-memory A
// operand and V as the MN-major B operand straight from its [key][dim] tile.  (A transposed form, with V as the MN-major A
// operand of 128 x 64 instructions, needed 160 cycles per instruction where K-major operands take 48: 38.6 us where this
// one takes 22.7.)  Where two CTAs per unit fit the GPU at once a cluster of two shares a unit's key tiles; the halves
// merge at the end through distributed shared memory, each CTA finishing 128 of the dims.
// P = hi + lo, both halves f16, two MMAs per 16 keys: together they miss p by at most one unit of its last f32 place.  The exponent
// carries +7, so that lo stays clear of f16's subnormals (the factor cancels in O / l); a p below 2^-32 of its row's reference
// maximum is in l but too small for lo.  The tensor pipe's truncation (2e-9 of the output per key, 2e-6 at 1024 keys) is left in: the error
// against 64 bits is f16's own, 2.069e-4, as on the streaming kernel.
// Roles: warps 0-7 softmax, one MMA warp, one K and one V loader; mbarriers only.
// Measured: 256 queries, 16 kv heads, ring + chunk: 795 us on the streaming kernel, 22.7 with one thread running the MMA loop, 20.7 with a
// warp (sgb_common.cuh); bound by the chain score -> softmax -> P V of eight tiles plus set-up and merge (the MMAs need 1800
// cycles a tile).
//
// What a tile reads beyond a query's own keys must not matter: scores are masked by selection, V rows that hold no key are
// zeroed.  A V row that is visible to some query of the tile and not finite is visible to all of them as 0 * Inf, so rows that are
// not finite are computed again by the streaming statement, which reads what each query sees (all of 256 queries over the
// ring: 807 us on the streaming kernel, 793 here; eight of them 238).
#include <mutex>
#include <string>

#include "attn_stream.cuh"
#include "sgb_common.cuh"
#include "sgb_kernels.h"

namespace sgb {

namespace {

constexpr int ROWS = 128;     // query rows per CTA (M)
constexpr int TILE_K = 64;    // keys per tile
constexpr int HD = 256, G = 2;
constexpr int SOFT_THREADS = 256;
constexpr int MMA_W = 8, K_W = 9, V_W = 10;
constexpr int WIDE_THREADS = 352;
constexpr int CHUNKS = 4, STAGES = 2;       // 128-byte chunks of a row of Q or K; K and V tiles in flight
constexpr uint32_t Q_CHUNK = ROWS * 128;    // 128 bytes of every row
constexpr uint32_t K_CHUNK = TILE_K * 128;
constexpr uint32_t V_CHUNK = TILE_K * 128;  // 64 dims f16 of every key
constexpr uint32_t V_TILE = 4 * V_CHUNK;
constexpr uint32_t TMEM_O = 0, TMEM_S = 256, TMEM_COLS = 512;
constexpr float EXP_BIAS = 7.0f, GROW_T = 8.0f;

struct WideSmem {
    uint8_t q[CHUNKS][Q_CHUNK];
    uint8_t k[STAGES][CHUNKS][K_CHUNK];  // afterwards the other CTA's O of this CTA's 128 dims
    uint8_t v[STAGES][V_TILE];
    float red[2][ROWS];
    float2 other_ml[ROWS];
    uint64_t q_bar, k_full[STAGES], k_free[STAGES], v_full[STAGES], v_free[STAGES], v_ok[STAGES], s_ready[2], p_ready[2], pv_done[2];
    uint32_t tmem_base, abort;
    __align__(16) uint32_t redo[2][2][ROWS / 32];  // rows that are not finite, a bit each: [found by this CTA or the other][dim half][row / 32]
};
static_assert(sizeof(WideSmem) <= 227 * 1024, "one CTA per SM");

struct WideParams {
    const uint32_t* step;
    __half* out;
    uint32_t* status;
    uint32_t m_tokens, n_kv, window, ring;
    float scale;
    uint32_t n_cta;          // CTAs of a cluster
    const void* q;           // for the streaming statement
    KvOperand k0, v0, k1, v1;
};

__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank)
{
    uint32_t out;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_addr), "r"(rank));
    return out;
}
__device__ __forceinline__ void st_cluster_f4(uint32_t addr, float4 v)
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t addr, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The rows that are not finite by the streaming statement, a warp per token (G = 2 rows); the CTAs of a cluster take turns.
template <bool TWO_SRC>
__device__ __noinline__ void stream_rows(const WideParams& prm, const WideSmem& sm, uint32_t m0, int kvh, uint32_t rank)
{
    const uint32_t q0 = prm.step[STEP_Q0];
    for (uint32_t tok = threadIdx.x >> 5; tok < ROWS / G; tok += WIDE_THREADS / 32) {
        const uint32_t i = tok / 16, redo = sm.redo[0][0][i] | sm.redo[0][1][i] | sm.redo[1][0][i] | sm.redo[1][1][i], which = (redo >> (2 * tok % 32)) & 3u;
        if (which == 0 || (prm.n_cta == 2 && tok % 2 != rank)) continue;
        stream_prefill_rows<HD, G, false, TWO_SRC>(prm.q, nullptr, prm.k0, prm.v0, prm.k1, prm.v1, prm.out, q0, m0 + tok, kvh * G, which, (int)prm.n_kv,
                                                   prm.window, prm.ring, prm.scale);
    }
}

struct WideTile {
    int src, row0;          // tensor-map row of key 0
    int64_t pos0, lo, hi;   // position of key 0; positions this source really holds
};

template <bool TWO_SRC>
__global__ void __launch_bounds__(WIDE_THREADS, 1)
    wide_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k0,
                        const __grid_constant__ CUtensorMap tm_v0, const __grid_constant__ CUtensorMap tm_k1,
                        const __grid_constant__ CUtensorMap tm_v1, const __grid_constant__ WideParams prm)
{
    constexpr int TOK = ROWS / G, CE = 64;  // tokens; elements of a 128-byte chunk
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    WideSmem& sm = *reinterpret_cast<WideSmem*>(smem_raw);
    const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
    const uint32_t rank = blockIdx.x % prm.n_cta, unit = blockIdx.x / prm.n_cta;
    const bool split = prm.n_cta == 2;  // the CTAs of a cluster share the keys
    const bool aligned = (smem_u32(smem_raw) & 1023u) == 0u;  // the swizzled tiles need it; never seen, but never assumed
    if (!aligned) {                                           // the same in every CTA: nobody waits for one that left
        if (tid == 0) report_error(prm.status, DEV_ERR_BOUNDS, 500, smem_u32(smem_raw), 0);
        return;
    }
    pdl_wait();  // the step words, q, K and V come from earlier kernels of the stream
    pdl_launch_dependents();
    const int kvh = unit % prm.n_kv;
    const uint32_t n_qt = (prm.m_tokens + TOK - 1) / TOK;
    const uint32_t m0 = (n_qt - 1 - unit / prm.n_kv) * TOK;  // latest query tile (most keys) first
    const uint32_t live_tok = min((uint32_t)TOK, prm.m_tokens - m0);
    const int64_t q0 = prm.step[STEP_Q0];
    const int64_t first_qpos = q0 + m0, last_qpos = first_qpos + live_tok - 1;
    const int64_t win = prm.window;
    const int64_t band_lo = (win && first_qpos + 1 > win) ? first_qpos + 1 - win : 0;
    const int64_t last_lo = (win && last_qpos + 1 > win) ? last_qpos + 1 - win : 0;
    const int64_t rows0 = (int64_t)min(prm.k0.rows, prm.v0.rows);
    int n_hist, n_tiles;
    const int64_t hist_pos0 = band_lo / TILE_K * TILE_K;
    int64_t chunk_c0 = 0;
    if (TWO_SRC) {
        n_hist = q0 > band_lo ? (int)((q0 - 1) / TILE_K - band_lo / TILE_K + 1) : 0;
        const int64_t c_lo = band_lo > q0 ? band_lo - q0 : 0, c_hi = last_qpos - q0;
        chunk_c0 = c_lo / TILE_K * TILE_K;
        n_tiles = n_hist + (int)(c_hi / TILE_K - c_lo / TILE_K + 1);
    } else {
        int64_t end = last_qpos;
        if (end >= rows0) {
            if (tid == 0) report_error(prm.status, DEV_ERR_BOUNDS, 211, (uint32_t)rows0, (uint32_t)rows0);
            end = rows0 - 1;
        }
        n_hist = end >= band_lo ? (int)(end / TILE_K - band_lo / TILE_K + 1) : 0;
        n_tiles = n_hist;
    }
    int t_begin = 0;
    if (split) {
        const int per = (n_tiles + 1) / 2;
        t_begin = min(n_tiles, (int)rank * per);
        n_tiles = min(n_tiles, t_begin + per) - t_begin;
    }
    auto tile_at = [&](int it) {
        WideTile t;
        it += t_begin;
        if (it < n_hist) {
            t.src = 0;
            t.pos0 = hist_pos0 + (int64_t)it * TILE_K;
            t.row0 = (int)(TWO_SRC ? t.pos0 % prm.ring : t.pos0);
            t.lo = 0;
            t.hi = TWO_SRC ? q0 - 1 : rows0 - 1;
        } else {
            t.src = 1;
            const int64_t c = chunk_c0 + (int64_t)(it - n_hist) * TILE_K;
            t.pos0 = q0 + c;
            t.row0 = (int)c;
            t.lo = q0;
            t.hi = INT64_MAX;
        }
        return t;
    };
    // positions of a tile that hold a key of this problem end here; V rows behind it are zeroed
    auto valid_end = [&](const WideTile& t) { return min(t.hi, q0 + (int64_t)prm.m_tokens - 1); };

    if (tid == 0) {
        mbar_init(&sm.q_bar, 1);
        for (int i = 0; i < STAGES; i++) {
            mbar_init(&sm.k_full[i], 1);
            mbar_init(&sm.k_free[i], 1);
            mbar_init(&sm.v_full[i], 1);
            mbar_init(&sm.v_free[i], 1);
            mbar_init(&sm.v_ok[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&sm.s_ready[i], 1);
            mbar_init(&sm.p_ready[i], SOFT_THREADS / 32);  // an arrival per warp: they serialise on the barrier's word
            mbar_init(&sm.pv_done[i], 1);
        }
        sm.abort = 0;
        mbar_fence_init();
    }
    if (tid < 4 * ROWS / 32) (&sm.redo[0][0][0])[tid] = 0;
    if (warp == 0) {
        tmem_alloc(&sm.tmem_base, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = sm.tmem_base;
    bool failed = false;

    const int kq = warp & 3, half = warp >> 2, row = kq * 32 + lane;  // softmax threads: row, keys 32 * half .. of a tile
    const uint32_t lane_addr = tmem + ((uint32_t)(kq * 32) << 16);
    float m_run = NEG_SENTINEL, l_run = 0.0f;

    if (warp == K_W) {
        // ======================= Q and K loads =======================
        if (lane == 0) {
            mbar_arrive_expect_tx(&sm.q_bar, CHUNKS * Q_CHUNK);
            for (int c = 0; c < CHUNKS; c++) tma_load_3d(sm.q[c], &tm_q, &sm.q_bar, c * CE, kvh * G, (int)m0);
            for (int j = 0; j < n_tiles; ++j) {
                const WideTile t = tile_at(j);
                const CUtensorMap* mk = (TWO_SRC && t.src) ? &tm_k1 : &tm_k0;
                const int st = j % STAGES;
                if (j >= STAGES) mbar_wait(&sm.k_free[st], (j / STAGES - 1) & 1, prm.status, 511, failed, 50);
                if (failed) break;  // never write into a buffer that may still be read
                mbar_arrive_expect_tx(&sm.k_full[st], CHUNKS * K_CHUNK);
                for (int c = 0; c < CHUNKS; c++) tma_load_3d(sm.k[st][c], mk, &sm.k_full[st], c * CE, kvh, t.row0);
            }
        }
    } else if (warp == V_W) {
        // ======================= V loads =======================
        for (int j = 0; j < n_tiles; ++j) {
            const WideTile t = tile_at(j);
            const CUtensorMap* mv = (TWO_SRC && t.src) ? &tm_v1 : &tm_v0;
            const int64_t last = valid_end(t);
            const bool tail = t.pos0 + TILE_K - 1 > last;  // the MMA warp computes the same
            const int st = j % STAGES;
            if (j >= STAGES && !mbar_wait_warp(&sm.v_free[st], (j / STAGES - 1) & 1, prm.status, 512, failed, 50)) break;
            if (lane == 0) {
                mbar_arrive_expect_tx(&sm.v_full[st], V_TILE);
                for (int c = 0; c < 4; c++) tma_load_3d(sm.v[st] + c * V_CHUNK, mv, &sm.v_full[st], c * 64, kvh, t.row0);
            }
            if (tail) {
                __syncwarp();
                if (!mbar_wait_warp(&sm.v_full[st], (j / STAGES) & 1, prm.status, 513, failed)) break;
                for (int r = lane; r < TILE_K; r += 32) {
                    if (t.pos0 + r <= last) continue;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        uint4* p = reinterpret_cast<uint4*>(sm.v[st] + c * V_CHUNK + r * 128);
#pragma unroll
                        for (int i = 0; i < 8; i++) p[i] = make_uint4(0u, 0u, 0u, 0u);
                    }
                }
                fence_proxy_async_smem();  // generic-proxy writes, read next by the tensor pipe
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.v_ok[st]);
            }
        }
    } else if (warp == MMA_W) {
        // ======================= MMA issue =======================
        {
            const uint32_t one = elect_one(), tm = warp_uniform(tmem);
            const int tiles = warp_uniform(n_tiles);
            constexpr uint32_t IDESC_QK = umma_idesc_f16(ROWS, TILE_K, 0, 0);
            constexpr uint32_t IDESC_PV = umma_idesc_f16(ROWS, HD, 0, 1);
            const uint64_t dq = umma_desc_sw128(smem_u32(sm.q[0]), 16, 1024), dk = umma_desc_sw128(smem_u32(sm.k[0][0]), 16, 1024);
            const uint64_t dv = umma_desc_sw128(smem_u32(sm.v[0]), V_CHUNK, 1024);
            uint32_t ok_phase = 0;  // of v_ok, a bit per stage: only tail tiles use it up
            // Q K^T of tile j, into S buffer j % 2 (free: P V of tile j - 2 was issued before)
            auto issue_tile = [&](int j) {
                const int st = j % STAGES;
                mbar_wait_warp(&sm.k_full[st], (j / STAGES) & 1, prm.status, 522, failed);
                if (failed) return;
                tc_fence_after_sync();
#pragma unroll
                for (int c = 0; c < CHUNKS; c++)
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)
                        umma_f16_ss(tm + TMEM_S + (j & 1) * 64, dq + c * (Q_CHUNK >> 4) + 2 * kk, dk + (st * CHUNKS + c) * (K_CHUNK >> 4) + 2 * kk,
                                    IDESC_QK, (c | kk) ? 1u : 0u, one);
                umma_commit(&sm.s_ready[j & 1], one);
                umma_commit(&sm.k_free[st], one);
            };
            mbar_wait_warp(&sm.q_bar, 0, prm.status, 520, failed);
            for (int j = 0; j < 2 && j < tiles; j++) issue_tile(j);
            for (int j = 0; j < tiles && !failed; ++j) {
                const WideTile t = tile_at(j);
                const bool tail = warp_uniform((int)(t.pos0 + TILE_K - 1 > valid_end(t))) != 0;
                const int st = j % STAGES;
                mbar_wait_warp(&sm.v_full[st], (j / STAGES) & 1, prm.status, 523, failed);
                if (tail) {
                    mbar_wait_warp(&sm.v_ok[st], (ok_phase >> st) & 1, prm.status, 524, failed);
                    ok_phase ^= 1u << st;
                }
                mbar_wait_warp(&sm.p_ready[j & 1], (j >> 1) & 1, prm.status, 525, failed);
                if (failed) break;
                tc_fence_after_sync();
                // O += P V in eight instructions (hi and lo of four 16-key steps)
                const uint32_t p = tm + TMEM_S + (j & 1) * 64;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int kk = i >> 1;
                    umma_f16_ts(tm + TMEM_O, p + (i & 1) * 32 + kk * 8, dv + (uint64_t)st * (V_TILE >> 4) + 128 * kk, IDESC_PV, (j > 0 || i > 0) ? 1u : 0u, one);
                }
                umma_commit(&sm.pv_done[j & 1], one);
                umma_commit(&sm.v_free[st], one);
                if (j + 2 < tiles) issue_tile(j + 2);
            }
        }
    } else {
        // ======================= softmax =======================
        const float scale2 = prm.scale * 1.4426950408889634f;  // > 0 (checked on the host)
        const uint32_t tok = m0 + row / G;
        const int64_t qpos = q0 + tok, row_lo = (win && qpos + 1 > win) ? qpos + 1 - win : 0;
        for (int it = 0; it < n_tiles; ++it) {
            const WideTile t = tile_at(it);
            const int b = it & 1;
            float s[32];
            {
                mbar_wait(&sm.s_ready[b], (it >> 1) & 1, prm.status, 531, failed);
                tc_fence_after_sync();
                uint32_t r[32];
                tmem_ld_32x32b_x32(lane_addr + TMEM_S + b * 64 + 32 * half, r);
                tc_wait_ld();
                tc_fence_before_sync();
#pragma unroll
                for (int i = 0; i < 32; i++) s[i] = __uint_as_float(r[i]);
            }
            // masks only where the tile crosses a band edge or the end of its source
            if (t.pos0 + TILE_K - 1 > first_qpos || t.pos0 < last_lo || t.pos0 < t.lo || t.pos0 + TILE_K - 1 > t.hi) {
                const int64_t at = t.pos0 + 32 * half;
                const int64_t lo64 = max(row_lo, t.lo) - at, hi64 = min(qpos, t.hi) - at;
                const int lo = (int)max((int64_t)-1, min((int64_t)64, lo64)), hi = (int)max((int64_t)-1, min((int64_t)64, hi64));
#pragma unroll
                for (int i = 0; i < 32; i++)
                    if (i < lo || i > hi) s[i] = -INFINITY;
            }
            float mx = max3(s[0], s[1], s[2]);
#pragma unroll
            for (int i = 3; i < 31; i += 2) mx = max3(mx, s[i], s[i + 1]);
            mx = fmaxf(mx, s[31]) * scale2;
            // The two threads of a row agree on its maximum; it moves only when a score exceeds it by 2^8.  The barrier also
            // stands between their reads of S and the writes of P over it.
            const bool raise = named_barrier_or(1 + kq, 64, mx > m_run + GROW_T);
            tc_fence_after_sync();
            if (raise) {
                sm.red[half][row] = mx;
                named_barrier_sync(5 + kq, 64);
                const float top = fmaxf(sm.red[0][row], sm.red[1][row]);
                const float now = top > m_run + GROW_T ? top : m_run;
                const float corr = ex2(m_run - now);
                m_run = now;
                l_run *= corr;
                if (it > 0) {
                    mbar_wait(&sm.pv_done[b ^ 1], ((it - 1) >> 1) & 1, prm.status, 532, failed);
                    tc_fence_after_sync();
#pragma unroll 1
                    for (int c = 0; c < 4; c++) {
                        uint32_t o[32];
                        tmem_ld_32x32b_x32(lane_addr + TMEM_O + 128 * half + 32 * c, o);
                        tc_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                        tmem_st_32x32b_x32(lane_addr + TMEM_O + 128 * half + 32 * c, o);
                    }
                    tc_wait_st();
                }
            }
            // P = 2^(s * scale2 - m + 7) as f16 hi + lo; l from the unrounded values
            uint32_t hi[16], lo[16];
            {
                const float2 sc2 = make_float2(scale2, scale2), neg = make_float2(EXP_BIAS - m_run, EXP_BIAS - m_run);
                float2 l2[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float2 x = __ffma2_rn(make_float2(s[2 * i], s[2 * i + 1]), sc2, neg);
                    const float2 p = make_float2(ex2(x.x), ex2(x.y));
                    l2[i & 1] = __fadd2_rn(l2[i & 1], p);
                    hi[i] = pack_half2(p.x, p.y);
                    const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi[i]));
                    lo[i] = pack_half2(p.x - h.x, p.y - h.y);
                }
                l_run += (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y);
            }
            const uint32_t p_at = lane_addr + TMEM_S + b * 64 + 16 * half;
            tmem_st_32x32b_x16(p_at, hi);
            tmem_st_32x32b_x16(p_at + 32, lo);
            tc_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.p_ready[b]);
        }
        if (n_tiles > 0) mbar_wait(&sm.pv_done[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1, prm.status, 534, failed);
        sm.red[half][row] = l_run;
    }
    if (failed) sm.abort = 1;
    tc_fence_before_sync();
    __syncthreads();
    if (prm.n_cta > 1) cluster_sync();  // neither CTA's shared memory is a target or a source any more
    tc_fence_after_sync();

    // ---- out = O / l --------------------------------------------------------------------------------------
    const bool soft = warp < SOFT_THREADS / 32;
    float l = 0.0f, w_own = 1.0f, w_other = 0.0f;
    if (soft) l = sm.red[0][row] + sm.red[1][row];
    float4* xo = reinterpret_cast<float4*>(sm.k[0][0]);  // split: the other CTA's O of this CTA's 128 dims, [half][16][row]
    static_assert(sizeof(WideSmem::k) >= 2 * 16 * ROWS * sizeof(float4), "the K stages hold it");
    if (split) {
        if (soft) {
            const uint32_t dst = map_to_rank(smem_u32(xo + half * 16 * ROWS + row), rank ^ 1u);
#pragma unroll 1
            for (int c = 0; c < 2; c++) {
                uint32_t o[32];
                if (n_tiles > 0) {  // uniform over the CTA
                    tmem_ld_32x32b_x32(lane_addr + TMEM_O + 128 * (rank ^ 1u) + 64 * half + 32 * c, o);
                    tc_wait_ld();
                } else {
#pragma unroll
                    for (int i = 0; i < 32; i++) o[i] = 0u;
                }
#pragma unroll
                for (int i = 0; i < 8; i++)
                    st_cluster_f4(dst + (8 * c + i) * ROWS * 16, make_float4(__uint_as_float(o[4 * i]), __uint_as_float(o[4 * i + 1]),
                                                                             __uint_as_float(o[4 * i + 2]), __uint_as_float(o[4 * i + 3])));
            }
            if (half == 0) {
                const uint32_t ml = map_to_rank(smem_u32(&sm.other_ml[row]), rank ^ 1u);
                asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(ml), "f"(m_run), "f"(l) : "memory");
            }
        }
        __syncwarp();
        cluster_sync();
        if (soft) {
            const float2 ml = sm.other_ml[row];
            const float top = fmaxf(m_run, ml.x);
            w_own = ex2(m_run - top);
            w_other = ex2(ml.x - top);
            l = rank == 0 ? fmaf(l, w_own, ml.y * w_other) : fmaf(ml.y, w_other, l * w_own);  // the same bits in both
        }
    }
    if (soft) {
        const float inv = 1.0f / l;
        const bool live = (uint32_t)(row / G) < live_tok;
        bool odd = false;
        const int n_c = split ? 2 : 4, col0 = split ? 128 * (int)rank + 64 * half : 128 * half;
        __half* orow = prm.out + ((size_t)(m0 + (live ? row / G : 0)) * (prm.n_kv * G) + kvh * G + row % G) * HD + col0;
#pragma unroll 1
        for (int c = 0; c < n_c; c++) {
            uint32_t o[32];
            if (n_tiles > 0) {  // uniform over the CTA
                tmem_ld_32x32b_x32(lane_addr + TMEM_O + col0 + 32 * c, o);
                tc_wait_ld();
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) o[i] = 0u;
            }
            float y[32];
#pragma unroll
            for (int i = 0; i < 32; i++) y[i] = __uint_as_float(o[i]);
            if (split) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 f = xo[(half * 16 + 8 * c + i) * ROWS + row];
                    y[4 * i] = fmaf(f.x, w_other, y[4 * i] * w_own);
                    y[4 * i + 1] = fmaf(f.y, w_other, y[4 * i + 1] * w_own);
                    y[4 * i + 2] = fmaf(f.z, w_other, y[4 * i + 2] * w_own);
                    y[4 * i + 3] = fmaf(f.w, w_other, y[4 * i + 3] * w_own);
                }
            }
            if (live) {
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    y[i] *= inv;
                    odd |= !(fabsf(y[i]) <= 3.4e38f);
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
                    *reinterpret_cast<uint4*>(orow + 32 * c + 8 * i) = make_uint4(pack_half2(y[8 * i], y[8 * i + 1]), pack_half2(y[8 * i + 2], y[8 * i + 3]),
                                                                                  pack_half2(y[8 * i + 4], y[8 * i + 5]), pack_half2(y[8 * i + 6], y[8 * i + 7]));
            }
        }
        const uint32_t rows_odd = __ballot_sync(0xffffffffu, odd);
        if (rows_odd != 0 && lane == 0) {
            sm.redo[0][half][kq] = rows_odd;
            if (split) st_cluster_u32(map_to_rank(smem_u32(&sm.redo[1][half][kq]), rank ^ 1u), rows_odd);
        }
    }
    // A wait that ran out leaves copies and MMAs of this CTA in flight that nobody will wait for: give them a bounded
    // time to land before the shared and tensor memory they target is handed to the next CTA.
    tc_fence_before_sync();
    __syncthreads();
    if (*(volatile uint32_t*)&sm.abort != 0u) {
        let_copies_land();
        __syncthreads();
    }
    if (warp == 0) tmem_dealloc(tmem, TMEM_COLS);
    if (prm.n_cta > 1) {
        // both CTAs have written their share and know of each other's rows: what is written again is the last
        __syncwarp();
        cluster_sync();
    }
    const uint4* redo = reinterpret_cast<const uint4*>(sm.redo);
    static_assert(sizeof(WideSmem::redo) == 4 * sizeof(uint4), "four words of rows / 32 bits each");
    uint32_t any = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) any |= redo[i].x | redo[i].y | redo[i].z | redo[i].w;
    if (any != 0) stream_rows<TWO_SRC>(prm, sm, m0, kvh, rank);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// [row][head][256] f16, boxes of 64 dims x box_heads x box_rows.
int encode_rows(const LaunchArgs& a, CUtensorMap* tm, const void* base, uint64_t rows, uint64_t heads, uint32_t box_heads, uint32_t box_rows)
{
    const uint64_t dims[3] = {HD, heads, rows};
    const uint64_t strides[2] = {HD * 2, heads * HD * 2};
    const uint32_t box[3] = {64, box_heads, box_rows};
    return encode_tensor_map(a, tm, 1, 3, const_cast<void*>(base), dims, strides, box, 3);
}

}  // namespace

// What the tensor-core kernel takes: a positive softmax scale (the row maximum is taken before it), operands whose rows the
// copies can address (K and V with at least one row, row indexes within an int; the launcher refuses bases that are not 16-byte
// aligned, which the streaming kernel's loads need too) and a 16-byte aligned output.  What else the launcher accepts stays on the
// streaming kernel.  So would calls with little history and few queries, were it known here (us, streaming | this one, 16 queries: 0 cached
// tokens 4.8 | 9.6, 64 cached 14 | 9.7, a full window 144 | 20).
template <bool TWO_SRC>
bool prefill_wide_takes(const KvOperand& k0, const KvOperand& v0, const KvOperand& k1, const KvOperand& v1, const void* q, const void* out, float scale)
{
    if (!(scale > 0.0f) || !(scale < 1e30f) || !aligned16(q) || !aligned16(out)) return false;
    const KvOperand* ops[4] = {&k0, &v0, &k1, &v1};
    for (int i = 0; i < (TWO_SRC ? 4 : 2); i++)
        if (ops[i]->rows == 0 || ops[i]->rows >= (1u << 30) || !aligned16(ops[i]->data)) return false;
    return true;
}

template <bool TWO_SRC>
int launch_prefill_wide(const LaunchArgs& a, const void* q, const KvOperand& k0, const KvOperand& v0, const KvOperand& k1, const KvOperand& v1, void* out,
                        const void* step, uint32_t n_kv, uint32_t m, uint32_t window, uint32_t ring, float scale)
{
    const uint32_t units = (m + ROWS / G - 1) / (ROWS / G) * n_kv;
    const uint32_t n_cta = 2 * units <= (uint32_t)a.sm_count ? 2 : 1;  // one CTA per SM: two per unit while they fit at once
    const WideParams prm{(const uint32_t*)step, (__half*)out, a.status, m, n_kv, window, ring, scale, n_cta, q, k0, v0, k1, v1};
    CUtensorMap tq, tk0, tv0, tk1, tv1;
    if (int r = encode_rows(a, &tq, q, m, n_kv * G, G, ROWS / G)) return r;
    if (int r = encode_rows(a, &tk0, k0.data, k0.rows, n_kv, 1, TILE_K)) return r;
    if (int r = encode_rows(a, &tv0, v0.data, v0.rows, n_kv, 1, TILE_K)) return r;
    tk1 = tk0;
    tv1 = tv0;
    if (TWO_SRC) {
        if (int r = encode_rows(a, &tk1, k1.data, k1.rows, n_kv, 1, TILE_K)) return r;
        if (int r = encode_rows(a, &tv1, v1.data, v1.rows, n_kv, 1, TILE_K)) return r;
    }
    auto kern = wide_prefill_kernel<TWO_SRC>;
    {
        static std::mutex attr_mutex;
        static bool attr_set[64] = {};
        std::lock_guard<std::mutex> lock(attr_mutex);
        if (a.device >= 64 || !attr_set[a.device]) {
            if (int r = check_cuda(a, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WideSmem)),
                                   "cudaFuncSetAttribute(wide_prefill)"))
                return r;
            if (a.device < 64) attr_set[a.device] = true;
        }
    }
    const cudaError_t err = launch_dependent_clusters(kern, n_cta, dim3(units * n_cta), dim3(WIDE_THREADS), sizeof(WideSmem), a.stream, tq, tk0, tv0, tk1,
                                                      tv1, prm);
    ++*a.launches;
    return check_cuda(a, err, "attn_prefill_sliding");
}
template bool prefill_wide_takes<false>(const KvOperand&, const KvOperand&, const KvOperand&, const KvOperand&, const void*, const void*, float);
template bool prefill_wide_takes<true>(const KvOperand&, const KvOperand&, const KvOperand&, const KvOperand&, const void*, const void*, float);
template int launch_prefill_wide<false>(const LaunchArgs&, const void*, const KvOperand&, const KvOperand&, const KvOperand&, const KvOperand&, void*,
                                        const void*, uint32_t, uint32_t, uint32_t, uint32_t, float);
template int launch_prefill_wide<true>(const LaunchArgs&, const void*, const KvOperand&, const KvOperand&, const KvOperand&, const KvOperand&, void*,
                                       const void*, uint32_t, uint32_t, uint32_t, uint32_t, float);

}  // namespace sgb
