// Flash-attention prefill on tcgen05, head_dim 128, GQA 2, for long key ranges: causal, one key source.  Same units, semantics and
// partials as attn_prefill_flash.cu (which says where the line between the two lies); a CTA has a whole SM.
//
// A unit's 128 rows meet 128 keys a tile: as M128 N128 K16 both products run at the tensor pipe's full rate, where Q K^T of a 64-key tile
// is bound by its operands in shared memory.  Two softmax groups of four warps take the tiles in turns, and three S buffers let
// Q K^T run two tiles ahead, so a tile's score -> softmax -> P V chain costs latency, not throughput.  A softmax thread has a
// row; 128 scores do not fit its registers, so the upper 64 come out of tensor memory twice.
// 4096 queries over 131072 keys, 16 kv heads: 1460 cycles a tile and SM, the special-function unit at 1024 of them and the tensor pipe too;
// the softmax groups take 1800 of 2900 cycles for the exponentials, and the board is at its power limit.  With the dequantisation
// 8211 us, where the 64-key kernel takes 8543.
#include <mutex>

#include "attn_flash.cuh"

namespace sgb {

namespace {

constexpr int HD = 128;
constexpr int G = 2;
constexpr int BLOCK_TOK = 64;   // query tokens per CTA
constexpr int BLOCK_M = 128;    // rows = tokens x G
constexpr int BLOCK_N = 128;    // keys per tile
constexpr int GROUP_THREADS = 128, SOFTMAX_THREADS = 2 * GROUP_THREADS;
constexpr int MMA_WARP = 8, LOAD_WARP = 9;
constexpr int FLASH_THREADS = 320;
constexpr int STAGES = 3;                           // tiles of K, of V and of S
constexpr uint32_t Q_HALF = 128 * 128;              // 64 dims of 128 rows
constexpr uint32_t Q_BYTES = 2 * Q_HALF;
constexpr uint32_t KV_HALF = BLOCK_N * 128;         // 64 dims of a tile's keys
constexpr uint32_t KV_TILE_BYTES = 2 * KV_HALF;
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t TMEM_O = 0;                      // O: 128 f32 columns
constexpr uint32_t TMEM_S = 128;                    // S: three buffers of 128
constexpr float RESCALE_T = 8.0f;

// The struct is not padded to its 1024-byte tile alignment: the dynamic shared-memory base is declared 1024-aligned instead (and
// checked at run time).
struct FlashSmem {
    uint8_t q[2][Q_HALF];                    // [dim half][128 rows x 128 B]
    uint8_t k[STAGES][2][KV_HALF];           // [stage][dim half][128 keys x 128 B]
    uint8_t v[STAGES][2][KV_HALF];
    float m_ref[BLOCK_M];                    // running maximum of a row, from one tile's softmax warp to the next's
    float l_sum[2][BLOCK_M];
    uint64_t full_k[STAGES];                 // TMA -> MMA warp
    uint64_t full_v[STAGES];
    uint64_t s_ready[STAGES];                // MMA commit: S[b] holds Q K^T of a tile
    uint64_t p_ready[STAGES][2];             // softmax warps: half the keys of P(j) are in tensor memory
    uint64_t pv_done[STAGES];                // MMA commit: O += P V of a tile has completed
    uint64_t m_known[2][4];                  // a softmax warp: m_ref of its rows is what its tile goes by, [tile parity][warp of the group]
    uint64_t q_bar;
    uint32_t tmem_base;
    uint32_t abort;                          // a bounded wait ran out somewhere in the CTA
};
static_assert(sizeof(FlashSmem) <= 227 * 1024, "one CTA per SM");

// Roles: warps 0-3 and 4-7 = two softmax groups that take the tiles in turns (thread r of either owns row r of S), warp 8 = MMA
// issue (the whole warp runs the loop, an elected lane issues), warp 9 = TMA loads (one thread).  The tensor pipe runs, in order, ... PV(j) QK(j+3) PV(j+1) QK(j+4) ...: with
// three S buffers the scores of the next two tiles are there when a group is done with its own, and the groups' special-function,
// conversion and hand-over phases overlap.  Both add to one O, so they go by one running maximum per row: it passes from tile to
// tile through m_ref, warp by warp, right after a tile's maximum is known.
__global__ void __launch_bounds__(FLASH_THREADS, 1)
    flash_long_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                      const FlashParams prm)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    FlashSmem& sm = *reinterpret_cast<FlashSmem*>(smem_raw);
    if ((smem_u32(smem_raw) & 1023u) != 0u) {  // the swizzled tiles need it; never seen, but never assumed
        if (threadIdx.x == 0) report_error(prm.status, DEV_ERR_BOUNDS, 400, smem_u32(smem_raw), 0);
        return;
    }

    const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < STAGES; i++) {
            mbar_init(&sm.full_k[i], 1);
            mbar_init(&sm.full_v[i], 1);
            mbar_init(&sm.s_ready[i], 1);
            mbar_init(&sm.p_ready[i][0], GROUP_THREADS / 32);  // an arrival per warp: they serialise on the barrier's word
            mbar_init(&sm.p_ready[i][1], GROUP_THREADS / 32);
            mbar_init(&sm.pv_done[i], 1);
        }
        for (int i = 0; i < 8; i++) mbar_init(&sm.m_known[i >> 2][i & 3], 1);
        mbar_init(&sm.q_bar, 1);
        sm.abort = 0;
        mbar_fence_init();
    }
    if (tid < BLOCK_M) sm.m_ref[tid] = NEG_SENTINEL;
    if (warp == 0) {
        tmem_alloc(&sm.tmem_base, TMEM_COLS);
        tmem_relinquish();
    }
    pdl_wait();  // the step words, q, K and V come from earlier kernels of the stream
    pdl_launch_dependents();
    // Launch order (blockIdx.x, then pieces): groups of `head_group` kv heads one after the other; inside a group the latest
    // query tile (the one with the most keys) of every head first, then the one before it, and so on.  The CTAs that run
    // together then read the K/V of one group, which the launcher sizes to stay in L2, and within the group the short
    // CTAs fill the end.
    const int n_qtiles = (int)((prm.m_tokens + BLOCK_TOK - 1) / BLOCK_TOK);
    const uint32_t per_group = prm.head_group * (uint32_t)n_qtiles;
    const uint32_t in_group = blockIdx.x % per_group;
    const int qt = n_qtiles - 1 - (int)(in_group / prm.head_group);
    const int kvh = (int)((blockIdx.x / per_group) * prm.head_group + in_group % prm.head_group);
    const uint32_t m0 = (uint32_t)qt * BLOCK_TOK;
    const int64_t q0 = ld_global(prm.step + STEP_Q0);
    const uint32_t tok_in_tile = min((uint32_t)BLOCK_TOK, prm.m_tokens - m0);

    // ---- which key tiles this CTA visits -------------------------------------------------------------
    const int64_t first_qpos = q0 + m0, last_qpos = q0 + m0 + tok_in_tile - 1;
    int n_tiles = (int)(last_qpos / BLOCK_N + 1);
    // gridDim.z pieces share a unit: piece z visits a contiguous run of its key tiles and leaves a partial
    // (unnormalised O, max, sum) that combine_pieces_kernel merges.  `it` below counts from the piece's
    // first tile, so barrier phases do not depend on the split.
    const int per_piece = (n_tiles + (int)gridDim.z - 1) / (int)gridDim.z;
    const int t_begin = min(n_tiles, (int)blockIdx.z * per_piece);
    n_tiles = min(n_tiles, t_begin + per_piece) - t_begin;
    auto pos_at = [&](int it) { return (int64_t)(t_begin + it) * BLOCK_N; };  // of a tile's first key

    // ---- the rest of the set-up -----------------------------------------------------------------------------
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = sm.tmem_base;
    bool failed = false;

    if (warp == LOAD_WARP) {
        // ======================= TMA loads =======================
        if (lane == 0) {
            tma_prefetch_desc(&tm_q);
            tma_prefetch_desc(&tm_k);
            tma_prefetch_desc(&tm_v);
            auto load = [&](bool is_v, int it) {
                if (it >= n_tiles) return;
                const int st = it % STAGES, row = (int)pos_at(it);
                const CUtensorMap* map = is_v ? &tm_v : &tm_k;
                uint64_t* bar = is_v ? &sm.full_v[st] : &sm.full_k[st];
                uint8_t* dst = is_v ? sm.v[st][0] : sm.k[st][0];
                mbar_arrive_expect_tx(bar, KV_TILE_BYTES);
                tma_load_3d(dst, map, bar, 0, kvh, row);
                tma_load_3d(dst + KV_HALF, map, bar, 64, kvh, row);
            };
            mbar_arrive_expect_tx(&sm.q_bar, Q_BYTES);
            tma_load_3d(sm.q[0], &tm_q, &sm.q_bar, 0, kvh * G, (int)m0);
            tma_load_3d(sm.q[1], &tm_q, &sm.q_bar, 64, kvh * G, (int)m0);
            load(false, 0);
            load(false, 1);
            load(true, 0);
            load(false, 2);
            load(true, 1);
            load(true, 2);
            // in the order in which the tensor pipe lets go of the stages: K(j) with QK(j), then V(j - 2) with PV(j - 2)
            for (int j = 0; j + 1 < n_tiles; ++j) {
                if (j + STAGES < n_tiles) {
                    mbar_wait(&sm.s_ready[j % STAGES], (j / STAGES) & 1, prm.status, 431, failed, 50);
                    if (failed) break;  // never write into a stage that may still be read
                    load(false, j + STAGES);
                }
                if (j >= 2) {
                    mbar_wait(&sm.pv_done[(j - 2) % STAGES], ((j - 2) / STAGES) & 1, prm.status, 432, failed, 50);
                    if (failed) break;
                    load(true, j + 1);
                }
            }
        }
    } else if (warp == MMA_WARP) {
        // ======================= MMA issue =======================
        {
            const uint32_t one = elect_one(), tm = warp_uniform(tmem);
            const int tiles = warp_uniform(n_tiles);
            constexpr uint32_t IDESC_QK = umma_idesc_f16(BLOCK_M, BLOCK_N, 0, 0);
            constexpr uint32_t IDESC_PV = umma_idesc_f16(BLOCK_M, HD, 0, 1);
            // Operand descriptors are built once; a step of 32 bytes along K (or of 16 keys of V) is an add to the
            // descriptor's address field (bytes >> 4).  Building them per instruction costs the issuing thread more
            // cycles than the tensor pipe needs for the instruction.
            const uint64_t dq = umma_desc_sw128(smem_u32(sm.q[0]), 16, 1024), dk = umma_desc_sw128(smem_u32(sm.k[0][0]), 16, 1024);
            const uint64_t dv = umma_desc_sw128(smem_u32(sm.v[0][0]), KV_HALF, 1024);
            // S[j % 3] = Q K(j)^T: 8 MMAs of K = 16, once K(j) has landed.
            auto issue_qk = [&](int j) {
                const int b = j % STAGES;
                mbar_wait_warp(&sm.full_k[b], (j / STAGES) & 1, prm.status, 422, failed);
                if (failed) return;
                tc_fence_after_sync();
                const uint64_t k = dk + (uint64_t)b * (KV_TILE_BYTES >> 4);
                const uint32_t d = tm + TMEM_S + b * BLOCK_N;
#pragma unroll
                for (int kk = 0; kk < 8; kk++)
                    umma_f16_ss(d, dq + (kk >> 2) * (Q_HALF >> 4) + 2 * (kk & 3), k + (kk >> 2) * (KV_HALF >> 4) + 2 * (kk & 3), IDESC_QK, kk ? 1u : 0u, one);
                umma_commit(&sm.s_ready[b], one);
            };
            mbar_wait_warp(&sm.q_bar, 0, prm.status, 421, failed);
            for (int j = 0; j < STAGES && j < tiles; ++j) issue_qk(j);
            for (int j = 0; j < tiles && !failed; ++j) {
                const int b = j % STAGES;
                mbar_wait_warp(&sm.full_v[b], (j / STAGES) & 1, prm.status, 425, failed);
                // P(j) lives in the first 64 columns of S[b] (packed f16 pairs), written by the softmax warps
                const uint64_t v = dv + (uint64_t)b * (KV_TILE_BYTES >> 4);
                const uint32_t p = tm + TMEM_S + b * BLOCK_N;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    mbar_wait_warp(&sm.p_ready[b][h], (j / STAGES) & 1, prm.status, 423, failed);
                    if (failed) break;
                    tc_fence_after_sync();
#pragma unroll
                    for (int kk = 4 * h; kk < 4 * h + 4; kk++) umma_f16_ts(tm + TMEM_O, p + kk * 8, v + 128 * kk, IDESC_PV, (j | kk) ? 1u : 0u, one);
                }
                if (failed) break;
                umma_commit(&sm.pv_done[b], one);
                // S[b] may be overwritten: the tensor pipe runs in order, and P V of this tile is ahead
                if (j + STAGES < tiles) issue_qk(j + STAGES);
            }
        }
    } else {
        // ======================= softmax: row r of the tile <-> TMEM lane r <-> thread r of a group =======================
        // token m0 + r/2, query head kvh*2 + r%2
        const int group = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t tok = m0 + (uint32_t)(r >> 1);
        const int64_t qpos = q0 + tok;
        const float scale2 = prm.scale * 1.4426950408889634f;  // > 0 (checked on the host)
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        float m_run = NEG_SENTINEL, l_run = 0.0f;

        for (int it = group; it < n_tiles; it += 2) {
            const int b = it % STAGES;
            const int64_t pos0 = pos_at(it);
            mbar_wait(&sm.s_ready[b], (it / STAGES) & 1, prm.status, 424, failed);
            tc_fence_after_sync();
            const uint32_t s_addr = lane_addr + TMEM_S + b * BLOCK_N;
            // Only a tile on the diagonal needs per-element masks: its keys before `end`, a bit each.
            const bool masked = pos0 + BLOCK_N - 1 > first_qpos;
            const int end = (int)min(max(qpos + 1 - pos0, (int64_t)0), (int64_t)BLOCK_N);
            float v[64];
            // the scores of 64 keys; the upper half comes twice (128 at once do not fit the registers), the first time for its maximum
            auto fetch = [&](int h) {
                uint32_t a0[32], a1[32];
                tmem_ld_32x32b_x32(s_addr + 64 * h, a0);
                tmem_ld_32x32b_x32(s_addr + 64 * h + 32, a1);
                tc_wait_ld();
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    v[j] = __uint_as_float(a0[j]);
                    v[32 + j] = __uint_as_float(a1[j]);
                }
                if (masked) {
#pragma unroll
                    for (int w = 0; w < 2; w++) {
                        const int e = min(max(end - 64 * h - 32 * w, 0), 32);
                        const uint32_t seen = e == 32 ? ~0u : (1u << e) - 1;
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (((seen >> j) & 1u) == 0) v[32 * w + j] = -INFINITY;
                    }
                }
            };
            // row max of the raw scores on four independent chains of three-input max; scale2 > 0
            // commutes with max
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            fetch(1);
#pragma unroll
            for (int j = 0; j < 64; j += 2) mx4[(j >> 1) & 3] = max3(mx4[(j >> 1) & 3], v[j], v[j + 1]);
            fetch(0);
#pragma unroll
            for (int j = 0; j < 64; j += 2) mx4[(j >> 1) & 3] = max3(mx4[(j >> 1) & 3], v[j], v[j + 1]);
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale2;
            // The running maximum as the tile before left it, with the other group.
            if (it > 0) {
                mbar_wait(&sm.m_known[(it - 1) & 1][quarter], ((it - 1) >> 1) & 1, prm.status, 426, failed);
                const float m_now = *(volatile float*)&sm.m_ref[r];
                l_run *= ex2(m_run - m_now);  // 1 while it stays
                m_run = m_now;
            }
            const bool grow = mx > m_run + RESCALE_T;
            const bool raised = __any_sync(0xffffffffu, grow);
            float corr = 1.0f;
            if (raised) {
                if (grow) {
                    corr = ex2(m_run - mx);
                    m_run = mx;
                    l_run *= corr;
                }
                *(volatile float*)&sm.m_ref[r] = m_run;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.m_known[it & 1][quarter]);
            // O is rescaled where a row's max moved (rare after the first tiles), and only once P V of the
            // previous tile has completed; P V of this one waits for its P.  (Most tiles skip this wait; its parity stays
            // unambiguous: P V(it - 4) is ahead of this tile's scores in the tensor pipe, P V(it + 2) needs this thread's P(it).)
            if (it > 0 && raised) {
                mbar_wait(&sm.pv_done[(it - 1) % STAGES], ((it - 1) / STAGES) & 1, prm.status, 427, failed);
                tc_fence_after_sync();
#pragma unroll 1
                for (int c = 0; c < 8; c++) {
                    uint32_t o[16];
                    tmem_ld_32x32b_x16(lane_addr + TMEM_O + 16 * c, o);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
                    tmem_st_32x32b_x16(lane_addr + TMEM_O + 16 * c, o);
                }
                tc_wait_st();
            }
            // Rows of the V tile that no query of this CTA sees are zeroed before P V reads them: their P is 0, but 0 times an Inf or
            // NaN there, or in what a caller's over-allocated buffer holds, would not be.
            if (pos0 + BLOCK_N - 1 > last_qpos) {  // uniform over the CTA
                mbar_wait(&sm.full_v[b], (it / STAGES) & 1, prm.status, 429, failed);
                if (pos0 + r > last_qpos) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint4* row = reinterpret_cast<uint4*>(sm.v[b][h] + r * 128);
#pragma unroll
                        for (int i = 0; i < 8; i++) row[i] = make_uint4(0u, 0u, 0u, 0u);
                    }
                }
                fence_proxy_async_smem();  // generic-proxy writes, read next by the tensor pipe
            }
            // p = 2^(s * scale2 - m) with the multiply-add and the running sums on packed f32x2 pipes; P row r goes back into tensor
            // memory over the first half of S[b] (this thread has S in registers), 64 keys at a time
            const float2 sc2 = make_float2(scale2, scale2), neg_m = make_float2(-m_run, -m_run);
            float2 ls4[4] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (h) fetch(1);
                uint32_t pk[32];
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const float2 x = __ffma2_rn(make_float2(v[2 * j], v[2 * j + 1]), sc2, neg_m);
                    const float2 pp = make_float2(ex2(x.x), ex2(x.y));
                    ls4[j & 3] = __fadd2_rn(ls4[j & 3], pp);  // l in f32 from the unrounded p (attn_prefill_global_flash_sp.wgsl:147-156)
                    pk[j] = pack_half2(pp.x, pp.y);
                }
                tmem_st_32x32b_x32(s_addr + 32 * h, pk);
                tc_wait_st();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.p_ready[b][h]);
            }
            l_run += ((ls4[0].x + ls4[0].y) + (ls4[1].x + ls4[1].y)) + ((ls4[2].x + ls4[2].y) + (ls4[3].x + ls4[3].y));
        }
        // ---- epilogue: out = O / l, or this piece's partial; a group has half the dims.  The TMEM loads are warp-wide, so every
        // thread takes part and only the stores are predicated (rows past the end of the chunk are not written). ----
        if (n_tiles > 0) {  // the groups' sums by the maximum that the last tile left
            mbar_wait(&sm.m_known[(n_tiles - 1) & 1][quarter], ((n_tiles - 1) >> 1) & 1, prm.status, 430, failed);
            const float m_now = *(volatile float*)&sm.m_ref[r];
            l_run *= ex2(m_run - m_now);
            m_run = m_now;
        }
        sm.l_sum[group][r] = l_run;
        named_barrier_sync(1, SOFTMAX_THREADS);
        l_run = sm.l_sum[0][r] + sm.l_sum[1][r];
        // the tensor pipe completes in order: the last P V done means all of them are
        if (n_tiles > 0) mbar_wait(&sm.pv_done[(n_tiles - 1) % STAGES], ((n_tiles - 1) / STAGES) & 1, prm.status, 428, failed);
        tc_fence_after_sync();
        const bool live = (uint32_t)(r >> 1) < tok_in_tile;
        const size_t row = (size_t)(live ? tok : m0) * (prm.n_kv * G) + kvh * G + (r & 1);
        const bool whole = gridDim.z == 1;
        const float mul = whole ? 1.0f / l_run : 1.0f;
        float* orow = (whole ? prm.out + row * HD : prm.part_acc + (row * gridDim.z + blockIdx.z) * HD) + 64 * group;
        if (!whole && live && group == 0) *reinterpret_cast<float2*>(prm.part_ml + (row * gridDim.z + blockIdx.z) * 2) = make_float2(m_run, l_run);
#pragma unroll
        for (int c = 0; c < 2; c++) {
            uint32_t o[32];
            if (n_tiles > 0) {  // uniform over the CTA
                tmem_ld_32x32b_x32(lane_addr + TMEM_O + 64 * group + 32 * c, o);
                tc_wait_ld();
            } else {
#pragma unroll
                for (int j = 0; j < 32; j++) o[j] = 0u;  // an empty piece: m = sentinel, l = 0, O = 0
            }
            if (live) {
#pragma unroll
                for (int j = 0; j < 8; j++)
                    *reinterpret_cast<float4*>(orow + 32 * c + 4 * j) =
                        make_float4(__uint_as_float(o[4 * j]) * mul, __uint_as_float(o[4 * j + 1]) * mul,
                                    __uint_as_float(o[4 * j + 2]) * mul, __uint_as_float(o[4 * j + 3]) * mul);
            }
        }
    }
    // A wait that ran out leaves copies and MMAs of this CTA in flight that nobody will wait for: give them
    // a bounded time to land before the shared and tensor memory they target is handed to the next CTA.
    if (failed) sm.abort = 1;
    tc_fence_before_sync();
    __syncthreads();
    if (*(volatile uint32_t*)&sm.abort != 0u) {
        for (int i = 0; i < 50; i++) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 0) tmem_dealloc(tmem, TMEM_COLS);
}

}  // namespace

cudaError_t launch_flash_long(const LaunchArgs& a, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashParams& prm,
                              uint32_t units, uint32_t pieces)
{
    const size_t smem = sizeof(FlashSmem);
    {
        static std::mutex attr_mutex;
        static bool attr_set[64] = {};
        std::lock_guard<std::mutex> lock(attr_mutex);
        if (a.device >= 64 || !attr_set[a.device]) {
            const cudaError_t e = cudaFuncSetAttribute(flash_long_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            if (a.device < 64) attr_set[a.device] = true;
        }
    }
    return launch_dependent(flash_long_kernel, dim3(units, 1, pieces), dim3(FLASH_THREADS), smem, a.stream, tq, tk, tv, prm);
}

}  // namespace sgb
