// Prefill attention for the reference model's global layers on tcgen05: head_dim 512, int8 Q and K with f16 block scales, f16 V,
// 8 query heads per kv head (attn_prefill_global_flash_sp_iq.wgsl).
//
// Two CTAs share one MMA (pair.cuh): 64 query rows each (8 tokens x the 8 query heads of one kv head), M = 128.  64 rows of 512 dims
// are 256 columns of tensor memory that way, so O fits beside the scores with the rows as the M side.  Per 128-key tile:
//   S[64 rows x 128 keys]  = Q K^T   per 32-value scale block, two blocks at a time into one of two buffers of 128 columns
//   O[64 rows x 512 dims] += P V     V as the MN-major B operand straight from its [key][dim] tile, 256 dims an instruction
// of which each CTA loads half the keys of K and half the dims of V.
// Scores: Q's quants are exact as f16.  A key's quants times their f16 scale are whole multiples of the scale's last place, 19 bits, which
// f16 hi + lo hold exactly (for scales above 511, whose quants overflow, in a second pass that splits otherwise); four warps make them from the cache's bytes.  A block's sum so lacks only the scale of Q, which is the
// row's, and the softmax threads have nothing left to do for it but one multiply-add.  The pipe adds the block's 64 products up in f32 and
// truncates, where a sum of int8 products is a whole number; the error against 64 bits is f16's own in both forms.  (Whole-number sums of int8 MMAs, scaled by
// both scales in the softmax threads: they then read 16 x 128 scales a tile through shared memory, which the MMAs read their
// operands from; 364 us.  The transposed form before it, keys and dims as M, took V as the MN-major A operand, 160 cycles
// an instruction where 48 would do, and converted every sum with an instruction of a sixteenth of the rate: 529 us.)
// P = hi + lo, both halves f16, two MMAs per V tile: together they miss p by at most one unit of its last f32 place.  The exponent
// carries +7, so that lo stays clear of f16's subnormals (the factor cancels in O / l); a p below 2^-32 of its row's reference
// maximum is in l but too small for lo.
// The tensor pipe truncates an accumulator each time it adds to it: in one accumulator, outputs shrank by 2e-9 of themselves per
// key (1.7e-5 at 8192 keys, 6.7e-5 at 33280, where the error against 64 bits was 2.22e-4 instead of f16's own 2.08e-4).  From the
// fifth tile on one of the two dim blocks of O is therefore settled in every other tile: the block, plus what was
// settled of it before, added in f32 with rounding, splits into its upper 16 bits, which stay in this CTA's share of the
// output, and the exact rest, from which the tensor pipe goes on; what it adds to stays as small as the sum of a few tiles.
// The block comes first in the products before it is settled, so the tensor pipe is at the other meanwhile, and the warps that make
// the keys do it, which have time (the softmax threads, whose chain the tile's time is, took 1500 cycles a tile for it).
// Roles: warps 0-7 softmax (a row in four threads), 8-11 K, one MMA warp (the even CTA's issues for both), one V loader; mbarriers only.
// Measured, 256 queries at 7936 + 256 keys with the appends and the quantisation of q: 13500 us on the streaming kernel, 529 in the
// transposed form, 345 here (floor 82).  The MMAs need 4900 cycles of a tile's 8500; the rest is the chain of the softmax threads: a
// hand-over of scores has to be read before the buffer takes the one after the next, eight times a tile.  Products issued one or
// two units earlier among the scores: 352 and 372 us for 346.
//
// What a tile reads beyond a query's own keys must not matter: scores are masked by selection, V rows that hold no key are
// zeroed.  A V row that is visible to some query of the tile and not finite is visible to all of them as 0 * Inf, so rows that are
// not finite are computed again by the streaming statement, which reads what each query sees (all of 256 queries at 8192
// keys: 13600 us on the streaming kernel, 12400 here).
#include <mutex>
#include <string>

#include "attn_stream.cuh"
#include "pair.cuh"
#include "sgb_common.cuh"
#include "sgb_kernels.h"

namespace sgb {

namespace {

constexpr int HD = 512, G = 8;
constexpr int ROWS = 64;       // query rows per CTA: 8 tokens x G heads
constexpr int PAIR_TOK = 2 * ROWS / G;  // tokens of a pair of CTAs
constexpr int TILE_K = 128;    // keys per tile
constexpr int SOFT_THREADS = 256, SOFT_WARPS = SOFT_THREADS / 32;
constexpr int K_WARPS = 4, MMA_W = SOFT_WARPS + K_WARPS, V_W = MMA_W + 1;
constexpr int INT8_THREADS = 32 * (V_W + 1);
constexpr int NK = 3;                          // K chunks in flight
constexpr int NV = 4;                          // V units in flight
constexpr uint32_t Q_CHUNK = ROWS * 128;       // 64 dims f16 of every row
constexpr uint32_t K_CHUNK = 64 * 128;         // 64 dims f16 of this CTA's half of a tile's keys
constexpr uint32_t V_UNIT = 64 * 256;          // 64 keys x 128 dims f16, as two [64 keys][128 B] halves
constexpr uint32_t P_HALF = ROWS * 128;        // [64 rows][64 keys] f16
constexpr uint32_t P_TILE = 2 * P_HALF;
constexpr int GROUPS = 8;                      // S hand-overs per tile, two scale blocks each
constexpr uint32_t S_COLS = 128;               // columns of one hand-over
constexpr uint32_t TMEM_O = 0, TMEM_S = 256, TMEM_COLS = 512;
static_assert(TMEM_S + 2 * S_COLS <= TMEM_COLS, "O and two S buffers fit");
constexpr int SETTLE_FROM = 4;                 // the first tile in which a dim block is settled; one in every other tile from there on
constexpr int SETTLE_CHUNK = 4;                // of K, even: the settling comes behind this one and the next
constexpr float EXP_BIAS = 7.0f, GROW_T = 8.0f;

struct Int8Barriers {
    uint64_t k_full[NK], k_free[NK], v_full[NV], v_free[NV], v_here[NV], v_ok[NV], s_ready[2], s_free[2], p_ready, first_done, pv_done,
        parts_here, settle_here, settle_ok;
};

struct Int8Smem {
    uint8_t q[HD / 64][Q_CHUNK];  // quants
    uint8_t k[NK][2][K_CHUNK];    // quants times scales: hi, lo
    uint8_t p[2][P_TILE];  // hi, lo; each [key half][row][64 keys]
    uint8_t v[NV][V_UNIT];
    float qs[HD / 32][ROWS];      // scales of Q, [block][row]
    float red[4][ROWS];
    Int8Barriers bars[2];         // of a pass each
    uint32_t tmem_base, abort;
    uint32_t gone, large, odd;  // of the pair: a wait ran out; a scale that takes quants beyond f16; a row that is not finite
    uint32_t redo[ROWS / 32];  // rows that are not finite, a bit each
};
static_assert(sizeof(Int8Smem) <= 227 * 1024, "one CTA per SM");

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

// Eight signed bytes as f16 pairs, exactly: 0x6400 | (q + 128) is the f16 of q + 1152, 0x4400 | (q + 128) that of q / 256 + 4.5.
template <bool IN_256THS = false>
__device__ __forceinline__ void whole_f16x8(uint2 q, __half2 (&out)[4])
{
    const uint32_t x[2] = {q.x ^ 0x80808080u, q.y ^ 0x80808080u};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t u = __byte_perm(x[i >> 1], IN_256THS ? 0x44444444u : 0x64646464u, (i & 1) ? 0x4342 : 0x4140);
        out[i] = __hsub2(*reinterpret_cast<const __half2*>(&u), __float2half2_rn(IN_256THS ? 4.5f : 1152.0f));
    }
}
__device__ __forceinline__ uint4 as_uint4(const __half2 (&h)[4])
{
    const uint32_t* w = reinterpret_cast<const uint32_t*>(h);
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Keeps what uses a load's registers behind the wait for it.
__device__ __forceinline__ void loaded(uint32_t (&r)[32])
{
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                      "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]));
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

// All roles of a CTA over its tiles.  WIDE takes keys whose scales times quants are beyond f16 as well (see the key warps), for two
// instructions more per pair of values of K, which the tile's time is: as the only pass it took 327 us instead of 317 (256 queries at
// 7936 + 256 keys), 1337 instead of 1235 (64 queries, 32768 keys).
template <bool WIDE>
__device__ __forceinline__ void int8_pass(const CUtensorMap& tm_v, const Int8Params& prm, Int8Smem& sm)
{
    const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
    const uint32_t rank = pair_rank();  // 0 issues the pair's MMAs
    Int8Barriers& bar = sm.bars[WIDE];
    const uint32_t pair = blockIdx.x / 2;
    const int kvh = pair % prm.n_kv;
    const uint32_t n_qt = prm.m_tokens / PAIR_TOK;
    const uint32_t pair_m0 = (n_qt - 1 - pair / prm.n_kv) * PAIR_TOK;  // latest query tile (most keys) first
    const uint32_t m0 = pair_m0 + rank * (ROWS / G);
    const int64_t q0 = prm.step[STEP_Q0];
    const int64_t first_qpos = q0 + m0, last_qpos = q0 + pair_m0 + PAIR_TOK - 1;
    const int64_t rows0 = (int64_t)min(prm.k0.rows, prm.v0.rows);
    int64_t end = last_qpos;  // positions that hold a visible key end here
    if (end >= rows0) {
        if (!WIDE && tid == 0) report_error(prm.status, DEV_ERR_BOUNDS, 211, (uint32_t)rows0, (uint32_t)rows0);
        end = rows0 - 1;
    }
    const int n_tiles = (int)(end / TILE_K + 1);
    // rows of a tile that hold a key of this problem end here; V rows behind it are zeroed
    const int64_t valid_end = min(rows0 - 1, q0 + (int64_t)prm.m_tokens - 1);

    // this CTA's query rows: quants as f16, which holds them exactly, K-major in 128-byte rows; scales in f32
    for (int i = tid; i < ROWS * (HD / 16); i += INT8_THREADS) {
        const int r = i / (HD / 16), c = i % (HD / 16);
        const size_t at = (size_t)(m0 + r / G) * (prm.n_kv * G) + kvh * G + r % G;
        const uint4 u = ld_global(reinterpret_cast<const uint4*>((const int8_t*)prm.q + at * HD) + c);
        __half2 h[2][4];
        whole_f16x8(make_uint2(u.x, u.y), h[0]);
        whole_f16x8(make_uint2(u.z, u.w), h[1]);
#pragma unroll
        for (int e = 0; e < 2; e++) *reinterpret_cast<uint4*>(sm.q[c / 4] + r * 128 + (((2 * (c & 3) + e) ^ (r & 7)) << 4)) = as_uint4(h[e]);
    }
    for (int i = tid; i < ROWS * (HD / 32); i += INT8_THREADS) {
        const int r = i / (HD / 32), b = i % (HD / 32);
        const size_t at = (size_t)(m0 + r / G) * (prm.n_kv * G) + kvh * G + r % G;
        sm.qs[b][r] = (WIDE ? 256.0f : 1.0f) * __half2float(ld_global(prm.q_scales + at * (HD / 32) + b));
    }
    fence_proxy_async_smem();  // read by the tensor pipe
    tc_fence_before_sync();
    __syncthreads();
    pair_sync();  // the other CTA's barriers are there
    tc_fence_after_sync();
    const uint32_t tmem = sm.tmem_base;
    bool failed = false;
    // V unit u of tile j: 64 keys (half u & 1) of this CTA's 128 of the 256 dims of block dim_block(j, u); the blocks take turns in
    // coming first, so that the first can be settled while the tensor pipe is at the other
    auto dim_block = [](int j, int u) { return ((u >> 1) + (j >> 1)) & 1; };

    // The settled part of O as 16-bit halves, in this CTA's own share of the output (64 rows x 512 dims x 2 bytes), which nobody reads
    // before the end: 8 values c of step h (16 of a row's dims) of softmax thread t at [2 * h + c][t].
    auto settled_at = [&](int t, int h, int c) {
        const int e = 2 * h + c;
        return reinterpret_cast<uint4*>(prm.out + ((size_t)(m0 + e / 2) * (prm.n_kv * G) + kvh * G) * HD) + (e & 1) * SOFT_THREADS + t;
    };
    auto fetch_settled = [&](int t, int h, uint4 (&u)[2]) {
        u[0] = *settled_at(t, h, 0);
        u[1] = *settled_at(t, h, 1);
    };
    auto add_settled = [&](const uint4 (&u)[2], uint32_t (&o)[16]) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t w = reinterpret_cast<const uint32_t*>(u)[i];
            o[2 * i] = __float_as_uint(__fadd_rn(__uint_as_float(o[2 * i]), __uint_as_float(w << 16)));
            o[2 * i + 1] = __float_as_uint(__fadd_rn(__uint_as_float(o[2 * i + 1]), __uint_as_float(w & 0xFFFF0000u)));
        }
    };
    auto settle = [&](int t, int h, uint32_t (&o)[16]) {  // o: whole values, left as the rest
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
            *settled_at(t, h, c) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    };
    // dim blocks that have a settled part once tile `it` has had its turn
    auto settled_by = [&](int it) { return it < SETTLE_FROM ? 0u : it < SETTLE_FROM + 2 ? 1u << dim_block(SETTLE_FROM - 1, 0) : 3u; };
    auto settles = [](int it) { return it >= SETTLE_FROM && (it & 1) == 0; };
    auto settle_phase = [](int it) { return ((it - SETTLE_FROM) >> 1) & 1; };  // of the last settling up to tile `it`
    // A CTA's settled parts change hands twice: the softmax threads, who rescale them where a tile raises a maximum, leave them to the key warps
    // with parts_here ahead of a settling, and get them back with settle_here.  Both are barriers of the CTA itself: the parts lie in
    // global memory, for which the pair's own hand-overs (pair.cuh) do not stand.

    if (warp >= SOFT_WARPS && warp < MMA_W) {
        // ======================= K: quants times scales as f16 hi + lo, 64 dims of this CTA's 64 keys at a time =======================
        // A thread has a key's 32-value block: hi = f16(s * q), lo = s * q - hi, which f16 holds exactly (s * q is a multiple of s's last
        // place, and hi misses it by 64 of those at most).  What overflows f16, or has a scale that is not finite, makes
        // infinities of both signs, so NaN scores, and its rows are computed again: by the WIDE pass where the scale is a number.
        // WIDE: hi = f16(s * q / 256), at most 2^15, and lo = s * q - 256 * hi, exact as well (where hi is subnormal, 256 * hi misses s * q by up to
        // 2^-17); the MMA that adds the first hi takes the sum of the lo by its 256th.  256 * hi is beyond f16 for a large s and a 256th of
        // a small one's last place is no f16, so lo comes in either order.
        const int t = tid - 32 * SOFT_WARPS, key = t >> 1, half = t & 1;
        const int64_t key_rows = rows0 - (int)rank * 64 - key;  // tiles that start before this hold the key
        const size_t row_q = (size_t)prm.n_kv * HD, row_s = (size_t)prm.n_kv * (HD / 32);
        const int8_t* quants = (const int8_t*)prm.k0.data + ((size_t)rank * 64 + key) * row_q + (size_t)kvh * HD + 32 * half;
        const __half* scales = prm.k0.scales + ((size_t)rank * 64 + key) * row_s + (size_t)kvh * (HD / 32) + half;
        const int n_chunks = n_tiles * (HD / 64);
        struct Block {
            uint4 q[2];
            __half s;
        };
        auto fetch = [&](int n, Block& b) {
            const int64_t pos0 = (int64_t)(n >> 3) * TILE_K;
            b.q[0] = b.q[1] = make_uint4(0u, 0u, 0u, 0u);
            b.s = __float2half_rn(0.0f);
            if (n >= n_chunks || pos0 >= key_rows) return;
            const uint4* p = reinterpret_cast<const uint4*>(quants + pos0 * row_q + 64 * (n & 7));
            b.q[0] = ld_global(p);
            b.q[1] = ld_global(p + 1);
            b.s = ld_global(scales + pos0 * row_s + 2 * (n & 7));
        };
        auto convert = [&](int n, const Block& b) {
            const int st = n % NK;
            if (n >= NK && !mbar_wait_warp(&bar.k_free[st], (n / NK - 1) & 1, prm.status, 511, failed)) return;
            const __half2 s2 = __half2half2(b.s);
            const bool upper = !(__habs(b.s) < __float2half_rn(64.0f));
            const __half2 f256 = __float2half2_rn(256.0f), f1 = __float2half2_rn(1.0f);
            const __half2 s_lo = upper ? s2 : __hmul2(s2, f256), less = __hneg2(upper ? f1 : f256), times = upper ? f256 : f1;  // WIDE
            const uint2* q = reinterpret_cast<const uint2*>(b.q);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                __half2 whole[4], hi[4], lo[4];
                whole_f16x8<WIDE>(q[c], whole);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    hi[i] = __hmul2(s2, whole[i]);
                    lo[i] = WIDE ? __hmul2(__hfma2(s_lo, whole[i], __hmul2(hi[i], less)), times) : __hfma2(s2, whole[i], __hneg2(hi[i]));
                }
                const uint32_t off = key * 128 + (((4 * half + c) ^ (key & 7)) << 4);
                *reinterpret_cast<uint4*>(sm.k[st][0] + off) = as_uint4(hi);
                *reinterpret_cast<uint4*>(sm.k[st][1] + off) = as_uint4(lo);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive_pair(at_leader(&bar.k_full[st]));
        };
        Block even, odd;  // two chunks' loads under way
        fetch(0, even);
        fetch(1, odd);
        for (int n = 0; n < n_chunks && !failed; n += 2) {
            convert(n, even);
            fetch(n + 2, even);
            if (failed) break;
            convert(n + 1, odd);
            fetch(n + 3, odd);
            const int it = n >> 3;
            if ((n & 7) == SETTLE_CHUNK && settles(it) && !failed) {
                // The products of the last tile's first block are done, or soon; the tensor pipe is at the other's and this tile's scores
                // meanwhile.  These warps have the time, and the 64 lanes and their twins that the softmax threads' parts are named by.
                const int db = dim_block(it - 1, 0), quarter = warp & 3;
                const uint32_t block = tmem + ((uint32_t)(quarter * 32) << 16) + TMEM_O + db * 128;
                const bool before = ((settled_by(it - 1) >> db) & 1) != 0;
                // One phase per settling, and the next one's needs chunks of K that these warps convert behind this wait.  It does not hold
                // them up: the buffer of the chunk just converted came free behind the last tile's p_ready.
                static_assert(SETTLE_CHUNK + 1 - NK >= 2, "chunks from the third on are multiplied behind the last tile's p_ready");
                mbar_wait_warp(&bar.parts_here, settle_phase(it), prm.status, 538, failed);
#pragma unroll 1
                for (int half = 0; half < 2; half++) {
                    const int owner = half * 128 + quarter * 32 + lane;
                    uint4 u[4][2] = {};  // asked for ahead of the wait below (behind it they cost 355 us for 345)
                    if (before)
#pragma unroll
                        for (int h = 0; h < 4; h++) fetch_settled(owner, 4 * db + h, u[h]);
                    if (half == 0) {
                        mbar_wait_warp(&bar.first_done, (it - 1) & 1, prm.status, 535, failed);
                        tc_fence_after_sync();
                    }
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        uint32_t o[16];
                        tmem_ld_32x32b_x16(block + 64 * half + 16 * h, o);
                        tc_wait_ld();
                        add_settled(u[h], o);
                        settle(owner, 4 * db + h, o);
                        tmem_st_32x32b_x16(block + 64 * half + 16 * h, o);
                    }
                }
                tc_wait_st();
                tc_fence_before_sync();
                __threadfence_block();  // the parts are read by the softmax threads
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&bar.settle_here);
                    mbar_arrive_pair(at_leader(&bar.settle_ok));
                }
            }
        }
    } else if (warp == V_W) {
        // ======================= V loads in units of 64 keys x 128 dims =======================
        int n = 0;
        for (int j = 0; j < n_tiles && !failed; ++j) {
            const int64_t pos0 = (int64_t)j * TILE_K;
            const bool tail = pos0 + TILE_K - 1 > valid_end;  // the last tile at most: v_here and v_ok of a slot have one phase.  The MMA warp computes the same
            for (int u = 0; u < 4; u++, n++) {
                const int st = n % NV;
                if (n >= NV && !mbar_wait_warp(&bar.v_free[st], (n / NV - 1) & 1, prm.status, 512, failed, 50)) break;
                const int kh = u & 1, dim = dim_block(j, u) * 256 + (int)rank * 128;
                if (!tail) {
                    if (lane == 0) {
                        if (rank == 0) mbar_arrive_expect_tx(&bar.v_full[st], 2 * V_UNIT);
                        tma_load_3d_pair(sm.v[st], &tm_v, at_leader(&bar.v_full[st]), dim, kvh, (int)pos0 + kh * 64);
                        tma_load_3d_pair(sm.v[st] + V_UNIT / 2, &tm_v, at_leader(&bar.v_full[st]), dim + 64, kvh, (int)pos0 + kh * 64);
                    }
                    continue;
                }
                if (lane == 0) {
                    mbar_arrive_expect_tx(&bar.v_here[st], V_UNIT);
                    tma_load_3d(sm.v[st], &tm_v, &bar.v_here[st], dim, kvh, (int)pos0 + kh * 64);
                    tma_load_3d(sm.v[st] + V_UNIT / 2, &tm_v, &bar.v_here[st], dim + 64, kvh, (int)pos0 + kh * 64);
                }
                __syncwarp();
                if (!mbar_wait_warp(&bar.v_here[st], 0, prm.status, 513, failed)) break;
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
                if (lane == 0) mbar_arrive_pair(at_leader(&bar.v_ok[st]));
            }
        }
    } else if (warp == MMA_W) {
        // ======================= MMA issue, for both CTAs =======================
        if (rank == 0) {
            const uint32_t one = elect_one(), tm = warp_uniform(tmem);
            const int tiles = warp_uniform(n_tiles);
            constexpr uint32_t IDESC_QK = umma_idesc_f16(2 * ROWS, TILE_K, 0, 0);
            constexpr uint32_t IDESC_PV = umma_idesc_f16(2 * ROWS, 256, 0, 1);
            const uint64_t dq = umma_desc_sw128(smem_u32(sm.q[0]), 16, 1024), dk = umma_desc_sw128(smem_u32(sm.k[0][0]), 16, 1024);
            const uint64_t dv = umma_desc_sw128(smem_u32(sm.v[0]), V_UNIT / 2, 1024);
            const uint64_t dp = umma_desc_sw128(smem_u32(sm.p[0]), 16, 1024);
            // S of (tile j, group g) into buffer n & 1, n = j * GROUPS + g
            auto issue_qk = [&](int j, int g) {
                const int n = j * GROUPS + g;
                if (n >= 2) mbar_wait_warp(&bar.s_free[n & 1], ((n - 2) >> 1) & 1, prm.status, 521, failed);
                const uint32_t d = tm + TMEM_S + (n & 1) * S_COLS;
                const int st = n % NK;
                mbar_wait_warp(&bar.k_full[st], (n / NK) & 1, prm.status, 522, failed);
                if (failed) return;
                tc_fence_after_sync();
#pragma unroll
                for (int e = 0; e < 2; e++)  // the scale blocks of the chunk
#pragma unroll
                    for (int i = 0; i < 4; i++) {  // lo, then hi
                        const uint32_t off = 2 * (2 * e + (i & 1)), hl = 1 - (i >> 1);
                        const uint64_t qd = dq + g * (Q_CHUNK >> 4) + off, kd = dk + (2 * st + hl) * (K_CHUNK >> 4) + off;
                        if (WIDE && i == 2)
                            umma2_f16_ss<8>(d + e * 64, qd, kd, IDESC_QK, 1u, one);
                        else
                            umma2_f16_ss(d + e * 64, qd, kd, IDESC_QK, i ? 1u : 0u, one);
                    }
                umma2_commit(&bar.k_free[st], one);
                umma2_commit(&bar.s_ready[n & 1], one);
            };
            // O += P V for one unit of tile j, the upper or lower halves of P
            auto issue_pv = [&](int j, int u, int half, bool tail) {
                const int n = 4 * j + u, st = n % NV, kh = u & 1;
                if (half == 0) {
                    if (tail)
                        mbar_wait_warp(&bar.v_ok[st], 0, prm.status, 524, failed);
                    else
                        mbar_wait_warp(&bar.v_full[st], (n / NV) & 1, prm.status, 523, failed);
                }
                if (failed) return;
                tc_fence_after_sync();
                const uint64_t v = dv + (uint64_t)st * (V_UNIT >> 4), p = dp + half * (P_TILE >> 4) + kh * (P_HALF >> 4);
                const uint32_t d = tm + TMEM_O + dim_block(j, u) * 128;
#pragma unroll
                for (int kk = 0; kk < 4; kk++) umma2_f16_ss(d, p + 2 * kk, v + 128 * kk, IDESC_PV, (j > 0 || kh || half || kk) ? 1u : 0u, one);
                if (half) umma2_commit(&bar.v_free[st], one);
            };
            for (int g = 0; g < GROUPS; g++) issue_qk(0, g);
            for (int j = 0; j < tiles && !failed; ++j) {
                const bool tail = warp_uniform((int)((int64_t)j * TILE_K + TILE_K - 1 > valid_end)) != 0, more = j + 1 < tiles;
                // the next tile's scores go ahead of this tile's products, and between them
                int g = 0;
                for (; more && g < 2; g++) issue_qk(j + 1, g);
                mbar_wait_warp(&bar.p_ready, j & 1, prm.status, 525, failed);
                if (failed) break;
                for (int i = 0; i < 8; i++) {
                    if (i == 4 && settles(j)) mbar_wait_warp(&bar.settle_ok, settle_phase(j), prm.status, 526, failed);  // the other block has been settled
                    issue_pv(j, i >> 1, i & 1, tail);
                    if (i == 3) umma2_commit(&bar.first_done, one);
                    if (i == 7) umma2_commit(&bar.pv_done, one);
                    if (more && g < GROUPS) issue_qk(j + 1, g++);
                }
            }
        }
    } else {
        // ======================= softmax: thread = (row, 32 keys of a tile; 64 dims of each block of O) =======================
        // A row is in lane `row` (keys 0..63, dims 0..127 of a block) and lane 64 + row (the others) of tensor memory, each shared by two warps.
        const int quarter = warp & 3, half = warp >> 2, tl = quarter * 32 + lane, row = tl & 63, kh = tl >> 6;
        const int key0 = 64 * kh + 32 * half;  // of the tile
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        const uint32_t s_free[2] = {at_leader(&bar.s_free[0]), at_leader(&bar.s_free[1])}, p_ready = at_leader(&bar.p_ready);
        const int64_t last_key = min(first_qpos + row / G, rows0 - 1) - key0;  // minus the tile's first: the last of this thread's keys that the row sees
        const float scale2 = prm.scale * 1.4426950408889634f;  // > 0 (checked on the host)
        const size_t out_row = ((size_t)(m0 + row / G) * (prm.n_kv * G) + kvh * G + row % G) * HD;
        bool odd = false;  // a scale or a result that is not finite
#pragma unroll
        for (int b = 0; b < 16; b++) odd |= !(fabsf(sm.qs[b][row]) <= 256.0f * 65504.0f);
        float m_ref = NEG_SENTINEL;
        float2 l2[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
        auto o_at = [&](int h) { return lane_addr + TMEM_O + (h >> 2) * 128 + 64 * half + 16 * (h & 3); };
        for (int it = 0; it < n_tiles; ++it) {
            float2 s[16];
#pragma unroll
            for (int i = 0; i < 16; i++) s[i] = make_float2(0.0f, 0.0f);
            // Block by block: the sums of the next are on their way out of tensor memory while one's are scaled by the row's scale.
            uint32_t r[2][32];
            auto ready = [&](int g) {
                mbar_wait(&bar.s_ready[g & 1], ((it * GROUPS + g) >> 1) & 1, prm.status, 531, failed);
                tc_fence_after_sync();
            };
            auto at = [&](int n) { return lane_addr + TMEM_S + ((n >> 1) & 1) * S_COLS + (n & 1) * 64 + 32 * half; };
            ready(0);
            tmem_ld_32x32b_x32(at(0), r[0]);
            tc_wait_ld();
            loaded(r[0]);
#pragma unroll
            for (int n = 0; n < 2 * GROUPS; n++) {
                const int g = n >> 1;
                if (n & 1) {
                    if (g + 1 < GROUPS) ready(g + 1);
                }
                if (n + 1 < 2 * GROUPS) tmem_ld_32x32b_x32(at(n + 1), r[(n + 1) & 1]);
                const float q = sm.qs[n][row];
#pragma unroll
                for (int i = 0; i < 16; i++)
                    s[i] = __ffma2_rn(make_float2(__uint_as_float(r[n & 1][2 * i]), __uint_as_float(r[n & 1][2 * i + 1])), make_float2(q, q), s[i]);
                if (n + 1 < 2 * GROUPS) {
                    tc_wait_ld();
                    loaded(r[(n + 1) & 1]);
                }
                if ((n & 1) == 0) {  // both blocks of the hand-over are in registers
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_pair(s_free[g & 1]);  // one arrival per warp: they serialise on the barrier's word
                }
            }

            // masks only where the tile crosses the diagonal or the end of the cache
            const int64_t pos0 = (int64_t)it * TILE_K;
            if (pos0 + TILE_K - 1 > min(first_qpos, rows0 - 1)) {
                const int last = (int)max((int64_t)-1, min((int64_t)TILE_K, last_key - pos0));
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    if (2 * i > last) s[i].x = -INFINITY;
                    if (2 * i + 1 > last) s[i].y = -INFINITY;
                }
            }
            // does any score exceed its row's reference by more than 2^8?
            const float2 sc2 = make_float2(scale2, scale2);
            float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 16; i++) top[i & 3] = max3(top[i & 3], s[i].x, s[i].y);
            const float most = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) * scale2;
            const bool raise = named_barrier_or(1, SOFT_THREADS, most > m_ref + GROW_T);
            if (raise) {
                sm.red[2 * kh + half][row] = most;
                named_barrier_sync(2, SOFT_THREADS);
                const float mx = fmaxf(fmaxf(sm.red[0][row], sm.red[1][row]), fmaxf(sm.red[2][row], sm.red[3][row]));
                const float now = mx > m_ref + GROW_T ? mx : m_ref;
                const float corr = ex2(m_ref - now);
                m_ref = now;
#pragma unroll
                for (int i = 0; i < 2; i++) l2[i] = __fmul2_rn(l2[i], make_float2(corr, corr));
                if (it > 0) {
                    mbar_wait(&bar.pv_done, (it - 1) & 1, prm.status, 532, failed);
                    // whoever settled last, in this tile or in the one before; pv_done says that the settling ahead of it is over
                    if (it >= SETTLE_FROM) mbar_wait(&bar.settle_here, settle_phase(it), prm.status, 536, failed);
                    tc_fence_after_sync();
#pragma unroll 1
                    for (int h = 0; h < 8; h++) {
                        const bool in_parts = (settled_by(it) >> (h >> 2)) & 1;
                        uint32_t o[16];
                        uint4 u[2];
                        tmem_ld_32x32b_x16(o_at(h), o);
                        if (in_parts) fetch_settled(tid, h, u);
                        tc_wait_ld();
                        if (in_parts) add_settled(u, o);
#pragma unroll
                        for (int i = 0; i < 16; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                        if (in_parts) settle(tid, h, o);
                        tmem_st_32x32b_x16(o_at(h), o);
                    }
                    tc_wait_st();
                    __threadfence_block();  // the parts are read by the warps that settle
                }
            }
            // P = 2^(s * scale2 - m + 7) as f16 hi + lo; l from the unrounded values
            uint32_t hi[16], lo[16];
            {
                const float2 less = make_float2(EXP_BIAS - m_ref, EXP_BIAS - m_ref);
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float2 x = __ffma2_rn(s[i], sc2, less);
                    const float2 p = make_float2(ex2(x.x), ex2(x.y));
                    l2[i & 1] = __fadd2_rn(l2[i & 1], p);
                    hi[i] = pack_half2(p.x, p.y);
                    const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi[i]));
                    lo[i] = pack_half2(p.x - h.x, p.y - h.y);
                }
            }
            if (it > 0) mbar_wait(&bar.pv_done, (it - 1) & 1, prm.status, 533, failed);  // P of the last tile has been read
            {
                uint8_t* to = sm.p[0] + kh * P_HALF + row * 128;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint32_t off = ((4 * half + c) ^ (row & 7)) << 4;
                    *reinterpret_cast<uint4*>(to + off) = make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
                    *reinterpret_cast<uint4*>(to + P_TILE + off) = make_uint4(lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]);
                }
            }
            fence_proxy_async_smem();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_pair(p_ready);
                if (settles(it + 1)) mbar_arrive(&bar.parts_here);
            }
        }

        // ---- epilogue -----------------------------------------------
        named_barrier_sync(2, SOFT_THREADS);  // every thread is done with red
        sm.red[2 * kh + half][row] = (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y);
        named_barrier_sync(2, SOFT_THREADS);
        const float inv = 1.0f / ((sm.red[0][row] + sm.red[1][row]) + (sm.red[2][row] + sm.red[3][row]));
        mbar_wait(&bar.pv_done, (n_tiles - 1) & 1, prm.status, 534, failed);
        tc_fence_after_sync();
        const uint32_t settled = settled_by(n_tiles - 1);
        if (settled != 0) {  // whole again before the first result is written over a settled part
            mbar_wait(&bar.settle_here, settle_phase(n_tiles - 1), prm.status, 537, failed);
#pragma unroll 1
            for (int h = 0; h < 8; h++) {
                if (((settled >> (h >> 2)) & 1) == 0) continue;
                uint32_t o[16];
                uint4 u[2];
                tmem_ld_32x32b_x16(o_at(h), o);
                fetch_settled(tid, h, u);
                tc_wait_ld();
                add_settled(u, o);
                tmem_st_32x32b_x16(o_at(h), o);
            }
            tc_wait_st();
            named_barrier_sync(2, SOFT_THREADS);
        }
#pragma unroll 1
        for (int h = 0; h < 8; h++) {
            uint32_t o[16], w[8];
            tmem_ld_32x32b_x16(o_at(h), o);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float a = __uint_as_float(o[2 * i]) * inv, b = __uint_as_float(o[2 * i + 1]) * inv;
                odd |= !(fabsf(a) <= 3.4e38f) || !(fabsf(b) <= 3.4e38f);
                w[i] = pack_half2(a, b);
            }
            uint4* to = reinterpret_cast<uint4*>(prm.out + out_row + (h >> 2) * 256 + kh * 128 + 64 * half + 16 * (h & 3));
            to[0] = make_uint4(w[0], w[1], w[2], w[3]);
            to[1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
        if (odd) {
            atomicOr(&sm.redo[row / 32], 1u << (row % 32));
            if (!WIDE) store_both(&sm.odd, 1);
        }
    }
    // A wait that ran out leaves copies and MMAs of this CTA in flight that nobody will wait for: give them a bounded
    // time to land before the shared and tensor memory they target is handed to the next CTA.
    if (failed) {
        sm.abort = 1;
        store_both(&sm.gone, 1);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (*(volatile uint32_t*)&sm.abort != 0u) {
        let_copies_land();
        __syncthreads();
    }
    pair_sync();  // the pair's MMAs and arrivals reach into both CTAs
}

// Keys that overflowed made NaN of every row that sees them: where a pair has such rows and such keys, all of it again, with the other split.
// (Looked for afterwards: one maximum per scale in the key warps cost 0.7 %.  Not inlined, for the registers of the pass that
// every call takes.)
__device__ __noinline__ void again_if_large(const CUtensorMap& tm_v, const Int8Params& prm, Int8Smem& sm, uint32_t pair_m0, int kvh)
{
    constexpr int BLOCKS = HD / 32, STEP = INT8_THREADS / BLOCKS;  // scales of a key; keys of a CTA at a time
    const int64_t keys = min((int64_t)min(prm.k0.rows, prm.v0.rows), (int64_t)prm.step[STEP_Q0] + pair_m0 + PAIR_TOK);
    bool large = false;
    for (int64_t key = threadIdx.x / BLOCKS + pair_rank() * STEP; key < keys; key += 2 * STEP) {
        const float s = fabsf(__half2float(ld_global(prm.k0.scales + ((size_t)key * prm.n_kv + kvh) * BLOCKS + threadIdx.x % BLOCKS)));
        large |= s >= 65504.0f / 128.0f && s <= 65504.0f;
    }
    if (large) store_both(&sm.large, 1);
    pair_sync();
    if (*(volatile uint32_t*)&sm.large == 0u) return;
    if (threadIdx.x == 0) sm.redo[0] = sm.redo[1] = 0;
    int8_pass<true>(tm_v, prm, sm);
}

__global__ void __launch_bounds__(INT8_THREADS, 1)
    int8_prefill_kernel(const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ Int8Params prm)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Int8Smem& sm = *reinterpret_cast<Int8Smem*>(smem_raw);
    if ((smem_u32(smem_raw) & 1023u) != 0u) {  // the swizzled tiles need it; never seen, but never assumed (the same in both CTAs)
        if (threadIdx.x == 0) report_error(prm.status, DEV_ERR_BOUNDS, 500, smem_u32(smem_raw), 0);
        return;
    }
    const int tid = threadIdx.x, warp = warp_uniform(tid >> 5);
    pdl_wait();  // the step words, q, K and V come from earlier kernels of the stream
    pdl_launch_dependents();
    if (tid < 2) {
        Int8Barriers& bar = sm.bars[tid];
        for (int i = 0; i < NK; i++) {
            mbar_init(&bar.k_full[i], 2 * K_WARPS);
            mbar_init(&bar.k_free[i], 1);
        }
        for (int i = 0; i < NV; i++) {
            mbar_init(&bar.v_full[i], 1);
            mbar_init(&bar.v_free[i], 1);
            mbar_init(&bar.v_here[i], 1);
            mbar_init(&bar.v_ok[i], 2);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&bar.s_ready[i], 1);
            mbar_init(&bar.s_free[i], 2 * SOFT_WARPS);
        }
        mbar_init(&bar.p_ready, 2 * SOFT_WARPS);
        mbar_init(&bar.first_done, 1);
        mbar_init(&bar.parts_here, SOFT_WARPS);
        mbar_init(&bar.settle_here, K_WARPS);
        mbar_init(&bar.settle_ok, 2 * K_WARPS);
        mbar_init(&bar.pv_done, 1);
        mbar_fence_init();
    }
    if (tid == 0) {
        sm.abort = sm.gone = sm.large = sm.odd = 0;
        sm.redo[0] = sm.redo[1] = 0;
    }
    if (warp == 0) {
        tmem_alloc_pair(&sm.tmem_base, TMEM_COLS);
    }
    int8_pass<false>(tm_v, prm, sm);
    const int kvh = (blockIdx.x / 2) % prm.n_kv;
    const uint32_t pair_m0 = (prm.m_tokens / PAIR_TOK - 1 - blockIdx.x / 2 / prm.n_kv) * PAIR_TOK, m0 = pair_m0 + pair_rank() * (ROWS / G);
    const volatile uint32_t &gone = sm.gone, &odd = sm.odd;  // a pair agrees: stored in both CTAs ahead of the cluster barrier
    if (odd != 0u && gone == 0u) again_if_large(tm_v, prm, sm, pair_m0, kvh);
    if (warp == 0) tmem_dealloc_pair(sm.tmem_base, TMEM_COLS);
    if ((*(volatile uint32_t*)&sm.redo[0] | *(volatile uint32_t*)&sm.redo[1]) != 0) stream_rows(prm, sm, m0, kvh);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// V as [row][head][512] f16, boxes of 64 dims x one head x 64 rows.
int encode_v(const LaunchArgs& a, CUtensorMap* tm, const KvOperand& v, uint64_t heads)
{
    const uint64_t dims[3] = {HD, heads, v.rows};
    const uint64_t strides[2] = {HD * 2, heads * HD * 2};
    const uint32_t box[3] = {64, 1, 64};
    return encode_tensor_map(a, tm, 1, 3, const_cast<void*>(v.data), dims, strides, box, 3);
}

}  // namespace

// What the tensor-core kernel takes: a positive softmax scale (the row maximum is taken before it), operands whose rows the
// copies can address (16-byte aligned bases, K and V with at least one row, row indexes within an int), an output that can be
// settled into (16-byte accesses, whole query tiles).  What else the launcher accepts stays on the streaming kernel: quants on 4
// bytes, an output on 2.  Scales are read one by one.
bool prefill_int8_takes(const KvOperand& k, const KvOperand& v, const void* q, const void* out, uint32_t m, float scale)
{
    if (!(scale > 0.0f) || !(scale < 1e30f) || !aligned16(q) || !aligned16(out) || m % PAIR_TOK != 0) return false;
    for (const KvOperand* o : {&k, &v})
        if (o->rows == 0 || o->rows >= (1u << 30) || !aligned16(o->data)) return false;
    return true;
}

int launch_prefill_int8(const LaunchArgs& a, const void* q, const __half* q_scales, const KvOperand& k, const KvOperand& v, void* out, const void* step,
                        uint32_t n_kv, uint32_t m, float scale)
{
    const Int8Params prm{(const uint32_t*)step, (__half*)out, a.status, q_scales, m, n_kv, scale, q, k, v};
    CUtensorMap tv;
    if (int r = encode_v(a, &tv, v, n_kv)) return r;
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
    const cudaError_t err = launch_dependent_clusters(int8_prefill_kernel, 2, dim3(2 * (m / PAIR_TOK) * n_kv), dim3(INT8_THREADS), sizeof(Int8Smem), a.stream,
                                                      tv, prm);
    ++*a.launches;
    return check_cuda(a, err, "attn_prefill_global_flash_sp_iq");
}

}  // namespace sgb
