// Scalar (CUDA-core) attention kernels: the statement of every reference-shaped registry name, for what the tensor-core kernels
// do not take, and the launchers that choose between the two.  They follow the reference's streaming-softmax statement per key
// (attn_decode_sliding.wgsl:84-107 and its siblings) with f32 math, one warp per key and the four
// warps of a block merged in a fixed order, so reruns are bit-identical.
#include "attn_merge.cuh"
#include "attn_stream.cuh"
#include "sgb_common.cuh"
#include "sgb_kernels.h"

namespace sgb {

namespace {

constexpr int GEN_THREADS = 128;
constexpr int GEN_WARPS = GEN_THREADS / 32;

// Merge the four warps' streaming states in warp order 0,1,2,3 through shared memory, leaving the
// result in warp 0's registers.  sm_acc holds G*HD floats, sm_ml holds 2*G floats.
template <int HD, int G, int DPL>
__device__ __forceinline__ void merge_warps(Stream<G, DPL>& st, float* sm_acc, float* sm_ml, int warp, int lane, int d0)
{
    for (int w = 1; w < GEN_WARPS; w++) {
        __syncthreads();
        if (warp == w) {
#pragma unroll
            for (int g = 0; g < G; g++) {
#pragma unroll
                for (int d = 0; d < DPL; d++) sm_acc[g * HD + d0 + d] = st.acc[g][d];
                if (lane == 0) {
                    sm_ml[2 * g] = st.m[g];
                    sm_ml[2 * g + 1] = st.l[g];
                }
            }
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int g = 0; g < G; g++) {
                const float ms = sm_ml[2 * g], ls = sm_ml[2 * g + 1];
                const float m_new = fmaxf(st.m[g], ms);
                const float ca = __expf(st.m[g] - m_new), cb = __expf(ms - m_new);
#pragma unroll
                for (int d = 0; d < DPL; d++) st.acc[g][d] = st.acc[g][d] * ca + sm_acc[g * HD + d0 + d] * cb;
                st.l[g] = st.l[g] * ca + ls * cb;
                st.m[g] = m_new;
            }
        }
    }
}

// Split-K decode partials.  Grid (kv head, split, query token); the reference's grid is the first
// two (attn_decode_sliding.wgsl:53-62).  part row = i * H + qh.
template <int HD, int G, int KFMT, int VFMT>
__global__ void __launch_bounds__(GEN_THREADS) decode_generic_kernel(const __half* q, KvOperand kop, KvOperand vop,
                                                                     float* __restrict__ part,
                                                                     const uint32_t* step, int step_slot,
                                                                     uint32_t n_splits, float scale, uint32_t* status)
{
    constexpr int DPL = HD / 32;
    __shared__ float sm_acc[G * HD];
    __shared__ float sm_ml[2 * G];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kvh = blockIdx.x, n_kv = gridDim.x, split = blockIdx.y;
    const uint32_t i = blockIdx.z, m_q = gridDim.z;
    const int n_q = n_kv * G;
    const int d0 = lane * DPL;

    const uint32_t kv_len = step[step_slot];
    const uint32_t chunk = (kv_len + n_splits - 1) / n_splits;
    const uint32_t t_begin = min((uint32_t)split * chunk, kv_len);
    uint32_t t_end = min(t_begin + chunk, kv_len);
    // query i of m_q sees keys t <= kv_len - m_q + i  (m_q = 1: every key)
    const uint32_t vis_end = kv_len + i >= m_q ? kv_len + i - m_q + 1 : 0;
    t_end = min(t_end, vis_end);

    float qr[G][DPL];
#pragma unroll
    for (int g = 0; g < G; g++) load_f16<DPL>(q + ((size_t)i * n_q + kvh * G + g) * HD + d0, qr[g]);

    Stream<G, DPL> st;
    st.init();
    for (uint32_t t = t_begin + warp; t < t_end; t += GEN_WARPS) {
        size_t krow, vrow;
        if (!resolve_row(kop, t, krow, status, 201) || !resolve_row(vop, t, vrow, status, 203)) break;
        float kk[DPL], vv[DPL];
        load_row<HD, KFMT, DPL>(kop, krow, kvh, n_kv, d0, kk);
        load_row<HD, VFMT, DPL>(vop, vrow, kvh, n_kv, d0, vv);
#pragma unroll
        for (int g = 0; g < G; g++) st.step(g, qr[g], kk, vv, scale);
    }
    merge_warps<HD, G, DPL>(st, sm_acc, sm_ml, warp, lane, d0);
    if (warp == 0) {
#pragma unroll
        for (int g = 0; g < G; g++) {
            float* row = part + (((size_t)i * n_q + kvh * G + g) * n_splits + split) * (HD + 2);
#pragma unroll
            for (int d = 0; d < DPL; d++) row[d0 + d] = st.acc[g][d];
            if (lane == 0) {
                row[HD] = st.m[g];
                row[HD + 1] = st.l[g];
            }
        }
    }
}

// Split-K combine (attn_reduce.wgsl:29-56): the splits of a row in ascending order with a running
// maximum, the reference's own op order (merge_splits_running).  Grid = rows, HD / 2 threads, two dims each.
// OUT_MODE 0: f16(acc/l) (the reference), 1: f32 acc/l, 2: merged (acc, m, l) as f32[HD+2].
// split_major = 0: part[(row*n + s)*(HD+2)]; 1: part[(s*rows + row)*(HD+2)] (per-rank blocks).
constexpr int REDUCE_MAX_SPLITS = 1024;

template <int HD, int OUT_MODE>
__global__ void __launch_bounds__(HD / 2) reduce_kernel(const float* part, void* __restrict__ out, uint32_t n_splits,
                                                       int split_major)
{
    const size_t row = blockIdx.x, rows = gridDim.x;
    const int d0 = 2 * threadIdx.x;
    pdl_wait();  // the partials come from the kernel before this one
    pdl_launch_dependents();
    const size_t s_stride = split_major ? rows * (HD + 2) : (size_t)(HD + 2);
    const float* base = part + (split_major ? row : row * n_splits) * (HD + 2);
    float acc[2];
    const MergeState st = merge_splits_running<HD, 2, 3>(base, s_stride, n_splits, d0, acc);  // up to 96 splits in one latency
    if constexpr (OUT_MODE == 2) {
        float* o = reinterpret_cast<float*>(out) + row * (HD + 2);
        *reinterpret_cast<float2*>(o + d0) = make_float2(acc[0], acc[1]);
        if (threadIdx.x == 0) *reinterpret_cast<float2*>(o + HD) = make_float2(st.m, st.l);
    } else if constexpr (OUT_MODE == 0) {
        reinterpret_cast<__half2*>(out)[(row * HD + d0) / 2] = __floats2half2_rn(acc[0] / st.l, acc[1] / st.l);
    } else {
        *reinterpret_cast<float2*>(reinterpret_cast<float*>(out) + row * HD + d0) = make_float2(acc[0] / st.l, acc[1] / st.l);
    }
}

// Streaming prefill.  Grid (kv head, query token).  TWO_RANGE: history [t_begin, min(q0, qpos+1))
// from `hist` at row t % ring, then chunk rows [max(q0, t_begin) - q0, i] from `chunk`
// (attn_prefill_sliding_ring.wgsl:88-140); otherwise one linear range [t_begin, qpos] from `hist`
// (attn_prefill_sliding.wgsl:53-57,78 / attn_prefill_global.wgsl:53,74).  window 0 = none.
// QFMT = FMT_Q8: q holds int8 quants [M x H x HD] with f16 scales q_scales [M x H x HD/32]
// (attn_prefill_global_flash_sp_iq.wgsl:24-25).
template <int HD, int G, int KFMT, int VFMT, int TWO_RANGE, int OUT_F32, int QFMT = FMT_F16>
__global__ void __launch_bounds__(GEN_THREADS) prefill_generic_kernel(const void* q, const __half* q_scales,
                                                                      KvOperand k_hist, KvOperand v_hist, KvOperand k_chunk,
                                                                      KvOperand v_chunk, void* __restrict__ out,
                                                                      const uint32_t* step, uint32_t window,
                                                                      uint32_t ring, float scale, uint32_t* status)
{
    constexpr int DPL = HD / 32;
    __shared__ float sm_acc[G * HD];
    __shared__ float sm_ml[2 * G];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kvh = blockIdx.x, n_kv = gridDim.x;
    const uint32_t i = blockIdx.y;
    const int n_q = n_kv * G;
    const int d0 = lane * DPL;
    const uint32_t q0 = step[STEP_Q0];
    const uint32_t qpos = q0 + i;
    const uint32_t t_begin = (window != 0 && qpos + 1 > window) ? qpos + 1 - window : 0;

    float qr[G][DPL];
#pragma unroll
    for (int g = 0; g < G; g++) {
        const size_t qrow = (size_t)i * n_q + kvh * G + g;
        if constexpr (QFMT == FMT_F16)
            load_f16<DPL>(reinterpret_cast<const __half*>(q) + qrow * HD + d0, qr[g]);
        else
            load_q8<DPL>(reinterpret_cast<const int8_t*>(q) + qrow * HD + d0, q_scales + qrow * (HD / 32), d0, qr[g]);
    }

    Stream<G, DPL> st;
    st.init();
    const uint32_t hist_end = TWO_RANGE ? min(q0, qpos + 1) : qpos + 1;
    for (uint32_t t = t_begin + warp; t < hist_end; t += GEN_WARPS) {
        const size_t lt = ring ? t % ring : t;
        size_t krow, vrow;
        if (!resolve_row(k_hist, lt, krow, status, 211) || !resolve_row(v_hist, lt, vrow, status, 213)) break;
        float kk[DPL], vv[DPL];
        load_row<HD, KFMT, DPL>(k_hist, krow, kvh, n_kv, d0, kk);
        load_row<HD, VFMT, DPL>(v_hist, vrow, kvh, n_kv, d0, vv);
#pragma unroll
        for (int g = 0; g < G; g++) st.step(g, qr[g], kk, vv, scale);
    }
    if (TWO_RANGE) {
        const uint32_t c_begin = t_begin > q0 ? t_begin - q0 : 0;
        for (uint32_t c = c_begin + warp; c <= i; c += GEN_WARPS) {
            size_t krow, vrow;
            if (!resolve_row(k_chunk, c, krow, status, 215) || !resolve_row(v_chunk, c, vrow, status, 217)) break;
            float kk[DPL], vv[DPL];
            load_row<HD, FMT_F16, DPL>(k_chunk, krow, kvh, n_kv, d0, kk);
            load_row<HD, FMT_F16, DPL>(v_chunk, vrow, kvh, n_kv, d0, vv);
#pragma unroll
            for (int g = 0; g < G; g++) st.step(g, qr[g], kk, vv, scale);
        }
    }
    merge_warps<HD, G, DPL>(st, sm_acc, sm_ml, warp, lane, d0);
    if (warp == 0) {
#pragma unroll
        for (int g = 0; g < G; g++) {
            const size_t o = ((size_t)i * n_q + kvh * G + g) * HD + d0;
#pragma unroll
            for (int d = 0; d < DPL; d++) {
                const float y = st.acc[g][d] / st.l[g];
                if (OUT_F32)
                    reinterpret_cast<float*>(out)[o + d] = y;
                else
                    reinterpret_cast<__half*>(out)[o + d] = __float2half_rn(y);
            }
        }
    }
}

struct PushSplitScale {
    uint32_t n_splits;
    float scale;
};

}  // namespace

// attn_decode_sliding / attn_decode_global / attn_decode_global_q8k and their d128 forms.
// bindings: q, k [, k_scales], v, part, step.  push {n_splits, scale}.  grid [n_kv, n_splits, m_q or 1].
template <int HD, int G, int KFMT, int VFMT, int STEP_SLOT>
int launch_decode_generic(const LaunchArgs& a)
{
    const PushSplitScale p = *(const PushSplitScale*)a.push;
    const int n_kv = (int)a.groups[0];
    const uint32_t m_q = a.groups[2] ? a.groups[2] : 1;
    if (n_kv <= 0 || p.n_splits == 0) return fail_validation(a, "decode: groups[0] (kv heads) and n_splits must be > 0");
    if (a.groups[1] != p.n_splits) return fail_validation(a, "decode: groups[1] must equal push.n_splits");
    int bi = 0;
    const BufView& q = a.b[bi++];
    KvOperand kop, vop;
    if (KFMT == FMT_Q8) {
        kop = linear_q8(a.b[bi], a.b[bi + 1], n_kv, HD);
        if (a.b[bi + 1].bytes / 2 < kop.rows * n_kv * (HD / 32)) return fail_validation(a, "decode: k_scales too short");
        bi += 2;
    } else {
        kop = linear_f16(a.b[bi++], n_kv, HD);
    }
    if (VFMT == FMT_Q8) {
        vop = linear_q8(a.b[bi], a.b[bi + 1], n_kv, HD);
        if (a.b[bi + 1].bytes / 2 < vop.rows * n_kv * (HD / 32)) return fail_validation(a, "decode: v_scales too short");
        bi += 2;
    } else {
        vop = linear_f16(a.b[bi++], n_kv, HD);
    }
    const int part_i = bi++, step_i = bi++;
    const size_t n_q = (size_t)n_kv * G;
    if (q.bytes < m_q * n_q * HD * 2) return fail_validation(a, "decode: q buffer too small");
    if (int r = need_bytes(a, part_i, m_q * n_q * p.n_splits * (HD + 2) * 4, "part")) return r;
    if (int r = need_bytes(a, step_i, 16, "step")) return r;
    static_assert(VFMT == FMT_F16, "the lists below name no V scales");
    constexpr uint32_t ROW = row_alignment(HD);
    if (int r = KFMT == FMT_Q8 ? need_aligned(a, {ROW, 4, 2, ROW, 4, 4}) : need_aligned(a, {ROW, ROW, ROW, 4, 4})) return r;
    // The tiled kernel pays its set-up for each of the many CTAs that many splits make (us, streaming | tiled, 1024 cached tokens: head_dim
    // 256, 16 splits 9.9 | 5.4, 32 splits 7.1 | 7.5, 256 splits 11 | 34; head_dim 128, 32 splits 6.4 | 4.1, 64 splits 5.0 | 6.3;
    // head_dim 512, 64 splits 19 | 16, 128 splits 28 | 32; 4096 tokens, 256 splits 66 | 55).  The length is on the device, the rows are known.
    constexpr size_t ROWS_PER_SPLIT = HD == 256 ? 64 : HD == 128 ? 32 : 16;
    if (min(kop.rows, vop.rows) >= ROWS_PER_SPLIT * p.n_splits && decode_rows_takes(kop, vop, q.ptr))
        return launch_decode_rows<HD, G, KFMT == FMT_Q8>(a, q.ptr, kop, vop, a.b[part_i].ptr, a.b[step_i].ptr, STEP_SLOT, n_kv, p.n_splits, m_q, p.scale);
    decode_generic_kernel<HD, G, KFMT, VFMT><<<dim3(n_kv, p.n_splits, m_q), GEN_THREADS, 0, a.stream>>>(
        (const __half*)q.ptr, kop, vop, (float*)a.b[part_i].ptr, (const uint32_t*)a.b[step_i].ptr, STEP_SLOT, p.n_splits,
        p.scale, a.status);
    ++*a.launches;
    return check_cuda(a, cudaGetLastError(), "attn_decode");
}
template int launch_decode_generic<256, 2, FMT_F16, FMT_F16, STEP_KV_LEN_SLIDING>(const LaunchArgs&);
template int launch_decode_generic<512, 8, FMT_F16, FMT_F16, STEP_KV_LEN_GLOBAL>(const LaunchArgs&);
template int launch_decode_generic<512, 8, FMT_Q8, FMT_F16, STEP_KV_LEN_GLOBAL>(const LaunchArgs&);
template int launch_decode_generic<128, 2, FMT_F16, FMT_F16, STEP_KV_LEN_SLIDING>(const LaunchArgs&);

struct PushDecodePaged {
    uint32_t n_splits;
    float scale;
    uint32_t page;
};

// The scalar statement of the paged Q8_0 decode (same bindings and push as the fast kernel):
// q, k_quants, k_scales, v_quants, v_scales, page_table, part, step.  push {n_splits, scale, page}.
int launch_decode_paged_q8kv_scalar_d128(const LaunchArgs& a)
{
    const PushDecodePaged p = *(const PushDecodePaged*)a.push;
    const int n_kv = (int)a.groups[0];
    const uint32_t m_q = a.groups[2] ? a.groups[2] : 1;
    if (n_kv <= 0 || p.n_splits == 0 || p.page == 0)
        return fail_validation(a, "decode_paged: kv heads, n_splits and page must be > 0");
    if (a.groups[1] != p.n_splits) return fail_validation(a, "decode_paged: groups[1] must equal push.n_splits");
    KvOperand kop = linear_q8(a.b[1], a.b[2], n_kv, 128), vop = linear_q8(a.b[3], a.b[4], n_kv, 128);
    if (a.b[2].bytes / 2 < kop.rows * n_kv * 4 || a.b[4].bytes / 2 < vop.rows * n_kv * 4)
        return fail_validation(a, "decode_paged: scales buffer too short for its quants buffer");
    kop.page_table = vop.page_table = (const uint32_t*)a.b[5].ptr;
    kop.table_len = vop.table_len = (uint32_t)(a.b[5].bytes / 4);
    kop.page = vop.page = p.page;
    const size_t n_q = (size_t)n_kv * 2;
    if (a.b[0].bytes < m_q * n_q * 128 * 2) return fail_validation(a, "decode_paged: q buffer too small");
    if (int r = need_bytes(a, 6, m_q * n_q * p.n_splits * 130 * 4, "part")) return r;
    if (int r = need_bytes(a, 7, 16, "step")) return r;
    if (int r = need_aligned(a, {row_alignment(128), 4, 2, 4, 2, 4, 4, 4})) return r;
    decode_generic_kernel<128, 2, FMT_Q8, FMT_Q8><<<dim3(n_kv, p.n_splits, m_q), GEN_THREADS, 0, a.stream>>>(
        (const __half*)a.b[0].ptr, kop, vop, (float*)a.b[6].ptr, (const uint32_t*)a.b[7].ptr, STEP_KV_LEN_GLOBAL, p.n_splits,
        p.scale, a.status);
    ++*a.launches;
    return check_cuda(a, cudaGetLastError(), "attn_decode_paged_q8kv_scalar_d128");
}

// attn_reduce_*: bindings part, out.  push {n_splits}.  grid [rows] (32 q heads in the reference).
template <int HD, int OUT_MODE>
int launch_reduce(const LaunchArgs& a)
{
    const uint32_t n_splits = *(const uint32_t*)a.push;
    const size_t rows = a.groups[0];
    if (rows == 0 || n_splits == 0 || n_splits > (uint32_t)REDUCE_MAX_SPLITS)
        return fail_validation(a, "attn_reduce: groups[0] (rows) must be > 0 and n_splits in 1..1024");
    if (int r = need_bytes(a, 0, rows * n_splits * (HD + 2) * 4, "part")) return r;
    const size_t out_bytes = OUT_MODE == 0 ? rows * HD * 2 : OUT_MODE == 1 ? rows * HD * 4 : rows * (HD + 2) * 4;
    if (int r = need_bytes(a, 1, out_bytes, "out")) return r;
    if (int r = need_aligned(a, {8, OUT_MODE == 0 ? 4u : 8u})) return r;
    const cudaError_t e = launch_dependent(reduce_kernel<HD, OUT_MODE>, dim3((uint32_t)rows), dim3(HD / 2), 0, a.stream, (const float*)a.b[0].ptr,
                                           a.b[1].ptr, n_splits, 0);
    ++*a.launches;
    return check_cuda(a, e, "attn_reduce");
}
template int launch_reduce<256, 0>(const LaunchArgs&);
template int launch_reduce<512, 0>(const LaunchArgs&);
template int launch_reduce<128, 0>(const LaunchArgs&);
template int launch_reduce<128, 1>(const LaunchArgs&);
template int launch_reduce<128, 2>(const LaunchArgs&);

// attn_combine_ranks_d128: bindings gathered [n_ranks][rows][130] f32, out f32 [rows][128].
// push {n_ranks}.  grid [rows].  Ranks are merged in rank order, so every rank computes the same bits.
int launch_combine_ranks_d128(const LaunchArgs& a)
{
    const uint32_t n_ranks = *(const uint32_t*)a.push;
    const size_t rows = a.groups[0];
    if (rows == 0 || n_ranks == 0 || n_ranks > (uint32_t)REDUCE_MAX_SPLITS)
        return fail_validation(a, "attn_combine_ranks: rows must be > 0 and n_ranks in 1..1024");
    if (int r = need_bytes(a, 0, rows * n_ranks * 130 * 4, "gathered partials")) return r;
    if (int r = need_bytes(a, 1, rows * 128 * 4, "out")) return r;
    if (int r = need_aligned(a, {8, 8})) return r;
    reduce_kernel<128, 1><<<(uint32_t)rows, 64, 0, a.stream>>>((const float*)a.b[0].ptr, a.b[1].ptr, n_ranks, 1);
    ++*a.launches;
    return check_cuda(a, cudaGetLastError(), "attn_combine_ranks_d128");
}

// attn_prefill_sliding / _sliding_ring / _global and the d128 f32-output forms.
// TWO_RANGE: bindings q, k_ring, v_ring, k_chunk, v_chunk, out, step; else q, k, v, out, step.
// push {scale}.  grid [n_kv, M].
template <int HD, int G, int WINDOW, int RING, int TWO_RANGE, int OUT_F32>
int launch_prefill_generic(const LaunchArgs& a)
{
    const float scale = *(const float*)a.push;
    const int n_kv = (int)a.groups[0];
    const size_t m = a.groups[1];
    if (n_kv <= 0 || m == 0) return fail_validation(a, "attn_prefill: groups must be [kv heads, query tokens]");
    const size_t n_q = (size_t)n_kv * G;
    KvOperand kh = linear_f16(a.b[1], n_kv, HD), vh = linear_f16(a.b[2], n_kv, HD), kc{}, vc{};
    int bi = 3;
    if (TWO_RANGE) {
        kc = linear_f16(a.b[3], n_kv, HD);
        vc = linear_f16(a.b[4], n_kv, HD);
        bi = 5;
        if (kh.rows < (size_t)RING || vh.rows < (size_t)RING) return fail_validation(a, "attn_prefill: ring buffers too small");
        if (kc.rows < m || vc.rows < m) return fail_validation(a, "attn_prefill: chunk K/V hold fewer than M rows");
    }
    if (a.b[0].bytes < m * n_q * HD * 2) return fail_validation(a, "attn_prefill: q buffer too small");
    if (int r = need_bytes(a, bi, m * n_q * HD * (OUT_F32 ? 4 : 2), "out")) return r;
    if (int r = need_bytes(a, bi + 1, 16, "step")) return r;
    constexpr uint32_t ROW = row_alignment(HD), OUT = OUT_F32 ? 4 : 2;
    if (int r = TWO_RANGE ? need_aligned(a, {ROW, ROW, ROW, ROW, ROW, OUT, 4}) : need_aligned(a, {ROW, ROW, ROW, OUT, 4})) return r;
    if constexpr (HD == 128 && TWO_RANGE) {
        // up to four queries are the eight rows of one MMA column; more queries are the streaming kernel's (or the flash kernel's)
        if (m <= 4 && decode_rows_takes(kh, vh, a.b[0].ptr) && decode_rows_takes(kc, vc, a.b[0].ptr))
            return launch_verify_ring_d128(a, a.b[0].ptr, kh, vh, kc, vc, a.b[bi].ptr, a.b[bi + 1].ptr, n_kv, (uint32_t)m, WINDOW, RING, scale);
    }
    if constexpr (HD == 256 && !OUT_F32) {
        if (prefill_wide_takes<TWO_RANGE != 0>(kh, vh, kc, vc, a.b[0].ptr, a.b[bi].ptr, scale))
            return launch_prefill_wide<TWO_RANGE != 0>(a, a.b[0].ptr, kh, vh, kc, vc, a.b[bi].ptr, a.b[bi + 1].ptr, n_kv, (uint32_t)m, WINDOW, RING,
                                                       scale);
    }
    prefill_generic_kernel<HD, G, FMT_F16, FMT_F16, TWO_RANGE, OUT_F32><<<dim3(n_kv, (uint32_t)m), GEN_THREADS, 0, a.stream>>>(
        a.b[0].ptr, nullptr, kh, vh, kc, vc, a.b[bi].ptr, (const uint32_t*)a.b[bi + 1].ptr, WINDOW, RING, scale,
        a.status);
    ++*a.launches;
    return check_cuda(a, cudaGetLastError(), "attn_prefill");
}
template int launch_prefill_generic<256, 2, 1024, 0, 0, 0>(const LaunchArgs&);     // attn_prefill_sliding
template int launch_prefill_generic<256, 2, 1024, 1024, 1, 0>(const LaunchArgs&);  // attn_prefill_sliding_ring
template int launch_prefill_generic<512, 8, 0, 0, 0, 0>(const LaunchArgs&);        // attn_prefill_global
template int launch_prefill_generic<128, 2, 1024, 0, 0, 1>(const LaunchArgs&);     // attn_prefill_sliding_f32_d128
template int launch_prefill_generic<128, 2, 1024, 1024, 1, 1>(const LaunchArgs&);  // attn_prefill_sliding_ring_f32_d128
template int launch_prefill_generic<128, 2, 0, 0, 0, 1>(const LaunchArgs&);        // attn_prefill_global_f32_d128

struct PushScalePage {
    float scale;
    uint32_t page;
};

// Scalar statement of the paged Q8_0 prefill: q, k_quants, k_scales, v_quants, v_scales,
// page_table, out f32, step.  push {scale, page}.  grid [n_kv, M].  Global causal.
int launch_prefill_paged_q8kv_scalar_d128(const LaunchArgs& a)
{
    const PushScalePage p = *(const PushScalePage*)a.push;
    const int n_kv = (int)a.groups[0];
    const size_t m = a.groups[1];
    if (n_kv <= 0 || m == 0 || p.page == 0) return fail_validation(a, "prefill_paged: kv heads, M and page must be > 0");
    KvOperand kop = linear_q8(a.b[1], a.b[2], n_kv, 128), vop = linear_q8(a.b[3], a.b[4], n_kv, 128);
    if (a.b[2].bytes / 2 < kop.rows * n_kv * 4 || a.b[4].bytes / 2 < vop.rows * n_kv * 4)
        return fail_validation(a, "prefill_paged: scales buffer too short for its quants buffer");
    kop.page_table = vop.page_table = (const uint32_t*)a.b[5].ptr;
    kop.table_len = vop.table_len = (uint32_t)(a.b[5].bytes / 4);
    kop.page = vop.page = p.page;
    const size_t n_q = (size_t)n_kv * 2;
    if (a.b[0].bytes < m * n_q * 128 * 2) return fail_validation(a, "prefill_paged: q buffer too small");
    if (int r = need_bytes(a, 6, m * n_q * 128 * 4, "out")) return r;
    if (int r = need_bytes(a, 7, 16, "step")) return r;
    if (int r = need_aligned(a, {row_alignment(128), 4, 2, 4, 2, 4, 4, 4})) return r;
    KvOperand none{};
    prefill_generic_kernel<128, 2, FMT_Q8, FMT_Q8, 0, 1><<<dim3(n_kv, (uint32_t)m), GEN_THREADS, 0, a.stream>>>(
        a.b[0].ptr, nullptr, kop, vop, none, none, a.b[6].ptr, (const uint32_t*)a.b[7].ptr, 0, 0, p.scale, a.status);
    ++*a.launches;
    return check_cuda(a, cudaGetLastError(), "attn_prefill_paged_q8kv_scalar_d128");
}

// The reference's tiled global-prefill names (crates/sg-gpu/build.rs:2207-2287), all hd 512 / 4 kv heads /
// 8 query heads per kv head, out f16, push {scale}, grid [32 query heads, M / 16] (one workgroup per query
// head and 16-row tile, attn_prefill_global_flash_sp.wgsl:68-75).  They differ in what they bind:
//   VARIANT 0  attn_prefill_global_flash, attn_prefill_global_flash_sp: q f16, k f16, v f16, out, step
//   VARIANT 1  attn_prefill_global_flash_sp_q8: q f16, k_quants, k_scales, v_quants, v_scales, out, step
//   VARIANT 2  attn_prefill_global_flash_sp_iq: q_i8, q_scales, k_quants, k_scales, v f16, out, step
// The first two are the streaming kernel's, on the dequantised values (the reference's own test compares the int8 kernel with
// attention over the dequantised Q and K, tests/parity_attn.rs:689-768); the third, the one the reference's graph
// dispatches, is int8_prefill_kernel's where that takes the call.  K/V need not be padded to a 64-key tile as the
// reference's callers do: rows past the last visible key do not count.
template <int VARIANT>
int launch_prefill_global_flash_ref(const LaunchArgs& a)
{
    constexpr int HD = 512, G = 8, N_KV = 4, M_Q = 16;
    const float scale = *(const float*)a.push;
    if (a.groups[0] != (uint32_t)(N_KV * G) || a.groups[1] == 0)
        return fail_validation(a, "attn_prefill_global_flash*: groups must be [32 query heads, M / 16]");
    const size_t m = (size_t)a.groups[1] * M_Q, n_q = (size_t)N_KV * G;
    KvOperand kop, vop, none{};
    const __half* q_scales = nullptr;
    int bi = 1;
    if (VARIANT == 2) {
        if (a.b[0].bytes < m * n_q * HD || a.b[1].bytes < m * n_q * (HD / 32) * 2)
            return fail_validation(a, "attn_prefill_global_flash_sp_iq: q_i8 / q_scales too small for M rows");
        q_scales = (const __half*)a.b[1].ptr;
        bi = 2;
    } else if (a.b[0].bytes < m * n_q * HD * 2) {
        return fail_validation(a, "attn_prefill_global_flash*: q buffer too small");
    }
    if (VARIANT == 0) {
        kop = linear_f16(a.b[bi], N_KV, HD);
        vop = linear_f16(a.b[bi + 1], N_KV, HD);
        bi += 2;
    } else {
        kop = linear_q8(a.b[bi], a.b[bi + 1], N_KV, HD);
        if (a.b[bi + 1].bytes / 2 < kop.rows * N_KV * (HD / 32)) return fail_validation(a, "attn_prefill_global_flash*: k_scales too short");
        bi += 2;
        if (VARIANT == 1) {
            vop = linear_q8(a.b[bi], a.b[bi + 1], N_KV, HD);
            if (a.b[bi + 1].bytes / 2 < vop.rows * N_KV * (HD / 32)) return fail_validation(a, "attn_prefill_global_flash*: v_scales too short");
            bi += 2;
        } else {
            vop = linear_f16(a.b[bi++], N_KV, HD);
        }
    }
    if (int r = need_bytes(a, bi, m * n_q * HD * 2, "out")) return r;
    if (int r = need_bytes(a, bi + 1, 16, "step")) return r;
    if (int r = VARIANT == 0   ? need_aligned(a, {16, 16, 16, 2, 4})
                : VARIANT == 1 ? need_aligned(a, {16, 4, 2, 4, 2, 2, 4})
                               : need_aligned(a, {4, 2, 4, 2, 16, 2, 4}))
        return r;
    if constexpr (VARIANT == 2) {
        if (prefill_int8_takes(kop, vop, a.b[0].ptr, a.b[bi].ptr, (uint32_t)m, scale))
            return launch_prefill_int8(a, a.b[0].ptr, q_scales, kop, vop, a.b[bi].ptr, a.b[bi + 1].ptr, N_KV, (uint32_t)m, scale);
    }
    const dim3 grid(N_KV, (uint32_t)m);
    void* out = a.b[bi].ptr;
    const uint32_t* step = (const uint32_t*)a.b[bi + 1].ptr;
    if (VARIANT == 0)
        prefill_generic_kernel<HD, G, FMT_F16, FMT_F16, 0, 0><<<grid, GEN_THREADS, 0, a.stream>>>(a.b[0].ptr, nullptr, kop, vop, none, none, out,
                                                                                               step, 0, 0, scale, a.status);
    else if (VARIANT == 1)
        prefill_generic_kernel<HD, G, FMT_Q8_F16, FMT_Q8_F16, 0, 0><<<grid, GEN_THREADS, 0, a.stream>>>(a.b[0].ptr, nullptr, kop, vop, none, none,
                                                                                                     out, step, 0, 0, scale, a.status);
    else
        prefill_generic_kernel<HD, G, FMT_Q8, FMT_F16, 0, 0, FMT_Q8><<<grid, GEN_THREADS, 0, a.stream>>>(a.b[0].ptr, q_scales, kop, vop, none,
                                                                                                      none, out, step, 0, 0, scale, a.status);
    ++*a.launches;
    return check_cuda(a, cudaGetLastError(), "attn_prefill_global_flash*");
}
template int launch_prefill_global_flash_ref<0>(const LaunchArgs&);
template int launch_prefill_global_flash_ref<1>(const LaunchArgs&);
template int launch_prefill_global_flash_ref<2>(const LaunchArgs&);

}  // namespace sgb
