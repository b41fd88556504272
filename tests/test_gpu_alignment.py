"""Adopted pointers carry no alignment of their own.  A binding that a kernel's accesses could not be aligned with is refused on the
host, before any launch; one that is aligned well enough, but not for the tensor-core kernels' copies, gives the streaming
kernel's result."""
import numpy as np
import pytest

from cases import assert_close, bind, normal_f16
from oracle import sg_oracle as O

pytestmark = pytest.mark.gpu

# name, push, groups, bytes of each binding, alignment asked of each binding
DEC = lambda hd, h, kv: [h * hd * 2, 64 * kv * hd * 2, 64 * kv * hd * 2, h * 2 * (hd + 2) * 4, 16]
PRE = lambda hd, h, kv, o: [16 * h * hd * 2, 64 * kv * hd * 2, 64 * kv * hd * 2, 16 * h * hd * o, 16]
RING = lambda hd, h, kv, o: [4 * h * hd * 2] + [1024 * kv * hd * 2] * 2 + [4 * kv * hd * 2] * 2 + [4 * h * hd * o, 16]
ROW = 2 * 128  # two kv heads
POOL = [64 * ROW, 64 * ROW // 16]  # quants, scales
CASES = [
    ("attn_decode_sliding", (2, 0.1), [2, 2, 1], DEC(256, 4, 2), [16, 16, 16, 4, 4]),
    ("attn_decode_global", (2, 0.1), [2, 2, 1], DEC(512, 16, 2), [16, 16, 16, 4, 4]),
    ("attn_decode_global_q8k", (2, 0.1), [2, 2, 1], [16 * 1024, 64 * 1024, 64 * 64, 64 * 2048, 16 * 2 * 514 * 4, 16], [16, 4, 2, 16, 4, 4]),
    ("attn_decode_sliding_d128", (2, 0.1), [2, 2, 1], DEC(128, 4, 2), [8, 8, 8, 4, 4]),
    ("attn_reduce_d256", 2, [4, 1, 1], [4 * 2 * 258 * 4, 4 * 512], [8, 4]),
    ("attn_reduce_d512", 2, [4, 1, 1], [4 * 2 * 514 * 4, 4 * 1024], [8, 4]),
    ("attn_reduce_f32_d128", 2, [4, 1, 1], [4 * 2 * 130 * 4, 4 * 512], [8, 8]),
    ("attn_reduce_partial_d128", 2, [4, 1, 1], [4 * 2 * 130 * 4, 4 * 520], [8, 8]),
    ("attn_combine_ranks_d128", 2, [4, 1, 1], [4 * 2 * 130 * 4, 4 * 512], [8, 8]),
    ("attn_prefill_sliding", 0.1, [2, 16, 1], PRE(256, 4, 2, 2), [16, 16, 16, 2, 4]),
    ("attn_prefill_global", 0.1, [2, 16, 1], PRE(512, 16, 2, 2), [16, 16, 16, 2, 4]),
    ("attn_prefill_sliding_ring", 0.1, [2, 4, 1], RING(256, 4, 2, 2), [16, 16, 16, 16, 16, 2, 4]),
    ("attn_prefill_sliding_f32_d128", 0.1, [2, 16, 1], PRE(128, 4, 2, 4), [8, 8, 8, 4, 4]),
    ("attn_verify_sliding_ring_d128", 0.1, [2, 4, 1], RING(128, 4, 2, 4), [8, 8, 8, 8, 8, 4, 4]),
    ("attn_prefill_global_flash", 0.1, [32, 1, 1], PRE(512, 32, 4, 2), [16, 16, 16, 2, 4]),
    ("attn_prefill_global_flash_sp_q8", 0.1, [32, 1, 1], [16 * 32 * 1024] + [64 * 2048, 64 * 128] * 2 + [16 * 32 * 1024, 16], [16, 4, 2, 4, 2, 2, 4]),
    ("attn_prefill_global_flash_sp_iq", 0.1, [32, 1, 1], [16 * 32 * 512, 16 * 32 * 32, 64 * 2048, 64 * 128, 64 * 4096, 16 * 32 * 1024, 16],
     [4, 2, 4, 2, 16, 2, 4]),
    ("attn_decode_paged_q8kv_d128", (2, 0.1, 16), [2, 2, 1], [4 * 256] + POOL * 2 + [16, 4 * 2 * 520, 16], [8, 16, 16, 16, 16, 4, 8, 4]),
    ("attn_decode_paged_q8kv_scalar_d128", (2, 0.1, 16), [2, 2, 1], [4 * 256] + POOL * 2 + [16, 4 * 2 * 520, 16], [8, 4, 2, 4, 2, 4, 4, 4]),
    ("attn_prefill_paged_q8kv_scalar_d128", (0.1, 16), [2, 16, 1], [16 * 4 * 256] + POOL * 2 + [16, 16 * 4 * 512, 16], [8, 4, 2, 4, 2, 4, 4, 4]),
    ("attn_prefill_flash_f16_d128", (0.1, 0), [2, 16, 1], PRE(128, 4, 2, 4), [16, 16, 16, 16, 4]),
    ("attn_prefill_sliding_ring_flash_d128", 0.1, [2, 4, 1], RING(128, 4, 2, 4), [16, 16, 16, 16, 16, 16, 4]),
    ("attn_prefill_paged_q8kv_flash_d128", (0.1, 16), [2, 16, 1], [16 * 4 * 256] + POOL * 2 + [16, 64 * ROW * 2, 64 * ROW * 2, 16 * 4 * 512, 16],
     [16, 16, 2, 16, 2, 4, 16, 16, 16, 4]),
    ("kv_append_sliding", None, [16, 1, 1], [8192, 1024 * 8192, 16], [16, 16, 4]),
    ("kv_append_global_q8", None, [1, 1, 1], [4096, 16 * 128, 16 * 2048, 16], [16, 2, 16, 4]),
    ("kv_append_paged_q8_d128", (ROW, 16), [1, 1, 1], [ROW * 2, POOL[1], POOL[0], 16, 16], [16, 2, 16, 4, 4]),
    ("kv_quant_q8", None, [1, 1, 1], [512, 16, 256], [16, 2, 16]),
    ("kv_dequant_q8", None, [1, 1, 1], [16, 256, 512], [2, 16, 16]),
    ("kv_dequant_paged_q8_d128", (ROW, 16), [1, 1, 1], [POOL[1], POOL[0], 16, 64 * ROW * 2, 16], [2, 16, 4, 16, 4]),
    ("rmsnorm_256", None, [4, 1, 1], [2048, 1024, 2048], [16, 4, 16]),
    ("rope_sliding_q", None, [16, 1, 1], [16384, 1024], [2, 8]),
    ("attn_norm_rope_d128", (2, 128, 0), [1, 1, 1], [512, 512, 512, 512], [16, 16, 16, 16]),
    ("kv_norm_rope_append_paged_q8_d128", (ROW, 16, 128, 0), [1, 1, 1], [ROW * 2, ROW * 2, 512, 512, POOL[1], POOL[0], POOL[1], POOL[0], 16, 16],
     [16, 16, 16, 16, 2, 8, 2, 8, 4, 4]),
    ("qkv_norm_rope_append_paged_q8_d128", (4, ROW, 16, 128, 0), [1, 1, 1],
     [1024, 512, 1024, ROW * 2, ROW * 2, 512, 512, POOL[1], POOL[0], POOL[1], POOL[0], 16, 16], [16, 16, 16, 16, 16, 16, 16, 2, 8, 2, 8, 4, 4]),
]


@pytest.fixture(scope="module")
def ctx():
    import super_gemma_b200 as sg

    return sg.GpuContext(0)


@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0])
def test_bindings_that_do_not_fit_are_refused_before_any_launch(ctx, case):
    import super_gemma_b200 as sg

    name, push, groups, sizes, align = case
    kernel = ctx.load_kernel(name)
    assert kernel.blob.bindings == len(sizes) == len(align)
    whole = [ctx.new_buffer(n + 64) for n in sizes]
    fit = [ctx.adopt(b.device_ptr, n, keep=b) for b, n in zip(whole, sizes)]
    ctx.dispatch_blocking(kernel, bind(*fit), push, groups)  # zeros everywhere: a valid call
    for i, a in enumerate(align):
        bad = list(fit)
        bad[i] = ctx.adopt(whole[i].device_ptr + a // 2, sizes[i], keep=whole[i])
        before = ctx.launch_count
        with pytest.raises(sg.Validation, match=f"binding {i} must be {a}-byte aligned"):
            ctx.dispatch(kernel, bind(*bad), push, groups)
        assert ctx.launch_count == before


def _moved(ctx, data, by):
    """The data at an address that is `by` bytes past a 16-byte boundary (and no better)."""
    raw = np.ascontiguousarray(data).reshape(-1).view(np.uint8)
    b = ctx.new_buffer(raw.size + 16)
    b.write(raw, by)
    return ctx.adopt(b.device_ptr + by, raw.size, keep=b)


def _step(ctx, **kw):
    import super_gemma_b200 as sg

    s = ctx.new_step_buffer()
    sg.StepState(**kw).write_to(s)
    return s


def test_decode_d128_rows_on_eight_bytes(ctx):
    n, kv, hd = 100, 2, 128
    q, k, v = normal_f16(1, 2 * kv, hd), normal_f16(2, n, kv, hd), normal_f16(3, n, kv, hd)
    part, out = ctx.new_buffer(2 * kv * 3 * (hd + 2), np.float32), ctx.new_buffer(2 * kv * hd, np.float32)
    ctx.dispatch(ctx.load_kernel("attn_decode_sliding_d128"), bind(*(_moved(ctx, x, 8) for x in (q, k, v)), part, _step(ctx, kv_len_sliding=n)),
                 (3, hd**-0.5), [kv, 3, 1])
    ctx.dispatch_blocking(ctx.load_kernel("attn_reduce_f32_d128"), bind(part, out), 3, [2 * kv, 1, 1])
    want = O.attention_f64(q.astype(np.float32)[None], k.astype(np.float32), v.astype(np.float32), 1, n - 1, 2 * kv, kv, hd, hd**-0.5)[0]
    assert_close(out.read().reshape(2 * kv, hd), want, 5e-5, 1e-5)


@pytest.mark.parametrize("which", range(6))
def test_global_int8_operands_on_their_own_alignment(ctx, which):
    """Quants on 4 bytes, scales and output on 2, one at a time: the streaming kernel, but for the scales, which the tensor-core kernel reads one by one."""
    m, q0 = 16, 100
    q, k, v = normal_f16(4, m, 32, 512).astype(np.float32), normal_f16(5, q0 + m, 4, 512).astype(np.float32), normal_f16(6, q0 + m, 4, 512)
    qs, qq, qd = O.q8_quant_div(q.ravel())
    ks, kq, kd = O.q8_quant_div(k.ravel())
    by = [4 if which == 0 else 0, 2 if which == 1 else 0, 4 if which == 2 else 0, 2 if which == 3 else 0, 0]
    bufs = [_moved(ctx, x, b) for x, b in zip((qq, qs, kq, ks, v), by)]
    whole = ctx.new_buffer(m * 32 * 512 * 2 + 16)
    out = ctx.adopt(whole.device_ptr + (2 if which == 4 else 8 if which == 5 else 0), m * 32 * 512 * 2, np.uint16, keep=whole)
    ctx.dispatch_blocking(ctx.load_kernel("attn_prefill_global_flash_sp_iq"), bind(*bufs, out, _step(ctx, q0=q0)), 512**-0.5, [32, 1, 1])
    want = O.attention_f64(qd.reshape(q.shape), kd.reshape(k.shape), v.astype(np.float32), m, q0, 32, 4, 512, 512**-0.5)
    assert_close(O.f16_bits_to_f32(out.read()).reshape(m, 32, 512), want, 5e-5, 2.0**-11)


@pytest.mark.parametrize("by", [2, 4, 8])
def test_global_int8_scales_of_k_on_two_bytes_keep_the_kernel(ctx, by):
    """... and so give the bits that scales on 16 bytes give (the streaming kernel's are others)."""
    m, q0 = 16, 300
    q, k, v = normal_f16(14, m, 32, 512).astype(np.float32), normal_f16(15, q0 + m, 4, 512).astype(np.float32), normal_f16(16, q0 + m, 4, 512)
    (qs, qq, _), (ks, kq, _) = O.q8_quant_div(q.ravel()), O.q8_quant_div(k.ravel())
    got = []
    for b in (0, by):
        out = ctx.new_buffer(m * 32 * 512, np.uint16)
        bufs = [_moved(ctx, x, y) for x, y in zip((qq, qs, kq, ks, v), (0, 0, 0, b, 0))]
        ctx.dispatch_blocking(ctx.load_kernel("attn_prefill_global_flash_sp_iq"), bind(*bufs, out, _step(ctx, q0=q0)), 512**-0.5, [32, 1, 1])
        got.append(out.read())
    assert np.array_equal(*got)


@pytest.mark.parametrize("name,n", [("rmsnorm_256", 256), ("rmsnorm_512_plus1", 512)])
def test_rmsnorm_weights_on_their_own_alignment(ctx, name, n):
    """Weights on 4 bytes come one by one, on 16 four at a time: the same bits, also past the first block of rows."""
    rows = 40
    x, w = normal_f16(7, rows, n), np.random.default_rng(8).standard_normal(n, dtype=np.float32)
    got = []
    for by in (0, 4):
        y = ctx.new_buffer(rows * n, np.uint16)
        ctx.dispatch_blocking(ctx.load_kernel(name), bind(ctx.buffer_from_iter(x), _moved(ctx, w, by), y), None, [rows, 1, 1])
        got.append(y.read())
    assert np.array_equal(*got) and np.any(got[0] != 0)


@pytest.mark.parametrize("name,n,by", [("rmsnorm_256", 256, 0), ("rmsnorm_256_plus1", 256, 4), ("rmsnorm_512", 512, 4), ("rmsnorm_512_plus1", 512, 0)])
def test_rmsnorm_of_many_rows_gives_the_bits_of_few(ctx, name, n, by):
    """Weights asked for ahead or behind the sum of squares, by the size of the launch: 3 / 2, 2 and 8 blocks an SM and one row more, and the
    same rows two thousand at a time."""
    import torch

    sms, per_block = torch.cuda.get_device_properties(0).multi_processor_count, 256 * 32 // n
    w = _moved(ctx, np.random.default_rng(n).standard_normal(n, dtype=np.float32), by)
    kernel = ctx.load_kernel(name)
    x = normal_f16(n, 8 * sms * per_block + 1, n)

    def run(rows):
        y = ctx.new_buffer(rows.size, np.uint16)
        ctx.dispatch_blocking(kernel, bind(ctx.buffer_from_iter(rows), w, y), None, [len(rows), 1, 1])
        return y.read().reshape(rows.shape)

    few = np.concatenate([run(x[i:i + 2000]) for i in range(0, len(x), 2000)])
    for blocks in (3 * sms // 2, 2 * sms, 8 * sms):
        for rows in (blocks * per_block, blocks * per_block + 1):
            assert np.array_equal(run(x[:rows]), few[:rows]), (blocks, rows)
