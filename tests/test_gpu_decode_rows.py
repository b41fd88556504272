"""Split-K decode over f16 values and the ring verify step where their 16-key tiles can go wrong: lengths around the tile and
the warps' strides, empty and one-key splits, rows past the end that hold NaN, the ring's wrap, values that are not finite,
lengths past the buffer.

Tolerance against the f64 oracle: P keeps f32's last place, sums and exponentials are f32 (1e-5 of the largest |v|, below 5 for these
normals), and the output's own f16 rounding (2^-11) where it is f16."""
import numpy as np
import pytest

from cases import assert_close, bind, normal_f16
from oracle import sg_oracle as O

pytestmark = pytest.mark.gpu
ATOL, R = 5e-5, 1024
NAN16 = 0x7E00
# name, reduce, kv heads, query heads per kv head, head_dim, Q8_0 keys, step slot
KINDS = [("attn_decode_sliding", "attn_reduce_d256", 16, 2, 256, False, "kv_len_sliding"),
         ("attn_decode_global", "attn_reduce_d512", 4, 8, 512, False, "kv_len_global"),
         ("attn_decode_global_q8k", "attn_reduce_d512", 4, 8, 512, True, "kv_len_global"),
         ("attn_decode_sliding_d128", "attn_reduce_f32_d128", 16, 2, 128, False, "kv_len_sliding")]


@pytest.fixture(scope="module")
def ctx():
    import super_gemma_b200 as sg

    return sg.GpuContext(0)


def _step(ctx, **kw):
    import super_gemma_b200 as sg

    s = ctx.new_step_buffer()
    sg.StepState(**kw).write_to(s)
    return s


def _spare(n, splits):
    """Rows behind the n keys: 64 per split in all, as many as the tiled kernels want."""
    return max(37, 64 * splits - n)


def _decode(ctx, kind, q, k, v, n, splits, rows=None, k_scale=None):
    name, red, n_kv, g, hd, q8, slot = kind
    up = lambda b: ctx.buffer_from_iter(np.ascontiguousarray(b))
    spare = _spare(n, splits)
    junk = np.full((spare, n_kv, hd), NAN16, np.uint16)
    v_up = up(np.concatenate([v.view(np.uint16), junk])[:rows])
    if q8:
        ks, kq, kd = O.q8_quant_div(k.astype(np.float32).ravel())
        kd = kd.reshape(k.shape)
        if k_scale is not None:
            ks = ks.copy()
            ks.view(np.uint16)[k_scale] = 0x7C00
        pad = lambda x, w, fill: up(np.concatenate([x.reshape(n, w), np.full((spare, w), fill, x.dtype)])[:rows])
        bufs = [pad(kq, n_kv * hd, 99), pad(ks.view(np.uint16), n_kv * hd // 32, NAN16)]
    else:
        kd, bufs = k.astype(np.float32), [up(np.concatenate([k.view(np.uint16), junk])[:rows])]
    part = ctx.new_buffer(n_kv * g * splits * (hd + 2), np.float32)
    out = ctx.new_buffer(n_kv * g * hd, np.float32 if "f32" in red else np.uint16)
    ctx.dispatch_blocking(ctx.load_kernel(name), bind(up(q), *bufs, v_up, part, _step(ctx, **{slot: n})), (splits, hd**-0.5), [n_kv, splits, 1])
    ctx.dispatch_blocking(ctx.load_kernel(red), bind(part, out), splits, [n_kv * g, 1, 1])
    got = out.read() if "f32" in red else O.f16_bits_to_f32(out.read())
    return got.reshape(n_kv * g, hd), kd, part.read().reshape(n_kv * g, splits, hd + 2)


def _case(kind, seed, n):
    _, _, n_kv, g, hd, _, _ = kind
    return normal_f16(seed, n_kv * g, hd), normal_f16(seed + 1, n, n_kv, hd), normal_f16(seed + 2, n, n_kv, hd)


@pytest.mark.parametrize("kind", KINDS, ids=lambda k: k[0])
@pytest.mark.parametrize("n,splits", [(1, 1), (1, 3), (15, 1), (16, 1), (17, 2), (64, 1), (65, 1), (129, 1), (300, 7), (1000, 16), (1024, 16), (1000, 1)])
def test_decode_lengths(ctx, kind, n, splits):
    _, _, n_kv, g, hd, _, _ = kind
    q, k, v = _case(kind, n + splits, n)
    got, kd, part = _decode(ctx, kind, q, k, v, n, splits)
    want = O.attention_f64(q.astype(np.float32)[None], kd, v.astype(np.float32), 1, n - 1, n_kv * g, n_kv, hd, hd**-0.5)[0]
    assert_close(got, want, ATOL, 1e-5 if got.dtype == np.float32 and "f32" in kind[1] else 2.0**-11, f"{kind[0]} n={n} splits={splits}")
    chunk = -(-n // splits)
    empty = [s for s in range(splits) if s * chunk >= n]
    assert np.all(part[:, empty, hd] == np.float32(-3.0e38)) and np.all(part[:, empty, hd + 1] == 0) and np.all(part[:, empty, :hd] == 0)


@pytest.mark.parametrize("kind", KINDS, ids=lambda k: k[0])
@pytest.mark.parametrize("n,splits,rows", [(300, 10, 639), (300, 10, 640), (300, 10, 319), (300, 10, 320), (150, 10, 159), (150, 10, 160), (300, 300, 300), (5, 64, 4096)])
def test_decode_few_rows_per_split(ctx, kind, n, splits, rows):
    """Both sides of the line between the streaming and the tiled kernel: 64 rows of the cache per split at head_dim 256, 32 at
    128, 16 at 512."""
    _, _, n_kv, g, hd, _, _ = kind
    q, k, v = _case(kind, rows, n)
    got, kd, part = _decode(ctx, kind, q, k, v, n, splits, rows=rows)
    want = O.attention_f64(q.astype(np.float32)[None], kd, v.astype(np.float32), 1, n - 1, n_kv * g, n_kv, hd, hd**-0.5)[0]
    assert_close(got, want, ATOL, 1e-5 if "f32" in kind[1] else 2.0**-11, f"{kind[0]} rows={rows}")
    empty = np.arange(splits) * -(-n // splits) >= n
    assert np.all(part[:, empty, hd] == np.float32(-3.0e38)) and np.all(part[:, empty, hd + 1] == 0) and np.all(part[:, empty, :hd] == 0)


@pytest.mark.parametrize("kind", KINDS, ids=lambda k: k[0])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_decode_value_that_is_not_finite(ctx, kind, value):
    _, _, n_kv, g, hd, _, _ = kind
    n, splits = 200, 3
    q, k, v = _case(kind, 77, n)
    clean, _, _ = _decode(ctx, kind, q, k, v, n, splits)
    v[90, 1, 5] = value
    got, _, _ = _decode(ctx, kind, q, k, v, n, splits)
    hit = got.reshape(n_kv, g, hd)[1, :, 5]
    assert np.all(np.isnan(hit) if np.isnan(value) else hit == value)
    got.reshape(n_kv, g, hd)[1, :, 5] = clean.reshape(n_kv, g, hd)[1, :, 5]
    assert_close(got, clean, ATOL, 2.0**-10, kind[0])  # two statements, each rounded to f16


@pytest.mark.parametrize("kind", KINDS, ids=lambda k: k[0])
def test_decode_length_past_the_buffer_is_reported(ctx, kind):
    import super_gemma_b200 as sg

    q, k, v = _case(kind, 5, 100)
    with pytest.raises(sg.GpuError):
        _decode(ctx, kind, q, k, v, 100, 2, rows=90)


@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("q0", [0, 1, 15, 16, 500, 1021, 1023, 1024, 1025, 66001])
def test_verify_ring(ctx, m, q0):
    n_kv, hd = 6, 128
    hist = min(q0, R)
    q, k, v = normal_f16(q0 + m, m, 2 * n_kv, hd), normal_f16(q0 + m + 1, hist + m, n_kv, hd), normal_f16(q0 + m + 2, hist + m, n_kv, hd)
    ring = [np.full((R, n_kv, hd), NAN16, np.uint16) for _ in range(2)]
    for i in range(hist):
        for r, x in zip(ring, (k, v)):
            r[(q0 - hist + i) % R] = x[i].view(np.uint16)
    up = lambda b: ctx.buffer_from_iter(np.ascontiguousarray(b))
    junk = np.full((20, n_kv, hd), NAN16, np.uint16)
    out = ctx.new_buffer(m * 2 * n_kv * hd, np.float32)
    ctx.dispatch_blocking(ctx.load_kernel("attn_verify_sliding_ring_d128"),
                          bind(up(q), up(ring[0]), up(ring[1]), up(np.concatenate([k[hist:].view(np.uint16), junk])),
                               up(np.concatenate([v[hist:].view(np.uint16), junk])), out, _step(ctx, q0=q0)), hd**-0.5, [n_kv, m, 1])
    want = O.attention_f64(q.astype(np.float32), k.astype(np.float32), v.astype(np.float32), m, hist, 2 * n_kv, n_kv, hd, hd**-0.5, window=1024)
    assert_close(out.read().reshape(m, 2 * n_kv, hd), want, ATOL, 1e-5, f"m={m} q0={q0}")


def test_verify_ring_keeps_the_precision_of_the_f32_statement(ctx):
    """The streaming kernel's 2-norm error on such inputs is 1.6e-7 of the result; scores summed in the tensor pipe gave 2.2e-7."""
    n_kv, hd, m, q0 = 16, 128, 4, 60
    q, k, v = normal_f16(1, m, 2 * n_kv, hd), normal_f16(2, q0 + m, n_kv, hd), normal_f16(3, q0 + m, n_kv, hd)
    up = lambda b: ctx.buffer_from_iter(np.ascontiguousarray(b))
    ring = lambda x: up(np.concatenate([x[:q0], np.zeros((R - q0, n_kv, hd), np.float16)]))
    out = ctx.new_buffer(m * 2 * n_kv * hd, np.float32)
    ctx.dispatch_blocking(ctx.load_kernel("attn_verify_sliding_ring_d128"), bind(up(q), ring(k), ring(v), up(k[q0:]), up(v[q0:]), out, _step(ctx, q0=q0)),
                          hd**-0.5, [n_kv, m, 1])
    q, k, v = (x.astype(np.float64) for x in (q, k, v))
    s = np.einsum("mhd,khd->mhk", q, np.repeat(k, 2, 1)) * hd**-0.5
    seen = np.arange(q0 + m)[None, None, :] <= q0 + np.arange(m)[:, None, None]
    p = np.where(seen, np.exp(s - s.max(-1, keepdims=True)), 0)
    want = np.einsum("mhk,khd->mhd", p / p.sum(-1, keepdims=True), np.repeat(v, 2, 1))
    got = out.read().reshape(want.shape).astype(np.float64)
    assert np.linalg.norm(got - want) < 1.8e-7 * np.linalg.norm(want)


def test_verify_ring_value_only_the_later_token_sees(ctx):
    """The draft's own last row holds Inf: earlier drafted tokens do not see it."""
    n_kv, hd, m, q0 = 2, 128, 4, 700
    q, k, v = normal_f16(1, m, 2 * n_kv, hd), normal_f16(2, q0 + m, n_kv, hd), normal_f16(3, q0 + m, n_kv, hd)
    up = lambda b: ctx.buffer_from_iter(np.ascontiguousarray(b))
    pad = lambda x: np.concatenate([x[:q0], np.zeros((R - q0, n_kv, hd), np.float16)])
    outs = []
    for value in (v[q0 + 3, 1, 9], np.float16(np.inf)):
        v[q0 + 3, 1, 9] = value
        out = ctx.new_buffer(m * 2 * n_kv * hd, np.float32)
        ctx.dispatch_blocking(ctx.load_kernel("attn_verify_sliding_ring_d128"),
                              bind(up(q), up(pad(k)), up(pad(v)), up(k[q0:]), up(v[q0:]), out, _step(ctx, q0=q0)), hd**-0.5, [n_kv, m, 1])
        outs.append(out.read().reshape(m, 2 * n_kv, hd))
    clean, got = outs
    assert np.all(got[3, 2:, 9] == np.inf)
    got[3, 2:, 9] = clean[3, 2:, 9]
    assert_close(got, clean, ATOL, 1e-5, "everything else")


@pytest.mark.parametrize("kind", KINDS, ids=lambda k: k[0])
def test_only_rows_that_are_not_finite_are_computed_again(ctx, kind):
    """A NaN in one query row leaves the other rows' bits alone."""
    _, _, n_kv, g, hd, _, _ = kind
    n, splits = 300, 3
    q, k, v = _case(kind, 91, n)
    clean, _, _ = _decode(ctx, kind, q, k, v, n, splits)
    row = n_kv * g - 1
    q[row, 3] = np.nan
    got, _, _ = _decode(ctx, kind, q, k, v, n, splits)
    assert np.all(np.isnan(got[row]))
    assert np.array_equal(got[:row].view(np.uint32), clean[:row].view(np.uint32))


@pytest.mark.parametrize("kind", KINDS, ids=lambda k: k[0])
@pytest.mark.parametrize("n,splits,m_q", [(50, 7, 4), (50, 7, 2), (17, 16, 3), (4, 2, 4), (200, 3, 2)])
def test_decode_of_a_draft_is_causal(ctx, kind, n, splits, m_q):
    """groups[2] query tokens: query i sees t <= n - m_q + i.  In (50, 7), (17, 16) and (4, 2) the last split begins between the
    queries' last visible keys, so that it is empty for the first of them."""
    name, red, n_kv, g, hd, q8, slot = kind
    q, k, v = normal_f16(n, m_q, n_kv * g, hd), normal_f16(n + 1, n, n_kv, hd), normal_f16(n + 2, n, n_kv, hd)
    up = lambda b: ctx.buffer_from_iter(np.ascontiguousarray(b))
    if q8:
        ks, kq, kd = O.q8_quant_div(k.astype(np.float32).ravel())
        bufs = [up(np.resize(x, (n + _spare(n, splits)) * (x.size // n))) for x in (kq, ks)]
    else:
        kd, bufs = k.astype(np.float32), [up(np.resize(k, (n + _spare(n, splits), n_kv, hd)))]
    rows = m_q * n_kv * g
    part, out = ctx.new_buffer(rows * splits * (hd + 2), np.float32), ctx.new_buffer(rows * hd, np.float32 if "f32" in red else np.uint16)
    ctx.dispatch(ctx.load_kernel(name), bind(up(q), *bufs, up(np.resize(v, (n + _spare(n, splits), n_kv, hd))), part,
                                            _step(ctx, **{slot: n})), (splits, hd**-0.5), [n_kv, splits, m_q])
    ctx.dispatch_blocking(ctx.load_kernel(red), bind(part, out), splits, [rows, 1, 1])
    got = out.read() if "f32" in red else O.f16_bits_to_f32(out.read())
    want = O.attention_f64(q.astype(np.float32), kd.reshape(k.shape), v.astype(np.float32), m_q, n - m_q, n_kv * g, n_kv, hd, hd**-0.5)
    assert_close(got.reshape(want.shape), want, ATOL, 1e-5 if "f32" in red else 2.0**-11, name)


@pytest.mark.parametrize("kind", KINDS[1:3], ids=lambda k: k[0])
@pytest.mark.parametrize("splits", [1, 32])
def test_every_tile_counts_once(ctx, kind, splits):
    """All scores equal, and the value of tile i is 1 in dim i % 512: over 32768 keys a dim's result is 4 tiles' worth, and one tile
    too few or twice is a quarter of it (allowed: the weights' f32 sums and the output's f16)."""
    _, _, n_kv, g, hd, _, _ = kind
    n = 32768
    q, _, _ = _case(kind, 3, 1)
    k, v = np.broadcast_to(normal_f16(4, 1, n_kv, hd), (n, n_kv, hd)), np.zeros((n, n_kv, hd), np.float16)
    v[np.arange(n), :, (np.arange(n) // 16) % hd] = 1
    got, _, _ = _decode(ctx, kind, q, k, v, n, splits)
    assert_close(got, np.full_like(got, 1 / hd), 0, 2.0**-11 + 1e-5, "equal weights")


def test_decode_infinite_scale_of_a_key(ctx):
    """The statement multiplies the scale with every quant: infinities of both signs, NaN for every head of that kv head."""
    n = 300
    q, k, v = _case(KINDS[2], 95, n)
    clean, _, _ = _decode(ctx, KINDS[2], q, k, v, n, 3)
    got, _, _ = _decode(ctx, KINDS[2], q, k, v, n, 3, k_scale=(170 * 4 + 1) * 16 + 9)
    assert np.all(np.isnan(got[8:16]))
    got[8:16] = clean[8:16]
    assert np.array_equal(got.view(np.uint32), clean.view(np.uint32))
