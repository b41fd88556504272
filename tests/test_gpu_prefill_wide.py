"""The tensor-core prefill of the reference-shaped heads (head_dim 256 f16 with a 1024-token window, head_dim 512 with int8
Q and K) where its tiles can go wrong: query counts around the 64- and 16-token tiles, histories around the 64-key tiles, one CTA and two per unit
and the ring's wrap, rows past the end that hold NaN, values that are not finite, and the calls it leaves to the streaming
kernel.

Tolerance against the f64 oracle: the output is f16 (relative 2^-11), P keeps f32's last place, sums and exponentials are f32:
1e-5 of the largest |v| (below 5 for these normals)."""
import numpy as np
import pytest

from cases import assert_close, bind
from oracle import sg_oracle as O

pytestmark = pytest.mark.gpu
RTOL, ATOL, R, W = 2.0**-11, 5e-5, 1024, 1024
NAN16 = 0x7E00


@pytest.fixture(scope="module")
def ctx():
    import super_gemma_b200 as sg

    return sg.GpuContext(0)


def _step(ctx, q0):
    import super_gemma_b200 as sg

    s = ctx.new_step_buffer()
    sg.StepState(pos=q0, q0=q0).write_to(s)
    return s


def _bits(x):
    return O.f32_to_f16_bits(np.ascontiguousarray(x, np.float32).ravel()).astype(np.uint16)


def _normal(seed, *shape):
    return np.random.default_rng(seed).standard_normal(shape, dtype=np.float32).astype(np.float16).astype(np.float32)


def _sliding(ctx, q, k, v, q0, m, n_kv, ring, scale=0.0625, poison=True):
    """k, v: rows of positions [first, q0 + m) with first = max(0, q0 - R); linear caches start at position 0 (q0 <= R)."""
    n_q, row = 2 * n_kv, n_kv * 256
    up = lambda b: ctx.buffer_from_iter(np.ascontiguousarray(b))
    out = ctx.new_buffer(m * n_q * 256, np.uint16)
    kb, vb = _bits(k).reshape(-1, row), _bits(v).reshape(-1, row)
    junk = np.full((70, row), NAN16, np.uint16) if poison else np.zeros((70, row), np.uint16)
    if ring:
        hist = len(kb) - m
        kr, vr = np.zeros((R, row), np.uint16), np.zeros((R, row), np.uint16)
        if poison and hist < R:
            kr[:], vr[:] = NAN16, NAN16
        for i in range(hist):
            kr[(q0 - hist + i) % R], vr[(q0 - hist + i) % R] = kb[i], vb[i]
        bufs = [up(kr), up(vr), up(np.vstack([kb[hist:], junk])), up(np.vstack([vb[hist:], junk]))]
        name = "attn_prefill_sliding_ring"
    else:
        bufs, name = [up(np.vstack([kb, junk])), up(np.vstack([vb, junk]))], "attn_prefill_sliding"
    ctx.dispatch_blocking(ctx.load_kernel(name), bind(up(_bits(q)), *bufs, out, _step(ctx, q0)), scale, [n_kv, m, 1])
    return O.f16_bits_to_f32(out.read()).reshape(m, n_q, 256)


def _sliding_case(seed, q0, m, n_kv):
    hist = min(q0, R)
    return _normal(seed, m, 2 * n_kv, 256), _normal(seed + 1, hist + m, n_kv, 256), _normal(seed + 2, hist + m, n_kv, 256), hist


@pytest.mark.parametrize("m", [1, 33, 63, 65, 200])
@pytest.mark.parametrize("q0", [0, 1, 127, 128, 1000, 1023, 1024])
@pytest.mark.parametrize("ring", [False, True])
def test_sliding_edges(ctx, m, q0, ring):
    q, k, v, hist = _sliding_case(m * 7 + q0, q0, m, 2)
    got = _sliding(ctx, q, k, v, q0, m, 2, ring)
    want = O.attention_f64(q, k, v, m, hist, 4, 2, 256, 0.0625, window=W)
    assert_close(got, want, ATOL, RTOL, f"m={m} q0={q0} ring={ring}")


@pytest.mark.parametrize("q0,m", [(1025, 5), (1531, 1300), (70001, 160)])
def test_sliding_ring_wrapped(ctx, q0, m):
    q, k, v, hist = _sliding_case(q0, q0, m, 16)
    got = _sliding(ctx, q, k, v, q0, m, 16, True)
    toks = np.unique([0, 1, m // 2, m - 1]).astype(np.uint32)
    want = O.attention_f64(q, k, v, m, hist, 32, 16, 256, 0.0625, window=W, tokens=toks)
    assert_close(got[toks], want, ATOL, RTOL, f"wrapped q0={q0} m={m}")


def _iq(ctx, q, k, v, q0, m, scale=0.044194174, pad=80, v_bits=None, poison=None, k_scale=None):
    qs, qq, qd = O.q8_quant_div(q.ravel())
    if poison is not None:  # a scale of q
        qs = qs.copy()
        qs.view(np.uint16)[poison] = NAN16
    ks, kq, kd = O.q8_quant_div(k.ravel())
    if k_scale is not None:  # an infinite scale of K
        ks = ks.copy()
        ks.view(np.uint16)[k_scale] = 0x7C00
    up = lambda b: ctx.buffer_from_iter(np.ascontiguousarray(b))
    tail = np.full(pad * 2048, NAN16, np.uint16)
    bufs = [up(qq), up(qs), up(np.concatenate([kq, np.full(pad * 2048, 77, np.int8)])),
            up(np.concatenate([ks.view(np.uint16), np.full(pad * 64, NAN16, np.uint16)])),
            up(np.concatenate([_bits(v) if v_bits is None else v_bits, tail]))]
    out = ctx.new_buffer(m * 32 * 512, np.uint16)
    ctx.dispatch_blocking(ctx.load_kernel("attn_prefill_global_flash_sp_iq"), bind(*bufs, out, _step(ctx, q0)), scale, [32, m // 16, 1])
    return O.f16_bits_to_f32(out.read()).reshape(m, 32, 512), qd.reshape(q.shape), kd.reshape(k.shape)


@pytest.mark.parametrize("m,q0", [(16, 0), (16, 47), (16, 48), (16, 111), (16, 112), (48, 1), (64, 2000), (144, 640)])
def test_global_int8_edges(ctx, m, q0):
    q, k, v = _normal(m + q0, m, 32, 512), _normal(m + q0 + 1, q0 + m, 4, 512), _normal(m + q0 + 2, q0 + m, 4, 512)
    got, qd, kd = _iq(ctx, q, k, v, q0, m)
    toks = np.unique([0, 1, 7, 8, m - 1]).astype(np.uint32)
    want = O.attention_f64(qd, kd, v, m, q0, 32, 4, 512, 0.044194174, tokens=toks)
    assert_close(got[toks], want, ATOL, RTOL, f"iq m={m} q0={q0}")
    assert np.all(np.isfinite(got))


def test_global_int8_long_history_is_not_biased(ctx):
    """Over 32768 keys the outputs must not shrink: their projection on the f64 result is off by at most what the products of four
    tiles, the longest sum left to the tensor pipe, lose to its truncation (64 additions of less than 2^-23 each: 7.6e-6), plus
    the mean of 32768 f16 roundings (4 sigma of 2.1e-4 / sqrt(32768): 4.6e-6).  In one sum it was 6.7e-5."""
    m, q0 = 16, 32752
    q, k, v = _normal(31, m, 32, 512), _normal(32, q0 + m, 4, 512), _normal(33, q0 + m, 4, 512)
    got, qd, kd = _iq(ctx, q, k, v, q0, m)
    toks = np.array([0, m - 1], np.uint32)
    want = O.attention_f64(qd, kd, v, m, q0, 32, 4, 512, 0.044194174, tokens=toks)
    d = got[toks] - want
    assert abs(np.vdot(d, want) / np.vdot(want, want)) <= 7.6e-6 + 4.6e-6
    assert_close(got[toks], want, 1e-6, 1.05 * RTOL, "32768 keys")  # outputs of some 0.006: their own rounding, barely more


@pytest.mark.parametrize("q0", [496, 500, 512, 624, 640, 1008, 1020, 1136, 2032])
def test_global_int8_settled_parts(ctx, q0):
    """Ends around the tiles in which a dim block is settled for the first or second time, with scores that keep raising the running maximum after parts were settled."""
    m = 16
    q, k, v = _normal(q0, m, 32, 512), _normal(q0 + 1, q0 + m, 4, 512), _normal(q0 + 2, q0 + m, 4, 512)
    q = np.repeat(q[:, ::8], 8, axis=1)
    for up, scale in ((0.0, 0.044194174), (1e-3, 200 / (q0 + m))):  # scores of up to some 100: rounded to 100 * 2^-24
        kk = (k + (np.arange(q0 + m)[:, None, None] * up * q.mean(0)[::8][None])).astype(np.float16).astype(np.float32)
        got, qd, kd = _iq(ctx, q, kk, v, q0, m, scale=scale)
        want = O.attention_f64(qd, kd, v, m, q0, 32, 4, 512, scale)
        assert_close(got, want, 2 * ATOL, RTOL, f"q0={q0} up={up}")


def test_global_int8_peaked_scores(ctx):
    """Scores that grow along the keys by far more than 2^8: every tile raises the running maximum."""
    m, q0 = 16, 700
    q, k, v = _normal(5, m, 32, 512), _normal(6, q0 + m, 4, 512), _normal(7, q0 + m, 4, 512)
    q = np.repeat(q[:, ::8], 8, axis=1)
    k += (np.arange(q0 + m)[:, None, None] * 1e-3 * q.mean(0)[::8][None]).astype(np.float16).astype(np.float32)
    got, qd, kd = _iq(ctx, q, k.astype(np.float16).astype(np.float32), v, q0, m, scale=0.5)
    want = O.attention_f64(qd, kd, v, m, q0, 32, 4, 512, 0.5)
    assert_close(got, want, 2 * ATOL, RTOL, "peaked")  # scores of some 60: their rounding moves the exponent by 60 * 2^-24


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_values_that_are_not_finite_reach_only_who_sees_them(ctx, value):
    m, q0, n_kv, at = 64, 300, 2, 330  # the key at position 330 is seen by queries 30 and later
    q, k, v, hist = _sliding_case(9, q0, m, n_kv)
    clean = _sliding(ctx, q, k, v, q0, m, n_kv, True)
    v2 = v.copy()
    v2[at, 1, 17] = value
    got = _sliding(ctx, q, k, v2, q0, m, n_kv, True)
    # both sides are rounded to f16, and the tile that sees the value is computed by another statement: one f16 step
    assert_close(got[:30], clean[:30], ATOL, 2 * RTOL, "queries before it")
    assert_close(got[30:, :2], clean[30:, :2], ATOL, 2 * RTOL, "the other kv head")
    hit = got[30:, 2:]
    assert np.all(np.isnan(hit[..., 17]) if np.isnan(value) else hit[..., 17] == value)
    rest = np.delete(np.arange(256), 17)
    assert_close(hit[..., rest], clean[30:, 2:][..., rest], ATOL, 2 * RTOL, "its other dims")


@pytest.mark.parametrize("scale", [-0.0625, 0.0])
def test_scales_the_tiles_do_not_take(ctx, scale):
    q, k, v, hist = _sliding_case(11, 200, 40, 2)
    got = _sliding(ctx, q, k, v, 200, 40, 2, True, scale=scale, poison=False)
    want = O.attention_f64(q, k, v, 40, hist, 4, 2, 256, scale, window=W)
    assert_close(got, want, ATOL, RTOL, f"scale {scale}")


def test_keys_past_the_end_of_the_cache_are_reported(ctx):
    import super_gemma_b200 as sg

    q, k, v, _ = _sliding_case(13, 100, 40, 2)
    up = lambda b: ctx.buffer_from_iter(np.ascontiguousarray(b))
    out = ctx.new_buffer(40 * 4 * 256, np.uint16)
    with pytest.raises(sg.GpuError):
        ctx.dispatch_blocking(ctx.load_kernel("attn_prefill_sliding"),
                              bind(up(_bits(q)), up(_bits(k[:120])), up(_bits(v[:120])), out, _step(ctx, 100)), 0.0625, [2, 40, 1])
    assert np.all(np.isfinite(O.f16_bits_to_f32(out.read())))


def test_reruns_give_the_same_bits(ctx):
    q, k, v, _ = _sliding_case(15, 1500, 96, 16)
    a, b = (_sliding(ctx, q, k, v, 1500, 96, 16, True) for _ in range(2))
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("n_kv", [2, 80])  # two CTAs per unit, one
def test_only_rows_that_are_not_finite_are_computed_again(ctx, n_kv):
    """A NaN in one query row leaves every other row's bits alone, also those of its own tile and of the other CTA of its cluster."""
    m, q0 = 64, 300
    q, k, v, _ = _sliding_case(21, q0, m, n_kv)
    clean = _sliding(ctx, q, k, v, q0, m, n_kv, True)
    for tok, head in ((37, 1), (0, 2), (63, 3)):
        q2 = q.copy()
        q2[tok, head, 100] = np.nan
        got = _sliding(ctx, q2, k, v, q0, m, n_kv, True)
        assert np.all(np.isnan(got[tok, head]))
        got[tok, head] = clean[tok, head]
        assert np.array_equal(got.view(np.uint32), clean.view(np.uint32))


def test_global_int8_only_rows_that_are_not_finite_are_computed_again(ctx):
    """... and of a row whose scales hold a NaN in the int8 form."""
    m, q0 = 16, 600
    q, k, v = _normal(41, m, 32, 512), _normal(42, q0 + m, 4, 512), _normal(43, q0 + m, 4, 512)
    clean, _, _ = _iq(ctx, q, k, v, q0, m)
    for tok, head in ((0, 0), (5, 13), (15, 31)):
        got, _, _ = _iq(ctx, q, k, v, q0, m, poison=(tok * 32 + head) * 16 + 7)
        assert np.all(np.isnan(got[tok, head]))
        got[tok, head] = clean[tok, head]
        assert np.array_equal(got.view(np.uint32), clean.view(np.uint32))


@pytest.mark.parametrize("n_kv", [2, 80])
def test_a_value_that_everybody_sees(ctx, n_kv):
    """Inf in the first visible value of one dim: all rows of that kv head are computed again, by both CTAs of a cluster."""
    m, q0 = 65, 200
    q, k, v, _ = _sliding_case(23, q0, m, n_kv)
    clean = _sliding(ctx, q, k, v, q0, m, n_kv, True)
    v[0, 1, 200] = np.inf
    got = _sliding(ctx, q, k, v, q0, m, n_kv, True)
    assert np.all(got[:, 2:4, 200] == np.inf)
    got[:, 2:4, 200] = clean[:, 2:4, 200]
    assert_close(got, clean, ATOL, 2 * RTOL, "everything else")  # two statements, each rounded to f16


def test_global_int8_value_that_everybody_sees(ctx):
    m, q0 = 16, 333
    q, k, v = _normal(51, m, 32, 512), _normal(52, q0 + m, 4, 512), _normal(53, q0 + m, 4, 512)
    clean, _, _ = _iq(ctx, q, k, v, q0, m)
    v[2, 3, 500] = -np.inf
    got, _, _ = _iq(ctx, q, k, v, q0, m)
    assert np.all(got[:, 24:, 500] == -np.inf)
    got[:, 24:, 500] = clean[:, 24:, 500]
    assert_close(got, clean, ATOL, 2 * RTOL, "everything else")


def test_global_int8_infinite_scale_of_a_key(ctx):
    """The statement multiplies the scale with every quant: infinities of both signs, NaN for every row that sees the key, also where
    the block's whole sum is negative."""
    m, q0 = 32, 200
    q, k, v = _normal(61, m, 32, 512), _normal(62, q0 + m, 4, 512), _normal(63, q0 + m, 4, 512)
    clean, _, _ = _iq(ctx, q, k, v, q0, m)
    got, _, _ = _iq(ctx, q, k, v, q0, m, k_scale=((q0 + 13) * 4 + 2) * 16 + 5)  # seen by queries 13 and later, kv head 2
    assert np.all(np.isnan(got[13:, 16:24]))
    assert_close(got[:13], clean[:13], ATOL, 2 * RTOL, "queries before it")
    assert np.array_equal(got[:, :16].view(np.uint32), clean[:, :16].view(np.uint32))
    assert np.array_equal(got[:, 24:].view(np.uint32), clean[:, 24:].view(np.uint32))


@pytest.mark.parametrize("m,q0,factor", [(16, 104, 1), (16, 112, 1), (16, 120, 1), (32, 120, 2.0**-12), (32, 1000, 2.0**13), (16, 200, 2.0**15)])
def test_global_int8_pairs_of_ctas(ctx, m, q0, factor):
    """The two CTAs of a pair end in different tiles (their queries lie on both sides of a multiple of 128), and keys whose scales are subnormal in
    f16, large, or so large that a quant times its scale is beyond f16."""
    q, k, v = _normal(m + q0, m, 32, 512), _normal(q0, q0 + m, 4, 512) * np.float32(factor), _normal(q0 + 2, q0 + m, 4, 512)
    scale = 0.044194174 / factor
    got, qd, kd = _iq(ctx, q, k, v, q0, m, scale=scale)
    assert_close(got, O.attention_f64(qd, kd, v, m, q0, 32, 4, 512, scale), ATOL, RTOL, f"m={m} q0={q0} factor={factor}")


@pytest.mark.parametrize("power,q0", [(-7, 300), (9, 300), (14, 300), (15, 1100), (20, 300)])
def test_global_int8_keys_of_any_scale_stay_on_the_tensor_cores(ctx, power, q0):
    """A power of two on the keys' scales that the softmax scale takes back changes no bit, also where quants times scales are beyond f16
    (from 2^14 on): no row is left to the streaming statement, whose bits are others."""
    m = 32
    q, k, v = _normal(71, m, 32, 512), _normal(72, q0 + m, 4, 512), _normal(73, q0 + m, 4, 512)
    clean, _, _ = _iq(ctx, q, k, v, q0, m, scale=2.0**-4)
    got, _, _ = _iq(ctx, q, k * np.float32(2.0**power), v, q0, m, scale=2.0 ** (-4 - power))
    assert np.array_equal(got.view(np.uint32), clean.view(np.uint32))
