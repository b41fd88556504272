"""The head_dim-128 flash prefill kernel where its tiles can go wrong: one to seven tiles of 64 keys, ends on both sides of a tile,
windows that begin inside one, the ring's wrap, pieces of the key range, maxima that rise from tile to tile, values that are not
finite, and key buffers that are longer than the keys.  SGB_FLASH_LONG, which some of the tests set, chose a second kernel with 128-key
tiles that is no longer there: nothing reads it, and what they ask holds for the one kernel.
Against the f64 oracle at the head_dim-128 tolerance (P is f16: 2^-11 of the largest |v|)."""
import numpy as np
import pytest

from cases import D, G, H, SCALE, assert_close, bind, normal_f16
from oracle import sg_oracle as O

pytestmark = pytest.mark.gpu
NKV, R, NAN16 = 2, 1024, 0x7E00


@pytest.fixture(scope="module")
def ctx():
    import super_gemma_b200 as sg

    return sg.GpuContext(0)


def _step(ctx, q0):
    import super_gemma_b200 as sg

    s = ctx.new_step_buffer()
    sg.StepState(pos=q0, q0=q0).write_to(s)
    return s


def _linear(ctx, q, k, v, m, q0, window, scale=SCALE, pad=130):
    up = ctx.buffer_from_iter
    junk = np.full((pad, NKV, D), NAN16, np.uint16)
    bufs = [up(q), up(np.concatenate([k.view(np.uint16), junk])), up(np.concatenate([v.view(np.uint16), junk]))]
    out = ctx.new_buffer(m * NKV * G * D, np.float32)
    ctx.dispatch_blocking(ctx.load_kernel("attn_prefill_flash_f16_d128"), bind(*bufs, out, _step(ctx, q0)), (scale, window), [NKV, m, 1])
    return out.read().reshape(m, NKV * G, D)


def _case(seed, m, q0):
    return normal_f16(seed, m, NKV * G, D), normal_f16(seed + 1, q0 + m, NKV, D), normal_f16(seed + 2, q0 + m, NKV, D)


def _want(q, k, v, m, q0, window, scale=SCALE):
    return O.attention_f64(q.astype(np.float32), k.astype(np.float32), v.astype(np.float32), m, q0, NKV * G, NKV, D, scale, window=window)


EDGES = [(1, 0), (1, 127), (1, 128), (64, 64), (65, 63), (63, 65), (64, 65), (130, 255), (64, 320), (1, 383), (1, 384), (129, 1151)]


@pytest.mark.parametrize("window", [100, 1024])
@pytest.mark.parametrize("m,q0", EDGES)
def test_windows(ctx, m, q0, window):
    q, k, v = _case(m + 3 * q0, m, q0)
    assert_close(_linear(ctx, q, k, v, m, q0, window), _want(q, k, v, m, q0, window), what=f"m={m} q0={q0} window={window}")


@pytest.mark.parametrize("long,pieces", [(0, 1), (1, 1), (1, 3)])
@pytest.mark.parametrize("m,q0", EDGES)
def test_tiles(ctx, monkeypatch, m, q0, long, pieces):
    monkeypatch.setenv("SGB_FLASH_LONG", str(long))
    monkeypatch.setenv("SGB_FLASH_PIECES", str(pieces))
    q, k, v = _case(m + 3 * q0, m, q0)
    got = _linear(ctx, q, k, v, m, q0, 0)
    assert_close(got, _want(q, k, v, m, q0, 0), what=f"m={m} q0={q0} long={long} pieces={pieces}")
    assert np.array_equal(got.view(np.uint32), _linear(ctx, q, k, v, m, q0, 0).view(np.uint32))


@pytest.mark.parametrize("q0,m", [(1, 65), (127, 2), (128, 64), (129, 130), (1023, 129), (1024, 1), (1151, 70), (2047, 66)])
def test_ring_and_chunk(ctx, q0, m):
    base = max(0, q0 - R)
    q, k, v = _case(q0 + m, m, q0 - base)
    ring = np.full((2, R, NKV, D), NAN16, np.uint16)
    for t in range(base, q0):
        ring[0, t % R], ring[1, t % R] = k[t - base].view(np.uint16), v[t - base].view(np.uint16)
    up, junk = ctx.buffer_from_iter, np.full((130, NKV, D), NAN16, np.uint16)
    chunk = [np.concatenate([x[q0 - base:].view(np.uint16), junk]) for x in (k, v)]
    out = ctx.new_buffer(m * NKV * G * D, np.float32)
    ctx.dispatch_blocking(ctx.load_kernel("attn_prefill_sliding_ring_flash_d128"), bind(up(q), up(ring[0]), up(ring[1]), up(chunk[0]), up(chunk[1]), out,
                                                                                        _step(ctx, q0)), SCALE, [NKV, m, 1])
    assert_close(out.read().reshape(m, NKV * G, D), _want(q, k, v, m, q0 - base, 1024), what=f"ring q0={q0} m={m}")


@pytest.mark.parametrize("long", [0, 1])
@pytest.mark.parametrize("m,q0", [(64, 100), (64, 300), (70, 900)])
def test_maxima_that_rise_in_every_tile(ctx, monkeypatch, m, q0, long):
    """Scores grow along the keys by far more than 2^8 a tile: every tile raises the maximum, rescales O and both groups' sums."""
    monkeypatch.setenv("SGB_FLASH_LONG", str(long))
    q, k, v = _case(7, m, q0)
    q = np.repeat(q[:, ::G], G, axis=1)
    k = (k.astype(np.float32) + np.arange(q0 + m)[:, None, None] * 0.02 * q.astype(np.float32).mean(0)[::G][None]).astype(np.float16)
    assert_close(_linear(ctx, q, k, v, m, q0, 0, scale=1.0), _want(q, k, v, m, q0, 0, 1.0), what=f"rising m={m} q0={q0}")


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_values_that_are_not_finite_stay_with_the_blocks_that_see_them(ctx, monkeypatch, value):
    """The long kernel: V rows of a tile that no query of a 64-token block sees leave its bits alone."""
    monkeypatch.setenv("SGB_FLASH_LONG", "1")
    m, q0, at = 256, 130, 250  # the row of position 250 is seen by queries 120 and later
    q, k, v = _case(11, m, q0)
    clean = _linear(ctx, q, k, v, m, q0, 0)
    v2 = v.copy()
    v2[at, 1, 5] = value
    got = _linear(ctx, q, k, v2, m, q0, 0)
    assert np.array_equal(got[:64].view(np.uint32), clean[:64].view(np.uint32))
    assert np.array_equal(got[:, :G].view(np.uint32), clean[:, :G].view(np.uint32))  # the other kv head
    assert not np.any(np.isfinite(got[120:, G:, 5]))


@pytest.mark.parametrize("pieces", [1, 3])
@pytest.mark.parametrize("m,q0", [(64, 100), (64, 300), (70, 900)])
def test_maxima_more_than_the_threshold_above_the_last_tiles(ctx, monkeypatch, m, q0, pieces):
    """Keys along the queries' common direction, longer with every position: each tile's maximum is more than 2^8 above the one before, so every
    tile of every row raises it and rescales O and the sum."""
    monkeypatch.setenv("SGB_FLASH_PIECES", str(pieces))
    q, k, v = _case(7, m, q0)
    along = normal_f16(8, NKV, D).astype(np.float32)
    q = (0.05 * q.astype(np.float32) + np.repeat(along, G, axis=0)[None]).astype(np.float16)
    k = (0.05 * k.astype(np.float32) + 0.16 / D * np.arange(q0 + m)[:, None, None] * along[None]).astype(np.float16)
    for h in range(NKV * G):  # the premise, in bits
        s = q[:, h].astype(np.float64) @ k[:, h // G].astype(np.float64).T * np.log2(np.e)
        for t in range(m):
            full = (q0 + t + 1) // 64
            assert np.all(np.diff(s[t, : 64 * full].reshape(full, 64).max(1)) > 8)
    assert_close(_linear(ctx, q, k, v, m, q0, 0, scale=1.0), _want(q, k, v, m, q0, 0, 1.0), what=f"rising m={m} q0={q0} pieces={pieces}")


def test_rows_behind_the_keys_do_not_change_the_bits(ctx, monkeypatch):
    """A program keeps one K and one V of its longest context: what they could hold says nothing about the keys of a call, so for the same
    pieces a call's kernel and with it its bits must not rest on that."""
    monkeypatch.setenv("SGB_FLASH_PIECES", "1")
    m, n_kv = 2368, 16
    q, k, v = normal_f16(21, m, n_kv * G, D), normal_f16(22, m, n_kv, D), normal_f16(23, m, n_kv, D)
    up, got = ctx.buffer_from_iter, []
    for rows in (m, 16384):
        kv = [up(np.concatenate([x, np.zeros((rows - m, n_kv, D), np.float16)])) for x in (k, v)]
        out = ctx.new_buffer(m * n_kv * G * D, np.float32)
        ctx.dispatch_blocking(ctx.load_kernel("attn_prefill_flash_f16_d128"), bind(up(q), *kv, out, _step(ctx, 0)), (SCALE, 0), [n_kv, m, 1])
        got.append(out.read())
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
