"""Recorded dispatches run in the order of their data, not of their recording: random programs over slices of one buffer
(reads after writes, writes after reads, writes over writes, partial overlaps, in-place steps, dispatches that keep hidden
state, timer stamps in between) leave the bits that the same dispatches leave one by one."""
import numpy as np
import pytest

from cases import bind, normal_f16

pytestmark = pytest.mark.gpu

ROW, ROWS = 8192, 24  # f16 values; a rope "token" of 32 heads x 256


@pytest.fixture(scope="module")
def ctx():
    import super_gemma_b200 as sg

    return sg.GpuContext(0)


def _program(rng, n):
    """(kernel, slots): slots are row ranges of the big buffer, at half-row offsets so that operands overlap in part."""
    out = []
    for _ in range(n):
        kind = rng.choice(["norm", "norm", "rope", "append", "quant", "flash", "stamp"], p=[0.3, 0.2, 0.15, 0.15, 0.1, 0.05, 0.05])
        halves = [int(x) for x in rng.choice(2 * ROWS - 8, 2, replace=False)]
        out.append((str(kind), halves))
    return out


@pytest.mark.parametrize("seed", range(8))
def test_random_programs_give_the_bits_of_the_serial_order(ctx, seed):
    import super_gemma_b200 as sg

    rng = np.random.default_rng(seed)
    prog = _program(rng, 60)
    init = normal_f16(seed, ROWS * ROW).view(np.uint16)
    w = ctx.buffer_from_iter(rng.standard_normal(256).astype(np.float32))
    cs = ctx.buffer_from_iter(rng.uniform(-1, 1, 128 * 2).astype(np.float32))
    step = ctx.new_step_buffer()
    sg.StepState(pos=0, kv_len_global=64).write_to(step)
    quants, scales = ctx.new_buffer(ROW, np.int8), ctx.new_buffer(ROW // 32, np.uint16)
    f_out = ctx.new_buffer(64 * 2 * 128, np.float32)
    big = ctx.buffer_from_iter(init)
    timer = ctx.new_timer(1)
    K = {n: ctx.load_kernel(n) for n in ("rmsnorm_256", "rope_sliding_q", "kv_append_global", "kv_quant_q8", "attn_prefill_flash_f16_d128")}
    half = ROW // 2

    def run(c, stamps):
        for kind, (a, b) in prog:
            sl = lambda h, n=ROW: big.slice(h * half, h * half + n)
            if kind == "norm":
                if abs(a - b) >= 2:  # source and result apart
                    c.dispatch(K["rmsnorm_256"], bind(sl(a), w, sl(b)), None, [32, 1, 1])
            elif kind == "rope":
                c.dispatch(K["rope_sliding_q"], bind(sl(a), cs), None, [16, 1, 1])
            elif kind == "append":
                if abs(a - b) >= 1:
                    c.dispatch(K["kv_append_global"], bind(sl(a, half), sl(b, half), step), None, [16, 1, 1])
            elif kind == "quant":
                c.dispatch(K["kv_quant_q8"], bind(sl(a), scales, quants), None, [1, 1, 1])
            elif kind == "flash":
                c.dispatch(K["attn_prefill_flash_f16_d128"], bind(sl(a, 64 * 256), sl(a, 64 * 128), sl(b, 64 * 128), f_out, step), (0.1, 0), [1, 64, 1])
            elif stamps:
                timer.stamp(0)

    run(ctx, False)
    ctx.sync()
    want = [x.read() for x in (big, quants, scales, f_out)]
    graph = ctx.record_graph(lambda c: run(c, True))
    for _ in range(3):
        for x in (quants, scales, f_out):
            x.zero()
        big.write(init)
        ctx.submit_blocking(graph)
        got = [x.read() for x in (big, quants, scales, f_out)]
        for g, e in zip(got, want):
            assert np.array_equal(g.view(np.uint8), e.view(np.uint8))
