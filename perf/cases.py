"""The attention path's work as a caller has it done, for timing and for comparing outputs between two builds.

Every case goes through the package's public entry points (``GpuContext.load_kernel`` / ``dispatch`` /
``record_graph`` / ``submit``, ``StepState.write_to``), on one context, the way a serving program drives them:
kernels, buffers and recorded graphs are made once, a pass only dispatches or replays.  Two geometries occur:

* head_dim 128, two query heads per kv head, paged Q8_0 cache: the shapes that ``bench.py`` quotes, and the kv-head
  slices that a rank of a sharded job owns (16, 8 or 4 kv heads);
* the reference model's own layers under the reference's kernel names: sliding layers of 32 query / 16 kv heads,
  head_dim 256 over a 1024-slot ring, global layers of 32 / 4 heads, head_dim 512 with Q8_0 keys and f16 values,
  prefilled in chunks of 256 tokens with 16 and 32 decode splits as its model graph records them.

Values are i.i.d. N(0, 1) rounded to f16 (post-norm activations), caches are filled by the package's own append.
"""
import math

import numpy as np
import torch

import super_gemma_b200 as sg

D, G, RING = 128, 2, 1024  # head_dim and query heads per kv head of the paged path; ring slots (= window) of a sliding layer
SLIDING_SPLITS, GLOBAL_SPLITS = 16, 32  # the split counts that the reference's model graph records
MOST_PAIRS = 4096 * 126976 + 4096 * 4097 // 2  # visible (query, key) pairs of the largest listed prefill


def listed():
    return [
        # One decoded token of a 16-kv-head layer early in a chat: one recorded launch sequence (norm + rope + append,
        # split-K decode, combine), replayed after the step words are written.  Latency and launches count.
        {"name": "token_1000", "kind": "token", "ctx": 1000, "kv": 16, "page": 256, "plus_one": False},
        # The same at the 32K context the benchmark quotes.
        {"name": "token_32768", "kind": "token", "ctx": 32768, "kv": 16, "page": 256, "plus_one": False},
        # A four-token draft verified against 64K cached tokens: the global layer's paged verify and combine, and the
        # sliding layer's verify over a wrapped ring; dispatched one by one, not recorded.
        {"name": "verify_65540", "kind": "decode", "ctx": 65540, "kv": 16, "page": 256, "queries": 4},
        # Decode over the longest context quoted.
        {"name": "decode_131072", "kind": "decode", "ctx": 131072, "kv": 16, "page": 256, "queries": 1},
        # A whole short prompt through a sliding layer: f16 K/V, 1024-token window, nothing cached before it.
        {"name": "prefill_window_512", "kind": "linear", "m": 512, "q0": 0, "kv": 16, "window": 1024},
        # A ragged chunk in mid-conversation through a sliding layer: ring history and chunk, then the ring append.
        {"name": "prefill_ring_1500", "kind": "ring", "m": 1500, "q0": 70001},
        # An 8192-token prompt through a global layer over the paged cache.
        {"name": "prefill_paged_8192", "kind": "paged", "m": 8192, "q0": 0, "kv": 16, "page": 256},
        # The last 4096-token chunk of a 128K prompt: the largest call.
        {"name": "prefill_paged_4096_of_131072", "kind": "paged", "m": 4096, "q0": 126976, "kv": 16, "page": 256},
        # The pre-attention step of a 4096-token chunk: norm, rope, quantise, paged append.
        {"name": "append_4096", "kind": "append", "m": 4096, "pos": 8000, "kv": 16, "page": 256, "plus_one": True},
        # One decoded token through one sliding and one global layer of the reference model, under its kernel names.
        {"name": "model_token_32768", "kind": "model_token", "ctx": 32768},
        # The reference model's 256-token prefill chunk at 8K context through a global layer: append, quantise q, int8 flash.
        {"name": "model_prefill_global_256", "kind": "model_global", "m": 256, "q0": 7936},
        # ... and through a sliding layer: ring history and chunk, then the ring append.
        {"name": "model_prefill_sliding_256", "kind": "model_sliding", "m": 256, "q0": 7936},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["token", "decode", "linear", "ring", "paged", "append", "model_token", "model_global", "model_sliding"])
    kv, page = rng.choice([16, 16, 8, 4]), rng.choice([64, 256, 512])
    if kind == "token":
        return {"kind": kind, "ctx": _log(rng, 64, 131072), "kv": kv, "page": page, "plus_one": rng.random() < 0.5}
    if kind == "decode":
        return {"kind": kind, "ctx": _log(rng, 64, 131072), "kv": kv, "page": page, "queries": rng.randint(1, 4)}
    if kind == "linear":
        return {"kind": kind, "m": _log(rng, 16, 8192), "q0": rng.choice([0, _log(rng, 64, 16384)]), "kv": kv, "window": rng.choice([0, 1024])}
    if kind == "ring":
        return {"kind": kind, "m": _log(rng, 16, 8192), "q0": _log(rng, 16, 131072)}
    if kind == "paged":
        m = _log(rng, 16, 8192)
        return {"kind": kind, "m": m, "q0": _log(rng, 16, min(122880, MOST_PAIRS // m - m)), "kv": kv, "page": page}
    if kind == "append":
        return {"kind": kind, "m": _log(rng, 1, 8192), "pos": _log(rng, 1, 65536), "kv": kv, "page": page, "plus_one": rng.random() < 0.5}
    if kind == "model_token":
        return {"kind": kind, "ctx": _log(rng, 64, 131072)}
    # the reference pads a chunk to a multiple of 64 rows
    return {"kind": kind, "m": 64 * rng.randint(1, 8), "q0": _log(rng, 16, 32768)}


# ---- what a program keeps: one context on one stream, kernel handles, device buffers --------------------------------
class _Session:
    def __init__(self):
        self.stream = torch.cuda.Stream()
        self.ctx = sg.GpuContext(torch.cuda.current_device(), stream=self.stream.cuda_stream)
        self._kernels = {}

    def kernel(self, name):
        if name not in self._kernels:
            self._kernels[name] = self.ctx.load_kernel(name)
        return self._kernels[name]


_session = None


def _open():
    global _session
    if _session is None:
        _session = _Session()
    return _session


class _State:
    """Named device tensors, their buffers, and the dispatches of one pass."""

    def __init__(self, seed):
        self.s = _open()
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.rng = np.random.default_rng(seed)
        self.t, self.b, self.calls, self.outputs = {}, {}, [], []
        self.graph = None
        self.step_words = None

    def put(self, name, tensor):
        self.t[name] = tensor
        self.b[name] = self.s.ctx.adopt(tensor.data_ptr(), tensor.numel() * tensor.element_size(), np.uint8, keep=tensor)
        return tensor

    def normal(self, name, *shape):
        return self.put(name, torch.randn(*shape, generator=self.gen, device="cuda").half())

    def zeros(self, name, *shape, dtype=torch.float16):
        return self.put(name, torch.zeros(*shape, dtype=dtype, device="cuda"))

    def norm_weight(self, name, n, plus_one):
        w = 0.1 * torch.randn(n, generator=self.gen, device="cuda")
        return self.put(name, w if plus_one else 1.0 + w)

    def cos_sin(self, name, pos, n, pairs, theta):
        """The host-filled rope table of `n` tokens from `pos`: (cos, sin) of pos * theta^(-i / pairs)."""
        at = torch.arange(pos, pos + n, device="cuda", dtype=torch.float64)[:, None]
        angle = at * torch.pow(theta, -torch.arange(pairs, device="cuda", dtype=torch.float64) / pairs)[None, :]
        return self.put(name, torch.stack([angle.cos(), angle.sin()], dim=-1).float().contiguous())

    def step(self, pos=0, sliding=0, glob=0, q0=0):
        self.step_words = sg.StepState(pos=pos, kv_len_sliding=sliding, kv_len_global=glob, q0=q0)
        self.put("step", torch.tensor([pos, sliding, glob, q0], dtype=torch.int32, device="cuda"))

    def call(self, kernel, names, push, groups):
        bindings = [sg.BufferBinding.buffer(i, self.b[n]) for i, n in enumerate(names.split())]
        self.calls.append((self.s.kernel(kernel), bindings, push, groups))

    def dispatch(self, ctx):
        for c in self.calls:
            ctx.dispatch(*c)

    def once(self, kernel, names, push, groups):
        """A dispatch of the preparation (filling a cache)."""
        torch.cuda.synchronize()
        self.s.ctx.dispatch_blocking(self.s.kernel(kernel), [sg.BufferBinding.buffer(i, self.b[n]) for i, n in enumerate(names.split())], push, groups)

    def drop(self, *names):
        for n in names:
            del self.b[n], self.t[n]

    def paged_cache(self, tokens, kv, page):
        """K and V of `tokens` tokens, Q8_0-quantised into a pool behind a shuffled page table."""
        pages = -(-tokens // page)
        row, rows = kv * D, (pages + 1) * page
        table = self.rng.permutation(pages + 1)[:pages].astype(np.int32)
        self.put("table", torch.from_numpy(table).cuda())
        self.zeros("fill_step", 4, dtype=torch.int32)
        for side in "kv":
            self.zeros(side + "q", rows * row, dtype=torch.int8)
            self.zeros(side + "s", rows * row // 32)
            self.normal("src", tokens, row)
            self.once("kv_append_paged_q8_d128", f"src {side}s {side}q table fill_step", (row, page), [1, 1, 1])
            self.drop("src")

    def ring(self, kv_dim):
        self.normal("k_ring", RING, kv_dim)
        self.normal("v_ring", RING, kv_dim)


# ---- the kinds of work -----------------------------------------------------------------------------------------------
def _token(st, ctx, kv, page, plus_one):
    heads, row = kv * G, kv * D
    st.paged_cache(ctx, kv, page)
    st.normal("q_raw", heads, D), st.normal("k_raw", row), st.normal("v_raw", row)
    st.norm_weight("q_w", D, plus_one), st.norm_weight("k_w", D, plus_one)
    st.cos_sin("cs", ctx - 1, 1, D // 2, 1e6)
    splits = st.s.ctx.decode_splits_hint(kv, ctx)
    st.zeros("q", heads, D)
    st.zeros("part", heads * splits * (D + 2), dtype=torch.float32)
    st.zeros("out", heads, D, dtype=torch.float32)
    st.step(pos=ctx - 1, glob=ctx)
    st.call("qkv_norm_rope_append_paged_q8_d128", "q_raw q_w q k_raw v_raw k_w cs ks kq vs vq table step",
            (heads, row, page, D, int(plus_one)), [1, 1, 1])
    st.call("attn_decode_paged_q8kv_d128", "q kq ks vq vs table part step", (splits, 1 / math.sqrt(D), page), [kv, splits, 1])
    st.call("attn_reduce_f32_d128", "part out", splits, [heads, 1, 1])
    st.outputs = ["out", "q", "kq", "ks", "vq", "vs"]
    return True


def _decode(st, ctx, kv, page, queries):
    heads = kv * G
    st.paged_cache(ctx, kv, page)
    st.normal("q", queries, heads, D)
    splits = st.s.ctx.decode_splits_hint(kv, ctx)
    st.zeros("part", queries * heads * splits * (D + 2), dtype=torch.float32)
    st.zeros("out", queries * heads, D, dtype=torch.float32)
    st.step(glob=ctx, q0=ctx - queries)
    st.call("attn_verify_paged_q8kv_d128" if queries > 1 else "attn_decode_paged_q8kv_d128", "q kq ks vq vs table part step",
            (splits, 1 / math.sqrt(D), page), [kv, splits, queries])
    st.call("attn_reduce_f32_d128", "part out", splits, [queries * heads, 1, 1])
    st.outputs = ["out"]
    if queries > 1:  # the draft through the sliding layer as well
        st.ring(kv * D)
        st.normal("q_sl", queries, heads, D), st.normal("k_new", queries, kv * D), st.normal("v_new", queries, kv * D)
        st.zeros("out_sl", queries, heads, D, dtype=torch.float32)
        st.call("attn_verify_sliding_ring_d128", "q_sl k_ring v_ring k_new v_new out_sl step", 1 / math.sqrt(D), [kv, queries, 1])
        st.outputs.append("out_sl")
    return False


def _linear(st, m, q0, kv, window):
    st.normal("q", m, kv * G, D), st.normal("k", q0 + m, kv, D), st.normal("v", q0 + m, kv, D)
    st.zeros("out", m, kv * G, D, dtype=torch.float32)
    st.step(pos=q0, q0=q0)
    st.call("attn_prefill_flash_f16_d128", "q k v out step", (1 / math.sqrt(D), window), [kv, m, 1])
    st.outputs = ["out"]
    return False


def _ring(st, m, q0):
    kv = 16
    st.ring(kv * D)
    st.normal("q", m, kv * G, D), st.normal("k", m, kv * D), st.normal("v", m, kv * D)
    st.zeros("out", m, kv * G, D, dtype=torch.float32)
    st.step(pos=q0, q0=q0)
    st.call("attn_prefill_sliding_ring_flash_d128", "q k_ring v_ring k v out step", 1 / math.sqrt(D), [kv, m, 1])
    _append_ring(st, "kv_append_sliding_d128", m, q0, kv * D)
    return False


def _append_ring(st, kernel, m, q0, row):
    """Attend, then append: the last RING tokens of the chunk go into the ring (at most one token per slot)."""
    st.outputs = ["out", "k_ring", "v_ring"]
    last, first = min(m, RING), q0 + m - min(m, RING)
    st.put("append_step", torch.tensor([first, 0, 0, 0], dtype=torch.int32, device="cuda"))
    for side in "kv":
        st.put(side + "_last", st.t[side][m - last:])
        st.call(kernel, f"{side}_last {side}_ring append_step", None, [-(-last * row // 256), 1, 1])


def _paged(st, m, q0, kv, page):
    total = q0 + m
    st.paged_cache(total, kv, page)
    st.normal("q", m, kv * G, D)
    padded = -(-total // 64) * 64
    st.zeros("k_lin", padded * kv * D), st.zeros("v_lin", padded * kv * D)
    st.zeros("out", m, kv * G, D, dtype=torch.float32)
    st.step(pos=q0, glob=total, q0=q0)
    st.call("attn_prefill_paged_q8kv_flash_d128", "q kq ks vq vs table k_lin v_lin out step", (1 / math.sqrt(D), page), [kv, m, 1])
    st.outputs = ["out"]
    return False


def _append(st, m, pos, kv, page, plus_one):
    heads, row = kv * G, kv * D
    pages = -(-(pos + m) // page)
    rows = (pages + 1) * page
    st.put("table", torch.from_numpy(st.rng.permutation(pages + 1)[:pages].astype(np.int32)).cuda())
    for side in "kv":
        st.zeros(side + "q", rows * row, dtype=torch.int8)
        st.zeros(side + "s", rows * row // 32)
    st.normal("q_raw", m, heads, D), st.normal("k_raw", m, row), st.normal("v_raw", m, row)
    st.norm_weight("q_w", D, plus_one), st.norm_weight("k_w", D, plus_one)
    st.cos_sin("cs", pos, m, D // 2, 1e6)
    st.zeros("q", m, heads, D)
    st.step(pos=pos)
    st.call("qkv_norm_rope_append_paged_q8_d128", "q_raw q_w q k_raw v_raw k_w cs ks kq vs vq table step",
            (heads, row, page, D, int(plus_one)), [1, 1, 1])
    st.outputs = ["q", "kq", "ks", "vq", "vs"]
    return False


def _model_cache(st, tokens):
    st.normal("src", tokens, 2048)
    st.zeros("gkq", tokens * 2048, dtype=torch.int8)
    st.zeros("gks", tokens * 64)
    st.zeros("fill_step", 4, dtype=torch.int32)
    st.once("kv_append_global_q8", "src gks gkq fill_step", None, [1, 1, 1])
    st.drop("src")
    st.normal("gv", tokens, 2048)


def _model_token(st, ctx):
    st.ring(16 * 256)
    _model_cache(st, ctx)
    st.step(pos=ctx - 1, sliding=min(ctx, RING), glob=ctx)
    for name, heads, hd in (("sq", 32, 256), ("sk", 16, 256), ("sv", 16, 256), ("gq", 32, 512), ("gk", 4, 512), ("gx", 4, 512)):
        st.normal(name + "_raw", heads, hd)
        st.zeros(name + "_n", heads, hd)
    st.norm_weight("sq_w", 256, False), st.norm_weight("sk_w", 256, False)
    st.norm_weight("gq_w", 512, False), st.norm_weight("gk_w", 512, False)
    st.put("ones", torch.ones(512, device="cuda"))
    st.cos_sin("s_cs", ctx - 1, 1, 128, 1e4), st.cos_sin("g_cs", ctx - 1, 1, 64, 1e6)
    st.zeros("s_part", 32 * SLIDING_SPLITS * 258, dtype=torch.float32), st.zeros("g_part", 32 * GLOBAL_SPLITS * 514, dtype=torch.float32)
    st.zeros("s_out", 32, 256), st.zeros("g_out", 32, 512)
    st.call("rmsnorm_256", "sq_raw sq_w sq_n", None, [32, 1, 1])
    st.call("rmsnorm_256", "sk_raw sk_w sk_n", None, [16, 1, 1])
    st.call("rmsnorm_256", "sv_raw ones sv_n", None, [16, 1, 1])
    st.call("rope_sliding_q", "sq_n s_cs", None, [16, 1, 1])
    st.call("rope_sliding_k", "sk_n s_cs", None, [8, 1, 1])
    st.call("kv_append_sliding", "sk_n k_ring step", None, [16, 1, 1])
    st.call("kv_append_sliding", "sv_n v_ring step", None, [16, 1, 1])
    st.call("attn_decode_sliding", "sq_n k_ring v_ring s_part step", (SLIDING_SPLITS, 0.0625), [16, SLIDING_SPLITS, 1])
    st.call("attn_reduce_d256", "s_part s_out", SLIDING_SPLITS, [32, 1, 1])
    st.call("rmsnorm_512", "gq_raw gq_w gq_n", None, [32, 1, 1])
    st.call("rmsnorm_512", "gk_raw gk_w gk_n", None, [4, 1, 1])
    st.call("rmsnorm_512", "gx_raw ones gx_n", None, [4, 1, 1])
    st.call("rope_global_q", "gq_n g_cs", None, [8, 1, 1])
    st.call("rope_global_k", "gk_n g_cs", None, [1, 1, 1])
    st.call("kv_append_global_q8", "gk_n gks gkq step", None, [1, 1, 1])
    st.call("kv_append_global", "gx_n gv step", None, [8, 1, 1])
    st.call("attn_decode_global_q8k", "gq_n gkq gks gv g_part step", (GLOBAL_SPLITS, 512 ** -0.5), [4, GLOBAL_SPLITS, 1])
    st.call("attn_reduce_d512", "g_part g_out", GLOBAL_SPLITS, [32, 1, 1])
    st.outputs = ["s_out", "g_out", "k_ring", "v_ring", "gkq", "gks", "gv"]
    return True


def _model_global(st, m, q0):
    total = q0 + m
    _model_cache(st, -(-total // 64) * 64)
    st.normal("q", m, 32, 512), st.normal("k", m, 2048), st.normal("v", m, 2048)
    st.zeros("qq", m * 32 * 512, dtype=torch.int8), st.zeros("qs", m * 32 * 16)
    st.zeros("out", m, 32, 512)
    st.step(pos=q0, q0=q0)
    st.call("kv_append_global_q8", "k gks gkq step", None, [-(-m * 64 // 256), 1, 1])
    st.call("kv_append_global", "v gv step", None, [m * 2048 // 256, 1, 1])
    st.call("kv_quant_q8", "q qs qq", None, [m * 2, 1, 1])
    st.call("attn_prefill_global_flash_sp_iq", "qq qs gkq gks gv out step", 512 ** -0.5, [32, m // 16, 1])
    st.outputs = ["out", "qq", "qs", "gkq", "gks", "gv"]
    return True


def _model_sliding(st, m, q0):
    st.ring(16 * 256)
    st.normal("q", m, 32, 256), st.normal("k", m, 4096), st.normal("v", m, 4096)
    st.zeros("out", m, 32, 256)
    st.step(pos=q0, q0=q0)
    st.call("attn_prefill_sliding_ring", "q k_ring v_ring k v out step", 0.0625, [16, m, 1])
    _append_ring(st, "kv_append_sliding", m, q0, 4096)
    return True


_KINDS = {"token": _token, "decode": _decode, "linear": _linear, "ring": _ring, "paged": _paged, "append": _append,
          "model_token": _model_token, "model_global": _model_global, "model_sliding": _model_sliding}


def _arguments(case):
    return {k: v for k, v in case.items() if k not in ("name", "kind")}


def prepare(case, seed):
    st = _State(seed)
    recorded = _KINDS[case["kind"]](st, **_arguments(case))
    torch.cuda.synchronize()
    if recorded:
        st.graph = st.s.ctx.record_graph(st.dispatch)
    return st


def run(state):
    if state.graph is not None:  # a recorded step: write the step words, replay
        state.step_words.write_to(state.b["step"])
        state.s.ctx.submit(state.graph)
    else:
        state.dispatch(state.s.ctx)
    return {n: state.t[n] for n in state.outputs}


# ---- the same in 64 bits, in plain torch -----------------------------------------------------------------------------
class _Plain(_State):
    """The inputs of a case without the package: no context, dispatches are dropped, caches are filled in torch."""

    class _Hint:
        @staticmethod
        def decode_splits_hint(kv, ctx):
            return 1

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.rng = np.random.default_rng(seed)
        self.t, self.b, self.outputs = {}, {}, []
        self.s = type("NoSession", (), {"ctx": self._Hint})
        self.cached = {}

    def put(self, name, tensor):
        self.t[name] = self.b[name] = tensor
        return tensor

    def call(self, kernel, names, push, groups):
        pass

    def once(self, kernel, names, push, groups):
        self.cached[names.split()[1][:-1]] = _q8(self.t["src"])  # "ks" -> k, "gks" -> gk


def _q8(x):
    """The values that Q8_0 keeps of f16 `x` (blocks of 32 along the last dim), as f64: f16 scale times whole number."""
    b = x.float().reshape(-1, 32)
    d = b.abs().amax(1, keepdim=True) * torch.tensor(1.0 / 127.0, dtype=torch.float32, device=x.device)
    whole = torch.round(b * torch.where(d > 0, 1.0 / d, torch.zeros_like(d)))
    return (d.half().double() * whole.double()).reshape(x.shape)


def _norm64(x, w, plus_one=False):
    x = x.double()
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6)
    return y if w is None else y * (w.double() + (1.0 if plus_one else 0.0))


def _rope64(x, cs):
    """x [tokens, heads, n]: pair i couples dims (i, i + n / 2); as many pairs turn as the table holds."""
    half, live = x.shape[-1] // 2, cs.shape[1]
    c, s = cs[:, None, :, 0].double(), cs[:, None, :, 1].double()
    lo, hi, y = x[..., :live], x[..., half:half + live], x.clone()
    y[..., :live], y[..., half:half + live] = lo * c - hi * s, hi * c + lo * s
    return y


def _f16(x):
    return x.half().double()


def _attention64(q, k, v, at, key_at, window=0):
    """q [m, heads, n] at positions `at`, k and v [keys, kv, n] at `key_at`: causal softmax attention in f64, scale 1 / sqrt(n)
    except head_dim 256 and 512, whose callers pass 1 / 16 and 512 ** -0.5 (the same values)."""
    m, heads, n = q.shape
    kv, out = k.shape[1], torch.empty(q.shape, dtype=torch.float64, device=q.device)
    rows = max(1, min(m, int(2e8) // k.shape[0]))
    for h in range(heads):
        kh, vh = k[:, h * kv // heads].double(), v[:, h * kv // heads].double()
        for i in range(0, m, rows):
            s = (q[i:i + rows, h].double() @ kh.T) / math.sqrt(n)
            back = at[i:i + rows, None] - key_at[None, :]
            s.masked_fill_((back < 0) | (back >= window) if window else back < 0, -math.inf)
            out[i:i + rows, h] = torch.softmax(s, -1) @ vh
    return out


def _range(a, b):
    return torch.arange(a, b, device="cuda")


def _over_ring(st, q, kn, vn, q0, n, ring=("k_ring", "v_ring")):
    """Sliding attention of a chunk from position q0: the ring holds what came before it."""
    m, first = q.shape[0], max(0, q0 - RING)
    slots, at = _range(first, q0) % RING, _range(first, q0 + m)
    k, v = (torch.cat([st.t[r][slots], new.reshape(m, -1)]).reshape(len(at), -1, n) for r, new in zip(ring, (kn, vn)))
    return _attention64(q, k, v, _range(q0, q0 + m), at, RING)


def _after_append(ring, new, q0):
    last = min(new.shape[0], RING)
    r = ring.double()
    r[_range(q0 + new.shape[0] - last, q0 + new.shape[0]) % RING] = new[new.shape[0] - last:].double().reshape(last, -1)
    return r


def exact(case, seed):
    """What `run` returns, from the same inputs, in f64.  Values that the path stores as f16 or Q8_0 between its steps (normed
    and rotated heads, caches) are stored so here too; quantised bytes and scales have no 64-bit value (None)."""
    st = _Plain(seed)
    c, kind = _arguments(case), case["kind"]
    _KINDS[kind](st, **c)
    t, out = st.t, {n: None for n in st.outputs}
    if kind in ("token", "append"):
        m, kv, pos = c.get("m", 1), c["kv"], c.get("pos", c.get("ctx", 1) - 1)
        q = _norm64(t["q_raw"].reshape(m, -1, D), t["q_w"], c["plus_one"])
        if kind == "append":
            out["q"] = _rope64(q, t["cs"])
            return out
        k = _f16(_rope64(_f16(_norm64(t["k_raw"].reshape(1, kv, D), t["k_w"], c["plus_one"])), t["cs"]))
        v = _f16(_norm64(t["v_raw"].reshape(1, kv, D), None))
        out["q"] = _rope64(_f16(q), t["cs"]).reshape(-1, D)
        keys, values = (torch.cat([st.cached[n][:pos], _q8(x.reshape(1, -1).half())]).reshape(-1, kv, D) for n, x in (("k", k), ("v", v)))
        out["out"] = _attention64(_f16(out["q"])[None], keys, values, _range(pos, pos + 1), _range(0, pos + 1))[0]
        return out
    if kind in ("decode", "paged"):
        kv, total = c["kv"], c["ctx"] if kind == "decode" else c["q0"] + c["m"]
        m = t["q"].shape[0]
        k, v = (st.cached[n].reshape(total, kv, D) for n in "kv")
        out["out"] = _attention64(t["q"], k, v, _range(total - m, total), _range(0, total))
        if kind == "decode":
            out["out"] = out["out"].reshape(-1, D)
            if m > 1:
                out["out_sl"] = _over_ring(st, t["q_sl"], t["k_new"], t["v_new"], total - m, D)
        return out
    if kind == "linear":
        out["out"] = _attention64(t["q"], t["k"], t["v"], _range(c["q0"], c["q0"] + c["m"]), _range(0, c["q0"] + c["m"]), c["window"])
        return out
    if kind in ("ring", "model_sliding"):
        out["out"] = _over_ring(st, t["q"], t["k"], t["v"], c["q0"], D if kind == "ring" else 256)
        out["k_ring"], out["v_ring"] = _after_append(t["k_ring"], t["k"], c["q0"]), _after_append(t["v_ring"], t["v"], c["q0"])
        return out
    if kind == "model_global":
        m, q0 = c["m"], c["q0"]
        k = torch.cat([st.cached["gk"][:q0], _q8(t["k"])]).reshape(-1, 4, 512)
        out["gv"] = t["gv"].double()
        out["gv"][q0:q0 + m] = t["v"].double()
        out["out"] = _attention64(_q8(t["q"]), k, out["gv"][:q0 + m].reshape(-1, 4, 512), _range(q0, q0 + m), _range(0, q0 + m))
        return out
    # model_token
    pos = c["ctx"] - 1
    n = {x: _f16(_norm64(t[x + "_raw"], t[x + "_w"] if x[1] in "qk" else None)) for x in ("sq", "sk", "sv", "gq", "gk", "gx")}
    for x in ("sq", "sk", "gq", "gk"):
        n[x] = _f16(_rope64(n[x][None], t[x[0] + "_cs"]))[0]
    out["s_out"] = _over_ring(st, n["sq"][None], n["sk"], n["sv"], pos, 256)[0]
    out["k_ring"], out["v_ring"] = _after_append(t["k_ring"], n["sk"].reshape(1, -1), pos), _after_append(t["v_ring"], n["sv"].reshape(1, -1), pos)
    out["gv"] = t["gv"].double()
    out["gv"][pos] = n["gx"].reshape(-1)
    keys = torch.cat([st.cached["gk"][:pos], _q8(n["gk"].reshape(1, -1).half())]).reshape(-1, 4, 512)
    out["g_out"] = _attention64(n["gq"][None], keys, out["gv"].reshape(-1, 4, 512), _range(pos, pos + 1), _range(0, pos + 1))[0]
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _pairs(m, q0, window=0):
    """Visible (query, key) pairs of m queries from q0 under the causal mask and the window."""
    if not window:
        return m * q0 + m * (m + 1) // 2
    full = max(0, min(m, q0 + m - window + 1))  # queries that see a whole window
    rest = m - full
    return full * window + rest * q0 + rest * (rest + 1) // 2


def work(case):
    c, kind = _arguments(case), case["kind"]
    if kind in ("token", "decode"):
        kv, ctx, n = c["kv"], c["ctx"], c.get("queries", 1)
        b = 2 * ctx * kv * (D + D // 16) + n * kv * G * D * (2 + 4)
        f = 4 * D * kv * G * _pairs(n, ctx - n)
        if kind == "token":
            b += kv * G * D * 2 + kv * D * 2 * 2 + 2 * kv * (D + D // 16)
        elif n > 1:
            b += 2 * (min(ctx - n, RING) + n) * kv * D * 2 + n * kv * G * D * (2 + 4)
            f += 4 * D * kv * G * _pairs(n, ctx - n, RING)
        return {"bytes": b, "flops": f}
    if kind in ("linear", "ring", "paged"):
        m, q0, kv = c["m"], c["q0"], c.get("kv", 16)
        window = RING if kind == "ring" else c.get("window", 0)
        keys = m + (min(q0, window - 1) if window else q0)
        per_key = 2 * kv * (D + D // 16) if kind == "paged" else 2 * kv * D * 2
        b = m * kv * G * D * (2 + 4) + keys * per_key
        if kind == "ring":
            b += 2 * min(m, RING) * kv * D * 2
        return {"bytes": b, "flops": 4 * D * kv * G * _pairs(m, q0, window)}
    if kind == "append":
        m, kv = c["m"], c["kv"]
        return {"bytes": m * (kv * G * D * 4 + 2 * kv * (2 * D + D + D // 16) + D * 4), "flops": m * kv * (G + 2) * D * 10}
    if kind == "model_token":
        n = min(c["ctx"], RING)
        return {"bytes": 2 * n * 4096 * 2 + c["ctx"] * 2048 * (1 + 1 / 16 + 2) + 32 * (256 + 512) * 4,
                "flops": 4 * 32 * (256 * n + 512 * c["ctx"])}
    m, q0 = c["m"], c["q0"]
    if kind == "model_global":
        b = (q0 + m) * 2048 * (1 + 1 / 16 + 2) + m * 2048 * (4 + 1 + 1 / 16 + 2) + m * 32 * 512 * (2 + 1 + 1 / 16 + 2)
        return {"bytes": b, "flops": 4 * 512 * 32 * _pairs(m, q0)}
    b = 2 * (m + min(q0, RING - 1)) * 4096 * 2 + m * 32 * 256 * (2 + 2) + 2 * min(m, RING) * 4096 * 2
    return {"bytes": b, "flops": 4 * 256 * 32 * _pairs(m, q0, RING)}


def tolerance(case):
    """About four times the error measured against the same path in float64 on each listed case (relative 2-norm error, largest
    error over the result's rms), rounded.  Quantised bytes and page placement are exact in every case."""
    kind = case["kind"]
    if kind in ("token", "decode"):
        # P and P * scale are f16 (5.4e-4 at 1000 tokens).  At long contexts the softmax of such values is nearly flat: the
        # output shrinks with 1 / sqrt(ctx) while the sums of P * (quant + offset) that it is the small difference of grow
        # with ctx, in f32: 2.6e-3 at 32768 tokens, 7.3e-3 at 65540, 2.2e-2 at 131072.
        r = max(2e-3, 0.09 * (case["ctx"] / 131072) ** 1.5)
        return {"rel": r, "max": 4 * r}
    if kind in ("linear", "ring", "paged"):
        return {"rel": 1.5e-3, "max": 5e-2}  # P in f16: 1.5e-4 to 3.8e-4, largest 1.3e-2
    if kind == "append":
        return {"rel": 1.2e-3, "max": 6e-3}  # f16 after the norm and again after the rotation: 2.9e-4, largest 1.6e-3
    return {"rel": 8e-4, "max": 2e-3}        # the reference's layers store f16: 2.1e-4, largest 4.9e-4
