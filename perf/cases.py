"""The work a user of this library has it do, as cases that can be timed.

A case is a dict of plain values with a "kind":

  layer    the seven projections of one transformer layer (or its attention input, or its MLP) over one batch of tokens,
           with what stands between them: the QKV consumer (prefill or decode form) and SwiGLU.  NVFP4 weights, a LoRA
           adapter per token, BF16 or FP4 activations.  The attention itself is not part of this library, so the output
           projection has an input of its own.
  linear   one fused linear call: NVFP4 or dense BF16 base plus the adapters of a mixed batch.
  staged   the operator pair of a caller that keeps base and adapters apart: `w4a16_gemm`, then `apply_lora_bgmv` (an
           adapter per token) or `apply_lora_delta` (one adapter for all rows) on its output.
  codec    what loading a checkpoint does: BF16 weight -> maximum -> tensor scale -> NVFP4, or NVFP4 -> BF16.

Sizes of the listed cases are those of the benchmark's workloads and of one decode step; draw() spreads over the models
and batches around them.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "apathy-atlas_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import atlas_b200 as ab  # noqa: E402

PAGE = 16                       # tokens per page of the K/V cache
EPS, THETA = 1e-6, 1e6
WEIGHT_RMS = math.sqrt(68.5 / 8)    # E2M1 codes uniform over 16 values, block scales |N(0,1)|

_8B = dict(hidden=4096, inter=14336, heads=32, kv_heads=8, head_dim=128)
_70B = dict(hidden=8192, inter=28672, heads=64, kv_heads=8, head_dim=128)


def listed():
    return [
        # one user, one token: the whole layer's calls at the size where latency and launches are all there is
        dict(name="decode_layer_1", kind="layer", part="all", form="decode", act="bf16", m=1, **_8B, rotary=128,
             adapters=8, max_rank=16, mixed_ranks=False, ids="uniform", none=0.0),
        # a decode batch in which every sequence has an adapter of its own, ranks 8 to 64: fused QKV and its consumer
        dict(name="decode_qkv_64", kind="layer", part="qkv", form="decode", act="bf16", m=64, **_8B, rotary=64,
             adapters=64, max_rank=64, mixed_ranks=True, ids="distinct", none=0.0),
        # a mid-sized mixed batch over an MLP-up-sized projection
        dict(name="linear_256", kind="linear", base="nvfp4", m=256, k=5120, n=17408, adapters=16, max_rank=32,
             mixed_ranks=False, ids="uniform", none=0.1),
        # the same call over an unquantised weight: a small decode batch
        dict(name="linear_dense_16", kind="linear", base="bf16", m=16, k=4096, n=4096, adapters=4, max_rank=16,
             mixed_ranks=False, ids="uniform", none=0.0),
        # a hidden size that is not a multiple of 256, and an odd batch
        dict(name="linear_odd_k_77", kind="linear", base="nvfp4", m=77, k=2880, n=2880, adapters=8, max_rank=16,
             mixed_ranks=False, ids="uniform", none=0.25),
        # a wide MLP, many small adapters with a skewed popularity, a quarter of the tokens without one
        dict(name="mlp_512", kind="layer", part="mlp", form="prefill", act="bf16", m=512, **_70B, rotary=128,
             adapters=128, max_rank=16, mixed_ranks=False, ids="zipf", none=0.25),
        # one chunk of a chunked prefill: ragged token count, mixed ranks, some sequences without an adapter
        dict(name="prefill_layer_1237", kind="layer", part="all", form="prefill", act="bf16", m=1237, **_8B, rotary=128,
             adapters=8, max_rank=64, mixed_ranks=True, ids="segments", none=0.1),
        # the largest: a full prefill batch of 32 sequences, exact activations
        dict(name="prefill_layer_8192", kind="layer", part="all", form="prefill", act="bf16", m=8192, **_8B, rotary=64,
             adapters=8, max_rank=64, mixed_ranks=False, ids="segments", none=0.0),
        # the same batch with activations quantised to FP4
        dict(name="prefill_layer_8192_fp4", kind="layer", part="all", form="prefill", act="fp4", m=8192, **_8B, rotary=64,
             adapters=8, max_rank=64, mixed_ranks=False, ids="segments", none=0.0),
        # base and adapters as separate operators: a decode batch with an adapter per token ...
        dict(name="staged_bgmv_37", kind="staged", op="bgmv", m=37, k=4096, n=4096, adapters=16, max_rank=32,
             mixed_ranks=False, ids="uniform", none=0.1),
        # ... and one adapter over the rows of a prefill
        dict(name="staged_delta_2048", kind="staged", op="delta", m=2048, k=4096, n=4096, adapters=1, max_rank=64,
             mixed_ranks=False, ids="uniform", none=0.0),
        # quantising one weight matrix at load time
        dict(name="quantize_weight", kind="codec", op="quantize", n=14336, k=4096),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _adapters(rng):
    max_rank = rng.choice((8, 16, 32, 64, 128))
    return dict(adapters=_log_int(rng, 1, min(128, 4096 // max_rank)), max_rank=max_rank, mixed_ranks=rng.random() < 0.4,
                none=rng.choice((0.0, 0.1, 0.25)))


def draw(rng):
    kind = rng.choices(("layer", "linear", "staged", "codec"), (5, 3, 2.5, 1.5))[0]
    if kind == "layer":
        form = rng.choice(("decode", "prefill"))
        head_dim = rng.choice((64, 128, 128, 256))
        heads = 256 * _log_int(rng, 4, 32) // head_dim
        hidden = heads * head_dim
        groups = [g for g in (1, 2, 4, 8) if heads % g == 0]
        case = dict(kind="layer", part=rng.choice(("all", "all", "qkv", "mlp")), form=form, act="fp4" if rng.random() < 0.25 else "bf16", m=1,
                    hidden=hidden, inter=256 * int(round(hidden * rng.uniform(2.0, 4.0) / 256)), heads=heads,
                    kv_heads=heads // rng.choice(groups), head_dim=head_dim, rotary=rng.choice((64, head_dim)), **_adapters(rng))
        # no more multiplications than the largest listed case
        most = int(8192 * _params(dict(_8B, part="all")) / _params(case))
        case["m"] = _log_int(rng, 1, 256) if form == "decode" else _log_int(rng, 128, min(8192, most))
        case["ids"] = rng.choice(("uniform", "distinct", "zipf")) if form == "decode" else "segments"
        if rng.random() < 0.1:      # the base model alone
            case.update(adapters=0, none=0.0, mixed_ranks=False)
        return case
    if kind == "linear":
        case = dict(kind="linear", base="bf16" if rng.random() < 0.25 else "nvfp4", m=1, k=256 * _log_int(rng, 4, 64), n=16 * _log_int(rng, 64, 1792),
                    **_adapters(rng))
        if rng.random() < 0.3:      # a contraction length that is a multiple of 32 only
            case["k"] = 32 * _log_int(rng, 32, 192) + 32
            case["n"] = min(case["n"], 8192)
        m_max = (1 << 32) // (case["k"] * case["n"]) if case["k"] % 256 else (1 << 38) // (case["k"] * case["n"])
        case["m"] = _log_int(rng, 1, max(1, min(4096, m_max)))
        case["ids"] = rng.choice(("uniform", "zipf", "segments"))
        return case
    if kind == "staged":
        case = dict(kind="staged", op=rng.choice(("bgmv", "delta")), m=_log_int(rng, 1, 2048), k=256 * _log_int(rng, 4, 32), n=16 * _log_int(rng, 64, 512),
                    **_adapters(rng), ids=rng.choice(("uniform", "zipf", "segments")))
        if case["op"] == "delta":
            case.update(adapters=1, none=0.0, mixed_ranks=False)
        return case
    return dict(kind="codec", op=rng.choice(("quantize", "dequant")), n=_log_int(rng, 256, 28672), k=16 * _log_int(rng, 32, 512))


# ---------------------------------------------------------------------------------------------------------------------
# shapes and work
# ---------------------------------------------------------------------------------------------------------------------
def _modules(case):
    """(name, N, K) of every projection of a layer case, in the order of the calls."""
    h, i, qw, kw = case["hidden"], case["inter"], case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"]
    attn = [("q", qw, h), ("k", kw, h), ("v", kw, h)]
    mlp = [("gate", i, h), ("up", i, h), ("down", h, i)]
    return {"all": attn + [("o", h, qw)] + mlp, "qkv": attn, "mlp": mlp}[case["part"]]


def _quantised_h(case):
    """With FP4 activations and no adapter nothing reads SwiGLU's result in BF16."""
    return case["act"] == "fp4" and case["adapters"] == 0


def _params(case):
    return sum(n * k for _, n, k in _modules(case))


def _rank(case):
    """Mean true rank of the case's adapters."""
    ranks = [r for r in (8, 16, 32, 64, 128) if r <= case["max_rank"]] if case["mixed_ranks"] else [case["max_rank"]]
    return sum(ranks) / len(ranks)


def _linear_work(case, m, n, k, base="nvfp4"):
    """(bytes of weights and adapters, flops) of one projection."""
    hit, r = min(case["adapters"], max(1, round(m * (1 - case["none"])))), _rank(case) if case["adapters"] else 0
    weights = n * k * (2 if base == "bf16" else 9 / 16) + hit * r * (k + n) * 2
    return weights, 2.0 * m * n * k + 2.0 * m * (1 - case["none"]) * r * (k + n)


def work(case):
    if case["kind"] == "codec":
        return {"bytes": case["n"] * case["k"] * (2 + 9 / 16), "flops": 0}
    m = case["m"]
    if case["kind"] in ("linear", "staged"):
        b, f = _linear_work(case, m, case["n"], case["k"], case.get("base", "nvfp4"))
        return {"bytes": b + 2.0 * m * (case["k"] + case["n"]) + 4 * m, "flops": f}
    total_b, total_f = 4.0 * m, 0.0
    for name, n, k in _modules(case):
        b, f = _linear_work(case, m, n, k)
        total_b, total_f = total_b + b + 2.0 * m * n, total_f + f        # every projection's output is written
        if name in ("q", "o", "gate"):                                   # inputs: x of q/k/v, of o, of gate/up
            total_b += 2.0 * m * k
        if name == "k":                                                  # the cache rows of K and V
            total_b += 2 * 2.0 * m * n
        if name == "down":                                               # SwiGLU's result
            total_b += (9 / 16 if _quantised_h(case) else 2.0) * m * k
    return {"bytes": total_b, "flops": total_f}


def tolerance(case):
    if case["kind"] == "codec":
        return "exact"
    # BF16 results of FP32 sums.  With FP4 activations, a value that another correct sum rounds to the next BF16 may fall
    # into the next of eight FP4 magnitudes before it is multiplied again.
    return {"rel": 2e-2 if case.get("act") == "fp4" else 1e-2}


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
class _Draw:
    """Seeded inputs on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def normal(self, *shape, std=1.0):
        return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=self.g)

    def uniform(self, *shape, limit):
        return torch.empty(shape, dtype=torch.bfloat16, device="cuda").uniform_(-limit, limit, generator=self.g)

    def integers(self, lo, hi, n):
        return torch.randint(lo, hi, (n,), generator=self.g, device="cuda")

    def nvfp4(self, n, k):
        """Codes uniform over the 16 E2M1 values, block scales E4M3(|N(0,1)|)."""
        packed = torch.empty((n, k // 2), dtype=torch.uint8, device="cuda").random_(0, 256, generator=self.g)
        scales = torch.empty((n, k // 16), dtype=torch.float32, device="cuda").normal_(generator=self.g).abs_()
        return packed, scales.to(torch.float8_e4m3fn).view(torch.uint8)

    def slots(self, case):
        """The adapter of every token, -1 for none: uniform, all different, Zipf(1.1), or contiguous sequences."""
        m, n_ad = case["m"], case["adapters"]
        if case["ids"] == "distinct":
            slot = torch.arange(m, device="cuda") % n_ad
        elif case["ids"] == "zipf":
            w = torch.arange(1, n_ad + 1, device="cuda", dtype=torch.float64) ** -1.1
            slot = torch.multinomial(w, m, replacement=True, generator=self.g)
        elif case["ids"] == "segments":
            start = self.starts(m)
            own = self.integers(0, n_ad, m)
            if case["none"]:
                own[torch.rand(m, generator=self.g, device="cuda") < case["none"]] = -1
            return own[start].to(torch.int32)
        else:
            slot = self.integers(0, n_ad, m)
        if case["none"]:
            slot[torch.rand(m, generator=self.g, device="cuda") < case["none"]] = -1
        return slot.to(torch.int32)

    def starts(self, m):
        """For every token the first token of its sequence: up to 32 sequences of random length."""
        cut = torch.zeros(m, dtype=torch.int64, device="cuda")
        cut[self.integers(0, m, min(31, m // 32))] = 1
        cut[0] = 1
        at = torch.arange(m, device="cuda")
        return torch.cummax(torch.where(cut == 1, at, 0), 0).values

    def pool(self, case, n, k, ranks):
        """One module's adapters: A uniform in +-1/sqrt(K), B ~ N(0, 0.02), scale alpha / r = 2."""
        pool = ab.LoraPool(k, n, case["max_rank"], case["adapters"])
        for s, r in enumerate(ranks):
            pool.pack(s, self.uniform(r, k, limit=k ** -0.5), self.normal(n, r, std=0.02), 2.0)
        return pool

    def ranks(self, case):
        if not case["mixed_ranks"]:
            return [case["max_rank"]] * case["adapters"]
        some = [r for r in (8, 16, 32, 64, 128) if r <= case["max_rank"]]
        return [some[i] for i in self.integers(0, len(some), case["adapters"]).tolist()]


def _scale2(k):
    """Tensor scale with which outputs have about unit variance."""
    return 1.0 / (WEIGHT_RMS * math.sqrt(k))


def _bf16(*shape):
    return torch.zeros(shape, dtype=torch.bfloat16, device="cuda")


def _desc(d, case, state, x, n, k, y, slot, ranks, ws, *, row_stride=None, flags=0, base="nvfp4"):
    """A projection's weight, adapters and call descriptor, as a program that keeps its model in memory has them."""
    kw = dict(w_bf16=d.normal(n, k, std=k ** -0.5)) if base == "bf16" else dict(zip(("w_packed", "w_scale"), d.nvfp4(n, k)), scale2=_scale2(k))
    if slot is not None:
        pool = d.pool(case, n, k, ranks)
        lora_t = _bf16(case["m"], case["max_rank"])
        state["keep"] += [pool, lora_t]
        kw.update(seq_slot=slot, route=pool.route(), lora_t=lora_t)
    state["keep"] += [x, y, slot, ws, *kw.values()]
    return ab.make_linear_desc(x=x, m=case["m"], k=k, n=n, y=y, out_row_stride=row_stride, flags=flags, ws=ws, ws_bytes=ws.numel(), **kw)


def _ws_bytes(case, k):
    need = ab.lora_ws_bytes(case["m"], case["adapters"], case["max_rank"]) if case["adapters"] else 256
    if case.get("act") == "fp4":
        need += (ab.act_fp4_ws_bytes(case["m"], k) + 255) // 256 * 256
    return need


def _prepare_layer(case, d):
    m, shapes = case["m"], {name: (n, k) for name, n, k in _modules(case)}
    slot, ranks = (d.slots(case), d.ranks(case)) if case["adapters"] else (None, None)
    s = {"case": case, "keep": [], "calls": {}, "out": {}}

    def scratch(k):
        return torch.empty(_ws_bytes(case, k), dtype=torch.uint8, device="cuda")

    fp4 = ab.FLAG_ACT_FP4 if case["act"] == "fp4" else 0
    ready = fp4 | (ab.FLAG_ACT_FP4_READY if fp4 else 0)      # a projection that reads the same x as the one before it

    if "q" in shapes:
        hidden, hd, nq, nkv = case["hidden"], case["head_dim"], case["heads"], case["kv_heads"]
        x, ws, width = d.normal(m, hidden), scratch(hidden), (nq + 2 * nkv) * hd
        qkv = _bf16(m, width)                                # one fused output, three column ranges
        at = {"q": qkv.data_ptr(), "k": qkv.data_ptr() + nq * hd * 2, "v": qkv.data_ptr() + (nq + nkv) * hd * 2}
        for name in ("q", "k", "v"):
            s["calls"][name] = _desc(d, case, s, x, *shapes[name], at[name], slot, ranks, ws, row_stride=width, flags=fp4 if name == "q" else ready)
        # paged K/V cache: a page of its own per sequence of a decode batch, consecutive tokens in a page for a prefill
        token = torch.arange(m, device="cuda")
        if case["form"] == "decode":
            pages = m
            page, offset, pos = token, d.integers(0, PAGE, m), d.integers(0, 8192, m)
        else:
            pages = (m + PAGE - 1) // PAGE
            page, offset, pos = token // PAGE, token % PAGE, token - d.starts(m)
        perm = torch.randperm(pages, generator=d.g, device="cuda")
        s.update(qkv=qkv, at=at, width=width, slots=perm[page] * PAGE + offset, pos=pos.to(torch.int32),
                 wq=d.normal(hd, std=0.1), wk=d.normal(hd, std=0.1),
                 inv_freq=(THETA ** (-torch.arange(0, case["rotary"], 2, device="cuda", dtype=torch.float64) / case["rotary"])).to(torch.float32),
                 k_cache=_bf16(pages, PAGE, nkv, hd), v_cache=_bf16(pages, PAGE, nkv, hd))
        s["out"].update(qkv=qkv, k_cache=s["k_cache"], v_cache=s["v_cache"])
    if "o" in shapes:
        n, k = shapes["o"]
        s["out"]["o"] = _bf16(m, n)
        s["calls"]["o"] = _desc(d, case, s, d.normal(m, k), n, k, s["out"]["o"], slot, ranks, scratch(k), flags=fp4)
    if "gate" in shapes:
        n, k = shapes["gate"]
        x, ws, ws_down, h = d.normal(m, k), scratch(k), scratch(n), _bf16(m, n)
        s.update(gate=_bf16(m, n), up=_bf16(m, n), h=h, ws_down=ws_down)
        s["out"].update(gate=s["gate"], up=s["up"], down=_bf16(m, k))
        if not _quantised_h(case):
            s["out"]["h"] = h
        s["calls"]["gate"] = _desc(d, case, s, x, n, k, s["gate"], slot, ranks, ws, flags=fp4)
        s["calls"]["up"] = _desc(d, case, s, x, n, k, s["up"], slot, ranks, ws, flags=ready)
        s["calls"]["down"] = _desc(d, case, s, h, *shapes["down"], s["out"]["down"], slot, ranks, ws_down, flags=ready if _quantised_h(case) else fp4)
    return s


def prepare(case, seed):
    d = _Draw(seed)
    if case["kind"] == "layer":
        return _prepare_layer(case, d)
    if case["kind"] == "codec":
        n, k = case["n"], case["k"]
        if case["op"] == "dequant":
            packed, scales = d.nvfp4(n, k)
            return {"case": case, "packed": packed, "scales": scales, "out": _bf16(n, k)}
        return {"case": case, "w": d.normal(n, k, std=k ** -0.5), "amax": torch.zeros(1, dtype=torch.float32, device="cuda"),
                "packed": torch.empty((n, k // 2), dtype=torch.uint8, device="cuda"), "scales": torch.empty((n, k // 16), dtype=torch.uint8, device="cuda")}
    m, n, k = case["m"], case["n"], case["k"]
    slot, ranks = d.slots(case), d.ranks(case)
    s = {"case": case, "keep": [], "y": _bf16(m, n)}
    if case["kind"] == "linear":
        ws = torch.empty(_ws_bytes(case, k), dtype=torch.uint8, device="cuda")
        s["call"] = _desc(d, case, s, d.normal(m, k), n, k, s["y"], slot, ranks, ws, base=case["base"])
        return s
    s["packed"], s["scales"] = d.nvfp4(n, k)
    s.update(x=d.normal(m, k), slot=slot, pool=d.pool(case, n, k, ranks), xa=_bf16(m, case["max_rank"]))
    s["route"] = s["pool"].route()
    return s


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def _run_layer(s):
    c, calls = s["case"], s["calls"]
    if "q" in calls:
        ab.nvfp4_lora_linear(calls["q"])
        ab.nvfp4_lora_linear(calls["k"])
        ab.nvfp4_lora_linear(calls["v"])
        at, width, dims = s["at"], s["width"], (c["kv_heads"], c["head_dim"], c["rotary"], PAGE, EPS)
        if c["form"] == "decode":
            ab.qkv_norm_rope_cache_write(at["q"], at["k"], at["v"], width, width, s["wq"], s["wk"], s["pos"], s["inv_freq"], s["slots"],
                                         s["k_cache"], s["v_cache"], c["m"], c["heads"], *dims)
        else:
            ab.kv_norm_rope_cache_write(at["k"], at["v"], width, s["wk"], s["pos"], s["slots"], s["k_cache"], s["v_cache"], c["m"], *dims, THETA)
    if "o" in calls:
        ab.nvfp4_lora_linear(calls["o"])
    if "gate" in calls:
        ab.nvfp4_lora_linear(calls["gate"])
        ab.nvfp4_lora_linear(calls["up"])
        if _quantised_h(c):
            ab.silu_mul_quant_nvfp4(s["gate"], s["up"], s["ws_down"], s["ws_down"].numel(), c["m"], c["inter"])
        else:
            ab.silu_mul(s["gate"], s["up"], s["h"], c["m"], c["inter"])
        ab.nvfp4_lora_linear(calls["down"])
    return s["out"]


def run(state):
    c = state["case"]
    if c["kind"] == "layer":
        return _run_layer(state)
    if c["kind"] == "linear":
        ab.nvfp4_lora_linear(state["call"])
        return state["y"]
    if c["kind"] == "staged":
        m, n, k, y = c["m"], c["n"], c["k"], state["y"]
        ab.w4a16_gemm(state["x"], state["packed"], state["scales"], _scale2(k), y, m, n, k)
        if c["op"] == "bgmv":
            ab.apply_lora_bgmv(state["route"], state["x"], y, state["slot"], m, k, n, state["xa"])
        else:
            pool = state["pool"]
            ab.apply_lora_delta(pool.a_pool[0], pool.b_pool[0], 2.0, k, n, c["max_rank"], state["x"], y, m, state["xa"])
        return y
    if c["op"] == "quantize":
        state["amax"].zero_()
        ab.nvfp4_global_absmax(state["w"], state["amax"], state["w"].numel())
        scale2 = ab.scale2_from_absmax(float(state["amax"]))
        ab.quantize_bf16_to_nvfp4(state["w"], state["packed"], state["scales"], scale2, c["n"], c["k"])
        return {"packed": state["packed"], "scales": state["scales"], "scale2": scale2}
    ab.dequant_nvfp4_to_bf16(state["packed"], state["scales"], state["out"], 1.0, c["n"], c["k"])
    return state["out"]
