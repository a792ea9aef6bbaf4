"""Calls one behind the other, without a synchronisation between them: kernels start while their predecessors drain, over
intermediates and scratch that every call and every pass shares.  The same bits as with the device synchronised behind each
call, also when the chain is captured into a graph."""
import pytest

pytestmark = pytest.mark.gpu

HIDDEN, INTER, HEADS, KV_HEADS, HEAD_DIM, PAGE = 1024, 2048, 8, 2, 128, 16
RANK, ADAPTERS, PASSES = 16, 4, 16


class Chain:
    """One layer's calls (fused QKV and its consumer, gate, up, SwiGLU, down), the staged operators and a dense linear, without adapters
    and with them (its base then starts beside the shrink)."""

    def __init__(self, torch, ab, m, fp4):
        self.torch, self.ab, self.m, self.fp4 = torch, ab, m, fp4
        g = self.g = torch.Generator(device="cuda")
        g.manual_seed(m)
        self.slot = torch.randint(-1, ADAPTERS, (m,), generator=g, device="cuda").to(torch.int32)
        self.x = [self.normal(m, HIDDEN) for _ in range(PASSES)]
        width = (HEADS + 2 * KV_HEADS) * HEAD_DIM
        self.weights = {name: self.linear(n, k) for name, n, k in (("q", HEADS * HEAD_DIM, HIDDEN), ("k", KV_HEADS * HEAD_DIM, HIDDEN),
                        ("v", KV_HEADS * HEAD_DIM, HIDDEN), ("gate", INTER, HIDDEN), ("up", INTER, HIDDEN), ("down", HIDDEN, INTER))}
        self.dense_pool = self.pool(512, HIDDEN)
        self.w_dense, self.wq, self.wk = self.normal(512, HIDDEN, std=0.03), self.normal(HEAD_DIM, std=0.1), self.normal(HEAD_DIM, std=0.1)
        self.pos = torch.randint(0, 4096, (m,), generator=g, device="cuda").to(torch.int32)
        self.cache_at = torch.randperm(m, generator=g, device="cuda")
        self.inv_freq = (1e6 ** (-torch.arange(0, 64, 2, device="cuda", dtype=torch.float64) / 64)).float()
        # shared by every pass
        need = ab.lora_ws_bytes(m, ADAPTERS, RANK) + (ab.act_fp4_ws_bytes(m, INTER) + 255) // 256 * 256
        self.ws, self.t = torch.empty(need, dtype=torch.uint8, device="cuda"), self.zeros(m, RANK)
        self.gate, self.up, self.h, self.qkv = self.zeros(m, INTER), self.zeros(m, INTER), self.zeros(m, INTER), self.zeros(m, width)

    def normal(self, *shape, std=1.0):
        return self.torch.empty(shape, dtype=self.torch.bfloat16, device="cuda").normal_(0.0, std, generator=self.g)

    def zeros(self, *shape):
        return self.torch.zeros(shape, dtype=self.torch.bfloat16, device="cuda")

    def linear(self, n, k):
        packed = self.torch.randint(0, 256, (n, k // 2), generator=self.g, device="cuda", dtype=self.torch.uint8)
        scales = self.torch.empty((n, k // 16), device="cuda").normal_(generator=self.g).abs_().to(self.torch.float8_e4m3fn).view(self.torch.uint8)
        return n, k, packed, scales, self.pool(n, k)

    def pool(self, n, k):
        pool = self.ab.LoraPool(k, n, RANK, ADAPTERS)
        for s in range(ADAPTERS):
            pool.pack(s, self.normal(RANK, k, std=k ** -0.5), self.normal(n, RANK, std=0.05), 2.0)
        return pool

    def call(self, name, x, y, stride=None, flags=0):
        n, k, packed, scales, pool = self.weights[name]
        d = self.ab.make_linear_desc(x=x, m=self.m, k=k, n=n, y=y, out_row_stride=stride, w_packed=packed, w_scale=scales, scale2=0.01,
                                     seq_slot=self.slot, route=pool.route(), lora_t=self.t, ws=self.ws, ws_bytes=self.ws.numel(), flags=flags)
        self.ab.nvfp4_lora_linear(d)

    def outputs(self):
        pages, cache = (self.m + PAGE - 1) // PAGE, (PAGE, KV_HEADS, HEAD_DIM)
        return [dict(qkv=self.zeros(*self.qkv.shape), k_cache=self.zeros(pages, *cache), v_cache=self.zeros(pages, *cache),
                     down=self.zeros(self.m, HIDDEN), staged=self.zeros(self.m, KV_HEADS * HEAD_DIM), dense=self.zeros(self.m, 512),
                     dense_lora=self.zeros(self.m, 512))
                for _ in range(PASSES)]

    def run(self, out, behind):
        """`behind` is called behind every call of the library."""
        ab, m, act = self.ab, self.m, self.ab.FLAG_ACT_FP4 if self.fp4 else 0
        ready = act | (self.ab.FLAG_ACT_FP4_READY if self.fp4 else 0)
        width = self.qkv.shape[1]
        at = {"q": 0, "k": HEADS * HEAD_DIM, "v": (HEADS + KV_HEADS) * HEAD_DIM}
        for x, o in zip(self.x, out):
            for name in ("q", "k", "v"):
                self.call(name, x, o["qkv"].data_ptr() + 2 * at[name], width, act if name == "q" else ready)
                behind()
            base = o["qkv"].data_ptr()
            ab.qkv_norm_rope_cache_write(base, base + 2 * at["k"], base + 2 * at["v"], width, width, self.wq, self.wk, self.pos, self.inv_freq,
                                         self.cache_at, o["k_cache"], o["v_cache"], m, HEADS, KV_HEADS, HEAD_DIM, 64, PAGE, 1e-6)
            behind()
            self.call("gate", x, self.gate, flags=act)
            behind()
            self.call("up", x, self.up, flags=ready)
            behind()
            ab.silu_mul(self.gate, self.up, self.h, m, INTER)
            behind()
            self.call("down", self.h, o["down"], flags=act)
            behind()
            n, k, packed, scales, pool = self.weights["k"]
            ab.w4a16_gemm(x, packed, scales, 0.01, o["staged"], m, n, k)
            behind()
            ab.apply_lora_bgmv(pool.route(), x, o["staged"], self.slot, m, k, n, self.t)
            behind()
            d = ab.make_linear_desc(x=x, m=m, k=HIDDEN, n=512, y=o["dense"], w_bf16=self.w_dense)
            ab.nvfp4_lora_linear(d)
            behind()
            d = ab.make_linear_desc(x=x, m=m, k=HIDDEN, n=512, y=o["dense_lora"], w_bf16=self.w_dense, seq_slot=self.slot,
                                    route=self.dense_pool.route(), lora_t=self.t)
            ab.nvfp4_lora_linear(d)
            behind()


class RewrittenRouting(Chain):
    """The same, with tokens routed anew and slots coming and going in the stream behind every call: what a kernel reads of the
    routing ahead of its wait is not what it is to use."""

    def __init__(self, torch, ab, m, fp4):
        super().__init__(torch, ab, m, fp4)
        self.pools = [w[4] for w in self.weights.values()] + [self.dense_pool]
        self.slots = [torch.randint(-1, ADAPTERS, (m,), generator=self.g, device="cuda").to(torch.int32) for _ in range(5)]
        self.tables = []
        for gone in range(3):                              # slot `gone` has no adapter, the one behind it half its ranks and another scale
            version = []
            for p in self.pools:
                a, b, scale, rank = p.a_table.clone(), p.b_table.clone(), p.scale_table.clone(), p.rank_table.clone()
                a[gone] = b[gone] = 0
                scale[gone + 1], rank[gone + 1] = 1.0 + gone, RANK // 2
                version.append((a, b, scale, rank))
            self.tables.append(version)

    def rewrite(self):
        self.slot.copy_(self.slots[self.calls % len(self.slots)])
        for p, (a, b, scale, rank) in zip(self.pools, self.tables[self.calls % len(self.tables)]):
            p.a_table.copy_(a)
            p.b_table.copy_(b)
            p.scale_table.copy_(scale)
            p.rank_table.copy_(rank)
        self.calls += 1

    def run(self, out, behind):
        def both():
            behind()
            self.rewrite()
        self.calls = 0
        self.rewrite()
        super().run(out, both)


@pytest.mark.parametrize("m,fp4", [(1, False), (8, False), (16, False), (40, True), (300, False), (1100, False), (1100, True)])
def test_a_chain_without_synchronisation(cuda, atlas, m, fp4):
    _same_bits(cuda, atlas, Chain(cuda, atlas, m, fp4))


@pytest.mark.parametrize("m,fp4", [(1, False), (8, False), (40, True), (300, False), (1100, False)])
def test_a_chain_over_rewritten_routing(cuda, atlas, m, fp4):
    _same_bits(cuda, atlas, RewrittenRouting(cuda, atlas, m, fp4))


def _same_bits(cuda, atlas, chain):
    want, got, captured = chain.outputs(), chain.outputs(), chain.outputs()
    chain.run(want, cuda.cuda.synchronize)
    chain.run(got, lambda: None)
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(graph):
        chain.run(captured, lambda: None)
    for _ in range(3):
        graph.replay()
    cuda.cuda.synchronize()
    for i in range(PASSES):
        for name, w in want[i].items():
            assert cuda.isfinite(w).all() and (w != 0).any()
            assert cuda.equal(got[i][name].view(cuda.int16), w.view(cuda.int16)), (i, name)
            assert cuda.equal(captured[i][name].view(cuda.int16), w.view(cuda.int16)), (i, name, "captured")
    assert atlas.device_status() == 0
