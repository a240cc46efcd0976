"""The work that a program gives this framework on one GPU, as timed cases.

Seven kinds of call, each with the values that it meets in use:

  decode   one token for each of `batch` sequences through `TPLlamaDecoder` (CUDA graph), contexts of different lengths
  prefill  `TPLlamaDecoder.prefill` of `batch` prompts of `seq` random ids
  mlp      forward and backward of `ParallelMLP` (bf16): the linear layers of tensor-parallel training
  gemm     `ops.gemm_bf16_tn`, the tcgen05 GEMM on its own
  moe      `ops.moe_dispatch` and `ops.moe_combine` around the experts of a mixture-of-experts layer
  fsdp     one full-shard training step (forward, backward with recomputation, gradient shards) of `FullyShardedSequential`
  c10d     one of each collective that data-parallel training issues, through `torch.distributed` on backend "ccl"

The process group has one rank: that is what one GPU can time. Its collectives take the same host path as those of a larger group
(checks, stream fork and join, Work, watchdog), and its fused kernels are the kernels of a larger group without the wait for peers.
"""
import math

import torch
import torch.distributed as dist
import torch.nn as nn
import torch.nn.functional as F

import oneccl_bindings_for_pytorch  # noqa: F401  (registers backend "ccl")
from torch_ccl_b200 import ops
from torch_ccl_b200.models.llama import LlamaConfig, TPLlamaDecoder
from torch_ccl_b200.parallel.fsdp import FullyShardedSequential
from torch_ccl_b200.parallel.tensor_parallel import ParallelMLP

BF16 = torch.bfloat16
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32, "i64": torch.int64}


def listed():
    llama = dict(hidden=4096, heads=32, kv_heads=32, inter=11008, vocab=32000)  # the 7B architecture of the benchmark
    gqa = dict(hidden=4096, heads=32, kv_heads=8, inter=14336, vocab=32003)      # grouped-query heads, a vocabulary with added ids
    return [
        # gradients of a small bucket: a 14336-element all_reduce is the decode-shaped message of the all_reduce benchmark
        dict(name="c10d_14336", kind="c10d", numel=14336, dtype="bf16"),
        # an interactive request on a small draft model: nothing but launches and latency
        dict(name="decode_tiny_b1", kind="decode", layers=2, hidden=512, heads=4, kv_heads=4, inter=1408, vocab=1024, batch=1, context=40, ragged=False),
        # one user on the full 7B model
        dict(name="decode_7b_b1", kind="decode", layers=32, batch=1, context=1024, ragged=False, **llama),
        # the headline of bench.py: 16 users
        dict(name="decode_7b_b16", kind="decode", layers=32, batch=16, context=1024, ragged=False, **llama),
        # a busy server: many sequences of very different lengths, grouped-query attention
        dict(name="decode_gqa_b33", kind="decode", layers=8, batch=33, context=2999, ragged=True, **gqa),
        # the prompts of bench.py (16 x 1024 ids) through a quarter of the layers
        dict(name="prefill_7b_16x1024", kind="prefill", layers=8, batch=16, seq=1024, **llama),
        # a few prompts of an odd length
        dict(name="prefill_gqa_3x777", kind="prefill", layers=4, batch=3, seq=777, **gqa),
        # the feed-forward block of a training step, one long sequence
        dict(name="mlp_8192", kind="mlp", tokens=8192, hidden=4096, inter=11008),
        # a short ragged micro-batch of a smaller model
        dict(name="mlp_1000", kind="mlp", tokens=1000, hidden=2048, inter=5504),
        # a projection with fp32 results and sizes that no tile divides
        dict(name="gemm_3000x5000x2048", kind="gemm", m=3000, n=5000, k=2048, out="f32"),
        # the Mixtral shape of the MoE benchmark: 8 experts, top 2, 4096 tokens
        dict(name="moe_4096", kind="moe", tokens=4096, hidden=4096, experts=8, topk=2),
        # two layers of the 7B model, sequence length 2048, as in the full-shard benchmark
        dict(name="fsdp_7b_2l", kind="fsdp", layers=2, hidden=4096, heads=32, inter=11008, seq=2048),
    ]


# ---- drawn cases -------------------------------------------------------------------------------------

def _log(rng, lo, hi, step=1):
    """A whole number between lo and hi, evenly spread over its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def _llama(rng):
    heads = rng.choice([4, 8, 12, 16, 24, 32, 40])
    kv = heads // rng.choice([g for g in (1, 1, 2, 4, 8) if heads % g == 0])
    return dict(hidden=heads * 128, heads=heads, kv_heads=kv, inter=_log(rng, 512, 14336, 8), vocab=_log(rng, 1000, 64000))


def _draw(rng, kind):
    if kind == "decode":
        return dict(kind=kind, layers=_log(rng, 1, 32), batch=_log(rng, 1, 128), context=_log(rng, 1, 4000), ragged=rng.random() < 0.5, **_llama(rng))
    if kind == "prefill":
        return dict(kind=kind, layers=_log(rng, 1, 8), batch=_log(rng, 1, 16), seq=_log(rng, 16, 4000), **_llama(rng))
    if kind == "mlp":
        return dict(kind=kind, tokens=_log(rng, 16, 8192) if rng.random() < 0.5 else _log(rng, 128, 8192, 128),
                    hidden=_log(rng, 512, 5120, 8), inter=_log(rng, 1024, 14336, 16))
    if kind == "gemm":
        return dict(kind=kind, m=_log(rng, 16, 8192), n=_log(rng, 16, 16384), k=_log(rng, 64, 16384, 8), out=rng.choice(["bf16", "f32"]))
    if kind == "moe":
        return dict(kind=kind, tokens=_log(rng, 16, 8192), hidden=_log(rng, 512, 8192, 8), experts=rng.choice([4, 8, 16, 64]), topk=rng.choice([1, 2, 4]))
    if kind == "fsdp":
        heads = rng.choice([4, 8, 16, 32])
        return dict(kind=kind, layers=rng.choice([1, 2, 3]), hidden=heads * 128, heads=heads, inter=_log(rng, 1024, 14336, 8), seq=_log(rng, 64, 2048))
    return dict(kind="c10d", numel=_log(rng, 16, 1 << 24), dtype=rng.choice(sorted(DTYPES)))


def _cost(case):
    w = work(case)
    return w["bytes"] / 6e12 + w["flops"] / 1e15


def draw(rng):
    kind = rng.choice(["decode", "prefill", "mlp", "gemm", "moe", "fsdp", "c10d"])
    most = max(_cost(c) for c in listed() if c["kind"] == kind)
    if kind in ("gemm", "moe", "c10d"):  # listed at an ordinary size: these go up to what the other kinds cost
        most = max(_cost(c) for c in listed())
    while True:
        c = _draw(rng, kind)
        if _cost(c) <= most and (kind != "moe" or c["tokens"] * c["topk"] * c["hidden"] * 2 <= 200 << 20):
            return c


# ---- the group and the inputs --------------------------------------------------------------------------

def _group():
    """The process group of the program; made once, as a program does."""
    if not dist.is_initialized():
        torch.cuda.set_device(0)
        dist.init_process_group("ccl", store=dist.HashStore(), rank=0, world_size=1)
    return dist.group.WORLD


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(gen, *shape, std=1.0, dtype=BF16):
    return (torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * std).to(dtype)


def _model(case, seed, max_seq):
    cfg = LlamaConfig(vocab=case["vocab"], hidden=case["hidden"], n_layers=case["layers"], n_heads=case["heads"],
                      n_kv_heads=case["kv_heads"], inter=case["inter"])
    m = TPLlamaDecoder(cfg, max_batch=case["batch"], max_seq=max_seq, seed=seed)
    # A trained model is mostly sure of its next token; one of random weights is not, and rounding would decide it. Here
    # each token has its own successor: the output head holds the embedding of the token before, in another order.
    g = _gen(seed + 17)
    table = _randn(g, cfg.vocab, cfg.hidden, std=4.0)
    before = torch.randperm(cfg.vocab, generator=g, device="cuda")
    m.embed.copy_(table)
    m.lm_head.copy_(ops.pack_weight(table[before] * (0.02 / 4.0)))
    return m, g


class _Norm(nn.Module):
    def __init__(self, d):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(d))

    def forward(self, x):
        return F.rms_norm(x, (x.shape[-1],), self.weight, 1e-5)


class _Block(nn.Module):
    """A Llama layer as a training program writes it."""

    def __init__(self, d, heads, ffn):
        super().__init__()
        self.heads = heads
        self.n1, self.n2 = _Norm(d), _Norm(d)
        self.qkv, self.o = nn.Linear(d, 3 * d, bias=False), nn.Linear(d, d, bias=False)
        self.gu, self.down = nn.Linear(d, 2 * ffn, bias=False), nn.Linear(ffn, d, bias=False)

    def forward(self, x):
        b, s, d = x.shape
        q, k, v = self.qkv(self.n1(x)).view(b, s, 3, self.heads, d // self.heads).unbind(2)
        a = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), is_causal=True)
        x = x + self.o(a.transpose(1, 2).reshape(b, s, d))
        g, u = self.gu(self.n2(x)).chunk(2, -1)
        return x + self.down(F.silu(g) * u)


def prepare(case, seed):
    kind = case["kind"]
    group = _group()
    if kind == "decode":
        ctx, b = case["context"], case["batch"]
        m, g = _model(case, seed, (ctx + 1 + 255) // 256 * 256)
        for layer in m.layers:  # what earlier tokens left in the caches
            layer["k"].normal_(generator=g)
            layer["v"].normal_(generator=g)
        pos = torch.full((b,), ctx, device="cuda", dtype=torch.int32)
        if case["ragged"]:  # the sequences of a server are at different places: one at the longest context, the others before it
            pos[1:] = torch.randint(0, ctx + 1, (b - 1,), generator=g, device="cuda", dtype=torch.int32)
        tok = torch.randint(0, case["vocab"], (b,), generator=g, device="cuda")
        m.positions.copy_(pos)
        m.tokens.copy_(tok)
        m.capture(b)
        return dict(case=case, model=m, pos=pos, tok=tok)
    if kind == "prefill":
        m, g = _model(case, seed, (case["seq"] + 255) // 256 * 256)
        prompt = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=torch.Generator().manual_seed(seed))
        return dict(case=case, model=m, prompt=prompt)
    g = _gen(seed)
    if kind == "mlp":
        mlp = ParallelMLP(case["hidden"], case["inter"], group=group, seed=seed, device="cuda", dtype=BF16)
        x = _randn(g, case["tokens"], case["hidden"]).requires_grad_()
        dy = _randn(g, case["tokens"], case["hidden"])
        return dict(case=case, mlp=mlp, x=x, dy=dy)
    if kind == "gemm":
        return dict(case=case, a=_randn(g, case["m"], case["k"]), b=_randn(g, case["n"], case["k"], std=0.02))
    if kind == "moe":
        t, e, k = case["tokens"], case["experts"], case["topk"]
        score = torch.randn(t, e, generator=g, device="cuda") + 0.3 * torch.randn(e, generator=g, device="cuda")  # some experts are busier
        w, idx = torch.topk(torch.softmax(score, -1), k, dim=-1)
        return dict(case=case, x=_randn(g, t, case["hidden"]), idx=idx.to(torch.int32).contiguous(),
                    gate=(w / w.sum(-1, keepdim=True)).contiguous(), group=group)
    if kind == "fsdp":
        torch.manual_seed(seed)
        with torch.device("cuda"):
            mods = [_Block(case["hidden"], case["heads"], case["inter"]) for _ in range(case["layers"])]
        for mod in mods:
            for p in mod.parameters():
                if p.dim() > 1:
                    nn.init.normal_(p, std=0.02)
        engine = FullyShardedSequential(mods, group=group)
        x = _randn(g, 1, case["seq"], case["hidden"]).requires_grad_()
        return dict(case=case, engine=engine, x=x, dy=_randn(g, 1, case["seq"], case["hidden"], std=0.01))
    dt = DTYPES[case["dtype"]]
    n = case["numel"]

    def vec():
        return torch.randint(-1000, 1000, (n,), generator=g, device="cuda") if dt == torch.int64 else _randn(g, n, dtype=dt)

    return dict(case=case, group=group, t=[vec() for _ in range(5)], out=[torch.empty(n, device="cuda", dtype=dt) for _ in range(3)])


# ---- one pass --------------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "decode":
        m, b = state["model"], case["batch"]
        m.positions.copy_(state["pos"])  # a server sets which sequences are in the batch and where they are
        m.tokens.copy_(state["tok"])
        ids = m.decode_step(b)
        every = max(1, case["layers"] // 8)  # caches: of a deep model those of eight layers
        return dict(ids=ids, logits=m.logits, positions=m.positions,
                    caches=[layer[c] for layer in m.layers[every - 1::every] for c in ("k", "v")])
    if kind == "prefill":
        m = state["model"]
        m.prefill(state["prompt"])
        return dict(tokens=m.tokens, positions=m.positions, caches=[layer[c] for layer in m.layers for c in ("k", "v")])
    if kind == "mlp":
        mlp, x = state["mlp"], state["x"]
        x.grad = mlp.up.weight.grad = mlp.down.weight.grad = None
        y = mlp(x)
        y.backward(state["dy"])
        return dict(y=y.detach(), dx=x.grad, dw_up=mlp.up.weight.grad, dw_down=mlp.down.weight.grad)
    if kind == "gemm":
        return ops.gemm_bf16_tn(state["a"], state["b"], out_dtype=DTYPES[case["out"]])
    if kind == "moe":
        x = state["x"]
        rows, meta, count = ops.moe_dispatch(x, state["idx"], case["experts"], case["tokens"] * case["topk"], group=state["group"])
        # here a program runs its experts on `rows`; their order is free, so what is compared is what comes back
        out = ops.moe_combine(rows, meta, count, state["gate"], group=state["group"])
        return dict(out=out, count=count)
    if kind == "fsdp":
        engine, x = state["engine"], state["x"]
        engine.after_step()  # the optimiser has just updated the master shards
        x.grad = None
        y = engine(x)
        y.backward(state["dy"])
        masters = engine.master_params()
        return dict(y=y.detach(), dx=x.grad, grads=[p.grad for p in masters], shards=[u.shard for u in engine.units])
    g, t, out = state["group"], state["t"], state["out"]
    dist.broadcast(t[0], 0, group=g)
    dist.all_reduce(t[1], group=g)
    dist.all_gather_into_tensor(out[0], t[2], group=g)
    dist.reduce_scatter_tensor(out[1], t[3], group=g)
    dist.all_to_all_single(out[2], t[4], group=g)
    return dict(broadcast=t[0], all_reduce=t[1], all_gather=out[0], reduce_scatter=out[1], all_to_all=out[2])


# ---- what a pass cannot do without -------------------------------------------------------------------------

def _params(c):
    """Weights of one layer, and of the output head."""
    hd = 128
    return (c["heads"] + 2 * c["kv_heads"]) * hd * c["hidden"] + c["heads"] * hd * c["hidden"] + 3 * c["inter"] * c["hidden"], c["vocab"] * c["hidden"]


def work(case):
    kind = case["kind"]
    if kind == "decode":
        layer, head = _params(case)
        b = case["batch"]
        ctx = case["context"] * ((1 + (b - 1) / 2) / b if case["ragged"] else 1) + 1
        cache = 2 * b * ctx * case["kv_heads"] * 128
        weights = layer * case["layers"] + head
        return dict(bytes=2 * (weights + cache * case["layers"]) + 4 * b * case["vocab"],
                    flops=2 * b * weights + case["layers"] * 4 * b * ctx * case["heads"] * 128)
    if kind == "prefill":
        layer, head = _params(case)
        b, s = case["batch"], case["seq"]
        cache = 2 * b * s * case["kv_heads"] * 128
        return dict(bytes=2 * (layer * case["layers"] + head + cache * case["layers"] + b * s * case["hidden"]),
                    flops=2 * b * s * layer * case["layers"] + case["layers"] * 2 * b * s * s * case["heads"] * 128 + 2 * b * head)
    if kind == "mlp":
        t, h, i = case["tokens"], case["hidden"], case["inter"]
        return dict(bytes=2 * (4 * t * h + 4 * h * i), flops=12 * t * h * i)
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return dict(bytes=2 * (m * k + n * k) + (2 if case["out"] == "bf16" else 4) * m * n, flops=2 * m * n * k)
    if kind == "moe":
        t, h, k = case["tokens"], case["hidden"], case["topk"]
        return dict(bytes=2 * (2 * t * h + 2 * t * k * h) + t * k * 8, flops=2 * t * k * h)
    if kind == "fsdp":
        h, i, s, n = case["hidden"], case["inter"], case["seq"], case["layers"]
        p = 4 * h * h + 3 * h * i + 2 * h
        # parameters from their master shard, gradients to their shard in fp32; forward, recomputation, two products of backward
        return dict(bytes=n * p * (4 + 2 + 4) + 2 * 4 * s * h, flops=n * (8 * p * s + 4 * 2 * s * s * h))
    size = torch.empty(0, dtype=DTYPES[case["dtype"]]).element_size()
    return dict(bytes=3 * 2 * case["numel"] * size, flops=0)  # with one rank three of the five move data


def tolerance(case):
    kind = case["kind"]
    if kind == "c10d":
        return "exact"
    if kind == "gemm":
        # fp32 sums of exact products, then rounded to the type of the result
        return dict(rel=1e-5) if case["out"] == "f32" else dict(rel=3e-3)
    if kind == "moe":
        return dict(rel=3e-3)  # one rounding to bf16
    return dict(rel=1e-2)      # bf16 between the operations
