"""The work a program gives this library on one GPU, as cases that can be timed and compared.

Each case names a public entry point (``kind``) and its sizes.  What runs on several GPUs only
(the collectives between ranks, the fused all-gather / reduce-scatter transfers) is not here: on
one GPU its ranks exist only as the test suite's emulation, which no program uses.  The same entry
points with a communicator of one rank are what a single-GPU job runs, and they are here.

``prepare`` makes the inputs of a case from a seed, ``run`` makes one pass through the entry
points, ``exact`` computes the same outputs in 64-bit floating point with plain torch.
"""
import math

import torch
import torch.nn.functional as F

from asystem_amem_b200 import Communicator, get_unique_id
from asystem_amem_b200.models import TPMLP, LlamaConfig, LlamaDecoder, MoELayer
from asystem_amem_b200.models.llama import rope_tables
from asystem_amem_b200.ops import MoeDispatcher, gemm_bf16
from asystem_amem_b200.parallel import FSDP, ShardedAdamW

BF16 = torch.bfloat16


def listed():
    return [
        # The gate / up projection of the 70B-shape MLP at tensor parallelism 8 (8192 -> 2 * 28672 / 8):
        # a decode step of 16 sequences ...
        {"name": "linear_decode", "kind": "linear", "M": 16, "N": 7168, "K": 8192},
        # ... a prompt chunk of odd length through the up projection alone ...
        {"name": "linear_ragged", "kind": "linear", "M": 1000, "N": 3584, "K": 8192},
        # ... and a full prefill or training batch of 8192 tokens.
        {"name": "linear_prefill", "kind": "linear", "M": 8192, "N": 7168, "K": 8192},
        # The tensor-parallel SwiGLU block of the 8B-shape decoder, both directions.
        {"name": "mlp_infer", "kind": "mlp", "T": 500, "dim": 4096, "ffn": 14336, "train": False},
        {"name": "mlp_train", "kind": "mlp", "T": 4096, "dim": 4096, "ffn": 14336, "train": True},
        # One expert-parallel rank's share of a mixture-of-experts layer (8 local experts of
        # 4096 x 1536): a decode step, a prefill, a training step.
        {"name": "moe_decode", "kind": "moe", "T": 32, "E": 8, "k": 2, "d": 4096, "ffn": 1536, "train": False},
        {"name": "moe_prefill", "kind": "moe", "T": 8192, "E": 8, "k": 2, "d": 4096, "ffn": 1536, "train": False},
        {"name": "moe_train", "kind": "moe", "T": 4096, "E": 8, "k": 2, "d": 4096, "ffn": 1536, "train": True},
        # Expert dispatch and combine alone at the full routing fan-out (64 experts, top-8, 16384 tokens).
        {"name": "moe_exchange", "kind": "exchange", "T": 16384, "E": 64, "k": 8, "d": 4096},
        # A sharded-data-parallel training step of a small decoder, optimizer included.
        {"name": "fsdp_step", "kind": "fsdp", "B": 2, "S": 1024, "dim": 2048, "layers": 2, "heads": 16, "kv": 4, "ffn": 7168, "vocab": 32768},
        # The gradient and parameter exchange of one shard unit: all-reduce, scaled and widened reduce-scatter, all-gather.
        {"name": "grad_exchange", "kind": "grads", "count": 50_000_003},
        # The library's reason to be: device memory handed back and restored, contents kept.
        {"name": "pause_resume", "kind": "pause", "mib": 256},
    ]


def _log_int(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "mlp", "mlp_train", "moe", "moe_train", "exchange", "fsdp", "grads", "pause"])
    if kind == "linear":
        return {"kind": kind, "M": _log_int(rng, 1, 8192), "N": _log_int(rng, 64, 8192, 8), "K": _log_int(rng, 64, 8192, 8)}
    if kind.startswith("mlp"):
        train = kind == "mlp_train"
        return {"kind": "mlp", "T": _log_int(rng, 32 if train else 1, 4096), "dim": _log_int(rng, 512, 4096, 64),
                "ffn": _log_int(rng, 1024, 14336, 64), "train": train}
    if kind.startswith("moe"):
        train = kind == "moe_train"
        return {"kind": "moe", "T": _log_int(rng, 32 if train else 1, 4096), "E": rng.choice([8, 16]), "k": rng.choice([1, 2, 4]),
                "d": _log_int(rng, 512, 4096, 64), "ffn": _log_int(rng, 128, 1024, 32), "train": train}
    if kind == "exchange":
        return {"kind": kind, "T": _log_int(rng, 1, 16384), "E": rng.choice([8, 16, 32, 64]), "k": rng.choice([1, 2, 4, 6, 8]),
                "d": _log_int(rng, 128, 4096, 8)}
    if kind == "fsdp":
        heads = rng.choice([8, 12, 16])
        return {"kind": kind, "B": rng.choice([1, 2]), "S": _log_int(rng, 128, 1024), "dim": heads * 128, "layers": 2, "heads": heads,
                "kv": rng.choice([2, 4]), "ffn": _log_int(rng, 1024, 6144, 64), "vocab": _log_int(rng, 4096, 32000, 64)}
    if kind == "grads":
        return {"kind": kind, "count": _log_int(rng, 1000, 50_000_000)}
    return {"kind": kind, "mib": _log_int(rng, 8, 250)}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, std=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * std).to(BF16)


class _Comm(Communicator):
    """A communicator of one rank that goes with the last state or output that holds it."""

    def __init__(self):
        super().__init__(1, 0, get_unique_id())

    def __del__(self):
        torch.cuda.synchronize()
        self.destroy()


class _Window:
    """Memory registered with a communicator, given back with the last state or output that holds it."""

    def __init__(self, comm, nbytes):
        self.comm, self.win = comm, comm.window_alloc(nbytes)

    def __del__(self):
        torch.cuda.synchronize()
        self.win.free()


def _linear_inputs(c, seed):
    g = _gen(seed)
    return _randn(g, c["M"], c["K"]), _randn(g, c["N"], c["K"], std=0.02)


def _mlp_inputs(c, seed):
    g = _gen(seed)
    return {"x": _randn(g, c["T"], c["dim"]), "w13": _randn(g, 2 * c["ffn"], c["dim"], std=0.02),
            "w2": _randn(g, c["dim"], c["ffn"], std=0.02), "g": _randn(g, c["T"], c["dim"])}


def _moe_inputs(c, seed):
    """Activations whose routing is decided, as a trained router's is: every token leans towards k
    experts by clearly more than the rounding of a bf16 logit, some experts being picked more often."""
    g = _gen(seed)
    T, E, k, d, ffn = c["T"], c["E"], c["k"], c["d"], c["ffn"]
    router = _randn(g, E, d, std=0.02)
    popularity = torch.rand(E, device="cuda", generator=g) + 0.25
    chosen = torch.multinomial(popularity.expand(T, E), k, generator=g)
    lean = (3.0 + 0.9 * torch.rand(T, k, device="cuda", generator=g)) / (0.0004 * d)
    x = 0.3 * torch.randn(T, d, device="cuda", generator=g)
    for j in range(k):
        x += lean[:, j:j + 1] * router[chosen[:, j]].float()
    return {"x": x.to(BF16), "router": router, "w13": _randn(g, E, 2 * ffn, d, std=0.02), "w2": _randn(g, E, d, ffn, std=0.02),
            "g": _randn(g, T, d)}


def _exchange_inputs(c, seed):
    g = _gen(seed)
    T, E, k, d = c["T"], c["E"], c["k"], c["d"]
    top = torch.randn(T, E, device="cuda", generator=g).topk(k, dim=1)
    return {"x": _randn(g, T, d), "idx": top.indices.to(torch.int32), "w": torch.softmax(top.values, dim=1), "y": _randn(g, T * k, d)}


def _llama_config(c):
    return LlamaConfig(vocab_size=c["vocab"], dim=c["dim"], n_layers=c["layers"], n_heads=c["heads"], n_kv_heads=c["kv"], ffn_dim=c["ffn"])


def _llama_inputs(c, seed):
    """(weights by name, unit after unit; token ids; labels)"""
    g = _gen(seed)
    d, hd, f, V = c["dim"], c["dim"] // c["heads"], c["ffn"], c["vocab"]
    w = {"units.0.tok.weight": _randn(g, V, d, std=0.02)}
    for i in range(1, c["layers"] + 1):
        p = f"units.{i}."
        w[p + "attn_norm.weight"] = torch.ones(d, device="cuda", dtype=BF16)
        w[p + "attn.wq.weight"] = _randn(g, c["heads"] * hd, d, std=0.02)
        w[p + "attn.wk.weight"] = _randn(g, c["kv"] * hd, d, std=0.02)
        w[p + "attn.wv.weight"] = _randn(g, c["kv"] * hd, d, std=0.02)
        w[p + "attn.wo.weight"] = _randn(g, d, c["heads"] * hd, std=0.02)
        w[p + "mlp_norm.weight"] = torch.ones(d, device="cuda", dtype=BF16)
        w[p + "mlp.w1.weight"] = _randn(g, f, d, std=0.02)
        w[p + "mlp.w3.weight"] = _randn(g, f, d, std=0.02)
        w[p + "mlp.w2.weight"] = _randn(g, d, f, std=0.02)
    p = f"units.{c['layers'] + 1}."
    w[p + "norm.weight"] = torch.ones(d, device="cuda", dtype=BF16)
    w[p + "out.weight"] = _randn(g, V, d, std=0.02)
    ids = torch.randint(0, V, (c["B"], c["S"] + 1), device="cuda", generator=g)
    return w, ids[:, :-1].contiguous(), ids[:, 1:].contiguous()


def _grads_inputs(c, seed):
    g = _gen(seed)
    return _randn(g, c["count"]), _randn(g, c["count"], std=0.02)


def _pause_contents(c, seed):
    return torch.randint(-2 ** 31, 2 ** 31 - 1, (c["mib"] << 18,), device="cuda", generator=_gen(seed), dtype=torch.int32)


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c, "kind": kind}
    if kind == "linear":
        s["a"], s["b"] = _linear_inputs(c, seed)
        return s
    if kind == "grads":
        s["comm"] = _Comm()
        s["grad"], s["param"] = _grads_inputs(c, seed)
        s["sum"], s["full"] = torch.empty_like(s["grad"]), torch.empty_like(s["param"])
        s["shard"] = torch.empty(c["count"], device="cuda", dtype=torch.float32)
        return s
    if kind == "pause":
        comm = _Comm()
        s["window"] = _Window(comm, c["mib"] << 20)
        s["comm"] = comm
        s["view"] = s["window"].win.tensor(torch.int32)
        s["view"].copy_(_pause_contents(c, seed))
        s["view"].owner = s["window"]       # the memory under it stays mapped while the view is held
        return s
    comm = s["comm"] = _Comm()
    if kind == "mlp":
        t = _mlp_inputs(c, seed)
        layer = s["layer"] = TPMLP(comm, c["dim"], c["ffn"])
        with torch.no_grad():
            layer.w13.weight.copy_(t["w13"])
            layer.w2.weight.copy_(t["w2"])
        s["x"], s["g"] = t["x"].requires_grad_(c["train"]), t["g"]
    elif kind == "moe":
        t = _moe_inputs(c, seed)
        layer = s["layer"] = MoELayer(comm, c["d"], c["ffn"], c["E"], c["k"], tokens_per_rank=c["T"], capacity_factor=1.0)
        with torch.no_grad():
            for name in ("router", "w13", "w2"):
                getattr(layer, name).copy_(t[name])
        s["x"], s["g"] = t["x"].requires_grad_(c["train"]), t["g"]
    elif kind == "exchange":
        t = _exchange_inputs(c, seed)
        disp = s["disp"] = MoeDispatcher(comm, c["E"], c["d"], c["T"] * c["k"])
        disp.y.copy_(t["y"])        # the experts' outputs that the combine gathers
        disp.recv_x.owner = comm    # the rows lie in the communicator's memory: mapped while they are held
        s.update(x=t["x"], idx=t["idx"], w=t["w"])
    elif kind == "fsdp":
        cfg = _llama_config(c)
        weights, s["ids"], s["labels"] = _llama_inputs(c, seed)
        model = LlamaDecoder(cfg)
        model.load_state_dict(weights)
        s["fsdp"] = FSDP(model, comm)
        s["opt"] = ShardedAdamW(s["fsdp"], lr=1e-4)
        s["rope"] = rope_tables(c["S"], cfg.dim // cfg.n_heads, cfg.rope_theta, "cuda")
    return s


# ------------------------------------------------------------------ one pass

def run(state):
    s, kind = state, state["kind"]
    if kind == "linear":
        return gemm_bf16(s["a"], s["b"])
    if kind in ("mlp", "moe"):
        layer, x = s["layer"], s["x"]
        if not s["case"]["train"]:
            with torch.no_grad():
                return layer(x)
        x.grad = None
        layer.zero_grad(set_to_none=True)
        out = layer(x)
        out.backward(s["g"])
        return [out.detach(), x.grad] + [p.grad for p in layer.parameters()]
    if kind == "exchange":
        res = s["disp"].dispatch(s["x"], s["idx"])
        out = s["disp"].combine(s["idx"], s["w"], res.send_pos)
        return [res.recv_x, res.expert_counts, res.expert_offsets, res.send_pos, out]
    if kind == "fsdp":
        fsdp = s["fsdp"]
        logits = fsdp.forward_units(s["ids"], *s["rope"])
        loss = F.cross_entropy(logits.float().view(-1, logits.shape[-1]), s["labels"].view(-1))
        fsdp.zero_grad()
        loss.backward()
        s["opt"].step()
        return [logits.detach(), loss.detach()] + [t for pair in fsdp.shards() for t in pair]
    if kind == "grads":
        comm = s["comm"]
        comm.all_reduce(s["grad"], s["sum"])
        comm.reduce_scatter(s["grad"], s["shard"], scale=0.25)
        comm.all_gather(s["param"], s["full"])
        return [s["sum"], s["shard"], s["full"]]
    s["comm"].pause()
    s["comm"].resume()
    return s["view"]


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    c, kind = case, case["kind"]
    if kind == "linear":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": 2 * (M * K + N * K + M * N), "flops": 2 * M * N * K}
    if kind == "mlp":
        T, d, f = c["T"], c["dim"], c["ffn"]
        weights, times = 3 * d * f, 3 if c["train"] else 1
        # training reads x, the output gradient and the weights, writes the output and every gradient
        return {"bytes": 2 * (2 * T * d + weights + (2 * T * d + weights if c["train"] else 0)), "flops": times * 2 * T * weights}
    if kind == "moe":
        T, E, k, d, f = c["T"], c["E"], c["k"], c["d"], c["ffn"]
        used = min(E, T * k)
        weights, times = 3 * d * f * used + E * d, 3 if c["train"] else 1
        return {"bytes": 2 * (2 * T * d + weights + (2 * T * d + 3 * d * f * E + E * d if c["train"] else 0)),
                "flops": times * (2 * T * k * 3 * d * f + 2 * T * E * d)}
    if kind == "exchange":
        T, k, d = c["T"], c["k"], c["d"]
        # tokens in, rows out; rows back, tokens out
        return {"bytes": 2 * (T * d + T * k * d) * 2 + T * k * (4 * 3 + 4), "flops": 2 * T * k * d}
    if kind == "fsdp":
        tok, d = c["B"] * c["S"], c["dim"]
        hd = d // c["heads"]
        block = d * hd * (2 * c["heads"] + 2 * c["kv"]) + 3 * d * c["ffn"]
        matmul = c["layers"] * block + c["vocab"] * d
        params = matmul + c["vocab"] * d
        attn = c["layers"] * 2 * tok * c["S"] * d        # both attention products, causal half
        # forward, recomputation, backward (twice a forward); per parameter: the shard read twice for the gathers, gradient
        # shard written, read and reset, master and both moments read and written, new shard written
        return {"bytes": params * (2 * 2 + 2 * 2 + 4 * 3 + 4 * 6 + 2) + 2 * 2 * tok * c["vocab"], "flops": 4 * (2 * tok * matmul + attn)}
    if kind == "grads":
        return {"bytes": c["count"] * ((2 + 2) + (2 + 4) + (2 + 2)), "flops": c["count"]}
    # out to the host and back: the device side of a copy each way (the host link, not this memory, sets the time)
    return {"bytes": 2 * (c["mib"] << 20), "flops": 0}


def tolerance(case):
    """About four times what one pass is measured to be away from 64 bits, less where two roundings of
    one sum to 16 bits are all that can differ; the two training paths carry several roundings on."""
    kind = case["kind"]
    if kind in ("grads", "pause"):
        return "exact"
    return {"linear": {"rel": 0.005, "max": 0.03}, "exchange": {"rel": 0.005, "max": 0.03}, "mlp": {"rel": 0.012},
            "moe": {"rel": 0.02}, "fsdp": {"rel": 0.03}}[kind]


# ------------------------------------------------------------------ the same in 64 bits

def _swiglu64(x, w13, w2, ffn):
    h = x @ w13.t()
    return (F.silu(h[:, :ffn]) * h[:, ffn:]) @ w2.t()


def _exact_mlp(c, seed):
    t = {n: v.double() for n, v in _mlp_inputs(c, seed).items()}
    if not c["train"]:
        return _swiglu64(t["x"], t["w13"], t["w2"], c["ffn"])
    leaves = [t[n].requires_grad_() for n in ("x", "w13", "w2")]
    out = _swiglu64(*leaves, c["ffn"])
    return [out.detach(), *torch.autograd.grad(out, leaves, t["g"])]


def _exact_moe(c, seed):
    t = {n: v.double() for n, v in _moe_inputs(c, seed).items()}
    leaves = [t[n].requires_grad_(c["train"]) for n in ("x", "router", "w13", "w2")]
    x, router, w13, w2 = leaves
    top = (x @ router.t()).topk(c["k"], dim=1)
    w = torch.softmax(top.values, dim=1)
    out = torch.zeros_like(x)
    for e in range(c["E"]):
        tok, j = (top.indices == e).nonzero(as_tuple=True)
        if tok.numel():
            out = out.index_add(0, tok, _swiglu64(x[tok], w13[e], w2[e], c["ffn"]) * w[tok, j].unsqueeze(1))
    if not c["train"]:
        return out
    return [out.detach(), *torch.autograd.grad(out, leaves, t["g"])]


def _exact_exchange(c, seed):
    t = _exchange_inputs(c, seed)
    T, k, d = c["T"], c["k"], c["d"]
    order = torch.argsort(t["idx"].reshape(-1).long(), stable=True)
    pos = torch.empty_like(order)
    pos[order] = torch.arange(T * k, device="cuda")
    out = torch.zeros(T, d, device="cuda", dtype=torch.float64)
    for j in range(k):
        out += t["w"][:, j:j + 1].double() * t["y"][pos.view(T, k)[:, j]].double()
    return [t["x"][order // k].double(), None, None, None, out]


def _norm64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + LlamaConfig.norm_eps) * w


def _rope64(x, cos, sin):
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * cos - b * sin, a * sin + b * cos), dim=-1).flatten(-2)


def _exact_fsdp(c, seed):
    weights, ids, labels = _llama_inputs(c, seed)
    w = {n: t.double().requires_grad_() for n, t in weights.items()}
    B, S, H, KV, hd = c["B"], c["S"], c["heads"], c["kv"], c["dim"] // c["heads"]
    inv = 1.0 / (LlamaConfig.rope_theta ** (torch.arange(0, hd, 2, device="cuda").double() / hd))
    ang = torch.outer(torch.arange(S, device="cuda").double(), inv)
    cos, sin = ang.cos(), ang.sin()
    hidden = torch.ones(S, S, device="cuda", dtype=torch.bool).triu(1)
    x = w["units.0.tok.weight"][ids]
    for i in range(1, c["layers"] + 1):
        p = f"units.{i}."
        h = _norm64(x, w[p + "attn_norm.weight"])
        q, k, v = ((h @ w[p + f"attn.{n}.weight"].t()).view(B, S, -1, hd).transpose(1, 2) for n in ("wq", "wk", "wv"))
        q, k = _rope64(q, cos, sin), _rope64(k, cos, sin)
        k, v = (t.repeat_interleave(H // KV, dim=1) for t in (k, v))
        a = torch.softmax((q @ k.transpose(-1, -2) / math.sqrt(hd)).masked_fill(hidden, float("-inf")), dim=-1) @ v
        x = x + a.transpose(1, 2).reshape(B, S, -1) @ w[p + "attn.wo.weight"].t()
        h = _norm64(x, w[p + "mlp_norm.weight"])
        x = x + (F.silu(h @ w[p + "mlp.w1.weight"].t()) * (h @ w[p + "mlp.w3.weight"].t())) @ w[p + "mlp.w2.weight"].t()
    p = f"units.{c['layers'] + 1}."
    logits = _norm64(x, w[p + "norm.weight"]) @ w[p + "out.weight"].t()
    loss = F.cross_entropy(logits.view(-1, c["vocab"]), labels.view(-1))
    grads = dict(zip(w, torch.autograd.grad(loss, list(w.values()))))
    out = [logits.detach(), loss.detach()]
    for i in range(c["layers"] + 2):
        names = [n for n in w if n.startswith(f"units.{i}.")]
        flat = [torch.cat([t[n].detach().reshape(-1) for n in names]) for t in (w, grads)]
        flat = [F.pad(t, (0, -t.numel() % 8)) for t in flat]
        # the first step of AdamW: both moments are the gradient's own, corrected for their start
        out += [flat[0] - 1e-4 * flat[1] / (flat[1].abs() + 1e-8), flat[1]]
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "linear":
        a, b = _linear_inputs(c, seed)
        return a.double() @ b.double().t()
    if kind == "mlp":
        return _exact_mlp(c, seed)
    if kind == "moe":
        return _exact_moe(c, seed)
    if kind == "exchange":
        return _exact_exchange(c, seed)
    if kind == "fsdp":
        return _exact_fsdp(c, seed)
    if kind == "grads":
        g, p = (t.double() for t in _grads_inputs(c, seed))
        return [g, 0.25 * g, p]
    return None
