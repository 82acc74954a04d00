"""The calls a user of this package makes, over the sizes they come in: what a timing or parity run goes through.

A case names a kind of call and its sizes:
  train      one MoE depth of MoE_Cascaded, forward and backward (outputs, input gradient, every parameter gradient)
  infer      the same depth, forward only, without gradients
  dense      a dense depth of MoE_Cascaded, forward and backward
  router     the step before the experts on given gate logits: softmax + top-k + GShard loss, its gradient, and the
             segmentation of the routed rows by expert
  operators  the operator-level interface (counter, ESMM, es_fused) for one route

Inputs are N(0,1) tokens and gradients; weights are scaled by 1/sqrt(fan-in) so that pre-activations are O(1) and both
branches of an activation are met.  `skew` puts a constant into the first token feature, whose gate weights are the
logarithms of a Zipf(1.2) distribution: some experts then receive a fifth of the rows and others none.
"""
import math

import torch
import torch.nn.functional as F

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ACTS = {"gelu": lambda t: F.gelu(t), "relu": F.relu, "silu": F.silu}
AUX_WEIGHT = 0.01          # weight of the auxiliary loss next to the loss of the outputs


def _moe(kind, name, tokens, dim, experts, top_k, dtype, act="gelu", fc1_bias=True, skew=False):
    c = dict(kind=kind, tokens=tokens, dim=dim, hidden=4 * dim, experts=experts, top_k=top_k, dtype=dtype, act=act,
             fc1_bias=fc1_bias, skew=skew)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the headline layer of the benchmark: large-model pre-training, one device's share of the tokens
        _moe("train", "train_large", 131072, 2048, 64, 2, "bf16"),
        # many experts under skewed routing (an untrained or collapsed gate): long and empty segments side by side
        _moe("train", "train_skewed", 65536, 1024, 64, 2, "bf16", skew=True),
        # the operator-sweep layer: a mid-size training step
        _moe("train", "train_mid", 16384, 768, 8, 2, "bf16"),
        # the last stage of the Swin-MoE-B-like network: 128 images x 36 tokens, top-1, no fc1 bias, ~144 rows per expert
        _moe("train", "train_vision", 4608, 1024, 32, 1, "bf16", fc1_bias=False),
        # nothing is a power of two or a multiple of a tile: a last, partial batch in fp16
        _moe("train", "train_ragged", 1000, 200, 7, 3, "fp16", act="relu"),
        # the README's module at its own size and default precision
        _moe("train", "train_readme", 4096, 128, 8, 1, "fp32"),
        # a full-precision training step without autocast
        _moe("train", "train_fp32", 8192, 512, 8, 2, "fp32"),
        # serving: a handful of tokens through a layer, where latency and the reading of the weights count
        _moe("infer", "infer_few", 16, 1024, 32, 1, "bf16"),
        # serving: a prompt batch in fp16
        _moe("infer", "infer_batch", 2048, 768, 8, 2, "fp16"),
        # the dense FFN either side of every MoE depth (stage 3 of the Swin-MoE-B-like network)
        dict(name="dense_vision", kind="dense", tokens=18432, dim=512, hidden=2048, dtype="bf16", act="gelu", fc1_bias=True),
        # the routing step of the headline layer by itself
        dict(name="router_large", kind="router", tokens=131072, experts=64, top_k=2),
        # code written against the reference's operators
        dict(name="operators_mid", kind="operators", tokens=2048, dim=256, hidden=1024, experts=8, dtype="fp16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "infer", "infer", "dense", "router", "operators"])
    if kind == "router":
        experts = rng.choice([4, 7, 8, 32, 64, 128])
        return dict(kind=kind, tokens=_log(rng, 1, 131072), experts=experts, top_k=rng.randint(1, min(4, experts)))
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    # now and then a width whose rows are not whole 16-byte chunks; such a call, and one in full precision, costs
    # several times as much as others
    odd = rng.random() < 0.1
    most_dim, most_flops = (512, 4e11) if dtype == "fp32" or odd else (1024, 1.2e13)
    dim = 8 * _log(rng, 8, most_dim // 8) - (rng.randint(1, 7) if odd else 0)
    if kind == "operators":
        return dict(kind=kind, tokens=_log(rng, 1, 16384), dim=min(dim, 512), hidden=4 * min(dim, 512),
                    experts=rng.choice([4, 7, 8, 32]), dtype=dtype)
    act = rng.choice(["gelu", "gelu", "relu", "silu"])
    if kind == "dense":
        most = min(65536, int(most_flops / (48 * dim * dim)))
        return dict(kind=kind, tokens=_log(rng, 1, most), dim=dim, hidden=4 * dim, dtype=dtype, act=act,
                    fc1_bias=rng.random() < 0.75)
    experts = rng.choice([4, 7, 8, 16, 32, 64])
    top_k = rng.randint(1, min(3, experts))
    per_token = (48 if kind == "train" else 16) * dim * dim * top_k
    most = min(65536, int(most_flops / per_token))
    c = _moe(kind, None, _log(rng, 1 if kind == "infer" else 64, most), dim, experts, top_k, dtype, act=act,
             fc1_bias=rng.random() < 0.75, skew=rng.random() < 0.25)
    return c


# ---- inputs --------------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _tokens(g, tokens, dim, dtype, skew=False):
    x = torch.randn(tokens, dim, generator=g, device="cuda", dtype=torch.float32).to(dtype)
    if skew:
        x[:, 0] = 1.0
    return x


def _zipf_logits(experts):
    return -1.2 * torch.log(torch.arange(1, experts + 1, device="cuda", dtype=torch.float32))


def _module(case, g, moe):
    """The module a program builds once, with its parameters filled from the generator."""
    from hexa_moe.moe import MoE_Cascaded
    dtype = DTYPES[case["dtype"]]
    gate = {"type": "top", "k": case.get("top_k", 1), "fp32_gate": True}
    with torch.device("cuda"):
        m = MoE_Cascaded(gate_type=gate, model_dim_list=[case["dim"]], moe_idx_list=[0] if moe else [], mlp_ratio=4,
                         num_global_experts=case.get("experts", 1), total_depth=1, data_centric=True,
                         mlp_fc1_bias=case["fc1_bias"], mlp_fc2_bias=True, activation_fn=ACTS[case["act"]])
    m = m.to(dtype)
    m.gates.float()
    d, H = case["dim"], case["hidden"]
    with torch.no_grad():
        for n, p in m.named_parameters():
            if "gates" in n:
                p.copy_(torch.randn(p.shape, generator=g, device="cuda") / math.sqrt(d))
                if case["skew"]:
                    p[:, 0] = _zipf_logits(case["experts"])
            elif "fc1_w" in n:
                p.normal_(0, 1 / math.sqrt(d), generator=g)
            elif "fc2_w" in n:
                p.normal_(0, 1 / math.sqrt(H), generator=g)
            else:
                p.normal_(0, 0.1, generator=g)
    return m.train() if case["kind"] != "infer" else m.eval()


def _operator_inputs(case, seed):
    g = _generator(seed)
    dtype, T, d, H, E = DTYPES[case["dtype"]], case["tokens"], case["dim"], case["hidden"], case["experts"]
    ids = torch.randint(0, E, (T,), generator=g, device="cuda").to(torch.int32)
    x = _tokens(g, T, d, dtype)
    w = (torch.randn(E, d, H, generator=g, device="cuda") / math.sqrt(d)).to(dtype)
    b = (torch.randn(E, H, generator=g, device="cuda") * 0.1).to(dtype)
    dy = _tokens(g, T, H, dtype)
    return dict(ids=ids, x=x, w=w, w_t=w.transpose(1, 2).contiguous(), b=b, dy=dy)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "router":
        g = _generator(seed)
        return dict(case=case, logits=torch.randn(case["tokens"], case["experts"], generator=g, device="cuda"),
                    d_loss=torch.full((), AUX_WEIGHT, device="cuda"))
    if kind == "operators":
        return dict(_operator_inputs(case, seed), case=case)
    g = _generator(seed)
    dtype = DTYPES[case["dtype"]]
    m = _module(case, g, kind != "dense")
    x = _tokens(g, case["tokens"], case["dim"], dtype, case.get("skew", False))
    state = dict(case=case, module=m, x=x)
    if kind != "infer":
        state["dy"] = _tokens(g, case["tokens"], case["dim"], dtype)
        state["x"] = x.requires_grad_(True)
    if kind == "train":
        state["d_loss"] = torch.full((), AUX_WEIGHT, device="cuda")
    return state


# ---- one pass --------------------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "router":
        from hexa_moe_b200 import ops
        ids, loss, first_count, mass = ops.gate_topk(state["logits"], case["top_k"])
        d_logits = ops.gate_loss_grad(state["logits"], first_count, state["d_loss"])
        r = ops.route(ids, case["experts"], route_major=True)
        return ids, loss, mass, d_logits, r.counts, r.pad_offsets, r.token_row
    if kind == "operators":
        from hexa_moe_b200.kernels.basics import counter
        from hexa_moe_b200.kernels.esmm import ESMM
        from hexa_moe_b200.kernels.fused import es_fused
        E = case["experts"]
        _, starts, toks, exps = counter(state["ids"], E)
        toks = toks + 1
        y = ESMM(state["x"], state["w"], state["b"], toks, exps)
        db, dx, dw = es_fused(state["dy"], state["x"], state["w_t"], toks, exps, starts, E)
        return y, db, dx, dw
    m, x = state["module"], state["x"]
    if kind == "infer":
        with torch.no_grad():
            y, l_aux = m(0, x)
        return y, l_aux
    m.zero_grad(set_to_none=True)
    x.grad = None
    y, l_aux = m(0, x)
    if kind == "dense":
        y.backward(state["dy"])
        return (y, x.grad) + tuple(p.grad for p in m.parameters())
    torch.autograd.backward([y, l_aux], [state["dy"], state["d_loss"]])
    return (y, l_aux, x.grad) + tuple(p.grad for p in m.parameters())


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def work(case):
    kind, T = case["kind"], case["tokens"]
    if kind == "router":
        E, k = case["experts"], case["top_k"]
        # logits read once, their gradient, the ids and the position of every routed row written
        return {"bytes": 8.0 * T * E + 8.0 * T * k, "flops": 12.0 * T * E}
    d, H, es = case["dim"], case["hidden"], 4 if case["dtype"] == "fp32" else 2
    if kind == "operators":
        E = case["experts"]
        # x, dy, two weight layouts and the ids in; y, dx, dw out
        return {"bytes": float(es * (3 * T * d + 2 * T * H + 3 * E * d * H) + 4 * T), "flops": 6.0 * T * d * H}
    E, k = case.get("experts", 1), case.get("top_k", 1)
    met = min(E, T * k)
    if kind == "infer":
        return {"bytes": float(es * (2 * T * d + 2 * met * d * H)), "flops": 4.0 * T * k * d * H + (2.0 * T * d * E)}
    gate = 0.0 if kind == "dense" else 6.0 * T * d * E
    return {"bytes": float(es * (4 * T * d + 2 * met * d * H + 2 * E * d * H)), "flops": 12.0 * T * k * d * H + gate}


def tolerance(case):
    # About four times the distance to a 64-bit evaluation (relative, 2-norm).  16-bit hidden activations and results set
    # it there; in full precision it is the summation order of sums up to a few thousand terms long.
    if case["kind"] == "router":
        return {"rel": 1.2e-5, "differ": 1e-4}    # ids and positions of equal scores
    return {"rel": {"bf16": 1.2e-2, "fp16": 1.6e-3, "fp32": 4e-6}[case["dtype"]]}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------------
def _gshard(scores, ids):
    T, E = scores.shape
    ce = torch.bincount(ids[:, 0], minlength=E).double() * (E / T)
    return (scores.sum(0) * ce).sum() / T


def exact(case, seed):
    kind = case["kind"]
    if kind == "router":
        s = prepare(case, seed)
        E, k, T = case["experts"], case["top_k"], case["tokens"]
        logits = s["logits"].double().requires_grad_(True)
        scores = F.softmax(logits, dim=1)
        ids = torch.topk(scores, k, dim=1).indices
        loss = _gshard(scores, ids)
        (d_logits,) = torch.autograd.grad(loss, logits, torch.tensor(AUX_WEIGHT, device="cuda").double())
        flat = ids.t().reshape(-1)                                   # routed rows numbered j * T + t
        counts = torch.bincount(flat, minlength=E)
        pad = torch.zeros(E + 1, dtype=torch.int64, device="cuda")
        pad[1:] = torch.cumsum((counts + 127) // 128 * 128, 0)
        first = torch.cumsum(counts, 0) - counts
        order = torch.argsort(flat, stable=True)
        row = torch.empty_like(flat)
        row[order] = torch.arange(T * k, device="cuda") - first[flat[order]] + pad[flat[order]]
        i32 = lambda t: t.to(torch.int32)
        return (i32(ids.t().contiguous()), loss.detach(), scores.detach().sum(0), d_logits, i32(counts), i32(pad),
                i32(row.view(k, T).t().reshape(-1)))
    if kind == "operators":
        s = _operator_inputs(case, seed)
        E = case["experts"]
        x, w, b, dy, ids = s["x"].double(), s["w"].double(), s["b"].double(), s["dy"].double(), s["ids"].long()
        y, dx = torch.zeros_like(dy), torch.zeros_like(x)
        db = torch.zeros_like(b)
        dw = torch.zeros(E, w.shape[2], w.shape[1], dtype=torch.float64, device="cuda")
        for e in range(E):
            t = torch.nonzero(ids == e).flatten()
            y[t] = x[t] @ w[e] + b[e]
            dx[t] = dy[t] @ w[e].t()
            db[e] = dy[t].sum(0)
            dw[e] = dy[t].t() @ x[t]
        return y, db, dx, dw
    if work(case)["flops"] > 1e13:
        return None
    s = prepare(case, seed)
    m, act = s["module"], ACTS[case["act"]]
    names, params = zip(*[(n, p.detach().double().requires_grad_(True)) for n, p in m.named_parameters()])
    P = dict(zip(names, params))
    x = s["x"].detach().double().requires_grad_(True)
    if kind == "dense":
        h = x @ P["mlp_fc1_w.0"].t()
        if case["fc1_bias"]:
            h = h + P["mlp_fc1_b.0"]
        y = act(h) @ P["mlp_fc2_w.0"] + P["mlp_fc2_b.0"]
        return (y.detach(),) + torch.autograd.grad(y, (x,) + params, s["dy"].double())
    k, E = case["top_k"], case["experts"]
    wg = next(p for n, p in P.items() if n.startswith("gates"))
    scores = F.softmax(x @ wg.t(), dim=1)
    ids = torch.topk(scores, k, dim=1).indices
    l_aux = _gshard(scores, ids)
    y = torch.zeros_like(x)
    for e in range(E):
        t = torch.nonzero((ids == e).any(1)).flatten()
        if t.numel() == 0:
            continue
        h = x[t] @ P["batched_fc1_w.0"][e].t()
        if case["fc1_bias"]:
            h = h + P["batched_fc1_bias.0"][e]
        y = y.index_add(0, t, act(h) @ P["batched_fc2_w.0"][e] + P["batched_fc2_bias.0"][e])
    if kind == "infer":
        return y.detach(), l_aux.detach()
    grads = torch.autograd.grad([y, l_aux], (x,) + params, [s["dy"].double(), torch.tensor(AUX_WEIGHT, device="cuda").double()])
    return (y.detach(), l_aux.detach()) + grads
