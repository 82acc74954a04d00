"""MoE_Cascaded on a B200 against (a) the golden activations of the reference's own module and
(b) the CPU oracle, including the parameter gradients the reference never delivers."""
import os

import numpy as np
import pytest
import torch
import torch.nn.functional as F

from oracle import hexa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def rel_err(got, want):
    got = got.detach().double().cpu(); want = want.detach().double().cpu()
    return float((got - want).abs().max() / want.abs().max().clamp_min(1e-30))


def _toy(k=1, d=32, E=4, **kw):
    from hexa_moe import moe as hmoe
    args = dict(gate_type={'type': 'top', 'k': k, 'gate_noise': 1.0, 'fp32_gate': True}, model_dim_list=[d] * 4,
                moe_idx_list=[2, 3], mlp_ratio=4, mlp_proportion=None, num_global_experts=E, total_depth=4,
                data_centric=True, mlp_fc1_bias=True, mlp_fc2_bias=True, activation_fn=lambda t: F.gelu(t))
    args.update(kw)
    return hmoe.MoE_Cascaded(**args)


@pytest.mark.parametrize("tag,k", [("top1", 1), ("top2", 2)])
def test_matches_reference_module_golden(golden_dir, tag, k):
    """Same parameters and input as the reference run that produced tests/golden/module.npz.
    The reference rounds both MMA operands to fp16 (its fp32 'full' flavour too), this module's fp32
    path does not, hence 5e-3 here; the 1e-5 check is the oracle test below."""
    z = np.load(os.path.join(golden_dir, "module.npz"))
    m = _toy(k=k)
    m.load_state_dict({n.split("param/")[1]: torch.from_numpy(z[n]) for n in z.files if n.startswith(tag + "/param/")})
    m = m.cuda().eval()
    x = torch.from_numpy(z[tag + "/x"]).cuda().requires_grad_(True)
    h, aux = x, 0
    for d in range(4):
        # feed the reference's own activations forward so that one flipped routing decision cannot cascade
        h_in = h if d == 0 else torch.from_numpy(z[f"{tag}/y{d - 1}"]).cuda()
        y, l = m(d, h_in)
        assert rel_err(y, torch.from_numpy(z[f"{tag}/y{d}"])) < 5e-3, d
        assert abs(float(l) - float(z[f"{tag}/l_aux{d}"])) < 1e-5
    h, aux = x, 0
    for d in range(4):
        h, l = m(d, h)
        aux = aux + l
    (h.sum() + aux).backward()
    assert rel_err(x.grad, torch.from_numpy(z[tag + "/x_grad"])) < 5e-3


@pytest.mark.parametrize("dtype,k,tol", [(torch.float32, 1, 1e-5), (torch.float32, 2, 1e-5), (torch.bfloat16, 2, 2e-2),
                                         (torch.float16, 1, 2e-2)])
def test_moe_depth_against_oracle(dtype, k, tol):
    torch.manual_seed(3)
    d, E, T = 64, 6, 700
    m = _toy(k=k, d=d, E=E)
    with torch.no_grad():
        for n_, p in m.named_parameters():
            p.normal_(0, 0.5 if "gates" in n_ else (0.1 if p.dim() < 3 else 0.15))
    m = m.to(dtype).cuda().eval()
    x = torch.randn(7, T // 7, d).to(dtype)
    xg = x.cuda().requires_grad_(True)
    y, l = m(2, xg)
    assert y.shape == xg.shape and y.dtype == dtype
    dy = torch.randn_like(y)
    (y * dy).sum().backward()
    i = 0
    P = {n_: p.detach().cpu() for n_, p in m.named_parameters()}
    ids_exp, l_exp, _ = O.gate_topk(x.reshape(-1, d), P["gates.0.wg.weight"], k)
    # the oracle gets the module's own routing decisions (a near-tie may resolve differently in another matmul
    # order); the two must still agree on all but a handful of tokens
    ids = torch.stack([i.cpu() for i in m.dispatch_params.indices_], dim=1)
    assert (ids == ids_exp).float().mean() > 0.99
    res = O.moe_layer(x.reshape(-1, d), ids, P["batched_fc1_w.0"], P["batched_fc2_w.0"], P["batched_fc1_bias.0"],
                      P["batched_fc2_bias.0"], F.gelu, dy.cpu().reshape(-1, d))
    assert abs(float(l) - float(l_exp)) < 1e-4
    assert rel_err(y.reshape(-1, d), res["y"]) < tol
    assert rel_err(xg.grad.reshape(-1, d), res["dx"]) < tol
    for name, key in (("batched_fc1_w.0", "dw1"), ("batched_fc2_w.0", "dw2"), ("batched_fc1_bias.0", "db1"), ("batched_fc2_bias.0", "db2")):
        g = dict(m.named_parameters())[name].grad
        assert g is not None and g.dtype == dtype, name          # the reference leaves these None
        assert rel_err(g, res[key]) < tol, (name, rel_err(g, res[key]))
    assert m.dispatch_params.stage == -1                          # decremented in backward like the reference


def test_model_centric_module_on_one_gpu_matches_data_centric():
    """data_centric=False without a process group: the model-centric branch (input gradients first, then the parameter
    gradients) must give what the data-centric branch gives on the same weights and tokens."""
    d, E, T, k = 64, 6, 900, 2
    outs = []
    for data_centric in (True, False):
        torch.manual_seed(11)
        m = _toy(k=k, d=d, E=E, data_centric=data_centric)
        with torch.no_grad():
            for n_, p in m.named_parameters():
                p.normal_(0, 0.5 if "gates" in n_ else (0.1 if p.dim() < 3 else 0.15))
        m = m.bfloat16().cuda().eval()
        x = torch.randn(T, d, generator=torch.Generator().manual_seed(4)).bfloat16().cuda().requires_grad_(True)
        y, _ = m(2, x)
        y2, _ = m(3, y)
        y2.float().square().mean().backward()
        outs.append([y2.detach(), x.grad] + [dict(m.named_parameters())[n_].grad for n_ in
                                             ("batched_fc1_w.0", "batched_fc2_w.1", "batched_fc1_bias.1", "batched_fc2_bias.0")])
    for a, b in zip(*outs):
        assert a is not None and b is not None
        assert rel_err(b, a) < 1e-2        # same kernels in another order; bf16 weight gradients round once either way


def test_training_mode_autocast_and_options():
    torch.manual_seed(0)
    m = _toy(k=2, d=64, E=8, result_func=lambda t: t * 2.0, is_gshard_loss=False).cuda().train()
    x = torch.randn(4, 50, 64, device="cuda", requires_grad=True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        h, aux = x, 0
        for d in range(4):
            h, l = m(d, h)
            aux = aux + (l if l is not None else 0)
    assert h.dtype == torch.float32 and h.shape == x.shape
    (h.float().sum() + aux).backward()
    for n_, p in m.named_parameters():
        assert p.grad is not None and torch.isfinite(p.grad).all(), n_
        assert p.grad.dtype == torch.float32
    assert torch.isfinite(x.grad).all()
    y1, _ = m(3, x.detach(), top_k=1)                              # per-call top_k override
    assert torch.isfinite(y1).all()


def test_unrecognised_activation_uses_the_callable():
    torch.manual_seed(1)
    act = lambda t: torch.tanh(t) * 1.3
    m = _toy(k=2, d=64, E=4, activation_fn=act)
    assert m.dispatch_params.act_id == -1
    with torch.no_grad():
        for n_, p in m.named_parameters():
            p.normal_(0, 0.3)
    m = m.cuda().eval()
    x = torch.randn(300, 64)
    xg = x.cuda().requires_grad_(True)
    y, _ = m(2, xg)
    y.sum().backward()
    P = {n_: p.detach().cpu() for n_, p in m.named_parameters()}
    ids, _, _ = O.gate_topk(x, P["gates.0.wg.weight"], 2)
    res = O.moe_layer(x, ids, P["batched_fc1_w.0"], P["batched_fc2_w.0"], P["batched_fc1_bias.0"], P["batched_fc2_bias.0"], act,
                      torch.ones(300, 64))
    assert rel_err(y, res["y"]) < 1e-5 and rel_err(xg.grad, res["dx"]) < 1e-5
    assert rel_err(m.batched_fc1_w[0].grad, res["dw1"]) < 1e-5


def test_inference_mode_and_gradient_accumulation():
    """no_grad forward keeps no state and equals the training forward; two backward passes accumulate into .grad."""
    torch.manual_seed(2)
    m = _toy(k=2, d=64, E=4)
    with torch.no_grad():
        for n_, p in m.named_parameters():
            p.normal_(0, 0.3)
    m = m.bfloat16().cuda().eval()
    x = torch.randn(3, 100, 64, device="cuda").bfloat16()
    with torch.no_grad():
        y0, _ = m(2, x)
    xg = x.clone().requires_grad_(True)
    y1, _ = m(2, xg)
    assert torch.equal(y0, y1)
    y1.float().sum().backward()
    g1 = m.batched_fc1_w[0].grad.clone()
    y2, _ = m(2, xg)
    y2.float().sum().backward()
    torch.testing.assert_close(m.batched_fc1_w[0].grad.float(), 2 * g1.float(), rtol=2e-2, atol=1e-3)


def test_split_precision_gate_matches_an_fp32_projection():
    """The bf16-token fast path of the fp32 gate (three bf16 terms of the fp32 weight, fp32 accumulation) against a
    float64 projection: logits and the weight gradient to fp32-GEMM accuracy (2e-5 of the largest value; a plain
    bf16 weight would be off by 4e-3), the token gradient to its own bf16 rounding (2^-8)."""
    from hexa_moe_b200.impls.gating import LinearTopKGate
    torch.manual_seed(3)
    g = LinearTopKGate(256, 16, k=2, fp32_gate=True).cuda()
    with torch.no_grad():
        g.wg.weight.normal_(0, 0.3)
    x = torch.randn(1000, 256, device="cuda").bfloat16().requires_grad_()
    logits = g(x)
    assert logits.dtype == torch.float32
    xr = x.detach().double().requires_grad_()
    wr = g.wg.weight.detach().double().requires_grad_()
    ref = xr @ wr.t()
    assert float((logits.double() - ref).abs().max()) <= 2e-5 * float(ref.abs().max())
    dl = torch.randn_like(logits)
    logits.backward(dl)
    ref.backward(dl.double())
    assert float((g.wg.weight.grad.double() - wr.grad).abs().max()) <= 2e-5 * float(wr.grad.abs().max())
    assert float((x.grad.double() - xr.grad).abs().max()) <= 2.0 ** -8 * float(xr.grad.abs().max())
    os.environ["HEXA_SPLIT_GATE"] = "0"
    try:
        plain = g(x.detach())
    finally:
        del os.environ["HEXA_SPLIT_GATE"]
    assert float((plain - logits).abs().max()) <= 2e-5 * float(ref.abs().max())


@pytest.mark.parametrize("dtype,tokens", [(torch.bfloat16, 96), (torch.bfloat16, 256), (torch.float16, 200)])
def test_dense_ffn_on_the_grouped_gemm_kernels(dtype, tokens):
    """A dense depth of MoE_Cascaded (reference layers.py:18-88) runs as a one-expert layer on the grouped-GEMM
    kernels for 16-bit tokens.  Checked against a float64 evaluation of the same FFN (2e-2 relative to the largest
    value, the 16-bit tolerance) and against the PyTorch-op path of the same module, for token counts that are and
    are not multiples of the 128-row tile."""
    torch.manual_seed(5)
    d, E = 64, 4
    m = _toy(k=1, d=d, E=E)
    with torch.no_grad():
        for n_, p in m.named_parameters():
            if n_.startswith("mlp_fc"):
                p.normal_(0, 0.1)
    m = m.to(dtype).cuda().train()
    x = torch.randn(tokens, d, device="cuda").to(dtype)
    dy = torch.randn(tokens, d, device="cuda").to(dtype)
    names = ["mlp_fc1_w.0", "mlp_fc2_w.0", "mlp_fc1_b.0", "mlp_fc2_b.0"]
    params = dict(m.named_parameters())

    def run():
        for p in m.parameters():
            p.grad = None
        xi = x.clone().requires_grad_(True)
        y, aux = m(0, xi)
        assert aux == 0
        y.backward(dy)
        return [y.detach(), xi.grad] + [params[n_].grad.clone() for n_ in names]

    from hexa_moe_b200 import ops
    os.environ["HEXA_DENSE_MIN_DIM"] = "0"          # by default only model dims >= 256 take the kernel path
    try:
        before = ops.LAUNCHES
        got = run()
        assert ops.LAUNCHES - before >= 9, "the dense depth did not run on this library's kernels"
        os.environ["HEXA_DENSE_KERNELS"] = "0"
        before = ops.LAUNCHES
        plain = run()
        assert ops.LAUNCHES == before
    finally:
        os.environ.pop("HEXA_DENSE_KERNELS", None)
        os.environ.pop("HEXA_DENSE_MIN_DIM", None)
    w1, w2, b1, b2 = [params[n_].detach().double().requires_grad_(True) for n_ in names]
    xr = x.double().requires_grad_(True)
    yr = F.gelu(xr @ w1.t() + b1) @ w2 + b2
    yr.backward(dy.double())
    want = [yr.detach(), xr.grad, w1.grad, w2.grad, b1.grad, b2.grad]
    for g, p_, w in zip(got, plain, want):
        assert g.shape == w.shape
        assert rel_err(g, w) <= 2e-2
        assert rel_err(g, p_) <= 3e-2


@pytest.mark.parametrize("dim,act,on_kernels", [(64, "gelu", True), (72, "silu", True), (56, "gelu", False), (64, "relu", False), (256, "relu", True)])
def test_dense_depth_widths_on_the_kernels(dim, act, on_kernels):
    """Which widths run as a one-expert layer, and that both ways agree to the 16-bit tolerance."""
    import os
    import torch.nn.functional as F
    from hexa_moe import moe as hmoe
    from hexa_moe_b200 import ops
    torch.manual_seed(dim)
    fn = {"gelu": lambda t: F.gelu(t), "silu": F.silu, "relu": F.relu}[act]
    m = hmoe.MoE_Cascaded(gate_type={'type': 'top', 'k': 1}, model_dim_list=[dim], moe_idx_list=[], mlp_ratio=4,
                          num_global_experts=1, total_depth=1, data_centric=True, activation_fn=fn)
    with torch.no_grad():
        for p in m.parameters():
            p.normal_(0, 0.1)
    m = m.to(torch.bfloat16).cuda()
    x, dy = torch.randn(333, dim, device="cuda").bfloat16(), torch.randn(333, dim, device="cuda").bfloat16()

    def run():
        m.zero_grad()
        xi = x.clone().requires_grad_(True)
        before = ops.LAUNCHES
        y, _ = m(0, xi)
        y.backward(dy)
        return ops.LAUNCHES > before, [y.detach(), xi.grad] + [p.grad for p in m.parameters()]

    used, got = run()
    assert used == on_kernels
    os.environ["HEXA_DENSE_KERNELS"] = "0"
    try:
        _, want = run()
    finally:
        del os.environ["HEXA_DENSE_KERNELS"]
    if act != "relu":
        for a, b in zip(got, want):
            assert float((a.float() - b.float()).norm()) <= 1.2e-2 * float(b.float().norm())
    if not on_kernels:
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        return
    # against 64 bits, a ReLU's mask included: the kernels round a pre-activation once, after the sum that decides its sign
    w1, w2, b1, b2 = P = [p.detach().double().requires_grad_(True) for p in m.parameters()]
    xd = x.double().requires_grad_(True)
    y = fn(xd @ w1.t() + b1) @ w2 + b2
    exact = [y.detach()] + list(torch.autograd.grad(y, [xd] + P, dy.double()))
    for a, b in zip(got, exact):
        assert float((a.double() - b).norm()) <= 1.2e-2 * float(b.norm())


def test_dense_routing_belongs_to_its_stream():
    """Tables built on one stream are not handed to another, and a captured graph has tables of its own."""
    from hexa_moe_b200 import _lib as L, ops
    dev = torch.device("cuda", torch.cuda.current_device())
    here = ops.dense_routing(300, dev)
    assert ops.dense_routing(300, dev) is here
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        there = ops.dense_routing(300, dev)
        assert there is not here and ops.dense_routing(300, dev) is there
    torch.cuda.synchronize()
    assert torch.equal(there.row_token[:300], here.row_token[:300]) and torch.equal(there.pad_offsets, here.pad_offsets)

    g = torch.Generator(device="cuda").manual_seed(0)
    x, w1, w2 = (torch.randn(*n, generator=g, device="cuda").bfloat16() for n in ((301, 64), (256, 64), (256, 64)))
    call = lambda: ops.dense_forward(x, w1, w2, None, None, L.ACT_GELU, need_state=False)[0]
    want = call().clone()
    before = len(ops._DENSE_ROUTING)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = call()
    assert len(ops._DENSE_ROUTING) == before
    ops._DENSE_ROUTING.clear()
    junk = [torch.full((4096,), 7, dtype=torch.int32, device="cuda") for _ in range(64)]
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want) and len(junk) == 64


@pytest.mark.parametrize("T,dim", [(256, 64), (333, 72)])
def test_narrow_dense_depths_keep_what_plain_operations_allow(T, dim):
    """Widths below 256 ran as PyTorch operations before they ran on the kernels: two passes over a kept graph, the check for
    changes in place, saved-tensor hooks, second derivatives, batched gradients, and tensors of any layout."""
    import os
    import torch.nn.functional as F
    from hexa_moe import moe as hmoe
    from hexa_moe_b200 import ops
    torch.manual_seed(dim)
    m = hmoe.MoE_Cascaded(gate_type={'type': 'top', 'k': 1}, model_dim_list=[dim], moe_idx_list=[], mlp_ratio=4,
                          num_global_experts=1, total_depth=1, data_centric=True, activation_fn=lambda t: F.gelu(t))
    with torch.no_grad():
        for p in m.parameters():
            p.normal_(0, 0.1)
    m = m.to(torch.bfloat16).cuda()
    params = list(m.parameters())
    flat = torch.randn(2 * T * dim + 2, device="cuda").bfloat16()
    x = flat[1: T * dim + 1].view(T, dim).requires_grad_(True)            # rows that start between 16-byte boundaries
    dy = flat[T * dim + 1: 2 * T * dim + 1].view(T, dim)
    grads = lambda y, d=dy, **kw: torch.autograd.grad(y, [x] + params, d, **kw)
    near = lambda a, b: float((a.float() - b.float()).norm()) <= 1.2e-2 * float(b.float().norm())

    def plain(f):
        os.environ["HEXA_DENSE_KERNELS"] = "0"
        try:
            return f()
        finally:
            del os.environ["HEXA_DENSE_KERNELS"]

    before = ops.LAUNCHES
    y = m(0, x)[0]
    first = grads(y, retain_graph=True)
    assert ops.LAUNCHES - before >= 8                                     # both directions on the kernels
    for a, b in zip(first, grads(y)):
        assert torch.equal(a, b)
    want = plain(lambda: grads(m(0, x)[0]))
    assert all(near(a, b) for a, b in zip(first, want))

    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(1), t.cpu())[1], lambda t: t.cuda()):
        y = m(0, x)[0]
    assert packed and all(torch.equal(a, b) for a, b in zip(first, grads(y)))

    second = lambda: torch.autograd.grad(grads(m(0, x)[0], create_graph=True)[0].float().square().sum(), params[0])[0]
    assert near(second(), plain(second))
    both = torch.stack([dy, -dy])
    batched = grads(m(0, x)[0], both, is_grads_batched=True)
    assert all(near(a[0], b) and near(a[1], -b) for a, b in zip(batched, want))

    w = params[0].data.clone()
    params[0].data = w.t().contiguous().t()                               # columns in memory
    assert all(torch.equal(a, b) for a, b in zip(first, grads(m(0, x)[0])))
    params[0].data = w

    y = m(0, x)[0]
    with torch.no_grad():
        params[0].add_(0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        grads(y)


def test_gelu_of_infinity_is_infinity():
    """As F.gelu has it, in the 16-bit epilogue too; -inf and NaN stay NaN."""
    from hexa_moe_b200 import _lib as L, ops
    r = ops.route(torch.zeros(128, 1, dtype=torch.int32, device="cuda"), 1)
    for dtype in (torch.bfloat16, torch.float16):
        x, w = torch.zeros(128, 64, device="cuda", dtype=dtype), torch.zeros(1, 128, 64, device="cuda", dtype=dtype)
        v = torch.tensor([float("inf"), float("-inf"), float("nan"), 3.0, -3.0, 60000.0], device="cuda").to(dtype)
        x[:6, 0], w[0, :, 0] = v, 1.0
        want = torch.nn.functional.gelu(v)
        for n in (128, 8):
            got = ops.esmm(x, w[:, :n], L.B_NK, r, None, L.EPI_ACT, L.ACT_GELU, engine=L.ENGINE_TCGEN05)[:6]
            assert torch.allclose(got, want[:, None].expand(6, n), rtol=1e-2, atol=1e-2, equal_nan=True)


def _filled(m, dtype, seed=0):
    torch.manual_seed(seed)
    with torch.no_grad():
        for n, p in m.named_parameters():
            p.normal_(0, 0.5 if "gates" in n else 0.1)
    m = m.to(dtype).cuda().eval()
    m.gates.float()
    return m


def _step(m, x, dy, depth=2, loss=True):
    x = x.detach().requires_grad_(True)
    m.zero_grad(set_to_none=True)
    y, l_aux = m(depth, x)
    stage = m.dispatch_params.stage
    torch.autograd.backward([y] + ([l_aux] if loss else []), [dy] + ([torch.ones_like(l_aux)] if loss else []))
    assert m.dispatch_params.stage == stage - 1
    return [y.detach(), l_aux.detach(), x.grad] + [p.grad for p in m.parameters()]


def _same(a, b):
    return len(a) == len(b) and all((u is None) == (v is None) and (u is None or (u.dtype == v.dtype and torch.equal(u, v))) for u, v in zip(a, b))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,d,E,k,b1,b2,act", [(1, 32, 4, 1, True, True, F.gelu), (300, 72, 5, 3, False, True, F.relu), (257, 50, 3, 2, True, False, F.silu),
                                               (4500, 64, 7, 2, True, True, F.gelu), (130, 64, 4, 1, False, False, lambda t: t.tanh())])
def test_native_layer_equals_the_general_path(dtype, T, d, E, k, b1, b2, act):
    """One GPU: the native autograd nodes against the Python functions over the same kernels (which a timed run takes), bit for
    bit, also without the loss, without gradients and for tokens in three dimensions."""
    from hexa_moe_b200 import ops
    m = _filled(_toy(k=k, d=d, E=E, mlp_fc1_bias=b1, mlp_fc2_bias=b2, activation_fn=act), dtype)
    x, dy = torch.randn(T, d, device="cuda").to(dtype), torch.randn(T, d, device="cuda").to(dtype)
    run = lambda: (_step(m, x, dy), _step(m, x, dy, loss=False), _step(m, x[None], dy[None], depth=3))
    native = run()
    with torch.no_grad():
        y = m(2, x)[0]
    assert not y.requires_grad and torch.equal(y, native[0][0])
    try:
        ops.PROFILE = []
        general = run()
    finally:
        ops.PROFILE = None
    assert all(_same(a, b) for a, b in zip(native, general))


def test_native_layer_under_hooks_checkpoints_and_failures():
    from hexa_moe_b200 import _lib as L
    from torch.utils.checkpoint import checkpoint
    m = _filled(_toy(k=2, d=64), torch.bfloat16)
    x, dy = torch.randn(500, 64, device="cuda").bfloat16(), torch.randn(500, 64, device="cuda").bfloat16()
    want = _step(m, x, dy)

    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(1), t.cpu())[1], lambda t: t.cuda()):
        assert _same(_step(m, x, dy), want) and len(packed) >= 4          # tokens and gate weight, logits and counts
    for reentrant in (True, False):
        xi = x.clone().requires_grad_(True)
        m.zero_grad(set_to_none=True)
        y, l_aux = checkpoint(lambda t: m(2, t), xi, use_reentrant=reentrant)
        torch.autograd.backward([y, l_aux], [dy, torch.ones_like(l_aux)])
        assert _same([y.detach(), l_aux.detach(), xi.grad] + [p.grad for p in m.parameters()], want)

    xi = x.clone().requires_grad_(True)
    y, l_aux = m(2, xi)
    with torch.no_grad():
        xi.add_(0)                                                        # the gate's tokens have changed
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        l_aux.backward()

    y, _ = m(2, x.clone().requires_grad_(True))
    y.backward(dy, retain_graph=True)
    with pytest.raises(RuntimeError, match="second time"):                # the layer keeps its state for one pass
        y.backward(dy)

    y, _ = m(2, x.clone().requires_grad_(True))
    word = L.ensure_status_word(0)
    try:
        word[0] = 3                                                       # as if an earlier kernel had given up a wait
        with pytest.raises(L.HexaError, match="gave up a bounded wait"):
            y.backward(dy)
    finally:
        L.clear_device_status(0)
    assert _same(_step(m, x, dy), want)


@pytest.mark.parametrize("T,dim,launches", [(256, 256, 2), (333, 256, 3), (256, 64, 2)])
def test_dense_depths_without_gradients_write_no_state(T, dim, launches):
    """Under no_grad a dense depth is its two GEMMs, after a gather where the tokens do not fill whole tiles, and the
    pre-activation, which only a backward pass reads, is not written; the output is that of a pass with gradients."""
    import torch.nn.functional as F
    from hexa_moe import moe as hmoe
    from hexa_moe_b200 import ops
    torch.manual_seed(dim)
    m = hmoe.MoE_Cascaded(gate_type={'type': 'top', 'k': 1}, model_dim_list=[dim], moe_idx_list=[], mlp_ratio=4,
                          num_global_experts=1, total_depth=1, data_centric=True, activation_fn=lambda t: F.gelu(t))
    m = m.to(torch.bfloat16).cuda()
    x = torch.randn(T, dim, device="cuda").bfloat16()
    want = m(0, x)[0].detach()
    kept = []
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            m(0, x)                                       # the routing's tables are built once
            torch.cuda.synchronize()
            torch.cuda.reset_peak_memory_stats()
            base, before = torch.cuda.memory_allocated(), ops.LAUNCHES
            y = m(0, x)[0]
            assert ops.LAUNCHES - before == launches and torch.equal(y, want)
            kept.append(torch.cuda.max_memory_allocated() - base)
    rows = (T + 127) // 128 * 128
    assert max(kept) < rows * (4 * dim + dim + dim + 2 * dim) * 2      # hidden, output, rows of its own; no second [rows, hidden]
