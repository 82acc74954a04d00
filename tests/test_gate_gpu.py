"""softmax + top-k + GShard loss kernels (hexa_gate_topk / hexa_gate_loss_grad) against the CPU oracle's restatement
of the reference chain F.softmax -> torch.topk -> gshard_loss (cascaded_moe.py:568-598, layers.py:480-489,
losses.py:12-19).  Index work is bit-exact; the float outputs are held to 1e-5 of their scale (fp32 summation order)."""
import pytest
import torch
import torch.nn.functional as F

from oracle import hexa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


CASES = [(1000, 64, 2), (257, 7, 1), (4096, 8, 4), (33, 300, 3), (5, 512, 8), (16, 1, 1), (1, 4, 4), (70000, 32, 1)]


@pytest.mark.parametrize("T,E,k", CASES)
def test_ids_loss_and_counts_match_the_oracle(T, E, k):
    from hexa_moe_b200 import ops
    g = torch.Generator().manual_seed(T * 31 + E)
    logits = torch.randn(T, E, generator=g) * 2.0
    ids, loss, first_count, mass = ops.gate_topk(logits.cuda(), k)
    scores = F.softmax(logits, dim=1)
    want = torch.topk(scores, k, dim=1)
    got = ids.cpu().t().long()                                   # [T, k]
    assert got.shape == (T, k) and ids.dtype == torch.int32
    same = got == want.indices
    if not bool(same.all()):
        # two scores within an ulp of each other may swap; nothing else may differ
        picked = scores.gather(1, got)
        assert torch.allclose(picked, want.values, rtol=1e-6, atol=0)
        assert float(same.float().mean()) > 0.999
    for t in range(0, T, max(T // 50, 1)):                       # k distinct experts per token
        assert len(set(got[t].tolist())) == k
    assert torch.equal(first_count.cpu().long(), torch.bincount(got[:, 0], minlength=E))
    assert torch.allclose(mass.cpu(), scores.sum(0), rtol=1e-5, atol=1e-6)
    want_loss = O.gshard_loss(scores.double(), got)
    assert abs(float(loss) - float(want_loss)) <= 1e-5 * abs(float(want_loss))


def test_equal_scores_go_to_the_lowest_expert_ids():
    from hexa_moe_b200 import ops
    logits = torch.zeros(64, 40, device="cuda")
    logits[:, 17] = 1.0                                         # one clear winner, everything else tied
    ids, _, first_count, _ = ops.gate_topk(logits, 3)
    assert ids.cpu().tolist() == [[17] * 64, [0] * 64, [1] * 64]
    assert int(first_count[17]) == 64 and int(first_count.sum()) == 64


@pytest.mark.parametrize("T,E,k", [(1000, 64, 2), (33, 300, 3), (4096, 8, 1)])
def test_loss_gradient_matches_autograd_of_the_reference_formulation(T, E, k):
    from hexa_moe_b200 import ops
    g = torch.Generator().manual_seed(7 + T)
    logits = torch.randn(T, E, generator=g)
    ref = logits.double().requires_grad_(True)
    scores = F.softmax(ref, dim=1)
    top = torch.topk(scores, k, dim=1).indices
    loss = O.gshard_loss(scores, top)
    (loss * 3.0).backward()
    dev = logits.cuda()
    _, _, first_count, _ = ops.gate_topk(dev, k)
    got = ops.gate_loss_grad(dev, first_count, torch.tensor(3.0, device="cuda"))
    scale = float(ref.grad.abs().max())
    assert float((got.cpu().double() - ref.grad).abs().max()) <= 1e-5 * scale


def test_module_routes_through_the_fused_gate_and_matches_the_pytorch_chain():
    """Same layer, same input: the fused gate step and the PyTorch-op chain give the same output, auxiliary loss and
    input gradient (2e-2, the bf16 tolerance of the layer; the gate itself is fp32 either way)."""
    import os
    from hexa_moe import moe as hmoe
    from hexa_moe_b200 import ops
    torch.manual_seed(11)
    m = hmoe.MoE_Cascaded(gate_type={'type': 'top', 'k': 2, 'fp32_gate': True}, model_dim_list=[64], moe_idx_list=[0],
                          mlp_ratio=4, num_global_experts=8, total_depth=1, data_centric=True,
                          activation_fn=lambda t: F.gelu(t))
    with torch.no_grad():
        for n_, p in m.named_parameters():
            p.normal_(0, 0.3 if "gates" in n_ else 0.1)
    m = m.to(torch.bfloat16).cuda().train()
    x = torch.randn(300, 64, device="cuda").bfloat16()

    def run():
        xi = x.clone().requires_grad_(True)
        y, aux = m(0, xi)
        (y.float().sum() + 5.0 * aux).backward()
        return y.detach().float(), float(aux), xi.grad.float(), m.gates[0].wg.weight.grad.clone()

    m.zero_grad()
    before = ops.LAUNCHES
    fused = run()
    n_fused = ops.LAUNCHES - before
    os.environ["HEXA_FUSED_GATE"] = "0"
    try:
        m.zero_grad()
        before = ops.LAUNCHES
        plain = run()
        n_plain = ops.LAUNCHES - before
    finally:
        del os.environ["HEXA_FUSED_GATE"]
    assert n_fused == n_plain + 2                                # one gate kernel each way
    assert abs(fused[1] - plain[1]) <= 1e-5 * abs(plain[1])
    for a, b in ((fused[0], plain[0]), (fused[2], plain[2]), (fused[3], plain[3])):
        assert float((a - b).abs().max()) <= 2e-2 * float(b.abs().max())


@pytest.mark.parametrize("T,E,k", [(1000, 64, 2), (257, 7, 1), (4096, 8, 4), (33, 300, 3), (70000, 32, 2)])
def test_load_importance_ids_loss_and_gradient_match_the_oracle(T, E, k):
    """The other auxiliary loss of the reference (is_gshard_loss=False, impls/losses.py:21-43): ids of the noisy logits
    bit-exact, loss and its gradient against float64 autograd of the oracle's restatement (1e-5 of their scale), and
    bit-identical outputs from run to run."""
    from hexa_moe_b200 import ops
    g = torch.Generator().manual_seed(T + E)
    logits = torch.randn(T, E, generator=g) * 0.05
    gate_noise = 1.0
    noisy = logits + gate_noise * torch.randn(T, E, generator=g) / E
    ids, loss, importance, load = ops.gate_topk_load_importance(logits.cuda(), noisy.cuda(), k, gate_noise / E)
    got = ids.cpu().t().long()
    assert torch.equal(got, torch.topk(noisy, k, dim=1).indices)          # the kernel ranks the noisy logits themselves
    # the reference ranks softmax(noisy) in fp32, where two different logits can round to the same score: the picks may
    # differ there, and only there (the picked scores agree to an ulp)
    scores = F.softmax(noisy, dim=1)
    ref_pick = torch.topk(scores, k, dim=1)
    assert torch.allclose(scores.gather(1, got), ref_pick.values, rtol=1e-6, atol=0)
    assert float((got == ref_pick.indices).float().mean()) > 0.99
    ref = logits.double().requires_grad_(True)
    noisy_ref = ref + (noisy.double() - logits.double())
    want = O.load_importance_loss(F.softmax(ref, dim=1), noisy_ref.gather(1, got), E, gate_noise)
    # the loss is a variance of nearly equal column sums over their squared mean: fp32 sums (1e-6 relative) are amplified
    # by mean / spread; the reference evaluates it in fp32 as well
    assert abs(float(loss) - float(want)) <= 2e-3 * abs(float(want)), (float(loss), float(want))
    assert torch.allclose(importance.cpu().double(), F.softmax(ref, dim=1).sum(0).detach(), rtol=1e-5, atol=1e-6)
    z = (F.softmax(ref, dim=1).detach() - noisy.double().gather(1, got)[:, -1:]) / (gate_noise / E)
    assert torch.allclose(load.cpu().double(), (0.5 * (1 + torch.erf(z / 2 ** 0.5))).sum(0), rtol=1e-4, atol=1e-5)
    (want * 3.0).backward()
    grad = ops.gate_load_importance_grad(logits.cuda(), noisy.cuda(), k, gate_noise / E, importance, load,
                                         torch.tensor(3.0, device="cuda"))
    scale = float(ref.grad.abs().max())
    # fp32 kernel against float64: the gradient factors of var / mean^2 are differences of nearly equal column sums
    assert float((grad.cpu().double() - ref.grad).abs().max()) <= 5e-3 * scale
    again = ops.gate_topk_load_importance(logits.cuda(), noisy.cuda(), k, gate_noise / E)
    for a, b in zip((ids, loss, importance, load), again):
        assert torch.equal(a, b)


def test_module_with_the_load_importance_loss_takes_the_fused_gate():
    """is_gshard_loss=False in training mode: the fused kernels and the PyTorch chain (HEXA_FUSED_GATE=0) see the same
    noise (same seed) and give the same output, auxiliary loss and gradients."""
    import os
    from hexa_moe import moe as hmoe
    from hexa_moe_b200 import ops
    torch.manual_seed(12)
    m = hmoe.MoE_Cascaded(gate_type={'type': 'top', 'k': 2, 'fp32_gate': True, 'gate_noise': 1.0}, model_dim_list=[64],
                          moe_idx_list=[0], mlp_ratio=4, num_global_experts=8, total_depth=1, data_centric=True,
                          is_gshard_loss=False, activation_fn=lambda t: F.gelu(t))
    with torch.no_grad():
        for n_, p in m.named_parameters():
            p.normal_(0, 0.02 if "gates" in n_ else 0.1)
    m = m.to(torch.bfloat16).cuda().train()
    x = torch.randn(300, 64, device="cuda").bfloat16()

    def run():
        torch.manual_seed(99)                        # the same noise draw both times
        xi = x.clone().requires_grad_(True)
        y, aux = m(0, xi)
        (y.float().sum() + 5.0 * aux).backward()
        return y.detach().float(), float(aux), xi.grad.float(), m.gates[0].wg.weight.grad.clone()

    m.zero_grad()
    before = ops.LAUNCHES
    fused = run()
    n_fused = ops.LAUNCHES - before
    os.environ["HEXA_FUSED_GATE"] = "0"
    try:
        m.zero_grad()
        before = ops.LAUNCHES
        plain = run()
        n_plain = ops.LAUNCHES - before
    finally:
        del os.environ["HEXA_FUSED_GATE"]
    assert n_fused == n_plain + 2                                # one gate kernel each way
    assert abs(fused[1] - plain[1]) <= 1e-4 * abs(plain[1])
    for a, b in ((fused[0], plain[0]), (fused[2], plain[2]), (fused[3], plain[3])):
        assert float((a - b).abs().max()) <= 2e-2 * float(b.abs().max())


# Edges of the group kernels: the lane-group widths (8 lanes up to 64 experts, 16 up to 128, 32 beyond), column counts
# around them, token counts around one block's sweeps and around a grid-stride step, and rows with a leading dimension.
@pytest.mark.parametrize("E", [1, 8, 9, 16, 17, 33, 64, 65, 128, 129, 256, 257, 512])
@pytest.mark.parametrize("T", [1, 33, 256, 257, 512, 513, 15000])
def test_group_kernels_at_their_edges(T, E):
    from hexa_moe_b200 import ops
    k = min(E, 3)
    g = torch.Generator(device="cuda").manual_seed(T * 1000 + E)
    wide = torch.randn(T, E + 3, generator=g, device="cuda") * 2.0
    logits = wide[:, :E]
    if E >= 4:
        logits[T // 2] = float("nan")                     # the lowest free ids, NaN only in the sums
    ids, loss, first_count, mass = ops.gate_topk(logits, k)
    live = torch.ones(T, dtype=torch.bool, device="cuda")
    if E >= 4:
        assert ids[:, T // 2].tolist() == list(range(k))
        assert torch.isnan(loss) and torch.isnan(mass).all()
        live[T // 2] = False
        ids2, loss, first2, mass = ops.gate_topk(logits[live], k) if T > 1 else (None, None, None, None)
        if T == 1:
            return
        assert torch.equal(ids2, ids[:, live])
        logits, ids, first_count = logits[live].contiguous(), ids2, first2
    n = logits.shape[0]
    scores = F.softmax(logits.double(), dim=1)
    want = torch.topk(scores, k, dim=1)
    picked = scores.gather(1, ids.t().long())
    assert torch.allclose(picked, want.values, rtol=1e-6, atol=0)       # equal up to scores within an ulp of each other
    assert torch.equal(first_count.long(), torch.bincount(ids[0].long(), minlength=E))
    assert torch.allclose(mass.double(), scores.sum(0), rtol=1e-5, atol=1e-6)
    ce = first_count.double() * (E / n)
    want_loss = (scores.sum(0) * ce).sum() / n
    assert abs(float(loss) - float(want_loss)) <= 1e-5 * float(want_loss)
    got = ops.gate_loss_grad(logits, first_count, torch.tensor(2.0, device="cuda"))
    ge = 2.0 * ce / n
    want_g = scores * (ge - (scores * ge).sum(1, keepdim=True))
    # products of fp32 scores (relative error ~1e-6 with expf and the division) with g up to max(g)
    assert float((got.double() - want_g).abs().max()) <= 4e-6 * float(ge.max())


@pytest.mark.parametrize("T,d,E", [(1, 8, 1), (37, 72, 7), (300, 64, 8), (1000, 40, 33)])
def test_split_precision_gate_terms(T, d, E):
    """The split projection equals the fp32 products to fp32 accuracy and its gradients agree with the formulation in
    plain operations that create_graph takes."""
    from hexa_moe_b200 import ops
    from hexa_moe_b200.impls.gating import _SplitPrecisionLinear, _split_terms
    g = torch.Generator(device="cuda").manual_seed(d)
    x = torch.randn(T, d, generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = torch.randn(E, d, generator=g, device="cuda").requires_grad_(True)
    t = _split_terms(w.detach(), torch.bfloat16, 3)
    assert torch.equal(ops.gate_split_terms(w.detach(), True), torch.cat([t[2], t[1], t[0], t[0]], dim=0))
    dy = torch.randn(T, E, generator=g, device="cuda")
    t = _split_terms(dy, torch.bfloat16, 3)
    assert torch.equal(ops.gate_split_terms(dy, False), torch.cat([t[0], t[0], t[1], t[2]], dim=1))
    y = _SplitPrecisionLinear.apply(x, w)
    exact = x.double() @ w.double().t()
    bound = (x.double().abs() @ w.double().abs().t()) * ((3 * d + 3) * 2.0 ** -24)      # 3d fp32 additions
    assert ((y.double() - exact).abs() <= bound + 1e-30).all()
    dx, dw = torch.autograd.grad(y, (x, w), dy)
    y2 = _SplitPrecisionLinear.apply(x, w)
    dx2, dw2 = torch.autograd.grad(y2, (x, w), dy, create_graph=True)
    # dw: 3T fp32 additions either way; dx: one bf16 rounding (2^-8 between neighbours) of sums of 3E terms
    bw = (dy.double().abs().t() @ x.double().abs()) * ((3 * T + 3) * 2.0 ** -23)
    assert ((dw - dw2).double().abs() <= bw + 1e-30).all()
    bx = (dy.double().abs() @ w.double().abs()) * ((3 * E + 3) * 2.0 ** -23)
    assert ((dx - dx2).double().abs() <= dx.double().abs() * 2.0 ** -7 + bx + 1e-30).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("T,d,E", [(1, 8, 1), (5, 264, 3), (63, 72, 7), (300, 64, 33), (4096, 200, 8), (130, 1024, 64)])
def test_direct_gate_projection(T, d, E, dtype):
    """Few-token projection and its gradients: within the bound of an fp32 sum of that many terms of the exact values, and
    in agreement with the formulation that create_graph takes."""
    from hexa_moe_b200.impls.gating import _DirectLinear, _direct_linear_applies
    g = torch.Generator(device="cuda").manual_seed(d + T)
    lin = torch.nn.Linear(d, E, bias=False, device="cuda")
    x = torch.randn(T, d + 8, generator=g, device="cuda").to(dtype)[:, :d].requires_grad_(True)      # a row pitch
    assert _direct_linear_applies(lin, x)
    w, dy = lin.weight, torch.randn(T, E, generator=g, device="cuda")
    y = _DirectLinear.apply(x, w)
    X, W, DY = x.detach().double(), w.detach().double(), dy.double()
    assert ((y.double() - X @ W.t()).abs() <= X.abs() @ W.abs().t() * (d * 2.0 ** -24) + 1e-30).all()
    dx, dw = torch.autograd.grad(y, (x, w), dy)
    assert dx.dtype == dtype and dw.dtype == torch.float32
    assert ((dw.double() - DY.t() @ X).abs() <= DY.abs().t() @ X.abs() * (max(T, 8) * 2.0 ** -24) + 1e-30).all()
    half = torch.finfo(dtype).eps / 2                      # one rounding of an fp32 sum of E terms (tiny: fp16's subnormals)
    want = DY @ W
    assert ((dx.double() - want).abs() <= want.abs() * half * 1.01 + DY.abs() @ W.abs() * (E * 2.0 ** -24) + 3e-8).all()
    dx2, dw2 = torch.autograd.grad(_DirectLinear.apply(x, w), (x, w), dy, create_graph=True)
    assert ((dx2 - dx).double().abs() <= want.abs() * half * 2.1 + DY.abs() @ W.abs() * (E * 2.0 ** -23) + 6e-8).all()
    assert ((dw2 - dw).double().abs() <= DY.abs().t() @ X.abs() * (max(T, 8) * 2.0 ** -23) + 1e-30).all()
    only = torch.autograd.grad(_DirectLinear.apply(x.detach(), w), w, dy)[0]
    assert torch.equal(only, dw)


def test_direct_gate_projection_leaves_the_linear_to_who_watches_it():
    """Backward hooks on the gate's linear fire whatever the batch size, torch.func and forward-mode AD pass through it, and
    rows without a pitch of their own (expanded tokens) are taken."""
    from hexa_moe_b200.impls import gating
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(64, 128, generator=g, device="cuda")
    for dtype in (torch.float32, torch.float16):
        gate = gating.LinearTopKGate(128, 8, fp32_gate=True).cuda()
        fired = []
        gate.wg.register_full_backward_hook(lambda *a: fired.append("post"))
        gate.wg.register_full_backward_pre_hook(lambda *a: fired.append("pre"))
        gate(x.to(dtype).clone().requires_grad_(True)).sum().backward()
        assert sorted(fired) == ["post", "pre"]
    gate = gating.LinearTopKGate(128, 8, fp32_gate=True).cuda()
    w = gate.wg.weight.detach()
    want = x @ w.t()
    # sums of 128 fp32 products of O(1) and O(0.1): within 1e-5 of each other in any order
    near = lambda a, b: torch.allclose(a, b, rtol=1e-5, atol=1e-5)
    assert near(torch.func.vmap(gate)(x.view(4, 16, 128)).view(64, 8), want)
    y, dy = torch.func.jvp(gate, (x,), (x,))
    assert near(y, want) and near(dy, want)
    row = x[:1].expand(64, 128)
    assert not gating._direct_linear_applies(gate.wg, row)
    assert near(gate(row), want[:1].expand(64, 8))
    # batched gradients and saved tensors that come back with another layout
    xi = x.clone().requires_grad_(True)
    assert gating._direct_linear_applies(gate.wg, xi)
    eye = torch.eye(8, device="cuda")[:, None].expand(8, 64, 8)
    (dx,) = torch.autograd.grad(gate(xi), xi, eye, is_grads_batched=True)
    assert near(dx, w[:, None].expand(8, 64, 128))
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.t().contiguous().t()):
        y = gate(xi)
    (dx,) = torch.autograd.grad(y.sum(), xi)
    assert near(dx, w.sum(0).expand(64, 128))


def test_split_precision_gate_under_modes_and_batched_gradients():
    """Tokens beyond the direct projection: dispatch modes see operations, and a batch of gradients passes through."""
    from torch.utils.flop_counter import FlopCounterMode
    from hexa_moe_b200.impls import gating
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(5000, 64, generator=g, device="cuda").bfloat16().requires_grad_(True)
    gate = gating.LinearTopKGate(64, 8, fp32_gate=True).cuda()
    w = gate.wg.weight
    dy = torch.randn(5000, 8, generator=g, device="cuda")
    y = gate(x)
    with FlopCounterMode(display=False) as flops:
        seen = gate(x)
    assert flops.get_total_flops() > 0 and torch.allclose(y, seen, rtol=1e-5, atol=1e-5)      # sums of 64 terms, in fp32
    dx, dw = torch.autograd.grad(y, (x, w), dy)
    bx, bw = torch.autograd.grad(gate(x), (x, w), torch.stack([dy, 2 * dy]), is_grads_batched=True)
    for b, d in ((bx, dx), (bw, dw)):
        assert float((b[0] - d).float().norm()) <= 1e-2 * float(d.float().norm())             # one bf16 rounding of dx
        assert float((b[1] - 2 * d).float().norm()) <= 1e-2 * float((2 * d).float().norm())


# The scores are quotients bit for bit, whatever way they are taken: a block's few tokens and several blocks of them, group sizes
# 8 to 32, ordinary rows and rows with exponentials too small for the remainder correction; equal scores go to the lowest id.
@pytest.mark.parametrize("E", [1, 7, 9, 33, 64, 100, 200, 500])
@pytest.mark.parametrize("T", [3, 2000])
def test_selection_follows_the_ieee_quotients(E, T):
    from hexa_moe_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(E + T)
    logits = torch.randint(-6, 7, (T, E), generator=g, device="cuda").float()          # many equal scores
    logits[::3] *= 20.0                                                                # e^-200: below 2^-90, down to zero
    k = min(4, E)
    ids, _, first, mass = ops.gate_topk(logits, k)
    order = torch.sort(logits, dim=1, descending=True, stable=True).indices[:, :k]     # integers: distinct logits, distinct scores
    # scores that underflow to zero tie as well, so compare where the k-th score is not zero
    live = (logits.gather(1, order[:, -1:]) - logits.max(1, keepdim=True).values)[:, 0] > -80
    assert bool(live.any()) and torch.equal(ids.t()[live].long(), order[live])
    assert torch.equal(first, torch.bincount(ids[0].long(), minlength=E).int())
    assert torch.allclose(mass.double(), torch.softmax(logits.double(), 1).sum(0), rtol=1e-5, atol=1e-6)


def _warp_order_sum(e):
    """fp32 sum of a row's exponentials in the kernel's order: columns c mod 32 in turn, then pairs 16, 8, 4, 2, 1 apart."""
    import numpy as np
    cls = np.zeros(32, np.float32)
    for c in range(0, len(e), 32):
        part = e[c:c + 32]
        cls[:len(part)] += part
    at = np.arange(32)
    for o in (16, 8, 4, 2, 1):
        cls = cls + cls[at ^ o]
    assert (cls == cls[0]).all()
    return cls[0]


# One token's column sums of the softmax are its scores.  Ordinary logits; exponentials on both sides of 2^-90 = e^-62.4 and down
# to zero; sums a few steps below whole numbers, whose significands are nearly all ones where the number is a power of two.
@pytest.mark.parametrize("E", [1, 2, 4, 7, 8, 9, 16, 31, 33, 64, 100, 200, 256, 500])
def test_scores_are_the_ieee_quotients_bit_for_bit(E):
    import numpy as np
    from hexa_moe_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(E)
    rand = lambda: torch.rand(1, E, generator=g, device="cuda")
    near = lambda: -torch.randint(0, 5, (1, E), generator=g, device="cuda").float() * 2.0 ** -23
    rows = []
    for _ in range(6):
        rows += [3 * torch.randn(1, E, generator=g, device="cuda"), -100 * rand(), -60 - 5 * rand(), near(),
                 torch.where(rand() < 0.3, -61.5 - 2 * rand(), near())]
        rows[-3][0, int(torch.randint(0, E, (1,), generator=g, device="cuda"))] = 0.0
    products_differ = 0
    for l in rows:
        mass = ops.gate_topk(l, min(4, E))[3]
        e = torch.exp(l - l.max())[0].cpu().numpy()
        total = _warp_order_sum(e)
        want = e / total
        assert want.dtype == np.float32 and np.array_equal(mass.cpu().numpy(), want)
        products_differ += int((e * (np.float32(1) / total) != want).sum())
    assert products_differ or E <= 2 or E in (4, 8)      # these rows tell quotients from products with the reciprocal


@pytest.mark.parametrize("E", [16, 64, 128, 200])
def test_equal_scores_of_lanes_that_go_different_ways(E):
    """Pairs of equal logits, one of them in a lane with an exponential below 2^-90: the lower id comes first."""
    from hexa_moe_b200 import ops
    T, lanes = 300, 8 if E <= 64 else 16 if E <= 128 else 32
    g = torch.Generator(device="cuda").manual_seed(E)
    logits = -20 - 10 * torch.rand(T, E, generator=g, device="cuda")
    cols = torch.stack([torch.randperm(E, generator=g, device="cuda") for _ in range(T)])
    at = torch.arange(T, device="cuda")
    for level in range(2):      # two pairs a token, e apart
        logits[at, cols[:, 2 * level]] = logits[at, cols[:, 2 * level + 1]] = -float(level)
    tiny = cols[:, 4:].clone()                            # of the other columns, those in the lane of the first pair's first
    tiny[(tiny % lanes) != (cols[:, :1] % lanes)] = -1
    for t in range(T):
        logits[t, tiny[t][tiny[t] >= 0]] = -70.0
    ids = ops.gate_topk(logits, 4)[0]
    assert torch.equal(ids.t().long(), torch.sort(logits, dim=1, descending=True, stable=True).indices[:, :4])
