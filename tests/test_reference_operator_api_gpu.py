"""The reference's operator-level API (`counter`, `ESMM`, `es_fused`: same names, arguments and return values) on
the CUDA kernels, checked against the golden outputs of the reference's own Triton kernels (tests/golden/*.npz)."""
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _cases(z):
    return sorted({k.split("/")[0] for k in z.files})


def test_counter_equals_reference_lists(golden_dir):
    from hexa_moe_b200.kernels.basics import counter
    z = np.load(os.path.join(golden_dir, "counter.npz"))
    for c in _cases(z):
        n, starts, tok, exp = counter(torch.from_numpy(z[c + "/routing"]).cuda(), int(z[c + "/E"]))
        assert n == int(z[c + "/n"])
        assert np.array_equal(starts.cpu().numpy(), z[c + "/starts"])
        assert np.array_equal(tok.cpu().numpy(), z[c + "/tok_ids"])       # ascending inside a segment = stable sort
        assert np.array_equal(exp.cpu().numpy(), z[c + "/exp_ids"])


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-3), (torch.float16, 2e-3)])
def test_esmm_and_fused_dx_equal_reference_outputs(golden_dir, dtype, tol):
    """The reference rounds both operands to fp16 and accumulates in fp32.  fp16 inputs here reproduce that rounding
    (the result differs only by the fp16 rounding of the output); fp32 inputs are NOT rounded by this library, so the
    distance to the golden values is the reference's own operand-rounding error (~1e-3)."""
    from hexa_moe_b200.kernels.basics import counter
    from hexa_moe_b200.kernels.esmm import ESMM
    from hexa_moe_b200.kernels.fused import es_fused
    z = np.load(os.path.join(golden_dir, "esmm.npz"))
    for c in _cases(z):
        x, w, b, dy = (torch.from_numpy(z[f"{c}/{k}"]).cuda() for k in ("x", "w", "b", "dy"))
        routing = torch.from_numpy(z[c + "/routing"]).cuda()
        E = int(z[c + "/E"])
        n, starts, tok, exp = counter(routing, E)
        y_b = ESMM(x.to(dtype), w.to(dtype), b, (tok + 1).contiguous(), exp)
        y_nb = ESMM(x.to(dtype), w.to(dtype), torch.empty(0, device="cuda"), (tok + 1).contiguous(), exp)
        wt = w.permute(0, 2, 1).contiguous()                    # es_fused takes [E, out, in] (reference layers.py:407)
        r_ess, dx, r_dw = es_fused(dy.to(dtype), x.to(dtype), wt.to(dtype), (tok + 1).contiguous(), exp, starts, E, bias=True)
        for got, key in ((y_b, "y_bias"), (y_nb, "y_nobias"), (dx, "dx")):
            want = torch.from_numpy(z[f"{c}/{key}"])
            err = float((got.float().cpu() - want).abs().max() / want.abs().max())
            assert err < tol, (c, key, err)
        assert y_b.dtype == dtype and y_b.shape == (x.shape[0], w.shape[2])


def test_fused_ess_estmm_equal_reference_where_it_is_correct(golden_dir):
    from hexa_moe_b200.kernels.basics import counter
    from hexa_moe_b200.kernels.fused import es_fused
    z = np.load(os.path.join(golden_dir, "estmm_ess.npz"))
    for c in _cases(z):
        x, w, dy = (torch.from_numpy(z[f"{c}/{k}"]).cuda() for k in ("x", "w", "dy"))
        routing = torch.from_numpy(z[c + "/routing"]).cuda()
        E = int(z[c + "/E"])
        n, starts, tok, exp = counter(routing, E)
        wt = w.permute(0, 2, 1).contiguous().half()
        r_ess, dx, r_dw = es_fused(dy.half(), x.half(), wt, (tok + 1).contiguous(), exp, starts, E, bias=True)
        ess_ref, dw_ref = z[c + "/ess"], z[c + "/estmm"]
        written = ~np.isnan(ess_ref).any(axis=1)              # the reference never writes trailing empty experts
        got_ess, got_dw = r_ess.float().cpu().numpy(), r_dw.float().cpu().numpy()
        assert np.abs(got_ess[written] - ess_ref[written]).max() / np.abs(ess_ref[written]).max() < 2e-3
        assert np.abs(got_dw[written] - dw_ref[written]).max() / np.abs(dw_ref[written]).max() < 2e-3
        counts = np.bincount(routing.cpu().numpy(), minlength=E)
        assert (got_ess[counts == 0] == 0).all() and (got_dw[counts == 0] == 0).all()


@pytest.mark.parametrize("T,n,dtype", [(1, 16, torch.int32), (300, 4096, torch.int32), (257, 320, torch.int64), (40, 0, torch.int32)])
def test_expert_ids_from_lists(T, n, dtype):
    """Pads (0), tokens in no segment, a list longer than a block and an empty one, against the indexing formulation."""
    from hexa_moe_b200.kernels.esmm import ids_from_lists
    g = torch.Generator().manual_seed(T + n)
    tok = torch.zeros(n, dtype=torch.int64)
    slots = torch.randperm(n, generator=g)[: min(T * 2 // 3 + 1, n)]
    tok[slots] = torch.randperm(T, generator=g)[: len(slots)] + 1
    exp = torch.randint(0, 9, (n // 16,), generator=g, dtype=torch.int32)
    want = torch.full((T + 1,), -1, dtype=torch.int32)
    want[tok] = exp.repeat_interleave(16)
    got = ids_from_lists(T, tok.to(dtype).cuda(), exp.cuda())
    assert got.dtype == torch.int32 and torch.equal(got.cpu(), want[1:])


def test_expert_ids_refuse_lists_on_another_device():
    from hexa_moe_b200 import _lib as L, ops
    tok, exp = torch.ones(16, dtype=torch.int32), torch.zeros(1, dtype=torch.int32)
    for a, b in ((tok.cuda(), exp), (tok, exp.cuda())):
        with pytest.raises(L.HexaError):
            ops.ids_from_lists(4, a, b, 16)
    with pytest.raises(L.HexaError, match="cover"):                   # 16 entries per expert id
        ops.ids_from_lists(4, tok.cuda().repeat(2), exp.cuda(), 16)


@pytest.mark.parametrize("bad,dtype", [(6, torch.int32), (-7, torch.int32), (6, torch.int64), ((1 << 32) + 2, torch.int64)])
def test_expert_ids_report_a_token_that_is_not_there(bad, dtype):
    """The kernel's bounds check skips the entry and leaves a code that the next call raises; entries that index, from
    either end, are taken."""
    from hexa_moe_b200 import _lib as L, ops
    tok = torch.tensor([1, 5, -1, -6] + [0] * 12, dtype=dtype)
    exp = torch.tensor([3], dtype=torch.int32).cuda()
    assert ops.ids_from_lists(5, tok.cuda(), exp, 16).tolist() == [3, -1, -1, -1, 3]
    tok[7] = bad
    ids = ops.ids_from_lists(5, tok.cuda(), exp, 16)
    torch.cuda.synchronize()
    assert ids.tolist() == [3, -1, -1, -1, 3] and L.device_status() == L.STATUS_BAD_TOKEN
    try:
        with pytest.raises(L.HexaError, match="index out of range"):
            ops.route(ids.view(-1, 1), 4)
    finally:
        L.clear_device_status()
    ops.route(ids.view(-1, 1), 4)
