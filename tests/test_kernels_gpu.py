"""Parity of every CUDA operator with the CPU oracle, called through the C ABI.  Needs a B200.

Tolerances (stated by the task): routing and indices bit-exact; fp32 within 1e-5 relative;
16-bit within 2e-2 relative.  "Relative" is measured against the largest magnitude of the
expected tensor (norm-wise), the usual meaning for accumulated dot products.
"""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from oracle import hexa_oracle as O

pytestmark = pytest.mark.gpu

REL = {torch.float32: 1e-5, torch.float16: 2e-2, torch.bfloat16: 2e-2}


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hexa_moe_b200 import ops as _ops
    return _ops


def L():
    from hexa_moe_b200 import _lib
    return _lib


def rel_err(got, want):
    got = got.detach().double().cpu(); want = want.detach().double().cpu()
    return float((got - want).abs().max() / want.abs().max().clamp_min(1e-30))


def make_ids(T, k, E, seed, skew=False, empty=()):
    g = torch.Generator().manual_seed(seed)
    if skew:
        p = torch.arange(1, E + 1, dtype=torch.float64) ** -1.2
    else:
        p = torch.ones(E, dtype=torch.float64)
    for e in empty:
        p[e] = 0
    ids = torch.multinomial(p.expand(T, E), k, replacement=False, generator=g)
    return ids.to(torch.int32)


# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("T,k,E,align", [(100, 1, 4, 16), (1000, 2, 8, 128), (4097, 2, 64, 128), (513, 4, 7, 128),
                                         (64, 1, 3, 128), (1, 1, 5, 128), (3000, 2, 300, 16)])
def test_route_bit_exact(ops, T, k, E, align):
    ids = make_ids(T, k, E, seed=T + k, skew=(E > 4), empty=(1,) if E > 2 else ())
    if T > 50:
        ids[5, 0] = -1          # out-of-range ids are skipped, as in the reference kernels
        ids[7, k - 1] = E
    r = ops.route(ids.cuda(), E, align)
    want = O.route(ids, E, align)
    n_pad = want["n_pad"]
    assert torch.equal(r.counts.cpu(), want["counts"])
    assert torch.equal(r.seg_offsets.cpu(), want["seg_offsets"])
    assert torch.equal(r.pad_offsets.cpu(), want["pad_offsets"])
    assert torch.equal(r.row_token.cpu()[:n_pad], want["row_token"])
    assert torch.equal(r.token_row.cpu()[: T * k], want["token_row"])
    te = r.tile_expert.cpu()
    assert torch.equal(te[: n_pad // align], want["tile_expert"])
    assert (te[n_pad // align: r.row_capacity // align] == -1).all()
    if align == 128:
        pb = r.pair_block.cpu()
        n_pairs = want["pair_block"].numel()
        assert torch.equal(pb[:n_pairs], want["pair_block"]) and (pb[n_pairs:] == -1).all() and pb.numel() > n_pairs
    else:
        assert r.pair_block is None
    # route-major ids ([k, T]) give the same answer
    r2 = ops.route(ids.t().contiguous().cuda(), E, align, route_major=True)
    assert torch.equal(r2.row_token.cpu()[:n_pad], want["row_token"])
    assert torch.equal(r2.token_row.cpu()[: T * k], want["token_row"])


def test_route_matches_reference_counter(ops, golden_dir):
    """align=16 reproduces the reference's own lists (golden fixture from kernels/basics.py:counter)."""
    import os
    z = np.load(os.path.join(golden_dir, "counter.npz"))
    for c in sorted({k.split("/")[0] for k in z.files}):
        routing = torch.from_numpy(z[c + "/routing"]); E = int(z[c + "/E"])
        r = ops.route(routing.view(-1, 1).cuda(), E, 16)
        n = int(z[c + "/n"])
        assert int(r.pad_offsets[-1]) == n
        assert np.array_equal(r.pad_offsets.cpu().numpy(), z[c + "/starts"])
        assert np.array_equal(r.row_token.cpu().numpy()[:n], z[c + "/tok_ids"])
        assert np.array_equal(r.tile_expert.cpu().numpy()[: n // 16], z[c + "/exp_ids"])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [64, 200, 3])
def test_gather_combine(ops, dtype, cols):
    T, k, E = 777, 2, 6
    ids = make_ids(T, k, E, 3, empty=(2,))
    r = ops.route(ids.cuda(), E)
    want = O.route(ids, E, 128)
    x = torch.randn(T, cols).to(dtype)
    xs = ops.gather_rows(x.cuda(), r).cpu()
    rt = want["row_token"].long()
    exp = torch.where((rt >= 0).unsqueeze(1), x[rt.clamp_min(0)], torch.zeros((), dtype=dtype))
    assert torch.equal(xs[: want["n_pad"]], exp)
    y = ops.combine_rows(xs.cuda(), r).cpu()
    exp_y = (x.double() * k).to(dtype) if dtype == torch.float32 else None
    # combine of gathered rows = k * x (each token appears once per route), fp32 accumulation then one rounding
    torch.testing.assert_close(y.double(), (x.double() * k).to(dtype).double(), rtol=0, atol=0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_ess(ops, dtype):
    T, k, E, n = 3000, 2, 16, 328
    ids = make_ids(T, k, E, 5, skew=True, empty=(3, 15))
    r = ops.route(ids.cuda(), E)
    dy = torch.randn(T, n).to(dtype)
    dys = ops.gather_rows(dy.cuda(), r)
    got = ops.ess(dys, r).cpu()
    want = sum(O.ess(dy, ids[:, j], E) for j in range(k))
    assert rel_err(got, want) < 1e-5          # fp32 accumulation for every input dtype
    assert (got[3] == 0).all() and (got[15] == 0).all()
    got2 = ops.ess(dys, r).cpu()
    assert torch.equal(got, got2)             # deterministic


def _esmm_case(ops, dtype, engine, T, k, E, K, N, b_layout, epilogue, act, seed=0, bias=True):
    Lb = L()
    ids = make_ids(T, k, E, seed, skew=True, empty=(1,))
    r = ops.route(ids.cuda(), E)
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(T, K, generator=g).to(dtype)
    w = (torch.randn(E, K, N, generator=g) / K ** 0.5).to(dtype)          # [E, K, N]
    b = torch.randn(E, N, generator=g) if bias else None
    wdev = (w.transpose(1, 2).contiguous() if b_layout == Lb.B_NK else w).cuda()
    xs = ops.gather_rows(x.cuda(), r)
    bdev = None if b is None else ops._f32(b.cuda())            # rows padded to whole 16-byte chunks when N % 4 != 0
    aux_pre = None
    if epilogue == Lb.EPI_DACT:
        pre = torch.randn(T, N, generator=g).to(dtype)
        aux_pre = ops.gather_rows(pre.cuda(), r)
        out = ops.esmm(xs, wdev, b_layout, r, bdev, epilogue, act, aux=aux_pre, engine=engine)
    elif epilogue == Lb.EPI_ACT:
        aux_pre = ops.sorted_buffer(r.row_capacity, N, dtype, "cuda")
        out = ops.esmm(xs, wdev, b_layout, r, bdev, epilogue, act, aux=aux_pre, engine=engine)
    else:
        out = ops.esmm(xs, wdev, b_layout, r, bdev, epilogue, act, engine=engine)
    torch_act = {Lb.ACT_NONE: lambda t: t, Lb.ACT_RELU: F.relu, Lb.ACT_GELU: F.gelu,
                 Lb.ACT_GELU_TANH: lambda t: F.gelu(t, approximate="tanh"), Lb.ACT_SILU: F.silu}[act]
    n_pad = int(r.pad_offsets[-1])
    tol = REL[dtype]
    for j in range(k):
        lin = O.esmm(x, w, b, ids[:, j])                                   # float64, token order
        rows = r.token_row.view(T, k)[:, j].cpu().long()
        got = out.cpu()[rows]
        if epilogue == Lb.EPI_LINEAR:
            want = lin
        elif epilogue == Lb.EPI_ACT:
            want = torch_act(lin)
            assert rel_err(aux_pre.cpu()[rows], lin) < tol
        else:
            _, gr = O.act_and_grad(torch_act, pre.double())
            want = lin * gr
        assert rel_err(got, want) < tol, (j, rel_err(got, want))
    # pad rows are zeros
    pad = (r.row_token[:n_pad] < 0).cpu()
    assert (out.cpu()[:n_pad][pad] == 0).all()
    return out


@pytest.mark.parametrize("b_layout", [0, 1])
@pytest.mark.parametrize("epilogue,act", [(0, 0), (1, 2), (2, 2), (1, 1), (2, 4), (1, 3)])
def test_esmm_simt_fp32(ops, b_layout, epilogue, act):
    _esmm_case(ops, torch.float32, L().ENGINE_SIMT, T=500, k=2, E=5, K=72, N=100, b_layout=b_layout, epilogue=epilogue, act=act)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("b_layout", [0, 1])
def test_esmm_tcgen05_linear(ops, dtype, b_layout):
    _esmm_case(ops, dtype, L().ENGINE_TCGEN05, T=1500, k=2, E=6, K=256, N=512, b_layout=b_layout, epilogue=0, act=0)


@pytest.mark.parametrize("b_layout,K,N", [(0, 200, 328), (1, 200, 328), (0, 64, 128), (1, 1024, 64), (0, 776, 2048)])
def test_esmm_tcgen05_ragged_dims(ops, b_layout, K, N):
    """K not a multiple of 64 (TMA zero fill), N not a multiple of the tile, both tile widths."""
    _esmm_case(ops, torch.bfloat16, L().ENGINE_TCGEN05, T=900, k=2, E=4, K=K, N=N, b_layout=b_layout, epilogue=0, act=0, seed=2)


@pytest.mark.parametrize("b_layout,K,N,epilogue", [(0, 128, 203, 0), (0, 128, 203, 1), (0, 256, 1639, 2), (1, 203, 128, 0),
                                                   (1, 1639, 256, 0), (0, 64, 1229, 1)])
def test_esmm_tcgen05_odd_widths(ops, b_layout, K, N, epilogue):
    """Output widths and contraction lengths that are not multiples of 8: a rank's slice of an unevenly split hidden
    dimension (8192 x 0.2 = 1639 columns).  The buffers keep a 16-byte row pitch, the tensor cores do the work."""
    _esmm_case(ops, torch.bfloat16, L().ENGINE_TCGEN05, T=700, k=2, E=3, K=K, N=N, b_layout=b_layout, epilogue=epilogue,
               act=2 if epilogue else 0, seed=6)


@pytest.mark.parametrize("epilogue,act", [(1, 2), (2, 2), (1, 1), (2, 1), (1, 4), (2, 3)])
def test_esmm_tcgen05_epilogues(ops, epilogue, act):
    _esmm_case(ops, torch.bfloat16, L().ENGINE_TCGEN05, T=700, k=1, E=3, K=128, N=384, b_layout=0, epilogue=epilogue, act=act, seed=4)


def test_esmm_tcgen05_equals_simt_many_tiles(ops):
    """More tiles than SMs so every CTA loops over several tiles and both accumulators are reused."""
    Lb = L()
    T, k, E, K, N = 12000, 2, 8, 192, 1024
    ids = make_ids(T, k, E, 9, skew=True)
    r = ops.route(ids.cuda(), E)
    x = torch.randn(T, K).bfloat16().cuda()
    w = (torch.randn(E, N, K) / K ** 0.5).bfloat16().cuda()
    b = torch.randn(E, N).cuda()
    xs = ops.gather_rows(x, r)
    a = ops.esmm(xs, w, Lb.B_NK, r, b, engine=Lb.ENGINE_TCGEN05)
    s = ops.esmm(xs, w, Lb.B_NK, r, b, engine=Lb.ENGINE_SIMT)
    n_pad = int(r.pad_offsets[-1])
    assert rel_err(a[:n_pad], s[:n_pad]) < 1e-2
    a2 = ops.esmm(xs, w, Lb.B_NK, r, b, engine=Lb.ENGINE_TCGEN05)
    assert torch.equal(a[:n_pad], a2[:n_pad])


def _estmm_case(ops, dtype, engine, T, k, E, M, N, out_dtype, seed=0):
    ids = make_ids(T, k, E, seed, skew=True, empty=(0, E - 1))
    r = ops.route(ids.cuda(), E)
    g = torch.Generator().manual_seed(seed)
    p = torch.randn(T, M, generator=g).to(dtype); q = torch.randn(T, N, generator=g).to(dtype)
    # every route sees its own p rows in the layer; here the same token rows are used for all routes
    ps = ops.gather_rows(p.cuda(), r); qs = ops.gather_rows(q.cuda(), r)
    got = ops.estmm(ps, qs, r, out_dtype=out_dtype, engine=engine)
    want = sum(O.estmm(p, q, ids[:, j], E) for j in range(k))            # [E, M, N]
    tol = REL[out_dtype] if out_dtype != torch.float32 else REL[dtype] if dtype != torch.float32 else 1e-5
    # 16-bit inputs are exact in the oracle, so an fp32 output must be accurate to fp32 accumulation
    if out_dtype == torch.float32:
        tol = 2e-5
    assert rel_err(got, want) < tol, rel_err(got, want)
    assert (got[0] == 0).all() and (got[E - 1] == 0).all()                 # empty experts are written as zeros
    got_b = ops.estmm(ps, qs, r, out=got.clone(), beta=1, engine=engine)
    assert rel_err(got_b, 2 * want) < max(tol, 1e-2 if out_dtype != torch.float32 else tol)
    return got


@pytest.mark.parametrize("dtype,engine", [(torch.bfloat16, 1), (torch.float32, 2)])
def test_estmm_rank_grouped_layout_and_copy_2d(ops, dtype, engine):
    """ranks=W writes the gradient as [W, E, m/W, n] (what a reduce-scatter over the hidden dimension reads);
    copy_2d moves hidden slices between that layout and [E, m, n]."""
    T, k, E, M, N, W = 1500, 2, 5, 512, 256, 4
    ids = make_ids(T, k, E, 8, skew=True)
    r = ops.route(ids.cuda(), E)
    p = ops.gather_rows(torch.randn(T, M).to(dtype).cuda(), r); q = ops.gather_rows(torch.randn(T, N).to(dtype).cuda(), r)
    plain = ops.estmm(p, q, r, out_dtype=torch.float32, engine=engine)
    grouped = ops.estmm(p, q, r, out_dtype=torch.float32, engine=engine, ranks=W)
    assert grouped.shape == (W, E, M // W, N)
    assert torch.equal(grouped.permute(1, 0, 2, 3).reshape(E, M, N), plain)
    back = torch.empty_like(plain)
    for w in range(W):
        ops.copy_2d(back[:, w * (M // W):(w + 1) * (M // W)], back.stride(0), grouped[w], grouped.stride(1), (M // W) * N, E)
    assert torch.equal(back, plain)


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,W", [(512, 4), (768, 2), (1024, 8)])
def test_estmm_scatter_to_per_owner_buffers(ops, out_dtype, M, W):
    """A list of W outputs: slice w of the hidden dimension is stored straight into out[w] ([E, M/W, N]).
    Bit-identical to the rank-grouped single-buffer layout, and nothing outside the slices is touched."""
    T, k, E, N = 1500, 2, 5, 256
    ids = make_ids(T, k, E, 8, skew=True)
    r = ops.route(ids.cuda(), E)
    p = ops.gather_rows(torch.randn(T, M).bfloat16().cuda(), r); q = ops.gather_rows(torch.randn(T, N).bfloat16().cuda(), r)
    grouped = ops.estmm(p, q, r, out_dtype=out_dtype, ranks=W)
    arena = torch.full((W, 2, E, M // W, N), 7.0, dtype=out_dtype, device="cuda")      # slot 1 of every owner is the target
    outs = [arena[w, 1] for w in range(W)]
    back = ops.estmm(p, q, r, ranks=W, out=outs)
    assert back is outs
    for w in range(W):
        assert torch.equal(outs[w], grouped[w])
        assert (arena[w, 0] == 7.0).all()
    with pytest.raises(L().HexaError):
        ops.estmm(p, q, r, ranks=W, out=outs[:-1])


def test_estmm_simt_fp32(ops):
    _estmm_case(ops, torch.float32, L().ENGINE_SIMT, T=900, k=2, E=6, M=100, N=72, out_dtype=torch.float32)


@pytest.mark.parametrize("dtype,out_dtype", [(torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16),
                                             (torch.float16, torch.float32)])
@pytest.mark.parametrize("M,N", [(256, 512), (200, 328), (128, 64), (1000, 136)])
def test_estmm_tcgen05(ops, dtype, out_dtype, M, N):
    _estmm_case(ops, dtype, L().ENGINE_TCGEN05, T=2500, k=2, E=7, M=M, N=N, out_dtype=out_dtype, seed=M)


@pytest.mark.parametrize("E,M,N,out_dtype,ranks", [(1, 256, 512, torch.float32, 1), (1, 512, 128, torch.bfloat16, 1),
                                                    (3, 256, 256, torch.float32, 2), (2, 200, 136, torch.bfloat16, 1)])
def test_estmm_split_segments(ops, E, M, N, out_dtype, ranks):
    """Few output tiles and long segments (the dense FFN's weight gradient is the E = 1 case): with scratch the kernel
    cuts every segment into chunks and adds the fp32 partial results in chunk order.  Same answer as the oracle and as
    the unsplit kernel, bit-identical from run to run, beta and the rank-grouped layout honoured, an expert without
    rows written as zeros."""
    Lb = L()
    T, k = 6000, 1
    g = torch.Generator().manual_seed(E * 100 + M)
    ids = torch.randint(0, max(E - 1, 1), (T, k), generator=g).to(torch.int32)          # the last of several experts stays empty
    r = ops.route(ids.cuda(), E)
    p = torch.randn(T, M, generator=g).bfloat16(); q = torch.randn(T, N, generator=g).bfloat16()
    ps, qs = ops.gather_rows(p.cuda(), r), ops.gather_rows(q.cuda(), r)
    lib = Lb.lib()
    need = lib.hexa_estmm_workspace_bytes(E, r.row_capacity, M, N, Lb.BF16)
    assert need > 0, "this shape is meant to take the split path"
    got = ops.estmm(ps, qs, r, out_dtype=out_dtype, engine=Lb.ENGINE_TCGEN05, ranks=ranks)
    flat = got.permute(1, 0, 2, 3).reshape(E, M, N) if ranks > 1 else got
    want = O.estmm(p, q, ids[:, 0], E)
    tol = 2e-5 if out_dtype == torch.float32 else 2e-2
    assert rel_err(flat, want) < tol, rel_err(flat, want)
    if E > 1:
        assert (flat[E - 1] == 0).all()
    for _ in range(3):
        assert torch.equal(ops.estmm(ps, qs, r, out_dtype=out_dtype, engine=Lb.ENGINE_TCGEN05, ranks=ranks), got)
    # the unsplit kernel (no scratch offered) on the same inputs
    plain = torch.empty(E, M, N, dtype=out_dtype, device="cuda")
    Lb.check(lib.hexa_estmm(ps.data_ptr(), ps.stride(0), qs.data_ptr(), qs.stride(0), r.pad_offsets.data_ptr(), E, r.row_capacity,
                            M, N, plain.data_ptr(), plain.stride(1), plain.stride(0), 0, 0, Lb.BF16, Lb.dt(plain), 0,
                            Lb.ENGINE_TCGEN05, None, 0, torch.cuda.current_stream().cuda_stream), "hexa_estmm")
    assert rel_err(flat, plain) < (2e-5 if out_dtype == torch.float32 else 1e-2)     # fp32: another summation order
    if ranks == 1:
        twice = ops.estmm(ps, qs, r, out=got.clone(), beta=1, engine=Lb.ENGINE_TCGEN05)
        assert rel_err(twice, 2 * want) < max(tol, 1e-2 if out_dtype != torch.float32 else tol)


@pytest.mark.parametrize("dtype,E,k,d,H,act", [(torch.float32, 8, 1, 128, 512, "gelu"), (torch.bfloat16, 8, 2, 256, 1024, "gelu"),
                                               (torch.float16, 5, 2, 128, 320, "relu"), (torch.bfloat16, 4, 2, 128, 256, "generic"),
                                               (torch.bfloat16, 4, 2, 128, 203, "gelu"), (torch.bfloat16, 3, 1, 256, 1639, "gelu"),
                                               (torch.bfloat16, 4, 2, 128, 203, "generic")])
def test_layer_forward_backward(ops, dtype, E, k, d, H, act):
    Lb = L()
    T = 1200
    ids = make_ids(T, k, E, 21, skew=True, empty=(2,))
    g = torch.Generator().manual_seed(1)
    x = torch.randn(T, d, generator=g).to(dtype)
    w1 = (torch.randn(E, H, d, generator=g) / d ** 0.5).to(dtype)
    w2 = (torch.randn(E, H, d, generator=g) / H ** 0.5).to(dtype)
    b1 = (torch.randn(E, H, generator=g) * 0.1).to(dtype); b2 = (torch.randn(E, d, generator=g) * 0.1).to(dtype)
    dy = torch.randn(T, d, generator=g).to(dtype)
    fn = {"gelu": F.gelu, "relu": F.relu, "generic": lambda t: torch.sigmoid(t) * t * 1.5}[act]
    act_id = {"gelu": Lb.ACT_GELU, "relu": Lb.ACT_RELU, "generic": -1}[act]
    # 16-bit data must run on the tensor-core kernels whatever the hidden width (no silent CUDA-core fallback)
    engine = Lb.ENGINE_TCGEN05 if dtype != torch.float32 else Lb.ENGINE_AUTO
    y, st = ops.moe_forward(x.cuda(), ids.cuda(), w1.cuda(), w2.cuda(), b1.cuda(), b2.cuda(), act_id, act_fn=fn, engine=engine)
    dx, dw1, dw2, db1, db2 = ops.moe_backward(st, dy.cuda(), w1.cuda(), w2.cuda(), act_id, grad_dtype=torch.float32,
                                              engine=engine)
    want = O.moe_layer(x, ids, w1, w2, b1, b2, fn, dy)
    tol = REL[dtype]
    for name, got, exp in (("y", y, want["y"]), ("dx", dx, want["dx"]), ("dw1", dw1, want["dw1"]), ("dw2", dw2, want["dw2"]),
                           ("db1", db1, want["db1"]), ("db2", db2, want["db2"])):
        e = rel_err(got, exp)
        assert e < tol, (name, e)


@pytest.mark.parametrize("dtype,n_out", [(torch.bfloat16, 512), (torch.bfloat16, 128), (torch.float32, 96)])
def test_esmm_by_expert_groups_equals_one_launch(ops, dtype, n_out):
    """hexa_esmm_experts: launching the operator once per group of experts (any order) writes exactly what one launch
    over all experts writes, and a group's launch leaves the rows of other experts untouched."""
    Lb = L()
    T, k, E, d = 3000, 2, 7, 256
    ids = make_ids(T, k, E, 4, skew=True, empty=(3,))
    r = ops.route(ids.cuda(), E)
    g = torch.Generator().manual_seed(n_out)
    xs = ops.gather_rows(torch.randn(T, d, generator=g).to(dtype).cuda(), r)
    w = (torch.randn(E, n_out, d, generator=g) / 16).to(dtype).cuda()
    b = (torch.randn(E, n_out, generator=g) * 0.1).cuda()
    n_pad = int(r.pad_offsets[-1])
    full_aux = torch.zeros(r.row_capacity, n_out, dtype=dtype, device="cuda")
    full = ops.esmm(xs, w, Lb.B_NK, r, b, Lb.EPI_ACT, Lb.ACT_GELU, aux=full_aux)
    out = torch.full((r.row_capacity, n_out), 7.0, dtype=dtype, device="cuda")
    aux = torch.full_like(out, 7.0)
    ops.esmm(xs, w, Lb.B_NK, r, b, Lb.EPI_ACT, Lb.ACT_GELU, aux=aux, out=out, experts=(4, 7))
    lo = int(r.pad_offsets[4])
    assert (out[:lo] == 7.0).all() and (aux[:lo] == 7.0).all()                    # experts 0..3 untouched
    assert torch.equal(out[lo:n_pad], full[lo:n_pad]) and torch.equal(aux[lo:n_pad], full_aux[lo:n_pad])
    for e0, e1 in ((2, 4), (0, 2)):                                              # the remaining groups, out of order
        ops.esmm(xs, w, Lb.B_NK, r, b, Lb.EPI_ACT, Lb.ACT_GELU, aux=aux, out=out, experts=(e0, e1))
    assert torch.equal(out[:n_pad], full[:n_pad]) and torch.equal(aux[:n_pad], full_aux[:n_pad])
    ops.esmm(xs, w, Lb.B_NK, r, b, out=out, experts=(3, 3))                        # an empty range launches nothing
    with pytest.raises(Lb.HexaError):
        ops.esmm(xs, w, Lb.B_NK, r, b, out=out, experts=(5, 9))


@pytest.mark.parametrize("dtype,K,N,epilogue,b_layout", [(torch.bfloat16, 256, 512, 2, 0), (torch.float16, 256, 512, 2, 0),
                                                          (torch.bfloat16, 512, 328, 0, 1), (torch.bfloat16, 128, 64, 1, 0),
                                                          (torch.bfloat16, 256, 1639, 2, 0), (torch.float32, 64, 96, 0, 0)])
def test_esmm_with_fused_column_sums(ops, dtype, K, N, epilogue, b_layout):
    """hexa_esmm_ess: the output is bit-identical to hexa_esmm's and the sums are ESS of that output - on the tcgen05
    engine from the epilogue's staging tile (ragged column tiles, an empty expert, both 16-bit types, all epilogues),
    on the other engine (fp32, odd pitches) as the two-pass fallback.  Deterministic."""
    Lb = L()
    T, k, E = 2500, 2, 7
    ids = make_ids(T, k, E, 11, skew=True, empty=(2,))
    r = ops.route(ids.cuda(), E)
    g = torch.Generator().manual_seed(3)
    xs = ops.gather_rows(torch.randn(T, K, generator=g).to(dtype).cuda(), r)
    w = (torch.randn(E, K, N, generator=g) / K ** 0.5).to(dtype)
    wdev = (w.transpose(1, 2).contiguous() if b_layout == Lb.B_NK else w).cuda()
    bias = ops._f32(torch.randn(E, N, generator=g).cuda()) if epilogue != Lb.EPI_DACT else None
    aux = None
    if epilogue == Lb.EPI_DACT:
        aux = ops.gather_rows(torch.randn(T, N, generator=g).to(dtype).cuda(), r)
    elif epilogue == Lb.EPI_ACT:
        aux = ops.sorted_buffer(r.row_capacity, N, dtype, xs.device)
    act = Lb.ACT_GELU if epilogue != Lb.EPI_LINEAR else Lb.ACT_NONE
    plain = ops.esmm(xs, wdev, b_layout, r, bias, epilogue, act, aux=aux)
    sums = torch.full((E, N), float("nan"), dtype=torch.float32, device="cuda")
    fused = ops.esmm(xs, wdev, b_layout, r, bias, epilogue, act, aux=aux, sums=sums)
    n_pad = int(r.pad_offsets[-1])
    assert torch.equal(fused[:n_pad], plain[:n_pad])
    want = ops.ess(plain, r)
    assert torch.isfinite(sums).all()
    assert rel_err(sums, want) < 1e-5
    assert (sums[2] == 0).all()                                   # the empty expert
    sums2 = torch.empty_like(sums)
    ops.esmm(xs, wdev, b_layout, r, bias, epilogue, act, aux=aux, sums=sums2)
    assert torch.equal(sums, sums2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("n_recv", [0, 1, 2, 3, 5, 7])
def test_mean_slices(ops, dtype, n_recv):
    """The reduction step of the peer-copy reduce-scatter: out = (local + received slices) / world with fp32
    accumulation in slice order, for slice counts with and without an unrolled variant and sizes that leave a tail."""
    world = n_recv + 1
    for elems in (8 * 1000, 8 * 128 * 8 * 37 + 8 * 5, 1 << 22):
        g = torch.Generator().manual_seed(elems % 1000 + n_recv)
        local = torch.randn(elems, generator=g).to(dtype).cuda()
        recv = torch.randn(max(n_recv, 1), elems, generator=g).to(dtype).cuda()
        out = torch.empty_like(local)
        ops.mean_slices(local, recv, n_recv, world, out)
        acc = local.float()
        for s_ in range(n_recv):
            acc = acc + recv[s_].float()
        want = (acc * (1.0 / world)).to(dtype)
        assert torch.equal(out, want), (elems, float((out.float() - want.float()).abs().max()))


def test_errors_are_reported_not_fatal(ops):
    Lb = L()
    ids = make_ids(64, 1, 4, 0)
    r = ops.route(ids.cuda(), 4)
    a = torch.zeros(r.row_capacity, 20, dtype=torch.bfloat16, device="cuda")      # lda = 20: not a multiple of 8
    b = torch.zeros(4, 16, 20, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(Lb.HexaError, match="tcgen05"):
        ops.esmm(a, b, Lb.B_NK, r, engine=Lb.ENGINE_TCGEN05)
    out = ops.esmm(a, b, Lb.B_NK, r)                # AUTO falls back to the CUDA-core kernel
    assert out.shape == (r.row_capacity, 16)
    with pytest.raises(Lb.HexaError):
        ops.route(ids.cuda().long(), 4)
    with pytest.raises(Lb.HexaError, match="CUDA tensors only"):
        ops.route(ids, 4)


# Both tile sizes of the CUDA-core kernels: every output is one FMA chain in ascending k whichever tile computes it, so a
# launch wide enough for 128-tiles must reproduce, bit for bit, what narrow launches over column slices (64-tiles) give.
@pytest.mark.parametrize("dtype,K,N", [(torch.float32, 36, 2052), (torch.float32, 37, 2051), (torch.bfloat16, 130, 2049)])
@pytest.mark.parametrize("nk", [True, False])
def test_simt_tile_sizes_agree(ops, dtype, K, N, nk):
    Lb = L()
    T, E = 5000, 5
    ids = make_ids(T, 1, E, 11, skew=True, empty=(2,))
    r = ops.route(ids.cuda(), E)
    assert (r.row_capacity // 128) * (-(-N // 128)) >= 2 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator().manual_seed(K)
    x = torch.randn(T, K, generator=g).to(dtype)
    w = torch.randn(E, N, K, generator=g).to(dtype)
    b = torch.randn(E, N, generator=g)
    xs = ops.gather_rows(x.cuda(), r)
    wd = w.cuda() if nk else w.transpose(1, 2).contiguous().cuda()
    bd = ops._f32(b.cuda())
    y1 = ops.sorted_buffer(r.row_capacity, N, dtype, "cuda")
    args = dict(epilogue=Lb.EPI_ACT, act=Lb.ACT_GELU, engine=Lb.ENGINE_SIMT)
    lay = Lb.B_NK if nk else Lb.B_KN
    wide = ops.esmm(xs, wd, lay, r, bd, aux=y1, **args)
    n_pad = int(r.pad_offsets[-1])
    for c0, c1 in ((0, 64), (1984, N), (N - 3, N)):
        sl = wd[:, c0:c1] if nk else wd[:, :, c0:c1]
        a1 = ops.sorted_buffer(r.row_capacity, c1 - c0, dtype, "cuda")
        got = ops.esmm(xs, sl, lay, r, ops._f32(b[:, c0:c1].cuda()), aux=a1, **args)
        assert torch.equal(got[:n_pad], wide[:n_pad, c0:c1]) and torch.equal(a1[:n_pad], y1[:n_pad, c0:c1])
    # the weight gradient, against float64 and slice by slice
    dw = ops.estmm(wide, xs, r, out_dtype=torch.float32, engine=Lb.ENGINE_SIMT)
    many = ops.estmm(wide, wide[:, :1024], r, out_dtype=torch.float32, engine=Lb.ENGINE_SIMT)        # 128-tiles
    few = ops.estmm(wide[:, :64], wide[:, :1024], r, out_dtype=torch.float32, engine=Lb.ENGINE_SIMT)   # 64-tiles
    assert torch.equal(many[:, :64], few)
    rows = r.row_token[:n_pad]
    po = r.pad_offsets.tolist()
    for e in range(E):
        want = wide[po[e]:po[e + 1]].double().t() @ xs[po[e]:po[e + 1]].double()
        # a chain of n fp32 FMAs is within n * 2^-24 of the sum of magnitudes; rows of an expert bound n
        bound = wide[po[e]:po[e + 1]].double().abs().t() @ xs[po[e]:po[e + 1]].double().abs() * ((po[e + 1] - po[e]) * 2.0 ** -24)
        assert ((dw[e].double() - want).abs() <= bound + 1e-30).all()


# One launch, two launches and three: sizes around a warp's chunk, the single block's capacity, a block's rows of the
# two-launch form, the expert limits of both, strided id tensors, ids out of range, no rows for most experts.
@pytest.mark.parametrize("T,k,E,launches", [(0, 2, 4, 1), (1, 1, 256, 1), (33, 3, 7, 1), (4096, 2, 64, 1), (8192, 1, 256, 1), (8193, 1, 64, 2),
                                            (9001, 1, 257, 2), (2048, 4, 512, 2), (70000, 3, 64, 2), (16385, 2, 8, 2),
                                            (600, 2, 513, 3), (200000, 4, 400, 3)])
@pytest.mark.parametrize("align", [128, 16])
def test_route_launch_forms(ops, T, k, E, launches, align):
    Lb = L()
    assert Lb.lib().hexa_route_launches(T, k, E) == launches
    g = torch.Generator().manual_seed(T + E)
    ids = torch.randint(-1, E + 1, (T, k), generator=g, dtype=torch.int32)
    if E > 8:
        ids[T // 2:] = ids[T // 2:] % 3
    dev = ids.cuda()
    wide = torch.full((T, 2 * k + 1), -7, dtype=torch.int32, device="cuda")
    wide[:, 1::2] = dev
    forms = [(dev, False), (dev.t().contiguous(), True), (wide[:, 1::2], False), (wide.t()[1::2], True)]
    want = O.route(ids, E, align)
    n_pad = want["n_pad"]
    for src, major in forms:
        r = ops.route(src, E, align, route_major=major)
        for name in ("counts", "seg_offsets", "pad_offsets"):
            assert torch.equal(getattr(r, name).cpu(), want[name]), name
        assert torch.equal(r.row_token.cpu()[:n_pad], want["row_token"])
        assert torch.equal(r.token_row.cpu()[: T * k], want["token_row"])
        te = r.tile_expert.cpu()
        assert torch.equal(te[: n_pad // align], want["tile_expert"]) and (te[n_pad // align: r.row_capacity // align] == -1).all()
        if align == 128:
            pb, n = r.pair_block.cpu(), want["pair_block"].numel()
            assert torch.equal(pb[:n], want["pair_block"]) and (pb[n:] == -1).all()


# Gather with column sums: whole and ragged 16-byte groups, more columns than one block's, empty experts, a row pitch.
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,cols", [(1, 8), (777, 264), (700, 203), (5000, 1032)])
def test_gather_with_sums_is_gather_then_ess(ops, dtype, T, cols):
    E, k = 6, 2
    ids = make_ids(T, k, E, 3, skew=True, empty=(2,))
    r = ops.route(ids.cuda(), E)
    x = torch.randn(T, cols + 8, generator=torch.Generator().manual_seed(T)).to(dtype).cuda()[:, :cols]
    n_pad = int(r.pad_offsets[-1])
    rows, sums = ops.gather_rows_ess(x, r)
    want = ops.gather_rows(x, r)
    assert torch.equal(rows[:n_pad], want[:n_pad])
    assert torch.equal(sums, ops.ess(want, r))
    # n additions of fp32 stay within n * 2^-24 of the sum of magnitudes
    for e in range(E):
        tok = r.row_token[r.pad_offsets[e]: r.pad_offsets[e + 1]].long()
        seg = x[tok[tok >= 0]].double()
        assert ((sums[e].double() - seg.sum(0)).abs() <= seg.abs().sum(0) * (len(seg) * 2.0 ** -24) + 1e-30).all()


# Biases and column sums of the data's own 16-bit type: the same values as the fp32 operands holding them / rounded once.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("K,N,engine", [(64, 264, "auto"), (72, 203, "auto"), (37, 41, "auto"), (64, 100, "simt"), (64, 96, "auto")])
def test_16_bit_bias_and_sums(ops, dtype, K, N, engine):
    Lb = L()
    eng = Lb.ENGINE_SIMT if engine == "simt" else Lb.ENGINE_AUTO
    T, k, E = 900, 2, 5
    r = ops.route(make_ids(T, k, E, 21, skew=True, empty=(1,)).cuda(), E)
    g = torch.Generator().manual_seed(N)
    xs = ops.gather_rows(torch.randn(T, K, generator=g).to(dtype).cuda(), r)
    w = torch.randn(E, N, K, generator=g).to(dtype).cuda()
    wide = torch.randn(E, N + 3, generator=g).to(dtype).cuda()
    n_pad = int(r.pad_offsets[-1])
    for b in (wide[:, :N], wide[:, 1:N + 1]):                       # rows that start and end anywhere
        outs = []
        for bias in (b, ops._f32(b)):
            s16, s32 = (torch.empty(E, N, dtype=t, device="cuda") for t in (dtype, torch.float32))
            y = ops.esmm(xs, w, Lb.B_NK, r, bias, Lb.EPI_ACT, Lb.ACT_GELU, engine=eng, sums=s32)
            y2 = ops.esmm(xs, w, Lb.B_NK, r, bias, Lb.EPI_ACT, Lb.ACT_GELU, engine=eng, sums=s16)
            assert torch.equal(y[:n_pad], y2[:n_pad]) and torch.equal(s16, s32.to(dtype))
            outs.append((y[:n_pad], s32))
        assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert torch.equal(ops.ess(xs, r, out_dtype=dtype), ops.ess(xs, r).to(dtype))
    x = torch.randn(T, K, generator=g).to(dtype).cuda()
    assert torch.equal(ops.gather_rows_ess(x, r, dtype)[1], ops.gather_rows_ess(x, r)[1].to(dtype))
    with pytest.raises(Lb.HexaError):
        ops.ess(xs, r, out_dtype=torch.float64)
    f = torch.zeros(r.row_capacity, 8, device="cuda")
    with pytest.raises(Lb.HexaError):
        ops.ess(f, r, out_dtype=torch.bfloat16)                     # only the data's own type


# Kernels take raw pointers: an operand left on the host is refused by the wrappers, whichever it is.
def test_operands_on_another_device_are_refused(ops):
    Lb = L()
    r = ops.route(make_ids(200, 1, 2, 3).cuda(), 2)
    x, w, b = torch.randn(200, 64), torch.randn(2, 32, 64), torch.randn(2, 32)
    xs = ops.gather_rows(x.cuda(), r)
    good = (xs, w.cuda(), Lb.B_NK, r, b.cuda())
    ops.esmm(*good)
    out, cpu_r = torch.empty(r.row_capacity, 32), type(r)(**{**vars(r), "pad_offsets": r.pad_offsets.cpu()})
    calls = [lambda: ops.esmm(xs, w, Lb.B_NK, r), lambda: ops.esmm(xs, w.cuda(), Lb.B_NK, r, b), lambda: ops.esmm(*good, out=out),
             lambda: ops.esmm(*good, epilogue=Lb.EPI_ACT, act=Lb.ACT_GELU, aux=out), lambda: ops.esmm(*good, sums=torch.empty(2, 32)),
             lambda: ops.esmm(xs, w.cuda(), Lb.B_NK, cpu_r), lambda: ops.estmm(xs, out, r), lambda: ops.ess(xs, cpu_r),
             lambda: ops.estmm(xs, xs, r, out=torch.empty(2, 64, 64)), lambda: ops.gather_rows(x.cuda(), cpu_r),
             lambda: ops.gather_rows_ess(x.cuda(), cpu_r), lambda: ops.combine_rows(xs, r, out=torch.empty(200, 64)),
             lambda: ops.gate_project(x.cuda(), w[0]), lambda: ops.gate_project_grad(b.cuda(), x.cuda()[:2], w[0], True, True),
             lambda: ops.gate_loss_grad(x.cuda(), torch.zeros(64, dtype=torch.int32), torch.ones((), device="cuda"))]
    for i, call in enumerate(calls):
        with pytest.raises(Lb.HexaError, match="different devices"):
            call()
            pytest.fail(f"call {i} went through")


def test_launches_are_counted_where_they_happen(ops):
    Lb = L()

    def count(call):
        before = ops.LAUNCHES
        call()
        return ops.LAUNCHES - before

    T, E = 12000, 4
    ids = make_ids(T, 1, E, 5).cuda()
    r = ops.route(ids, E)
    xs, w = ops.gather_rows(torch.randn(T, 256, device="cuda"), r), torch.randn(E, 2048, 256, device="cuda")
    h = ops.esmm(xs, w, Lb.B_NK, r)
    y1 = torch.empty_like(h)
    assert count(lambda: ops.esmm(xs, w, Lb.B_NK, r)) == 3                     # split, GEMM, the CUDA cores' stand-by
    assert count(lambda: ops.esmm(xs, w, Lb.B_NK, r, None, Lb.EPI_ACT, Lb.ACT_GELU, aux=y1)) == 4
    assert count(lambda: ops.esmm(xs, w, Lb.B_NK, r, engine=Lb.ENGINE_SIMT)) == 1
    assert count(lambda: ops.estmm(h, xs, r)) == 3
    xb, hb, wb = xs.bfloat16(), h.bfloat16(), w.bfloat16()
    assert count(lambda: ops.esmm(xb, wb, Lb.B_NK, r)) == 1
    assert count(lambda: ops.estmm(hb, xb, r)) == (2 if Lb.lib().hexa_estmm_workspace_bytes(E, r.row_capacity, 2048, 256, Lb.BF16) else 1)
    assert count(lambda: ops.estmm(hb[:, :256], xb, r)) == 2                    # chunks and their sum
    assert count(lambda: ops.esmm(xb, wb, Lb.B_NK, r, sums=torch.empty(E, 2048, device="cuda"))) == 2
    assert count(lambda: ops.ess(xb, r)) == 2 and count(lambda: ops.gather_rows_ess(xb[:T], r)) == 2
    assert count(lambda: ops.gather_rows(xb[:T], r)) == 1 and count(lambda: ops.combine_rows(xb, r)) == 1
    for rows, kernels in ((512, 1), (513, 2)):
        assert count(lambda: ops.gate_topk(torch.randn(rows, 64, device="cuda"), 2)) == kernels
    for rows, kernels in ((8192, 1), (8193, 2)):
        assert count(lambda: ops.route(torch.zeros(rows, 1, dtype=torch.int32, device="cuda"), E)) == kernels


# Column sums keep one order of additions, which the bias gradients are rounded from: within a 128-row tile rows r mod 4 in
# ascending order and the four sums in turn, then the tiles of an expert in ascending order.
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,E,cols", [(1, 1, 8), (1000, 3, 264), (18432, 1, 520), (9000, 2, 203), (8200, 1, 32)])
def test_column_sums_keep_their_order(ops, dtype, T, E, cols):
    ids = make_ids(T, 1, E, 3, skew=True)
    r = ops.route(ids.cuda(), E)
    x = torch.randn(T, cols, generator=torch.Generator().manual_seed(T)).to(dtype).cuda()
    rows, both = ops.gather_rows_ess(x, r)
    n_pad, po = int(r.pad_offsets[-1]), r.pad_offsets.tolist()
    tiles = rows[:n_pad].float().view(-1, 32, 4, cols)
    acc = torch.zeros(tiles.shape[0], 4, cols, device="cuda")
    for i in range(32):
        acc = acc + tiles[:, i]
    part = ((acc[:, 0] + acc[:, 1]) + acc[:, 2]) + acc[:, 3]
    want = torch.zeros(E, cols, device="cuda")
    for e in range(E):
        for t in range(po[e] // 128, po[e + 1] // 128):
            want[e] += part[t]
    assert torch.equal(both, want) and torch.equal(ops.ess(rows, r), want)


# fp32 weight gradients of 16-bit data (fp32 parameters under autocast): the accumulator truncates, half an ulp (2^-24 of a sum
# of positive terms, at most) per 16-row MMA of a chain on average, so the chunks that a long segment is cut into bound it.
@pytest.mark.parametrize("T,E,m,n,chunks", [(18432, 1, 2048, 512, 10), (32768, 8, 1024, 256, 5)])
def test_fp32_weight_gradient_of_16_bit_data(ops, T, E, m, n, chunks):
    g = torch.Generator(device="cuda").manual_seed(m)
    r = ops.route((torch.arange(T, device="cuda") % E).to(torch.int32).view(-1, 1), E)
    p, q = (ops.gather_rows(torch.randn(T, c, generator=g, device="cuda").abs().bfloat16(), r) for c in (m, n))
    got = ops.estmm(p, q, r, out_dtype=torch.float32)
    po = r.pad_offsets.tolist()
    exact = torch.stack([p[po[e]:po[e + 1]].double().t() @ q[po[e]:po[e + 1]].double() for e in range(E)])
    chain = -(-(T // E // 64) // chunks) * 4
    assert float((got.double() - exact).norm() / exact.norm()) <= (chain + chunks) * 2.0 ** -24


# A split weight gradient: tiles past m and n, empty and short segments next to long ones, every form of the output.  Bound: half
# an ulp per MMA of a chain (as above; chains of at most 32 k-blocks here), one per partial sum, the rounding of the output.
@pytest.mark.parametrize("T,E,m,n,skew", [(8200, 1, 136, 40, False), (5000, 3, 264, 520, True), (16384, 5, 640, 128, True), (2200, 2, 96, 1000, False)])
def test_split_weight_gradient_forms(ops, T, E, m, n, skew):
    ids = make_ids(T, 1, E, 5, skew=skew)
    if E > 2:
        ids[ids == 1] = 0
    r = ops.route(ids.cuda(), E)
    g = torch.Generator(device="cuda").manual_seed(T)
    p, q = (ops.gather_rows(torch.randn(T, c, generator=g, device="cuda").half(), r) for c in (m, n))
    assert r.row_capacity // 64 // E >= 16      # long enough to be split
    po = r.pad_offsets.tolist()
    exact = torch.stack([p[po[e]:po[e + 1]].double().t() @ q[po[e]:po[e + 1]].double() for e in range(E)])
    size = torch.stack([p[po[e]:po[e + 1]].double().abs().t() @ q[po[e]:po[e + 1]].double().abs() for e in range(E)])
    bound = size * (32 * 4 + 32) * 2.0 ** -24
    got = ops.estmm(p, q, r, out_dtype=torch.float32)
    assert bool(((got.double() - exact).abs() <= bound).all())
    half = ops.estmm(p, q, r)
    assert bool(((half.double() - exact).abs() <= bound + exact.abs() * 2.0 ** -11 + 2.0 ** -25).all())
    assert torch.equal(ops.estmm(p, q, r, out=got.clone(), beta=1), got + got)
    assert torch.equal(ops.estmm(p, q, r, out_dtype=torch.float32, ranks=2), torch.stack(got.split(m // 2, dim=1)))


# Kernels may be launched while the one before drains: a chain over ever new data and reused memory, enqueued without a stop and
# next to PyTorch kernels, against the same chain with the host waiting behind every operator.
@pytest.mark.parametrize("dtype,T,d,H", [(torch.bfloat16, 300, 64, 256), (torch.float32, 900, 72, 200), (torch.float32, 4000, 256, 1024), (torch.float16, 5000, 128, 512)])
def test_chains_without_a_stop(ops, dtype, T, d, H):
    Lb, E, k = L(), 5, 2
    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)
    data = [(torch.randn(T, E, generator=g, device="cuda"), rand(T, d), rand(E, H, d), rand(E, H, d)) for _ in range(6)]

    def chain(logits, x, w1, w2, stop):
        ids = ops.gate_topk(logits * 1.0, k)[0]; stop()
        r = ops.route(ids, E, route_major=True); stop()
        xs, sums = ops.gather_rows_ess(x + 0, r); stop()
        y1 = ops.sorted_buffer(r.row_capacity, H, dtype, "cuda")
        h = ops.esmm(xs, w1, Lb.B_NK, r, None, Lb.EPI_ACT, Lb.ACT_GELU, aux=y1); stop()
        dw = ops.estmm(h, xs, r); stop()
        ys = ops.esmm(h, w2, Lb.B_KN, r); stop()
        return [ids, r.token_row, sums, dw, ops.combine_rows(ys, r), ops.ess(h, r)]

    want = [chain(*a, torch.cuda.synchronize) for a in data]
    got = [chain(*a, lambda: None) for _ in range(5) for a in data]
    for i, out in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(out, want[i % len(data)])), i


# Few rows take 128-column tiles of one CTA, more take CTA pairs: either side of the rule, against single-CTA tiles of the other
# width (no pair list), bit for bit.
@pytest.mark.parametrize("T,E,n,k", [(1, 3, 136, 64), (96 * 4, 4, 520, 72), (97 * 4, 4, 520, 72), (700, 7, 800, 200), (300, 1, 264, 128), (3000, 2, 2048, 64), (20000, 4, 256, 64)])
def test_few_rows_take_small_tiles(ops, T, E, n, k):
    from dataclasses import replace
    Lb = L()
    r = ops.route(make_ids(T, 1, E, 9, skew=True).cuda(), E)
    plain = replace(r, pair_block=None)
    g = torch.Generator(device="cuda").manual_seed(n)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, wt, b = ops.gather_rows(rand(T, k), r), rand(E, n, k), rand(E, k, n), rand(E, n)
    rows = int(r.pad_offsets[-1])

    def both(layout, wgt, epilogue):
        out = []
        for table in (r, plain):
            aux = ops.sorted_buffer(r.row_capacity, n, x.dtype, "cuda")
            aux.copy_(saved) if epilogue == Lb.EPI_DACT else aux.zero_()
            sums = torch.empty(E, n, device="cuda")
            c = ops.esmm(x, wgt, layout, table, None if epilogue == Lb.EPI_DACT else b, epilogue, Lb.ACT_GELU if epilogue else Lb.ACT_NONE,
                         aux=aux if epilogue else None, sums=sums)
            out.append((c[:rows], aux[:rows], sums))
        return out

    saved = ops.esmm(x, w, Lb.B_NK, r, b)
    for layout, wgt in ((Lb.B_NK, w), (Lb.B_KN, wt)):
        for epilogue in (Lb.EPI_LINEAR, Lb.EPI_ACT, Lb.EPI_DACT):
            a, c = both(layout, wgt, epilogue)
            assert all(torch.equal(u, v) for u, v in zip(a, c)), (layout, epilogue)


@pytest.mark.parametrize("dtype,T", [(torch.bfloat16, 131072), (torch.float32, 32768)])
def test_sms_left_free_stay_free(ops, dtype, T):
    """With an SM limit, the kernels that follow a GEMM in its stream do not take up the SMs that it leaves to other streams: a
    kernel of another stream that becomes ready in the first of two GEMMs runs then, not behind it."""
    from hexa_moe_b200 import _lib as L
    d = 4096
    r = ops.route(torch.zeros(T, 1, dtype=torch.int32, device="cuda"), 1)
    xs = torch.randn(r.row_capacity, d, dtype=dtype, device="cuda")
    w = torch.randn(1, d, d, dtype=dtype, device="cuda")
    out = torch.empty_like(xs)
    host, dev = torch.empty(4 << 20, dtype=torch.float32).pin_memory(), torch.empty(4 << 20, device="cuda")
    small = torch.zeros(64, device="cuda")
    side = torch.cuda.Stream()
    start, ran, end = (torch.cuda.Event(enable_timing=True) for _ in range(3))

    def both():
        torch.cuda._sleep(2_000_000)                  # the host is ahead of the device
        start.record()
        for _ in range(2):
            ops.esmm(xs, w, L.B_NK, r, out=out)
        end.record()
        with torch.cuda.stream(side):                 # a copy engine's work, then a kernel
            side.wait_event(start)
            dev.copy_(host, non_blocking=True)
            small.add_(1)
            ran.record(side)
        torch.cuda.synchronize()
        return start.elapsed_time(ran) / start.elapsed_time(end)

    try:
        L.lib().hexa_set_sm_limit(torch.cuda.get_device_properties(0).multi_processor_count - 16)
        both()
        share = min(both() for _ in range(3))
    finally:
        L.lib().hexa_set_sm_limit(0)
    assert share < 0.4, share                         # behind the first GEMM: at least half


@pytest.mark.parametrize("T,E,n,limit,experts,small", [
    (2048, 8, 1536, 0, (0, 8), False), (2048, 8, 1536, 132, (0, 8), True),            # a cap on the SMs
    (4608, 32, 1024, 0, (0, 32), False), (4608, 32, 1024, 0, (8, 16), True),          # some of the experts
    (2048, 32, 1024, 0, (0, 32), True), (2048, 32, 1024, 1, (0, 32), True),           # a cap that leaves no pair
])
def test_small_tiles_follow_the_launch(ops, T, E, n, limit, experts, small):
    """Waves of small tiles and of pairs are those of the SMs and the experts that a launch has; results are the same bit for bit."""
    from torch.profiler import ProfilerActivity, profile
    from hexa_moe_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(T)
    r = ops.route(torch.randint(0, E, (T, 1), generator=g, device="cuda").to(torch.int32), E)
    xs = ops.gather_rows(torch.randn(T, 128, generator=g, device="cuda").bfloat16(), r)
    w = torch.randn(E, n, 128, generator=g, device="cuda").bfloat16()
    n_pad = int(r.pad_offsets[-1])
    rows = slice(int(r.pad_offsets[experts[0]]), int(r.pad_offsets[experts[1]]))
    want = ops.esmm(xs, w, L.B_NK, r)
    try:
        L.lib().hexa_set_sm_limit(limit)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            got = ops.esmm(xs, w, L.B_NK, r, experts=experts)
            torch.cuda.synchronize()
    finally:
        L.lib().hexa_set_sm_limit(0)
    assert rows.stop <= n_pad and torch.equal(got[rows], want[rows])
    names = [e.key for e in prof.key_averages() if "gemm_tc_kernel<" in e.key]
    if not names:
        pytest.skip("no kernel records on this machine")
    ctas = int(names[0].split("gemm_tc_kernel<")[1].split(",")[2])
    assert (ctas == 1) == small, names


@pytest.mark.parametrize("T,E,m,n", [(18432, 1, 512, 2048), (8192, 2, 256, 512), (30000, 1, 256, 128), (16384, 8, 1024, 256)])
def test_scratch_that_holds_the_chunks_is_enough(ops, T, E, m, n):
    """A split weight gradient takes any scratch that holds what it writes, which may be less than the query asks for."""
    from hexa_moe_b200 import _lib as L
    lib = L.lib()
    g = torch.Generator(device="cuda").manual_seed(T)
    r = ops.route(torch.randint(0, E, (T, 1), generator=g, device="cuda").to(torch.int32), E)
    p, q = (ops.gather_rows(torch.randn(T, w, generator=g, device="cuda").bfloat16(), r) for w in (m, n))
    plane = E * m * n
    most = lib.hexa_estmm_workspace_bytes(E, r.row_capacity, m, n, L.BF16) // (4 * plane)
    assert most > 1
    mark = 0x7fc12345                                     # a NaN that no sum is

    def run(planes):
        ws = torch.full((most, plane), mark, dtype=torch.int32, device="cuda")
        out, before = torch.empty(E, m, n, device="cuda"), ops.LAUNCHES
        assert lib.hexa_estmm(p.data_ptr(), m, q.data_ptr(), n, r.pad_offsets.data_ptr(), E, r.row_capacity, m, n, out.data_ptr(), n,
                              m * n, 0, 0, L.BF16, L.F32, 0, L.ENGINE_AUTO, ws.data_ptr(), planes * plane * 4,
                              torch.cuda.current_stream().cuda_stream) == 0
        return out, ops.LAUNCHES - before, int((ws != mark).all(1).sum()), int((ws != mark).any(1).sum())

    want, launches, whole, touched = run(most)
    assert launches == 2 and whole == touched >= 2
    got, launches, *used = run(whole)
    assert launches == 2 and used == [whole, whole] and torch.equal(got, want)
    _, launches, *used = run(whole - 1)                   # the unsplit kernel
    assert launches == 1 and used == [0, 0]
