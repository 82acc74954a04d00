"""fp32 ESMM / ESTMM on the tensor cores (three bf16 planes per operand, fp32 additions between k-blocks) against float64 and
against the CUDA-core kernel: never further from the exact result than the FMA chain, zero pad rows, and the FMA chain's own
answer wherever an operand holds a value that has no planes.  Sizes are just beyond the point where the path is taken."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _mods():
    from hexa_moe_b200 import _lib as L, ops
    return L, ops


def _routing(ops, T, E, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    logits = torch.randn(T, E, generator=g, device="cuda") - 0.3 * torch.arange(E, device="cuda")
    logits[:, min(1, E - 1)] = -100.0 if E > k else 0.0                     # an empty expert
    return ops.route(torch.topk(logits, k, dim=1).indices.to(torch.int32), E), g


def _data(shape, g, kind):
    x = torch.randn(shape, generator=g, device="cuda")
    return {"normal": x, "positive": x.abs(), "wide": x * torch.exp2(torch.randint(-20, 20, shape, generator=g, device="cuda").float())}[kind]


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("kind", ["normal", "positive", "wide"])
@pytest.mark.parametrize("T,K,N,nk", [(12000, 256, 512, True), (12000, 250, 1028, False), (9000, 321, 1000, True), (9000, 324, 1012, False),
                                      (7000, 1088, 272, False), (6000, 200, 2048, True), (32768, 92, 4096, True)])
def test_esmm_is_closer_than_the_fma_chain(T, K, N, nk, kind):
    L, ops = _mods()
    r, g = _routing(ops, T, 5, 2, K)
    assert L.lib().hexa_esmm_f32_workspace_bytes(5, r.row_capacity, N, K) > 0
    x = _data((T, K), g, kind)
    w = torch.randn(5, N, K, generator=g, device="cuda")
    if kind == "positive":
        w = w.abs()
    b = torch.randn(5, N, generator=g, device="cuda")
    xs = ops.gather_rows(x, r)
    wd, lay = (w, L.B_NK) if nk else (w.transpose(1, 2).contiguous(), L.B_KN)
    n_pad = int(r.pad_offsets[-1])
    po = r.pad_offsets.tolist()
    exact = torch.zeros(n_pad, N, dtype=torch.float64, device="cuda")
    for e in range(5):
        exact[po[e]:po[e + 1]] = xs[po[e]:po[e + 1]].double() @ w[e].double().t()
    got = ops.esmm(xs, wd, lay, r)[:n_pad]
    chain = ops.esmm(xs, wd, lay, r, engine=L.ENGINE_SIMT)[:n_pad]
    assert not torch.equal(got, chain)                      # the other path did run
    assert _rel(got, exact) <= _rel(chain, exact) and _rel(got, exact) < 4e-7
    live = r.row_token[:n_pad] >= 0
    assert (got[~live] == 0).all()
    exact[live] += b.double()[r.tile_expert[: n_pad // 128].repeat_interleave(128).long()][live]
    # epilogues: both ways round the same formulas in fp32 from sums that close (1e-5 is the fp32 tolerance of the operators)
    for epi, act in ((L.EPI_ACT, L.ACT_GELU), (L.EPI_ACT, L.ACT_SILU), (L.EPI_DACT, L.ACT_GELU), (L.EPI_DACT, L.ACT_RELU)):
        outs = []
        for eng in (L.ENGINE_AUTO, L.ENGINE_SIMT):
            aux = ops.sorted_buffer(r.row_capacity, N, torch.float32, "cuda")
            if epi == L.EPI_DACT:
                aux.copy_(torch.randn(aux.shape, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda"))
            y = ops.esmm(xs, wd, lay, r, b, epi, act, aux=aux, engine=eng)
            outs.append((y[:n_pad], aux[:n_pad]))
        (y0, a0), (y1, a1) = outs
        assert (y0[~live] == 0).all()
        assert float((y0 - y1).norm() / y1.norm()) < 3e-6 and float((a0 - a1).norm() / a1.norm()) < 3e-6
        if epi == L.EPI_ACT:
            assert _rel(a0, exact) <= _rel(a1, exact)


@pytest.mark.parametrize("kind", ["normal", "positive", "wide"])
@pytest.mark.parametrize("T,m,n,E", [(9000, 516, 1000, 4), (9000, 1001, 260, 7), (20000, 1001, 500, 7), (30000, 1000, 700, 3)])
def test_estmm_is_closer_than_the_fma_chain(T, m, n, E, kind):
    L, ops = _mods()
    r, g = _routing(ops, T, E, 2, m)
    assert L.lib().hexa_estmm_workspace_bytes(E, r.row_capacity, m, n, L.F32) > 0
    p, q = ops.gather_rows(_data((T, m), g, kind), r), ops.gather_rows(_data((T, n), g, kind), r)
    got = ops.estmm(p, q, r)
    chain = ops.estmm(p, q, r, engine=L.ENGINE_SIMT)
    po = r.pad_offsets.tolist()
    exact = torch.stack([p[po[e]:po[e + 1]].double().t() @ q[po[e]:po[e + 1]].double() for e in range(E)])
    if n % 4 == 0:
        assert not torch.equal(got, chain)
    assert _rel(got, exact) <= _rel(chain, exact) and _rel(got, exact) < 6e-7
    assert (got[1] == 0).all() or E <= 2


@pytest.mark.parametrize("kind", ["normal", "positive"])
@pytest.mark.parametrize("T,E", [(1016, 64), (400, 24)])
def test_estmm_of_few_rows_per_expert(T, E, kind):
    """From 16 rows per expert on planes are closer than a chain of so few FMAs; below, the chain computes the call."""
    L, ops = _mods()
    g = torch.Generator(device="cuda").manual_seed(E)
    ids = (torch.arange(T, device="cuda") % E).to(torch.int32).view(-1, 1)
    r = ops.route(ids, E)
    assert L.lib().hexa_estmm_workspace_bytes(E, r.row_capacity, 2048, 1024, L.F32) > 0
    assert L.lib().hexa_estmm_workspace_bytes(E, L.lib().hexa_route_row_capacity(8 * E, 1, E, 128), 2048, 1024, L.F32) == 0
    p, q = ops.gather_rows(_data((T, 2048), g, kind), r), ops.gather_rows(_data((T, 1024), g, kind), r)
    po = r.pad_offsets.tolist()
    exact = torch.stack([p[po[e]:po[e + 1]].double().t() @ q[po[e]:po[e + 1]].double() for e in range(E)])
    got, chain = ops.estmm(p, q, r), ops.estmm(p, q, r, engine=L.ENGINE_SIMT)
    assert not torch.equal(got, chain) and _rel(got, exact) <= _rel(chain, exact)


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("where", ["a", "b"])
def test_values_without_planes_take_the_fma_chain(bad, where):
    L, ops = _mods()
    T, K, N, E = 12000, 256, 512, 4
    r, g = _routing(ops, T, E, 2, 3)
    x = torch.randn(T, K, generator=g, device="cuda")
    w = torch.randn(E, N, K, generator=g, device="cuda")
    (x if where == "a" else w[2])[17, 5] = bad
    xs = ops.gather_rows(x, r)
    n_pad = int(r.pad_offsets[-1])
    y1, y2 = torch.empty(r.row_capacity, N, device="cuda"), torch.empty(r.row_capacity, N, device="cuda")
    got = ops.esmm(xs, w, L.B_NK, r, None, L.EPI_ACT, L.ACT_GELU, aux=y1)[:n_pad]
    want = ops.esmm(xs, w, L.B_NK, r, None, L.EPI_ACT, L.ACT_GELU, aux=y2, engine=L.ENGINE_SIMT)[:n_pad]
    assert torch.equal(got.nan_to_num(7.0, 8.0, 9.0), want.nan_to_num(7.0, 8.0, 9.0))
    assert torch.equal(y1[:n_pad].nan_to_num(7.0, 8.0, 9.0), y2[:n_pad].nan_to_num(7.0, 8.0, 9.0))
    dw, dw2 = ops.estmm(y1, xs, r), ops.estmm(y1, xs, r, engine=L.ENGINE_SIMT)
    if where == "a":
        assert torch.equal(dw.nan_to_num(7.0, 8.0, 9.0), dw2.nan_to_num(7.0, 8.0, 9.0))


def _scaled(x, e):
    """x * 2^e with the exponent in two steps (2^e alone may be out of range)."""
    return x * 2.0 ** (e // 2) * 2.0 ** (e - e // 2)


# Exponents of two operands of normal data: inside the range where planes hold, at both of its ends, and beyond.  Where
# they do not hold the answer is the FMA chain's own: bits are lost, products overflow in terms of either sign, or all fall
# below the normal range.
@pytest.mark.parametrize("ea,eb,planes", [(0, 0, True), (-80, 0, True), (-80, 60, True), (90, 20, True), (-60, -36, True), (55, 55, True),
                                          (-100, 0, False), (0, -112, False), (-116, 20, False), (-124, 100, False), (-140, 0, False),
                                          (-60, -50, False), (-64, -64, False), (-66, -66, False), (60, 60, False), (62, 62, False),
                                          (100, 20, False), (100, 100, False), (0, 126, False)])
def test_magnitudes_decide_between_planes_and_chain(ea, eb, planes):
    L, ops = _mods()
    T, K, N, E = 12000, 256, 512, 4
    r, g = _routing(ops, T, E, 2, 5)
    xs = ops.gather_rows(_scaled(torch.randn(T, K, generator=g, device="cuda"), ea), r)
    w = _scaled(torch.randn(E, N, K, generator=g, device="cuda"), eb)
    n_pad = int(r.pad_offsets[-1])
    po = r.pad_offsets.tolist()
    got, chain = (ops.esmm(xs, w, L.B_NK, r, engine=e)[:n_pad] for e in (L.ENGINE_AUTO, L.ENGINE_SIMT))
    if not planes:
        assert torch.equal(got.nan_to_num(7.0, 8.0, 9.0), chain.nan_to_num(7.0, 8.0, 9.0))
        return
    exact = torch.cat([xs[po[e]:po[e + 1]].double() @ w[e].double().t() for e in range(E)])
    assert not torch.equal(got, chain) and _rel(got, exact) <= _rel(chain, exact)


@pytest.mark.parametrize("value,planes", [(2.0 ** -109, True), (-2.0 ** -109 * (1 - 2.0 ** -24), False), (2.0 ** -149, False), (0.0, True),
                                          (3.3895e38, False), (2.0 ** 105, True), (2.0 ** 127, False)])
@pytest.mark.parametrize("op", ["a", "b", "tn"])
def test_one_value_decides(value, planes, op):
    """A single value at the ends of the range among normal data, in either operand of ESMM or one of ESTMM."""
    L, ops = _mods()
    T, K, N, E = 12000, 256, 2048, 4
    r, g = _routing(ops, T, E, 2, 3)
    x, w = torch.randn(T, K, generator=g, device="cuda"), torch.randn(E, N, K, generator=g, device="cuda")
    (w[2] if op == "b" else x)[17, 5] = value
    xs = ops.gather_rows(x, r)
    n_pad = int(r.pad_offsets[-1])
    if op == "tn":
        q = ops.gather_rows(torch.randn(T, N, generator=g, device="cuda"), r)
        got, chain = (ops.estmm(xs, q, r, engine=e) for e in (L.ENGINE_AUTO, L.ENGINE_SIMT))
    else:
        got, chain = (ops.esmm(xs, w, L.B_NK, r, engine=e)[:n_pad] for e in (L.ENGINE_AUTO, L.ENGINE_SIMT))
    assert torch.equal(got.nan_to_num(7.0, 8.0, 9.0), chain.nan_to_num(7.0, 8.0, 9.0)) != planes


def test_tiny_values_keep_their_products():
    """Operands around 1e-30, some of which lie below the range of planes: the result stays as close as the FMA chain's."""
    L, ops = _mods()
    r, g = _routing(ops, 12000, 4, 2, 5)
    x = torch.randn(12000, 256, generator=g, device="cuda") * 1e-30
    w = torch.randn(4, 512, 256, generator=g, device="cuda")
    xs = ops.gather_rows(x, r)
    n_pad = int(r.pad_offsets[-1])
    po = r.pad_offsets.tolist()
    exact = torch.cat([xs[po[e]:po[e + 1]].double() @ w[e].double().t() for e in range(4)])
    got = _rel(ops.esmm(xs, w, L.B_NK, r)[:n_pad], exact)
    assert got <= _rel(ops.esmm(xs, w, L.B_NK, r, engine=L.ENGINE_SIMT)[:n_pad], exact)


def test_relu_masks_do_not_depend_on_the_path():
    L, ops = _mods()
    r, g = _routing(ops, 12000, 5, 2, 9)
    x = torch.randn(12000, 256, generator=g, device="cuda")
    w = torch.randn(5, 512, 256, generator=g, device="cuda")
    xs = ops.gather_rows(x, r)
    n_pad = int(r.pad_offsets[-1])
    a = [torch.empty(r.row_capacity, 512, device="cuda") for _ in range(2)]
    y = [ops.esmm(xs, w, L.B_NK, r, None, L.EPI_ACT, L.ACT_RELU, aux=a[i], engine=e)[:n_pad] for i, e in enumerate((L.ENGINE_AUTO, L.ENGINE_SIMT))]
    assert torch.equal(y[0], y[1]) and torch.equal(a[0][:n_pad], a[1][:n_pad])


def test_without_room_for_planes_the_chain_computes_the_call():
    """The scratch is optional: when the allocator cannot give it, the CUDA cores do what they did without any."""
    L, ops = _mods()
    T, K, N, E = 60000, 512, 2048, 4
    r, g = _routing(ops, T, E, 1, 1)
    xs = ops.gather_rows(torch.randn(T, K, generator=g, device="cuda"), r)
    w = torch.randn(E, N, K, generator=g, device="cuda")
    n_pad = int(r.pad_offsets[-1])
    h, dw = torch.empty(r.row_capacity, N, device="cuda"), torch.empty(E, N, K, device="cuda")
    need = min(L.lib().hexa_esmm_f32_workspace_bytes(E, r.row_capacity, N, K), L.lib().hexa_estmm_workspace_bytes(E, r.row_capacity, N, K, L.F32))
    assert need > 128 << 20
    want = ops.esmm(xs, w, L.B_NK, r, engine=L.ENGINE_SIMT)[:n_pad].clone()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
    try:
        ops.esmm(xs, w, L.B_NK, r, out=h)
        ops.estmm(h, xs, r, out=dw)
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(h[:n_pad], want)
    assert torch.equal(dw, ops.estmm(h, xs, r, engine=L.ENGINE_SIMT))
    assert not torch.equal(ops.esmm(xs, w, L.B_NK, r)[:n_pad], want)      # with room the planes are taken
