"""The routed feed-forward's small kernels and the elementwise kernels with wide accesses: several tokens a block, odd
counts, sizes that take the wide and the element-by-element forms, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def ops():
    from llm_infer_engine_b200.kernels import ops as o
    return o


@pytest.mark.parametrize("T", [1, 295, 297, 411])
@pytest.mark.parametrize("d,E,top", [(64, 16, 3), (100, 7, 2), (130, 33, 5), (2048, 3, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_route(T, d, E, top, dtype):
    g = torch.Generator().manual_seed(T + d)
    x = torch.randn(T, d, generator=g).to(dtype).to(DEV)
    w, b = torch.randn(E, d, generator=g).to(DEV), torch.randn(E, generator=g).to(DEV)
    ids = torch.empty(T, top, dtype=torch.int32, device=DEV)
    wt = torch.empty(T, top, device=DEV)
    ops().moe_route(x, w, b, ids, wt)
    z = x.double() @ w.double().T + b.double()
    bound = d * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T).max() + 1e-6     # sums of d products in float32
    best = z.topk(top, dim=1)
    picked = z.gather(1, ids.long())
    assert bool(((picked - best.values).abs() <= bound).all())          # the largest, or one that ties with it
    assert bool((wt.double() - picked.softmax(1)).abs().max() <= 4 * bound)
    one, one_w = torch.empty(1, top, dtype=torch.int32, device=DEV), torch.empty(1, top, device=DEV)
    ops().moe_route(x[T // 2:T // 2 + 1], w, b, one, one_w)             # a token alone: the same bits
    assert torch.equal(one[0], ids[T // 2]) and torch.equal(one_w[0], wt[T // 2])


@pytest.mark.parametrize("T", [3, 297])
@pytest.mark.parametrize("rule", ["all", "sigmoid", "groups"])
@pytest.mark.parametrize("d,E,top", [(64, 16, 3), (100, 8, 2), (136, 40, 5)])
def test_route_rules(T, rule, d, E, top):
    """The other choices and weights, a token and two tokens a block: scores that each token's own part of shared memory holds."""
    g = torch.Generator().manual_seed(T + E)
    x, w = torch.randn(T, d, generator=g).to(torch.bfloat16).to(DEV), (torch.randn(E, d, generator=g) / d ** 0.5).to(DEV)
    correction = None if rule == "sigmoid" else (torch.randn(E, generator=g) * 0.1).to(DEV)
    mode = {"all": True, "sigmoid": ops().ROUTE_SIGMOID, "groups": ops().ROUTE_SIGMOID_GROUPS}[rule]
    groups = (4, 2) if rule == "groups" else (1, 1)

    def route(rows):
        ids = torch.empty(len(rows), top, dtype=torch.int32, device=DEV)
        wt = torch.empty(len(rows), top, device=DEV)
        ops().moe_route(rows, w, None, ids, wt, mode, correction, 1.7, groups)
        return ids, wt

    ids, wt = route(x)
    z = x.double() @ w.double().T
    score = z.softmax(1) if rule == "all" else torch.sigmoid(z)
    choice = z.clone() if rule == "sigmoid" else score + correction.double()
    if rule == "groups":
        best = choice.view(T, 4, -1).topk(2, dim=2).values.sum(2).topk(2, dim=1).indices
        kept = torch.zeros(T, 4, dtype=torch.bool, device=DEV).scatter(1, best, True)
        choice = choice.masked_fill(~kept.repeat_interleave(E // 4, 1), -1e9)
    bound = d * 2.0 ** -23 * float((x.double().abs() @ w.double().abs().T).max()) + 1e-6     # sums of d products in float32
    assert bool(((choice.gather(1, ids.long()) - choice.topk(top, dim=1).values).abs() <= bound).all())
    picked = score.gather(1, ids.long())
    want = picked / picked.sum(1, keepdim=True) * 1.7 if rule == "all" else picked * 1.7
    assert bool(((wt.double() - want).abs() <= 4 * bound).all())
    for t in (0, T // 2, T - 1):                                             # a token alone: the same bits
        one, one_w = route(x[t:t + 1].contiguous())
        assert torch.equal(one[0], ids[t]) and torch.equal(one_w[0], wt[t])


@pytest.mark.parametrize("T,d,top", [(1, 8, 1), (5, 2056, 3), (3, 100, 9), (70, 264, 2)])
@pytest.mark.parametrize("y_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("identity", [False, True])
def test_combine(T, d, top, y_dtype, identity):
    g = torch.Generator().manual_seed(T * d)
    n_real = 4
    ids = torch.randint(0, n_real + (2 if identity else 0), (T, top), generator=g, dtype=torch.int32).to(DEV)
    y = torch.randn(T * top + 3, d, generator=g).to(y_dtype).to(DEV)
    pos = torch.randperm(T * top + 3, generator=g)[:T * top].to(torch.int32).to(DEV)
    wt, x = torch.rand(T, top, generator=g).to(DEV), torch.randn(T, d, generator=g).to(torch.bfloat16).to(DEV)
    shared, out = torch.randn(T, d, generator=g).to(DEV), torch.empty(T, d, device=DEV)
    rows = y.double()[pos.long()].view(T, top, d)
    if identity:
        ops().moe_combine_identity(y, wt, ids, n_real, x, out, pos)
        rows = torch.where((ids >= n_real)[..., None], x.double()[:, None, :], rows)
        ref = (wt.double()[..., None] * rows).sum(1)
    else:
        ops().moe_combine(y, wt, shared, out, pos)
        ref = (wt.double()[..., None] * rows).sum(1) + shared.double()
    bound = (top + 2) * 2.0 ** -23 * ((wt.double()[..., None] * rows.abs()).sum(1) + shared.double().abs())
    assert bool(((out.double() - ref).abs() <= bound + 1e-7).all())


@pytest.mark.parametrize("T,n,extra", [(1, 8, 0), (3, 2056, 8), (33, 264, 4), (2, 100, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gate_per_element(T, n, extra, dtype):
    g = torch.Generator().manual_seed(n)
    out = torch.randn(T, n, generator=g).to(dtype).to(DEV)
    wide = (torch.randn(T, n + extra, generator=g) * 3).to(dtype).to(DEV)
    ref = out.double() * torch.sigmoid(wide[:, extra:].double())
    ops().sigmoid_gate(out, wide[:, extra:])
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    assert bool(((out.double() - ref).abs() <= rel * ref.abs() + 1e-30).all())


@pytest.mark.parametrize("Dv", [32, 64, 128, 48, 256])
@pytest.mark.parametrize("items,per_row", [(1, 1), (7, 7), (66, 3)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("gated", [False, "sigmoid", "silu"])
@pytest.mark.parametrize("per_head", [False, True])
def test_head_norm(Dv, items, per_row, dtype, gated, per_head):
    g = torch.Generator().manual_seed(Dv + items)
    rows = items // per_row
    o = torch.randn(rows, per_row * Dv, generator=g).to(DEV)
    w = (torch.rand(Dv * (per_row if per_head else 1), generator=g) + 0.5).to(DEV)      # of all heads, or one a head
    gate = torch.randn(rows, per_row * Dv + 5, generator=g).to(dtype).to(DEV)[:, 5:] if gated else None
    y = ops().head_rmsnorm(o, w, 1e-6, torch.empty(rows, per_row * Dv, dtype=dtype, device=DEV), Dv, gate=gate,
                           gate_silu=gated == "silu")
    x = o.double().view(rows, per_row, Dv)
    ref = (x / (x.square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double().view(-1, Dv)).view(rows, -1)
    if gated:
        ref = ref * torch.sigmoid(gate.double()) * (gate.double() if gated == "silu" else 1)
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -18
    assert bool(((y.double() - ref).abs() <= rel * ref.abs() + 1e-30).all())


@pytest.mark.parametrize("T,n,q_off,f_off,pad", [(1, 8, 0, 8, 0), (70, 1032, 8, 1048, 8), (3, 100, 0, 100, 0), (2, 64, 4, 72, 4)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gates_of_a_recurrence(T, n, q_off, f_off, pad, dtype):
    g = torch.Generator().manual_seed(T + n)
    proj = (torch.randn(T, f_off + n + pad, generator=g) * 3).to(dtype).to(DEV)
    bias, lower = torch.randn(n, generator=g).to(DEV), (torch.rand(n, generator=g) * 0.9).to(DEV)
    q, f = torch.empty(T, n, device=DEV), torch.empty(T, n, device=DEV)
    ops().matrix_gates(proj, q_off, f_off, bias, lower, q, f)
    x, z = proj[:, q_off:q_off + n].double(), proj[:, f_off:f_off + n].double() + bias.double()
    want_q, want_f = x * torch.sigmoid(x), lower.double() + (1 - lower.double()) * torch.sigmoid(z)
    assert bool(((q.double() - want_q).abs() <= 2.0 ** -19 * want_q.abs() + 1e-30).all())
    assert bool(((f.double() - want_f).abs() <= 2.0 ** -19 * (want_f.abs() + z.abs())).all())
