"""The prompts' grouped bfloat16 products on tcgen05 at the edges of their tiles (128 rows, 64 to 256 weight rows, 64 k): groups
without rows, remainders of rows, N and K, more tiles than blocks; against float64 sums, and against the kernel of fewer rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
U = 2.0 ** -8          # unit roundoff of bfloat16: 8 significant bits, round to nearest


def ops():
    from llm_infer_engine_b200.kernels import ops as o
    return o


def _sum_bound(x, w):
    """float32 sums of K products: relative to the sum of the products' magnitudes, as for the other grouped products."""
    return 2.0 ** -16 * (x.abs() @ w.abs().T) + 1e-6


@pytest.mark.parametrize("rows", [(64, 0, 128, 1, 0), (0, 0, 0, 300, 257), (1, 1, 1, 1, 1), (0, 0, 0, 0, 0), (640, 0, 64, 129, 127)])
@pytest.mark.parametrize("N,K", [(8, 8), (256, 64), (120, 200), (264, 72), (2048, 320)])
@pytest.mark.parametrize("form", ["plain", "relu", "dual"])
def test_routed(rows, N, K, form):
    o, E, P = ops(), len(rows), sum(rows) + 70
    g = torch.Generator().manual_seed(P + N + K)
    a = torch.randn(P, K, generator=g).to(torch.bfloat16)
    w = torch.randn(E, (2 if form == "dual" else 1) * N, K, generator=g).to(torch.bfloat16)
    end = torch.tensor(rows).cumsum(0)
    out = torch.full((P, N), 7.0, dtype=torch.bfloat16, device=DEV)
    o.routed_gemm_tc(a.to(DEV), w.to(DEV), out, end.int().to(DEV), form == "dual",
                     o.ACT_NONE if form == "plain" else o.ACTIVATIONS["relu"])
    got = out.cpu().double()
    assert bool((got[int(end[-1]):] == 7.0).all())                     # nothing behind the last group's rows
    for e in range(E):
        x, y = a[int(end[e]) - rows[e]:int(end[e])].double(), w[e].double()
        s, b = x @ y.T, _sum_bound(x, y)
        mine = got[int(end[e]) - rows[e]:int(end[e])]
        if form == "dual":
            # both products rounded to bfloat16 (U each, and the sums' own error), their product rounded again
            (gate, up), (bg, bu) = s.split(N, 1), b.split(N, 1)
            eg, eu = bg + U * (gate.abs() + bg), bu + U * (up.abs() + bu)
            s, b = gate.clamp(min=0) * up, eg * up.abs() + eu * gate.abs() + eg * eu
        elif form == "relu":
            b, s = b + U * (s.abs() + b), s.clamp(min=0)
        assert bool(((mine - s).abs() <= b + U * (s.abs() + b)).all()), float((mine - s).abs().max())


@pytest.mark.parametrize("T", [128, 129, 255, 1000])
@pytest.mark.parametrize("G,N,K", [(3, 64, 64), (2, 72, 128), (5, 8, 64), (2, 264, 192), (32, 256, 64), (40, 64, 256)])
def test_batched(T, G, N, K):
    o = ops()
    assert T >= o.BATCHED_TC_FROM
    g = torch.Generator().manual_seed(T + N + K)
    a = torch.randn(T, G * (K + 8) + 8, generator=g).to(torch.bfloat16)
    w = torch.randn(G, N, K, generator=g).to(torch.bfloat16)
    out = torch.zeros(T, G * (N + 8) + 8, dtype=torch.bfloat16, device=DEV)
    few = torch.zeros(64, G * (N + 8) + 8, dtype=torch.bfloat16, device=DEV)
    o.batched_gemm_nt(a.to(DEV)[:, 8:], w.to(DEV), out[:, 8:], K + 8, N + 8, K)
    o.batched_gemm_nt(a.to(DEV)[:64, 8:], w.to(DEV), few[:, 8:], K + 8, N + 8, K)          # the kernel of fewer rows
    assert not bool(out[:, :8].any())
    for i in range(G):
        x, y = a[:, 8 + i * (K + 8):8 + i * (K + 8) + K].double(), w[i].double()
        mine = out[:, 8 + i * (N + 8):8 + (i + 1) * (N + 8)].cpu().double()
        s, b = x @ y.T, _sum_bound(x, y)
        assert bool(((mine[:, :N] - s).abs() <= b + U * (s.abs() + b)).all())
        assert not bool(mine[:, N:].any())                            # nothing beside the columns
        f = few[:, 8 + i * (N + 8):8 + i * (N + 8) + N].cpu().double()
        assert bool(((mine[:64, :N] - f).abs() <= 2 * b[:64] + 2 * U * (s[:64].abs() + b[:64])).all())


@pytest.mark.parametrize("T", [128, 300])
def test_batched_rows_that_overlap(T):
    """One row for all (stride 0), and windows of a sequence: what the kernel of fewer rows takes, whatever their number."""
    o = ops()
    G, N, K = 3, 64, 64
    w = torch.randn(G, N, K, device=DEV).to(torch.bfloat16)
    flat = torch.randn(T * 8 + G * K, device=DEV).to(torch.bfloat16)
    for a in (flat[:G * K].expand(T, G * K), flat.as_strided((T, G * K), (8, 1))):
        out = torch.zeros(T, G * N, dtype=torch.bfloat16, device=DEV)
        o.batched_gemm_nt(a, w, out, K, N, K)
        want = torch.zeros_like(out)
        o.batched_gemm_nt(a.contiguous(), w, want, K, N, K)
        assert torch.equal(out, want)


@pytest.mark.parametrize("G,N,K", [(3, 64, 64), (2, 72, 128), (5, 8, 64), (2, 264, 192), (32, 256, 64), (40, 64, 256), (2, 512, 1024)])
@pytest.mark.parametrize("spread", [0.0, 3.0])
def test_batched_rows_do_not_depend_on_the_step(G, N, K, spread):
    """A row's bits in a step of few rows (tiles of 16, of 64) and of many (tcgen05); numbers alike, and over many powers of two."""
    o, T = ops(), 400
    g = torch.Generator().manual_seed(G + N + K)
    a = (torch.randn(T, G * K, generator=g) * torch.exp(spread * torch.randn(T, G * K, generator=g))).to(torch.bfloat16).to(DEV)
    w = (torch.randn(G, N, K, generator=g) * torch.exp(spread * torch.randn(G, N, K, generator=g))).to(torch.bfloat16).to(DEV)

    def product(rows):
        out = torch.zeros(rows, G * N, dtype=torch.bfloat16, device=DEV)
        return o.batched_gemm_nt(a[:rows], w, out, K, N, K)

    many = product(T)
    for rows in (1, 16, 64, 65, 127, 128):
        assert torch.equal(product(rows), many[:rows]), rows


def test_no_finite_value_crosses_rows_or_groups():
    o = ops()
    a = torch.ones(256, 72, dtype=torch.bfloat16, device=DEV)
    a[130] = float("nan")
    w = torch.ones(2, 64, 72, dtype=torch.bfloat16, device=DEV)
    w[1, 5] = float("inf")
    out = torch.zeros(256, 64, dtype=torch.bfloat16, device=DEV)
    o.routed_gemm_tc(a, w, out, torch.tensor([100, 256], dtype=torch.int32, device=DEV))
    bad = ~torch.isfinite(out)
    want = torch.zeros_like(bad)
    want[130] = True
    want[100:, 5] = True
    assert torch.equal(bad, want)


@pytest.mark.parametrize("form", ["routed", "dual", "batched"])
def test_a_block_that_gives_up_leaves_no_numbers(form):
    """Waits that run out (no polls at all here): NaN in every row that has a group, also in tiles that a block never came to, an
    error for whoever asks, and the next call is none the worse."""
    o = ops()
    E, K = 5, 128
    N = 4104 if form == "routed" else 2056 if form == "dual" else 64        # more tiles than blocks; the batched form has fewer
    rows = torch.tensor([640, 0, 64, 129, 127])
    end = rows.cumsum(0).int().to(DEV)
    P = int(rows.sum()) + 30
    a = torch.randn(P, E * K if form == "batched" else K, device=DEV).to(torch.bfloat16)
    w = torch.randn(E, 2 * N if form == "dual" else N, K, device=DEV).to(torch.bfloat16)
    out = torch.full((P, E * N if form == "batched" else N), 3.0, dtype=torch.bfloat16, device=DEV)
    status = o.tc_status_word(torch.device(DEV, 0))
    groups = (None, E, P, N, K, 0, 0) if form == "batched" else (end.data_ptr(), E, P, N, K, int(form == "dual"), 0)
    cols = (K, N) if form == "batched" else (0, 0)
    f = o._fn("grouped_gemm_tc", "llmie_grouped_gemm_tc_form",
              [o._c_void_p, o._c_ll, o._c_ll, o._c_void_p, o._c_void_p, o._c_ll, o._c_ll, o._c_void_p] + [o._c_int] * 6
              + [o._c_void_p, o._c_int, o._c_void_p])

    def call(no_wait):
        assert f(a.data_ptr(), a.shape[1], cols[0], w.data_ptr(), out.data_ptr(), out.shape[1], cols[1], *groups, status.data_ptr(),
                 no_wait, o._stream()) == 0
        torch.cuda.synchronize()
        return out[:P if form == "batched" else int(rows.sum())]

    assert bool(call(1).isnan().all())
    with pytest.raises(o.KernelError):
        o.check_tc_status(torch.device(DEV, 0))
    assert bool(call(0).isfinite().all()) and (form == "batched" or bool((out[int(rows.sum()):] == 3.0).all()))
    o.check_tc_status(torch.device(DEV, 0))


@pytest.mark.parametrize("experts", [4, 8, 16])
@pytest.mark.parametrize("rows", [32, 33, 64, 65, 127, 128, 129, 400])
def test_down_products_of_few_pairs_are_not_rounded(experts, rows):
    """Routed experts around the sizes where their kernels change. Inputs and weights are small whole numbers, so everything up to
    the down products is exact, and those are whole numbers that bfloat16 does not hold: up to 256 pairs only the weighted sum rounds."""
    from test_parts_gpu import build
    d, ff, top = 64, 32, 2
    part, _ = build("feed_forward", "routed_experts", {"hidden": d, "n_experts": experts, "top": top, "expert_ff": ff,
                                                       "activation": "relu", "router_bias": False}, "bfloat16", seed=1)
    g = torch.Generator().manual_seed(rows)
    whole = lambda lo, hi, *s: torch.randint(lo, hi + 1, s, generator=g).double()                    # noqa: E731
    router, x = torch.randn(experts, d, generator=g).double() / 8, whole(-1, 1, rows, d)
    gate, up = (whole(-1, 1, experts, ff, d) * (torch.rand(experts, ff, d, generator=g) < 0.1) for _ in range(2))
    down = whole(-200, 200, experts, d, ff)
    tensors = {"router": router.float()}
    for e in range(experts):
        tensors.update({f"e{e}.gate": gate[e], f"e{e}.up": up[e], f"e{e}.down": down[e]})
    part.load({k: v.to(torch.float32 if k == "router" else torch.bfloat16).to(DEV) for k, v in tensors.items()})
    got = part.forward(x.to(torch.bfloat16).to(DEV), None).cpu().double()
    scores, ids = (x @ router.float().double().T).topk(top, 1)
    weights = scores.softmax(1)
    act = torch.einsum("td,efd->tef", x, gate).clamp(min=0) * torch.einsum("td,efd->tef", x, up)
    assert float(act.abs().max()) <= 256
    y = torch.einsum("tef,edf->ted", act, down)
    assert float(y.abs().max()) > 512
    y = y.gather(1, ids[:, :, None].expand(-1, -1, d))
    want, size = (weights[:, :, None] * y).sum(1), (weights[:, :, None] * y.abs()).sum(1)
    # float32 scores of 64 terms (their size times 2^-17 at most), exponentials, two products and a sum
    bound = 1e-4 * size + 1e-6 if rows * top <= 256 else (1e-4 + U) * size + 1e-6
    assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() / (size + 1)).max())
