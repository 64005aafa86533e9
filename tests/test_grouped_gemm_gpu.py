"""The grouped bfloat16 products at the edges of their tiles: remainders of K, N and rows, columns that do not start on 16
bytes, tiles with gaps, both tile heights; against float64 sums, and the two heights against one another bit by bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def ops():
    from llm_infer_engine_b200.kernels import ops as o
    return o


def _close(got, ref, absolute, out_dtype):
    """float32 sums of K products, and one rounding of a bfloat16 result."""
    bound = 2.0 ** -16 * absolute + (2.0 ** -8 * ref.abs() if out_dtype == torch.bfloat16 else 0) + 1e-6
    assert bool(((got.double() - ref).abs() <= bound).all()), float((got.double() - ref).abs().max())


@pytest.mark.parametrize("T", [1, 16, 17, 64, 65, 200])
@pytest.mark.parametrize("G,N,K,shift", [(3, 64, 64, 0), (2, 72, 8, 0), (4, 130, 200, 0), (2, 33, 65, 0), (3, 64, 128, 1),
                                         (2, 70, 712, 0)])                   # rings that come round more than once
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_batched(T, G, N, K, shift, out_dtype):
    g = torch.Generator().manual_seed(T + N + K)
    a = torch.randn(T, G * K + 8 + shift, generator=g).to(torch.bfloat16)
    w = torch.randn(G, N, K, generator=g).to(torch.bfloat16)
    wide = torch.zeros(T, G * (N + 4) + 8 + shift, dtype=out_dtype, device=DEV)
    out = wide[:, shift:]                                     # shift 1: neither A's nor C's columns start on 16 bytes
    ops().batched_gemm_nt(a.to(DEV)[:, shift:], w.to(DEV), out, K, N + 4, K)
    for i in range(G):
        x, y = a[:, shift + i * K:shift + (i + 1) * K].double(), w[i].double()
        _close(out[:, i * (N + 4):i * (N + 4) + N].cpu(), x @ y.T, x.abs() @ y.abs().T, out_dtype)
        assert not bool(out[:, i * (N + 4) + N:(i + 1) * (N + 4)].any())        # nothing beside the columns


@pytest.mark.parametrize("pairs", [5, 63, 150])
@pytest.mark.parametrize("N,K", [(64, 64), (100, 72), (40, 37), (70, 712)])
@pytest.mark.parametrize("dual", [False, True])
def test_routed_tiles_of_both_heights(pairs, N, K, dual):
    E, o = 5, ops()
    g = torch.Generator().manual_seed(pairs + N)
    x = torch.randn(pairs, K, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(E, (2 if dual else 1) * N, K, generator=g).to(torch.bfloat16).to(DEV)
    expert = torch.randint(0, E, (pairs,), generator=g)
    expert[: pairs // 2] = 1                                  # one expert with several slices of rows, maybe some without
    results = []
    for small in (True, False):
        tile = o.grouped_tile_rows(small)
        rows, groups = [], []
        for e in range(E):
            mine = (expert == e).nonzero().flatten().tolist()
            mine += [-1] * (-len(mine) % tile)
            rows, groups = rows + mine, groups + [e] * (len(mine) // tile)
        groups.append(-1)                                     # a tile that is not used
        rows += [-1] * tile
        pos = torch.tensor(rows, dtype=torch.int32, device=DEV)
        out = torch.full((pairs, N), 7.0, device=DEV, dtype=torch.float32)
        o.routed_gemm_nt(x, pos, w, out, pos, torch.tensor(groups, dtype=torch.int32, device=DEV), len(rows), small,
                         dual=dual, act=o.ACT_SILU if dual else o.ACT_NONE)
        results.append(out)
    assert torch.equal(*results)
    z = torch.einsum("pk,pnk->pn", x.double(), w.double()[expert.to(DEV)])
    a = torch.einsum("pk,pnk->pn", x.double().abs(), w.double()[expert.to(DEV)].abs())
    if dual:
        gate, up = z[:, :N], z[:, N:]
        ref = gate * torch.sigmoid(gate) * up
        _close(results[0], ref, 2.0 ** 3 * (a[:, :N] * up.abs() + a[:, N:] * gate.abs() + 1), torch.float32)
    else:
        _close(results[0], z, a, torch.float32)
