"""Decode attention of long sequences of unequal lengths: six warps a block, the longest sequences served first. Against the
plain kernel: every sequence is served, by both entry points, up to 64 sequences and above, with equal lengths among them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _step(hd, n, longest, n_q=32, n_kv=8):
    """A step of n sequences: the blocks' runs, and both entry points against the plain kernel."""
    from llm_infer_engine_b200.kernels import ops
    g = torch.Generator().manual_seed(n * hd)
    lens = torch.randint(1, longest + 1, (n,), generator=g)
    lens[n // 2], lens[3], lens[n - 1], lens[5] = longest, lens[7], 1, lens[7]          # the longest, the shortest, equal ones
    pages = (lens + 63) // 64
    total, most = int(pages.sum()), int(pages.max())
    table, at, order = torch.zeros(n, most, dtype=torch.int32), 0, torch.randperm(total, generator=g)
    for i, p in enumerate(pages.tolist()):
        table[i, :p] = order[at:at + p].int()
        at += p
    k = torch.randn(total + 1, n_kv, 64, hd, generator=g).to(torch.bfloat16).to(DEV)
    v = torch.randn(total + 1, n_kv, 64, hd, generator=g).to(torch.bfloat16).to(DEV)
    table, kvlen = table.to(DEV), lens.int().to(DEV)
    slots, seq = torch.arange(n, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV)
    qkv = torch.randn(n, (n_q + 2 * n_kv) * hd, generator=g).to(torch.bfloat16).to(DEV)
    still = torch.zeros(longest, hd // 2, 2, device=DEV)
    still[..., 0] = 1.0                                               # a rotation by nothing
    per = ops.attention_decode_mma_pages(n, n_q, n_kv, longest)
    runs = (most + per - 1) // per
    counters = torch.zeros(4096, dtype=torch.int32, device=DEV)
    got = torch.full((n, n_q * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.attention_decode_mma_rope(qkv, k, v, got, still, slots, kvlen, table, 64, n_q, n_kv, hd, hd ** -0.5, 0, per, runs, True,
                                  counters=counters)                  # writes the new keys and values into the cache
    q = qkv[:, :n_q * hd].contiguous()
    want, plain = torch.full_like(got, float("nan")), torch.full_like(got, float("nan"))
    ops.attention_decode_mma(q, k, v, want, slots, kvlen, table, 64, n_q, n_kv, hd, hd ** -0.5, 0, per, runs, counters=counters)
    ops.attention_paged(q, k, v, plain, kvlen - 1, seq, slots, table, 64, n_q, n_kv, hd, hd ** -0.5, 0)
    assert torch.equal(got, want) and not bool(counters.any())
    # outputs and probabilities are bfloat16: as in the other tests of this kernel
    assert torch.allclose(want.float(), plain.float(), atol=2e-2, rtol=1.6e-2)
    return runs


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("n,longest", [(19, 2100), (36, 2113), (40, 2113), (49, 2100), (64, 2300), (65, 2200), (33, 1100)])
def test_every_sequence_is_served(hd, n, longest):
    _step(hd, n, longest)


@pytest.mark.parametrize("hd,n,longest,runs", [(128, 16, 4300, 2), (128, 15, 8300, 2), (128, 17, 4200, 2), (64, 9, 8300, 4)])
def test_runs_that_meet(hd, n, longest, runs):
    """Sequences in several runs, whose blocks meet by the counters, the longest first (head size 128: more blocks than SMs)."""
    assert _step(hd, n, longest) == runs


@pytest.mark.parametrize("hd", [64, 128])
def test_a_key_head_for_every_query_head(hd):
    """Many more blocks than fit at once: few warps a block, the longest sequences first."""
    _step(hd, 40, 2100, 32, 32)
