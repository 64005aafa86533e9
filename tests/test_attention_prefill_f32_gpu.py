"""The float32 path's prompt attention in tiles against the plain kernel's math in float64: edges of pages and tiles, pieces
behind held tokens, windows and chunks, both tile heights and both head sizes; a row's bits whatever is in the step; values
that are not finite stay with the rows that see them."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(lens, held, n_q, n_kv, hd, seed=0):
    g = torch.Generator().manual_seed(seed)
    need = [(h + l + 63) // 64 for h, l in zip(held, lens)]
    order = torch.randperm(sum(need) + 2, generator=g).tolist()
    table = torch.full((len(lens) + 1, max(need)), sum(need) + 2, dtype=torch.int32)
    k, v = (torch.full((sum(need) + 3, n_kv, 64, hd), float("nan")) for _ in "kv")       # nobody's rows are never read
    q = torch.randn(sum(lens), n_q * hd, generator=g)
    rows, at = [], 0
    for i in range(len(lens)):
        kv = torch.randn(2, n_kv, held[i] + lens[i], hd, generator=g)
        rows.append(kv)
        for j in range(need[i]):
            page, part = order[at], kv[:, :, 64 * j:64 * j + 64]
            table[i, j], at = page, at + 1
            k[page, :, :part.shape[2]], v[page, :, :part.shape[2]] = part[0], part[1]
    return q.to(DEV), k.to(DEV), v.to(DEV), rows, table.to(DEV)


def _run(q, k, v, table, lens, held, slots, n_q, n_kv, hd, scale, window):
    from llm_infer_engine_b200.kernels import ops
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)              # noqa: E731
    cu = [0]
    for l in lens:
        cu.append(cu[-1] + l)
    out = torch.full((sum(lens), n_q * hd), float("nan"), device=DEV)
    return ops.attention_prefill_f32(q, k, v, out, i32(cu), i32(slots), i32(held), table, 64, len(lens), max(lens), n_q, n_kv,
                                     hd, scale, window)


def _reference(q, rows, lens, held, n_q, n_kv, hd, scale, window):
    out, at = [], 0
    for kv, l, h in zip(rows, lens, held):
        k, v = (t.double().to(DEV).repeat_interleave(n_q // n_kv, 0) for t in kv)
        x = q[at:at + l].double().view(l, n_q, hd).transpose(0, 1)
        at += l
        pos, key = torch.arange(h, h + l, device=DEV)[:, None], torch.arange(h + l, device=DEV)[None, :]
        lo = pos - window + 1 if window > 0 else pos - pos % -window if window < 0 else 0 * pos
        s = (x @ k.transpose(1, 2) * scale).masked_fill((key > pos) | (key < lo), -math.inf)
        out.append((s.softmax(-1) @ v).transpose(0, 1).reshape(l, n_q * hd))
    return torch.cat(out)


@pytest.mark.parametrize("n_q,n_kv,hd", [(4, 2, 64), (3, 1, 128)])
@pytest.mark.parametrize("lens,held", [([1, 16, 9], [0, 700, 63]), ([65, 1, 200, 128, 9], [0, 63, 130, 64, 300]), ([17], [0])])
@pytest.mark.parametrize("window", [0, 70, -96])
def test_prompts(n_q, n_kv, hd, lens, held, window):
    q, k, v, rows, table = _case(lens, held, n_q, n_kv, hd)
    scale = 1.5 * hd ** -0.5
    out = _run(q, k, v, table, lens, held, list(range(len(lens))), n_q, n_kv, hd, scale, window)
    want = _reference(q, rows, lens, held, n_q, n_kv, hd, scale, window)
    # scores: hd products; weights: their absolute error relative to the weight; sums of at most 900 weighted values
    bound = (hd * 2.0 ** -24 * 12 + 2.0 ** -21) * 5
    assert bool(((out.double() - want).abs() <= bound).all()), float((out.double() - want).abs().max())
    at = 0
    for i, l in enumerate(lens):                                   # each alone: the same bits, whichever tile height
        one = _run(q[at:at + l].contiguous(), k, v, table, [l], [held[i]], [i], n_q, n_kv, hd, scale, window)
        assert torch.equal(one, out[at:at + l]), i
        at += l


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_what_is_not_finite_stays_behind(bad):
    lens, held, n_q, n_kv, hd = [100], [30], 4, 2, 64
    q, k, v, rows, table = _case(lens, held, n_q, n_kv, hd, seed=3)
    want = _run(q, k, v, table, lens, held, [0], n_q, n_kv, hd, 0.2, 0)
    for cache in (k, v):
        spoiled = cache.clone()
        spoiled[int(table[0, 1]), :, 90 - 64] = bad                # position 90: the step's token 60
        a, b = (spoiled, v) if cache is k else (k, spoiled)
        out = _run(q, a, b, table, lens, held, [0], n_q, n_kv, hd, 0.2, 0)
        assert torch.equal(out[:60], want[:60]) and not bool(torch.isfinite(out[60:]).all())


@pytest.mark.parametrize("dtype,heads,hd,hdv", [("float32", 4, 64, 64), ("bfloat16", 4, 96, 64)])
def test_an_output_that_does_not_start_on_16_bytes(dtype, heads, hd, hdv):
    """As a layer calls it: float32 prompts, and latent rows in bfloat16. The kernels with 16-byte stores refuse such an output
    and others take it."""
    import types
    from llm_infer_engine_b200.parts.base import AttentionOptions
    from test_parts_gpu import DTYPES, kernel_plan, make_ctx
    g, dt = torch.Generator().manual_seed(3), DTYPES[dtype]
    k = torch.randn(4, 1, 64, hd, generator=g).to(dt).to(DEV)
    v = k[..., :hdv] if hdv != hd else torch.randn(4, 1, 64, hd, generator=g).to(dt).to(DEV)
    kv = types.SimpleNamespace(k=k, v=v, page_size=64, block_table=torch.tensor([[0, 1, 2]], dtype=torch.int32, device=DEV))
    q = torch.randn(130, heads * hd, generator=g).to(dt).to(DEV)
    ctx = make_ctx([130], [0], [0], dtype, kernel_plan(dtype))
    whole, odd = torch.empty(130, heads * hdv, dtype=dt, device=DEV), torch.empty(130 * heads * hdv + 4, dtype=dt, device=DEV)
    outs = whole, odd[4 if dtype == "bfloat16" else 1:][:whole.numel()].view_as(whole)
    for out in outs:
        ctx.attention(q, kv, out, heads, 1, hd, AttentionOptions(scale=0.1))
    # two kernels: sums in another order, and in bfloat16 a rounding of the weights and of the result each
    assert float((outs[0].float() - outs[1].float()).abs().max()) <= (2e-5 if dtype == "float32" else 3e-2)
