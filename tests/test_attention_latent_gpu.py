"""Prompts of latent attention on the tensor cores against float64 attention: head counts that do and do not divide a tile
of 128 rows, the edges of pages and tiles, pieces behind held tokens, windows, chunks and sinks, scores that grow along
the sequence so that a row's reference maximum has to move, and the sizes at the ends of what the kernel takes."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(lens, held, heads, hd, hdv, seed=0, growth=0.0):
    g = torch.Generator().manual_seed(seed)
    n = len(lens)
    need = [(h + l + 63) // 64 for h, l in zip(held, lens)]
    order = torch.randperm(sum(need) + 2, generator=g).tolist()          # scrambled pages
    table = torch.full((n + 1, max(need)), sum(need) + 2, dtype=torch.int32)
    cache = torch.randn(sum(need) + 3, 1, 64, hd, generator=g) * 3       # what is not written over belongs to nobody
    q = torch.randn(sum(lens), heads * hd, generator=g).to(torch.bfloat16)
    rows, at = [], 0
    for i in range(n):
        k = torch.randn(held[i] + lens[i], hd, generator=g)
        k = (k * (1 + growth * torch.arange(len(k))[:, None])).to(torch.bfloat16)
        rows.append(k)
        for j in range(need[i]):
            page, part = order[at], k[64 * j:64 * j + 64]
            table[i, j], at = page, at + 1
            cache[page, 0, :len(part)] = part.float()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)              # noqa: E731
    cu = [0]
    for l in lens:
        cu.append(cu[-1] + l)
    return q.to(DEV), cache.to(torch.bfloat16).to(DEV), rows, i32(cu), i32(list(range(n))), i32(held), table.to(DEV)


def _reference(q, rows, lens, held, heads, hd, hdv, scale, window, sink):
    out, at = [], 0
    for k, l, h in zip(rows, lens, held):
        k = k.double().to(DEV)
        x = q[at:at + l].double().view(l, heads, hd)
        at += l
        s = torch.einsum("thd,kd->htk", x, k) * scale
        pos, key = torch.arange(h, h + l, device=DEV)[:, None], torch.arange(h + l, device=DEV)[None, :]
        seen = key <= pos
        if window > 0:
            seen &= key > pos - window
        if window < 0:
            seen &= key >= pos - pos % -window
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.double().view(heads, 1, 1).expand(heads, l, 1)], dim=2)
        p = s.softmax(-1)[..., :h + l]
        out.append(torch.einsum("htk,kd->thd", p, k[:, :hdv]).reshape(l, heads * hdv))
    return torch.cat(out)


@pytest.mark.parametrize("heads,hd,hdv", [(32, 288, 256), (3, 80, 64), (1, 320, 256), (5, 144, 128), (128, 64, 64),
                                          (40, 208, 192)])
@pytest.mark.parametrize("window,sink", [(0, False), (70, True), (-96, False)])
@pytest.mark.parametrize("growth", [0.0, 0.02])
def test_prompts(heads, hd, hdv, window, sink, growth):
    from llm_infer_engine_b200.kernels import ops
    lens, held = [65, 1, 200, 128, 9], [0, 63, 130, 64, 700]
    q, cache, rows, cu, slot, start, table = _case(lens, held, heads, hd, hdv, growth=growth)
    values = cache[..., :hdv]
    scale = 1.7 * hd ** -0.5
    sinks = torch.linspace(-2, 5, heads, device=DEV) if sink else None
    assert ops.attention_latent_tc_supported(q, cache, values, 64, heads, 1, hd, max(lens), scale)
    out = torch.full((sum(lens), heads * hdv), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.attention_latent_tc(q, cache, values, out, cu, slot, start, table, 64, len(lens), max(lens), heads, hd, scale,
                            window, sinks)
    ops.check_tc_status(torch.device(DEV, 0))
    want = _reference(q, rows, lens, held, heads, hd, hdv, scale, window, sinks)
    # probabilities and the result are rounded to bfloat16 (2^-9 each, relative), sums are float32
    bound = 2.0 ** -7 * torch.cat([r.abs().max().expand(l) for r, l in zip(rows, lens)])[:, None].double().to(DEV)
    diff = (out.double() - want).abs()
    assert bool((diff <= bound).all()), (float((diff / bound).max()), int((diff > bound).sum()))
    # a sequence alone: the same bits
    one = torch.empty(200, heads * hdv, dtype=torch.bfloat16, device=DEV)
    a = 66 * 1
    ops.attention_latent_tc(q[a:a + 200].contiguous(), cache, values, one, torch.tensor([0, 200], dtype=torch.int32, device=DEV),
                            slot[2:3].contiguous(), start[2:3].contiguous(), table, 64, 1, 200, heads, hd, scale, window, sinks)
    assert torch.equal(one, out[a:a + 200])


@pytest.mark.parametrize("heads,hd,hdv", [(32, 288, 256), (3, 80, 64), (1, 144, 128)])
@pytest.mark.parametrize("window", [0, 70, -96])
@pytest.mark.parametrize("value", [math.nan, math.inf, -math.inf])
def test_values_that_are_not_finite_stay_with_the_rows_that_see_them(heads, hd, hdv, window, value):
    """A key that went wrong, at places where a page's first tokens do not see it yet or its last no longer do, in a first and
    in a later page; and whatever the last page holds behind the sequence, and pages of nobody."""
    from llm_infer_engine_b200.kernels import ops
    lens, held = [65, 1, 200, 9], [0, 63, 130, 700]
    wrong = [20, None, 200, 650]
    q, cache, rows, cu, slot, start, table = _case(lens, held, heads, hd, hdv, seed=7)
    used = torch.zeros(cache.shape[0], 64, dtype=torch.bool)
    for i, k in enumerate(rows):
        for t in range(len(k)):
            used[table[i, t // 64], t % 64] = True
    cache[~used[:, None].to(DEV)] = value
    for i, t in enumerate(wrong):
        if t is not None:
            cache[table[i, t // 64], 0, t % 64, ::5] = value
    values, scale = cache[..., :hdv], 1.7 * hd ** -0.5
    out = torch.full((sum(lens), heads * hdv), 3.0, dtype=torch.bfloat16, device=DEV)
    ops.attention_latent_tc(q, cache, values, out, cu, slot, start, table, 64, len(lens), max(lens), heads, hd, scale, window)
    ops.check_tc_status(torch.device(DEV, 0))
    want = _reference(q, rows, lens, held, heads, hd, hdv, scale, window, None)
    at = 0
    for i, (l, h) in enumerate(zip(lens, held)):
        pos = torch.arange(h, h + l)
        sees = torch.zeros(l, dtype=torch.bool)
        if wrong[i] is not None:
            sees = pos >= wrong[i]
            if window > 0:
                sees &= wrong[i] > pos - window
            if window < 0:
                sees &= wrong[i] >= pos - pos % -window
        sees, got, ref = sees.to(DEV), out[at:at + l].double(), want[at:at + l]
        at += l
        bound = 2.0 ** -7 * rows[i].abs().max().double().to(DEV)             # as in test_prompts
        diff = (got - ref)[~sees].abs()
        assert bool((diff <= bound).all()), (i, float(diff.max()), int((~(diff <= bound)).any(1).sum()))
        if value != value and bool(sees.any()):
            assert bool(got[sees].isnan().all())


def test_a_block_that_gives_up_leaves_no_numbers():
    """A wait that runs out (no polls at all here): NaN in every row and an error for whoever asks, not what was there."""
    from llm_infer_engine_b200.kernels import ops
    lens, held, heads, hd, hdv = [130, 40], [0, 300], 5, 144, 128
    q, cache, rows, cu, slot, start, table = _case(lens, held, heads, hd, hdv)
    out = torch.full((sum(lens), heads * hdv), 3.0, dtype=torch.bfloat16, device=DEV)
    status = ops.tc_status_word(torch.device(DEV, 0))
    p = [t.data_ptr() for t in (q, cache, out, cu, slot, start, table)]
    f = ops._fn("attention_latent_tc", "llmie_attention_latent_tc_form",
                [ops._c_void_p] * 7 + [ops._c_int] * 8 + [ops._c_float, ops._c_int, ops._c_void_p, ops._c_int, ops._c_void_p,
                                                          ops._c_int, ops._c_void_p])
    assert f(*p, table.shape[1], cache.shape[0], sum(lens), 2, 130, heads, hd, hdv, 0.1, 0, None, 0, status.data_ptr(), 1,
             ops._stream()) == 0
    torch.cuda.synchronize()
    assert bool(out.isnan().all())
    with pytest.raises(ops.KernelError):
        ops.check_tc_status(torch.device(DEV, 0))
    ops.check_tc_status(torch.device(DEV, 0))                            # raised once
    ops.attention_latent_tc(q, cache, cache[..., :hdv], out, cu, slot, start, table, 64, 2, 130, heads, hd, 0.1)
    assert bool(out.isfinite().all())


@pytest.mark.parametrize("heads,hd,hdv", [(32, 288, 256), (2, 80, 64)])
@pytest.mark.parametrize("gated", [False, True])
def test_a_piece_gets_the_same_bits_beside_others(heads, hd, hdv, gated):
    """Pieces of one to five tokens, alone (a step of one token, a short prompt) and beside a long one, as a layer calls it."""
    import types
    from llm_infer_engine_b200.parts.base import AttentionOptions
    from test_parts_gpu import kernel_plan, make_ctx
    lens, held = [1, 2, 5, 300], [90, 0, 700, 20]
    q, cache, rows, cu, slot, start, table = _case(lens, held, heads, hd, hdv, seed=11)
    kv = types.SimpleNamespace(k=cache, v=cache[..., :hdv], page_size=64, block_table=table)
    gate = torch.randn(sum(lens), heads * hdv, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    plan, options = kernel_plan("bfloat16"), AttentionOptions(scale=hd ** -0.5)

    def run(which):
        at = torch.cat([torch.arange(sum(lens[:i]), sum(lens[:i + 1])) for i in which]).to(DEV)
        out = torch.empty(len(at), heads * hdv, dtype=torch.bfloat16, device=DEV)
        ctx = make_ctx([lens[i] for i in which], [held[i] for i in which], which, "bfloat16")
        assert plan.attention(ctx, q[at].contiguous(), kv, out, heads, 1, hd, options, gate[at].contiguous() if gated else None)
        return list(out.split([lens[i] for i in which]))

    whole = run([0, 1, 2, 3])
    for which in ([0], [1], [2], [0, 1], [1, 2]):
        assert all(torch.equal(a, whole[i]) for i, a in zip(which, run(which))), which


def test_both_kernels_agree():
    """The kernel of 32 rows takes the same calls (and all that this one refuses)."""
    from llm_infer_engine_b200.kernels import ops
    heads, hd, hdv, lens, held = 32, 288, 256, [130, 300], [0, 77]
    q, cache, rows, cu, slot, start, table = _case(lens, held, heads, hd, hdv, seed=5)
    values, outs = cache[..., :hdv], []
    for f in (lambda o: ops.attention_latent_tc(q, cache, values, o, cu, slot, start, table, 64, 2, 300, heads, hd, 0.06),
              lambda o: ops.attention_rows_mma(q, cache, values, o, cu, slot, start, table, 64, 2, 300, heads, 1, hd, 0.06)):
        outs.append(torch.empty(sum(lens), heads * hdv, dtype=torch.bfloat16, device=DEV))
        f(outs[-1])
    want = _reference(q, rows, lens, held, heads, hd, hdv, 0.06, 0, None)
    errors = [float((o.double() - want).norm() / want.norm()) for o in outs]
    assert errors[0] <= 1.2 * errors[1] and errors[1] < 5e-3, errors


def test_what_it_refuses():
    from llm_infer_engine_b200.kernels import ops
    q, cache, *_ = _case([130], [0], 4, 96, 64)
    ok = lambda **kw: ops.attention_latent_tc_supported(**{**dict(q=q, k_cache=cache, v_cache=cache[..., :64], page_size=64,  # noqa: E731
                                                                  n_q=4, n_kv=1, head_dim=96, max_q_len=130, scale=1.0), **kw})
    assert ok()
    assert not ok(v_cache=cache[..., :48]) and not ok(v_cache=cache[..., 32:])
    assert ok(max_q_len=1) and not ok(max_q_len=1 << 30)
    assert not ok(scale=0.0) and not ok(page_size=32) and not ok(n_kv=2) and not ok(q=q.float())
