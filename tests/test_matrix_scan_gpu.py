"""The matrix-state scans against float64, token by token: sizes that take the kernel with 8 rows and 4 columns a thread (one
to 32 lanes a column, narrow and wide heads, columns that do not fill a block) and sizes that do not, gates, constant decays
and stepped forms, pieces of one token to several chunks, values as columns of wider rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D,Dv", [(8, 4), (16, 12), (32, 64), (64, 36), (128, 8), (256, 68), (24, 20), (32, 30)])
@pytest.mark.parametrize("form", ["gates", "decay", "stepped"])
@pytest.mark.parametrize("lens", [[1, 1, 1], [5, 1, 40], [3, 0, 70, 200]])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_scan(D, Dv, form, lens, dtype):
    from llm_infer_engine_b200.kernels import ops
    H, G = 4, 2 if form == "stepped" else 4
    g = torch.Generator().manual_seed(D + Dv + len(lens))
    T, n = sum(lens), len(lens)
    q = torch.randn(T, G * D, generator=g).to(DEV)
    f = (torch.rand(T, G * D, generator=g) if form == "gates" else torch.randn(T, G * D, generator=g) * 0.3).to(DEV)
    wide = torch.randn(T, H * Dv + 8, generator=g).to(dtype).to(DEV)
    v = wide[:, 8:]
    decay = (torch.rand(H, generator=g) if form == "decay" else torch.rand(T, H, generator=g)).to(DEV) if form != "gates" else None
    factor = torch.rand(T, H, generator=g).to(DEV) if form == "stepped" else None
    slots = torch.randperm(n + 2, generator=g)[:n].to(torch.int32).to(DEV)
    state = torch.randn(n + 2, H, D, Dv, generator=g).to(DEV)
    cu = [0]
    for l in lens:
        cu.append(cu[-1] + l)

    def run(state, q, f, v, cu, slots, decay, factor):
        out = torch.full((q.shape[0], H * Dv), float("nan"), device=DEV)
        ops.matrix_scan(q, f, v, state, torch.tensor(cu, dtype=torch.int32, device=DEV), slots, out, len(cu) - 1, H, D, Dv,
                        max_len=max(b - a for a, b in zip(cu, cu[1:])), head_decay=decay, key_factor=factor,
                        groups=G if form == "stepped" else None)
        return out

    got_state = state.clone()
    out = run(got_state, q, f, v, cu, slots, decay, factor)
    want_state, mag_state = state.double().clone(), state.double().abs()
    k64 = f.double().view(T, G, D).repeat_interleave(H // G, 1)
    q64 = q.double().view(T, G, D).repeat_interleave(H // G, 1)
    v64 = v.double().reshape(T, H, Dv)
    for i in range(n):
        S, M = want_state[int(slots[i])], mag_state[int(slots[i])]
        for t in range(cu[i], cu[i + 1]):
            gate = k64[t][..., None] if form == "gates" else (decay if form == "decay" else decay[t]).double()[:, None, None]
            write = 1 - k64[t] if form == "gates" else k64[t] * (factor[t].double()[:, None] if form == "stepped" else 1)
            S, add = gate * S, write[..., None] * v64[t][:, None, :]
            S, M = S + add, gate.abs() * M + add.abs()
            o = torch.einsum("hd,hdv->hv", q64[t], S).reshape(-1)
            # each of a state's terms carries the roundings of the steps behind it; a read-out adds D products more
            bound = (l_ + D + 8) * 2.0 ** -24 * torch.einsum("hd,hdv->hv", q64[t].abs(), M).reshape(-1) if (l_ := t - cu[i] + 4) else None
            assert bool(((out[t].double() - o).abs() <= bound + 1e-6).all()), (i, t)
        want_state[int(slots[i])], mag_state[int(slots[i])] = S, M
    assert bool(((got_state.double() - want_state).abs() <= 300 * 2.0 ** -24 * mag_state + 1e-6).all())
    i = max(range(n), key=lambda k: lens[k])                 # the longest piece alone: the same bits
    a, b = cu[i], cu[i + 1]
    alone = state.clone()
    one = run(alone, q[a:b].contiguous(), f[a:b].contiguous(), v[a:b], [0, b - a], slots[i:i + 1].contiguous(),
              decay if form != "stepped" else decay[a:b].contiguous(), factor[a:b].contiguous() if form == "stepped" else None)
    assert torch.equal(one, out[a:b]) and torch.equal(alone[int(slots[i])], got_state[int(slots[i])])


@pytest.mark.parametrize("H,D,Dv,n", [(4, 8, 4, 3), (2, 16, 16, 2), (16, 64, 32, 5), (32, 32, 64, 60), (32, 64, 128, 3), (32, 64, 128, 40),
                                      (2, 128, 64, 2)])
@pytest.mark.parametrize("form", ["gates", "decay", "stepped"])
def test_both_kernels_give_the_same_bits(H, D, Dv, n, form):
    """One-token steps go to either kernel by their size and pieces beside a long one to the chunked one: the same bits, values
    that do not start on 16 bytes (never the kernel with 16-byte loads) included."""
    from llm_infer_engine_b200.kernels import ops
    g = torch.Generator().manual_seed(D + Dv)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                              # noqa: E731
    T = n + 90                                                     # the last piece is long where it is there
    q, f = torch.randn(T, H * D, generator=g).to(DEV), torch.rand(T, H * D, generator=g).to(DEV)
    wide = torch.randn(T, H * Dv + 9, generator=g).to(torch.bfloat16).to(DEV)
    odd, even = wide[:, 9:], torch.cat([wide[:, 9:]], 1).contiguous()
    decay = None if form == "gates" else (torch.rand(H, generator=g) if form == "decay" else torch.rand(T, H, generator=g)).to(DEV)
    factor = torch.rand(T, H, generator=g).to(DEV) if form == "stepped" else None
    first = torch.randn(n + 1, H, D, Dv, generator=g).to(DEV)

    def run(v, lens):
        t, state = sum(lens), first.clone()
        cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
        out = torch.empty(t, H * Dv, device=DEV)
        ops.matrix_scan(q[:t], f[:t], v[:t], state, i32(cu), i32(list(range(len(lens)))), out, len(lens), H, D, Dv,
                        max_len=max(lens), head_decay=decay if form != "stepped" else decay[:t],
                        key_factor=factor[:t] if form == "stepped" else None)
        return out[:n], state[:n]

    a, b, c = run(even, [1] * n), run(odd, [1] * n), run(even, [1] * n + [90])
    assert all(torch.equal(a[k], b[k]) and torch.equal(a[k], c[k]) for k in (0, 1))
