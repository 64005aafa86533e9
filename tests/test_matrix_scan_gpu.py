"""The matrix-state scans against float64, token by token: sizes that take the kernel with 8 rows and 4 columns a thread (one
to 32 lanes a column, narrow and wide heads, columns that do not fill a block) and sizes that do not, gates, constant decays
and stepped forms, pieces of one token to several chunks, values as columns of wider rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D,Dv", [(8, 4), (16, 12), (32, 64), (64, 36), (128, 8), (256, 68), (24, 20), (32, 30)])
@pytest.mark.parametrize("form", ["gates", "decay", "stepped"])
@pytest.mark.parametrize("lens", [[1, 1, 1], [3, 0, 70, 200]])
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
