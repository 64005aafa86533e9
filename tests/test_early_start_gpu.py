"""Kernels that begin while the product in front of them still runs read that product's rows only behind their wait: the
same launches with and without the early start, bit for bit. One buffer takes the projections of all rounds, so rows that
are read too soon are those of the round before."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROUNDS = 60


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _consumer(kind, rows, n, g, dtype):
    """A function of the projection [rows, n] whose result is new for every call; rows are sequences of one token."""
    from llm_infer_engine_b200.kernels import ops
    rand = lambda *s: torch.randn(*s, generator=g).to(DEV)                                       # noqa: E731
    cu, seq, slot = _i32(list(range(rows + 1))), _i32(list(range(rows))), _i32(list(range(rows)))
    if kind == "conv":
        taps, bias, cb = rand(4, n), rand(n), rand(n)
        held = rand(rows, 3, n)

        def call(proj):
            out = torch.empty(rows, n, device=DEV)
            ops.causal_conv(proj, 0, bias, taps, cb, held.clone(), cu, seq, slot, out, act=ops.ACT_SILU, single=True)
            return out
    elif kind == "conv_prompt":
        taps, bias, cb = rand(4, n), rand(n), rand(n)
        held = rand(1, 3, n)

        def call(proj):
            out = torch.empty(rows, n, device=DEV)
            ops.causal_conv(proj, 0, bias, taps, cb, held, _i32([0, rows]), torch.zeros_like(seq), _i32([0]), out)
            return out
    elif kind in ("conv_qk", "conv_qk_odd"):
        hd = 64 if kind == "conv_qk" else 16 * 3 - 4        # eight channels a lane, or two
        heads = n // hd
        n_kv = 1
        C = heads * hd
        taps, bias, held = rand(4, C), rand(C), rand(rows, 3, C)
        qw, kw, table = rand(hd), rand(hd), rand(64, hd // 4, 2)
        pages = _i32([[i] for i in range(rows)])

        def call(proj):
            q = torch.empty(rows, (heads - n_kv) * hd, dtype=dtype, device=DEV)
            k, v = (torch.zeros(rows, n_kv, 64, hd, dtype=dtype, device=DEV) for _ in range(2))
            ops.conv_qk_store(proj, bias, taps, held.clone(), qw, kw, 1e-5, table, hd // 2 // 2 * 2, cu, torch.zeros_like(seq),
                              seq, slot, pages, 64, q, k, v, heads - n_kv, n_kv, hd, single=True)
            return torch.cat([q.flatten(), k.flatten(), v.flatten()])
    else:
        bias, A = rand(n), rand(n).abs()

        def call(proj):
            dt, decay = torch.empty(rows, n, device=DEV), torch.empty(rows, n, device=DEV)
            ops.ssm_steps(proj, 0, bias, A, dt, decay)
            return torch.cat([dt, decay])
    return call


@pytest.mark.parametrize("product", ["skinny", "float32"])
@pytest.mark.parametrize("kind", ["conv", "conv_prompt", "conv_qk", "conv_qk_odd", "steps"])
@pytest.mark.parametrize("rows,k,n", [(1, 128, 512), (3, 2048, 2816), (8, 96, 448), (40, 128, 640), (17, 1024, 512), (301, 2048, 2816)])
def test_rows_behind_a_product_are_that_products(product, kind, rows, k, n):
    from llm_infer_engine_b200.kernels import ops
    if product == "skinny" and rows > 8:
        pytest.skip("the library's product from 9 rows on")
    g = torch.Generator().manual_seed(rows + n)
    dt = torch.bfloat16 if product == "skinny" else torch.float32
    call = _consumer(kind, rows, n, g, dt)
    w = (torch.randn(n, k, generator=g) / k ** 0.5).to(dt).to(DEV)
    xs = [torch.randn(rows, k, generator=g).to(dt).to(DEV) for _ in range(ROUNDS)]
    proj = torch.empty(rows, n, dtype=dt, device=DEV)

    def rounds():
        got = []
        for x in xs:
            if product == "skinny":
                ops.gemm_skinny(x, w, proj, ops.SKINNY_STORE_BF16)
            else:
                ops.gemm_f32_nt(x, w, out=proj)
            got.append(call(proj))
        torch.cuda.synchronize()
        return torch.stack(got)

    was = ops.PDL
    try:
        ops.set_pdl(False)
        want = rounds()
        ops.set_pdl(True)
        for _ in range(3):
            assert torch.equal(rounds(), want)
    finally:
        ops.set_pdl(was)


@pytest.mark.parametrize("rows,k,n", [(3, 2048, 2816), (16, 1024, 256), (16, 1024, 8192), (17, 1024, 512), (90, 1152, 300), (301, 2048, 2816),
                                      (3, 96, 448)])
def test_a_matrix_that_a_kernel_in_front_writes(rows, k, n):
    """A float32 product reads ahead only what its caller calls a stored weight: here its matrix is scaled by the kernel in front,
    which lets it start early."""
    from llm_infer_engine_b200.kernels import ops
    g = torch.Generator().manual_seed(rows + n)
    w = torch.randn(n, k, generator=g).to(DEV)
    xs = [torch.randn(rows, k, generator=g).to(DEV) for _ in range(ROUNDS)]

    def rounds():
        got = []
        for i, x in enumerate(xs):
            ops.scale_rows(w, 0.5 if i % 2 else 2.0)            # exact, and back where it was after two rounds
            got.append(ops.gemm_f32_nt(x, w))
        torch.cuda.synchronize()
        return torch.stack(got)

    was = ops.PDL
    try:
        ops.set_pdl(False)
        want = rounds()
        ops.set_pdl(True)
        for _ in range(3):
            assert torch.equal(rounds(), want)
    finally:
        ops.set_pdl(was)
