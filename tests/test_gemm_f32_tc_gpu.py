"""The float32 product on the tensor cores against 64-bit sums and against itself: every form gives the same bits, at the edges
of tiles, slices and chains, with rows that start on 32 bytes and rows that do not; infinities and overflow."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
FORMS = (1008, 1016, 2016, 4016, 1064, 2064, 4064, 1080, 2080, 4080, 0)


def _form(a, w, form, ld_extra=0):
    from llm_infer_engine_b200.kernels import ops
    f = ops._fn("gemm_f32_tc", "llmie_gemm_f32_tc_form", [ctypes.c_void_p] * 4 + [ctypes.c_int] * 7 + [ctypes.c_void_p] * 2)
    (M, K), N = a.shape, w.shape[0]
    out = torch.full((M, N + ld_extra), float("nan"), device=DEV)
    parts = torch.empty(3 * M * K, dtype=torch.bfloat16, device=DEV)
    status = f(a.data_ptr(), w.data_ptr(), out.data_ptr(), parts.data_ptr(), M, N, K, a.stride(0), w.stride(0), N + ld_extra,
               form, ops.tc_status_word(torch.device(DEV, 0)).data_ptr(), ops._stream())
    return status, out[:, :N]


@pytest.mark.parametrize("M,N,K", [(1, 128, 1024), (3, 2369, 1152), (8, 300, 2048), (9, 129, 1408), (16, 640, 3072), (17, 200, 1024),
                                   (64, 257, 1280), (65, 1000, 1024), (80, 384, 8192), (81, 130, 1536), (301, 640, 2048)])
@pytest.mark.parametrize("offset", [0, 1])
def test_every_form_gives_the_same_bits(M, N, K, offset):
    from llm_infer_engine_b200.kernels import ops
    g = torch.Generator().manual_seed(M * 1000 + K)
    a = (torch.randn(M, K + 8 + offset, generator=g) * torch.exp(torch.randn(M, 1, generator=g))).to(DEV)[:, :K]
    w = torch.randn(N, K + 8 + offset, generator=g).to(DEV)[:, :K]       # offset 1: rows that do not start on 16 bytes
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    status, first = _form(a, w, 1064)
    assert status == 0
    # 17 terms a product and 8 products a slice, each cut off at 2^-24 of the largest; the parts left out; the sums behind
    bound = (17 * 8 + 6 + K / 512 + 4) * 2.0 ** -24 * size
    assert bool(((first.double() - ref).abs() <= bound).all())
    # what is seen, beside sums in one float32 chain each
    assert float((first.double() - ref).norm() / ref.norm()) < 2e-7
    for form in FORMS:
        status, out = _form(a, w, form, ld_extra=3)
        if form == 1008 and M > 16:
            assert status == -2
            continue
        assert status == 0, form
        assert torch.equal(out, first), form
    status, some = _form(a[M // 2:M // 2 + 1], w, 0)          # a row alone
    assert status == 0 and torch.equal(some[0], first[M // 2])
    if offset:
        assert torch.equal(ops.gemm_f32_nt(a.contiguous(), w.contiguous()), first)
    ops.check_tc_status(torch.device(DEV, 0))


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(128, 1024), (1185, 1152), (300, 2048), (2369, 1408), (129, 2176), (640, 8192), (300, 14336), (130, 20480)])
@pytest.mark.parametrize("offset", [0, 1])
def test_two_items_at_a_time(M, N, K, offset):
    """The form for up to four rows, with an odd number of slices too: the bits of the others, and what is not finite where it belongs."""
    g = torch.Generator().manual_seed(M * 1000 + K)
    a = torch.randn(M, K + offset, generator=g).to(DEV)[:, :K]
    w = torch.randn(N, K + offset, generator=g).to(DEV)[:, :K]
    status, want = _form(a, w, 1016)
    for form in (1004, 1008, 0):
        status, out = _form(a, w, form, ld_extra=3)
        assert status == 0 and torch.equal(out, want), form
    assert _form(torch.cat([a] * 5), w, 1004)[0] == -2
    a[M - 1, K - 1], w[N - 1, 0] = float("inf"), float("nan")
    ref, out = a.double() @ w.double().T, _form(a, w, 1004)[1].double()
    fine = torch.isfinite(ref)
    assert torch.equal(torch.isnan(out), torch.isnan(ref)) and torch.equal(out[~fine & ~torch.isnan(ref)], ref[~fine & ~torch.isnan(ref)])
    assert torch.equal(out[fine], want.double()[fine])


def test_infinities_nan_overflow_and_nothing():
    torch.manual_seed(5)
    a, w = torch.randn(40, 1152, device=DEV), torch.randn(200, 1152, device=DEV)
    w[7, 1151], w[130, 5] = float("inf"), float("nan")
    a[3, 600] = float("-inf")
    a[5, 0] = 3e38                                            # times 100: a product that float32 does not hold
    w[:, 0] = w[:, 0].clamp(-1, 1)
    w[9, 0] = 100.0                                           # and the only one (beside an infinity it would make NaN, in float32)
    want = a.double() @ w.double().T
    for rows in (6, 14, 40):
        for form in FORMS[(0 if rows <= 16 else 1):]:
            out = _form(a[:rows], w, form)[1]
            nan = torch.isnan(want[:rows])
            assert torch.equal(torch.isnan(out), nan), form
            huge = want[:rows].abs() > 3.4e38
            assert torch.equal(torch.isinf(out), huge & ~nan) and bool((out[huge & ~nan].sign() == want[:rows][huge & ~nan].sign()).all())
            fine = ~nan & ~huge
            assert bool(((out.double() - want[:rows])[fine].abs() <= 1e-5 * (want[:rows][fine].abs() + 1e3)).all())
    assert _form(a[:0], w, 0)[0] == 0


def test_what_it_takes():
    from llm_infer_engine_b200.kernels import build, ops
    takes = build.load("gemm_f32_tc").llmie_gemm_f32_tc_takes
    for n in (1, 127, 128, 5000):
        for k in (128, 896, 1024, 1025, 1152, 8192):
            assert bool(takes(n, k)) == ops.gemm_f32_tc_takes(n, k)
    a, w = torch.randn(3, 1024, device=DEV), torch.randn(100, 1024, device=DEV)
    assert _form(a, w, 0)[0] == -2                            # fewer rows than a tile


@pytest.mark.parametrize("form", [1016, 4016, 1064, 1080, 2080, 4080])
def test_waits_that_run_out(form):
    """No polls at all: an error for whoever asks, plain sums in place of those that did not come, and the next call is none the worse."""
    from llm_infer_engine_b200.kernels import ops
    M, N, K = 16 if form % 1000 == 16 else 90, 300, 1152
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    status, out = _form(a, w, 10000 + form)
    torch.cuda.synchronize()
    assert status == 0 and bool(((out.double() - ref).abs() <= K * 2.0 ** -24 * size).all())
    with pytest.raises(ops.KernelError):
        ops.check_tc_status(torch.device(DEV, 0))
    status, out = _form(a, w, form)
    assert status == 0 and torch.equal(out, ops.gemm_f32_nt(a, w))
    ops.check_tc_status(torch.device(DEV, 0))


@pytest.mark.parametrize("K", [1024, 1152, 2048, 8192])
@pytest.mark.parametrize("kind", ["normal", "positive", "uniform", "common", "constant", "rising", "falling", "spread"])
def test_error_beside_fma_sums(K, kind):
    """Relative error against 64-bit sums beside that of the FMA kernel for the same numbers, of random and of one sign. The accumulator
    of the tensor cores cuts off towards zero, which for sums of one sign adds up (1.4e-7 to 1.7e-7, all of it bias, where every
    slice starts from zero; FMA 0.5e-7 to 1.3e-7)."""
    from llm_infer_engine_b200.kernels import ops
    f = ops._fn("gemm_simt", "llmie_gemm_f32_nt", [ctypes.c_void_p] * 3 + [ctypes.c_int] * 6 + [ctypes.c_void_p])
    M, N = 64, 512
    g = torch.Generator().manual_seed(K)

    def data(rows):
        x = torch.randn(rows, K, generator=g)
        along = torch.linspace(0, 1, K)
        return {"normal": x, "positive": x.abs(), "uniform": torch.rand(rows, K, generator=g), "common": 1 + 0.01 * x,
                "constant": (0.5 + torch.rand(rows, 1, generator=g)).expand(rows, K).contiguous(), "spread": x.exp(),
                "rising": torch.rand(rows, K, generator=g) * along, "falling": torch.rand(rows, K, generator=g) * (1 - along)}[kind].to(DEV)

    a, w = data(M), data(N)
    ref, fma = a.double() @ w.double().T, torch.empty(M, N, device=DEV)
    assert f(a.data_ptr(), w.data_ptr(), fma.data_ptr(), M, N, K, K, K, N, ops._stream()) == 0
    out = ops.gemm_f32_nt(a, w)
    error = lambda o: float((o.double() - ref).norm() / ref.norm())                                  # noqa: E731
    # measured: 0.03 to 0.95 of the FMA kernel's, rising numbers with a K of 1,024 or 1,152 1.05 and 1.07
    assert error(out) <= 1.15 * error(fma)
    if kind != "normal":
        assert abs(float(((out.double() - ref) / ref).mean())) <= 0.5e-7      # half a unit of float32 is 0.6e-7; measured 0.37e-7
    assert torch.equal(ops.gemm_f32_nt(a[:5].contiguous(), w), out[:5])


@pytest.mark.parametrize("M", [3, 301])
@pytest.mark.parametrize("what", ["nan", "inf"])
def test_rows_that_are_not_finite_are_not_slow(M, what):
    """One such row, and all of them: a thread a sum took 30 and 430 times as long as the finite product; now at most 6 and 40 times."""
    N, K = 4096, 2048
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)

    def seconds():
        _form(a, w, 0)
        times = []
        for _ in range(5):
            first, last = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            first.record()
            for _ in range(4):
                _form(a, w, 0)
            last.record()
            torch.cuda.synchronize()
            times.append(first.elapsed_time(last))
        return min(times)

    fine = seconds()
    a[0, 5] = float(what)
    one = seconds()
    a[:, 7] = float(what)
    assert one < 12 * fine and seconds() < 80 * fine


@pytest.mark.parametrize("M", [1, 17, 161, 400, 1000])
def test_scratch_is_bounded(M, monkeypatch):
    """More rows than the scratch for their parts holds: several launches, the same bits."""
    from llm_infer_engine_b200.kernels import ops
    K, N = 1152, 300
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    want = ops.gemm_f32_nt(a, w)
    monkeypatch.setattr(ops, "F32_PARTS_BYTES", 6 * K * 170)
    used = []
    empty = torch.empty
    monkeypatch.setattr(ops.torch, "empty", lambda *s, **kw: (used.append(s[0]) if kw.get("dtype") == torch.bfloat16 else None) or empty(*s, **kw))
    got = ops.gemm_f32_nt(a, w)
    monkeypatch.undo()
    assert all(n * 2 <= 6 * K * 170 for n in used) and len(used) == (M > 16)
    assert torch.equal(got, want)


def test_first_call_under_capture(monkeypatch):
    """A call that a graph captures first leaves nothing behind that is read before a replay has set it."""
    from llm_infer_engine_b200.kernels import ops
    a, w = torch.randn(40, 1024, device=DEV), torch.randn(256, 1024, device=DEV)
    want = ops.gemm_f32_nt(a, w)
    monkeypatch.setattr(ops, "_tc_status", {})
    out = torch.zeros_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.gemm_f32_nt(a, w, out)
    captured = [t for t in ops._tc_status.values()]
    word = ops.tc_status_word(torch.device(DEV, 0))
    assert len(captured) == 1 and all(word is not t for t in captured) and int(word) == 0
    graph.replay()
    ops.check_tc_status(torch.device(DEV, 0))
    assert torch.equal(out, want)


@pytest.mark.parametrize("scale", [0, -100, -108])
def test_small_numbers_keep_their_bits(scale):
    """The third part of a number is there down to 2^-110 (the numbers here reach some binary orders below their scale), on either side."""
    from llm_infer_engine_b200.kernels import ops
    g = torch.Generator().manual_seed(3)
    a, w = torch.randn(64, 2048, generator=g).to(DEV), torch.randn(256, 2048, generator=g).to(DEV)
    for x, y in ((a * 2.0 ** scale, w * 2.0 ** 60), (a * 2.0 ** 60, w * 2.0 ** scale)):
        ref, out = x.double() @ y.double().T, ops.gemm_f32_nt(x, y)
        assert float((out.double() - ref).norm() / ref.norm()) < 2e-7        # measured 1.2e-7; 2.2e-6 at 2^-116
        assert torch.equal(ops.gemm_f32_nt(x[:5].contiguous(), y), out[:5])
