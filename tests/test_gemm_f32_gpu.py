"""The float32 product's kernels against 64-bit sums and against one another: every form that takes a size gives the same
bits, at the edges of tiles, slices and stages, with rows that start on 16 bytes and rows that do not."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
FEW, TILES = (10, 20, 30), (51, 54, 58, 61, 64, 68)


def _form(a, w, form, ld_extra=0):
    from llm_infer_engine_b200.kernels import ops
    f = ops._fn("gemm_simt", "llmie_gemm_f32_nt_form",
                [ctypes.c_void_p] * 3 + [ctypes.c_int] * 7 + [ctypes.c_void_p])
    (M, K), N = a.shape, w.shape[0]
    out = torch.full((M, N + ld_extra), float("nan"), device=DEV)
    status = f(a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), w.stride(0), N + ld_extra, form,
               ops._stream())
    return status, out[:, :N]


@pytest.mark.parametrize("M,N,K", [(1, 2500, 96), (2, 33, 130), (4, 130, 1031), (8, 2369, 128), (9, 100, 1152),
                                   (16, 70, 2052), (17, 129, 4097), (33, 64, 1), (64, 65, 1024), (130, 999, 777),
                                   (301, 640, 2048), (64, 130, 16), (13, 4800, 40), (9, 5000, 160), (70, 200, 33),
                                   (700, 900, 250), (301, 1000, 513), (24, 2100, 384)])
@pytest.mark.parametrize("offset", [0, 1])
def test_every_form_gives_the_same_bits(M, N, K, offset):
    g = torch.Generator().manual_seed(M * 1000 + K)
    lda, ldw = K + (-K) % 4 + 4 * offset + offset, K + (-K) % 4 + offset    # offset 1: rows that do not start on 16 bytes
    a = torch.randn(M, lda, generator=g).to(DEV)[:, :K]
    w = torch.randn(N, ldw, generator=g).to(DEV)[:, :K]
    ref = a.double() @ w.double().T
    status, first = _form(a, w, 61)
    assert status == 0
    # a sum of K products, each chain at most K / 16 long: rounding errors of the chain and of the nine sums behind it
    bound = (K / 16 + 10) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T) + 1e-30
    assert bool(((first.double() - ref).abs() <= bound).all())
    taken = 0
    for form in FEW + TILES + (0,):
        status, out = _form(a, w, form, ld_extra=3)
        if form in FEW and status == -2:
            continue                                          # a form for fewer rows
        assert status == 0, form
        taken += 1
        assert torch.equal(out, first), form
    assert taken >= len(TILES) + 1 + (2 if M in (1, 2, 4, 8) else 1 if M <= 16 else 0)
    status, some = _form(a[M // 2:M // 2 + 1], w, 0)          # a row alone
    assert status == 0 and torch.equal(some[0], first[M // 2])


def test_zeros_infinities_and_nothing():
    a, w = torch.zeros(3, 200, device=DEV), torch.randn(40, 200, device=DEV)
    assert torch.equal(_form(a, w, 0)[1], torch.zeros(3, 40, device=DEV))
    a = torch.ones(20, 200, device=DEV)
    w[7, 199] = float("inf")
    for rows in (3, 20):
        out = _form(a[:rows], w, 0)[1]
        assert bool(torch.isinf(out[:, 7]).all()) and int(torch.isfinite(out).sum()) == rows * 39
    assert _form(a[:0], w, 0)[0] == 0
