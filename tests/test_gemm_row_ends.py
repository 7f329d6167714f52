"""Results of the tcgen05 GEMM whose rows end within 16 bytes, inside wider matrices: what lies beside them stays."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [1, 3])
@pytest.mark.parametrize("m, n, k", [(1, 1, 8), (64, 3, 64), (130, 9, 40), (86, 304, 96), (176, 87, 320), (129, 102, 72),
                                     (200, 150, 192), (346, 4, 33), (64, 130, 64), (300, 1001, 64)])
def test_rows_that_end_within_16_bytes(m: int, n: int, k: int, groups: int) -> None:
    """Against FP64 sums of the BF16 operands, 2e-6 of 4 sqrt(k) as for whole rows; the other columns of a
    matrix 16 wider, and the rows after the transposed result's, hold what they held."""
    from open_analysis_gb300 import native

    lib = native.load()
    up = lambda v: (v + 7) // 8 * 8  # noqa: E731
    lda, ldc, ldct = up(k), up(n) + 16, up(m) + 16
    gen = torch.Generator("cuda").manual_seed(m + n + k)
    randn = lambda *s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    a, b, bias = randn(groups, m, lda).bfloat16(), randn(groups, n, lda).bfloat16(), randn(groups, n)
    c32 = torch.full((groups, m, ldc), 7.0, device="cuda")
    c16 = c32.bfloat16()
    c16t = torch.full((groups, n, ldct), 7.0, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    native.check(lib.oafdtd_mlp_gemm_tn(a.data_ptr(), b.data_ptr(), c32.data_ptr(), c16.data_ptr(), c16t.data_ptr(),
                                        bias.data_ptr(), None, m, n, k, lda, lda, ldc, ldct, 0, 0.0, groups, m * lda,
                                        n * lda, m * ldc, n * ldct, n, status.data_ptr(), None), "gemm")
    torch.cuda.synchronize()
    assert int(status) == 0
    ref = torch.bmm(a[..., :k].double(), b[..., :k].double().transpose(1, 2)) + bias[:, None].double()
    assert (c32[..., :n].double() - ref).abs().max() <= 2e-6 * 4 * k**0.5
    assert torch.equal(c16[..., :n], c32[..., :n].bfloat16())
    assert torch.equal(c16t[..., :m], c16[..., :n].transpose(1, 2))
    for rest in (c32[..., n:], c16[..., n:], c16t[..., m:]):
        assert bool((rest == 7).all())
