"""The tcgen05 GEMM off its tile sizes: ragged M, N and K, one row, layer inputs 8 wide, several
groups, transposed results whose rows TMA cannot address. Against FP64 sums of the BF16 operands, and
bit for bit against the mma.sync kernel, which takes the same K steps of 16 in the same order."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SHAPES = [  # groups, M, N, K
    (1, 412, 512, 8), (3, 412, 512, 512), (2, 64, 512, 512), (2, 512, 512, 64), (2, 1, 8, 8), (1, 130, 72, 136),
    (2, 200, 1024, 256), (1, 129, 520, 72), (4, 40, 40, 40), (20, 127, 264, 88),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("act", [0, 1, 2, 3, 4])
def test_ragged_gemm_tn(shape: tuple[int, int, int, int], act: int) -> None:
    from open_analysis_gb300 import native

    lib = native.load()
    g, m, n, k = shape
    gen = torch.Generator(device="cuda")
    gen.manual_seed(act + m + n + k)

    def randn(*s: int):  # type: ignore[no-untyped-def]
        return torch.randn(s, generator=gen, device="cuda")

    a, b, bias = randn(g, m, k).bfloat16(), randn(g, n, k).bfloat16(), randn(g, n)
    mask = randn(g, m, n).bfloat16()
    pad = 64  # elements between the groups' results, which stay as they are
    c32 = torch.full((g, m * n + pad), 7.0, device="cuda")
    c16 = torch.full((g, m * n + pad), 7.0, device="cuda").bfloat16()
    c16t = torch.full((g, m * n + pad), 7.0, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    one = torch.full((m, n), 7.0, device="cuda")
    # the mask moves with C: its groups lie as far apart
    masks = torch.zeros((g, m * n + pad), device="cuda").bfloat16()
    masks[:, : m * n] = mask.reshape(g, -1)
    need = act in (2, 4)
    assert lib.oafdtd_mlp_gemm_tn(a.data_ptr(), b.data_ptr(), c32.data_ptr(), c16.data_ptr(), c16t.data_ptr(),
                                  bias.data_ptr(), masks.data_ptr() if need else None, m, n, k, k, k, n, m, act, 0.0,
                                  g, m * k, n * k, m * n + pad, m * n + pad, n, status.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(status) == 0
    mk = mask.double()
    ref = torch.bmm(a.double(), b.double().transpose(1, 2)) + bias[:, None].double()
    ref = {0: ref, 1: ref.clamp(min=0), 2: torch.where(mk > 0, ref, 0 * ref), 3: torch.tanh(ref),
           4: ref * (1 - mk * mk)}[act]
    scale = 4 * k**0.5 * (1.0 if act != 4 else float((mk * mk).max()) + 1.0)
    got = c32[:, : m * n].reshape(g, m, n)
    assert (got.double() - ref).abs().max() <= 2e-6 * scale
    assert torch.equal(c16[:, : m * n].reshape(g, m, n), got.bfloat16())
    assert torch.equal(c16t[:, : m * n].reshape(g, n, m), got.bfloat16().transpose(1, 2))
    for c in (c32, c16, c16t):
        assert bool((c[:, m * n :] == 7).all())
    for gi in range(g):
        assert lib.oafdtd_mlp_gemm(a[gi].data_ptr(), b[gi].data_ptr(), one.data_ptr(), None, bias[gi].data_ptr(),
                                   mask[gi].data_ptr() if need else None, m, n, k, k, k, n, 0, 1, act, 0.0, None) == 0
        torch.cuda.synchronize()
        assert torch.equal(one, got[gi]), gi
