"""The kernels that a training step takes in one pass each, against the separate ones they stand for."""

import ctypes as C

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _lib():
    from open_analysis_gb300 import native

    return native, native.load()


@pytest.mark.parametrize("sizes,members", [([8, 8], 1), ([24, 72, 8], 3), ([64, 128, 64], 2), ([8, 1032, 200], 1)])
def test_adam_of_a_whole_net_matches_adam_and_a_transpose(sizes, members):
    # tiles of 64 x 64: whole ones, ragged ones (72, 200), single 8-wide ones; > 256 biases (1032)
    native, lib = _lib()
    layers, off = [], 0
    for a, b in zip(sizes, sizes[1:]):
        layers.append((off, a, b, off + a * b))
        off += a * b + b
    gen = torch.Generator("cuda").manual_seed(1)
    r = lambda: torch.randn(members * off, generator=gen, device="cuda")  # noqa: E731
    w, grad, m1, m2 = r(), r(), r(), r().abs()
    lr = torch.full((1,), 1e-3, device="cuda")
    step = torch.full((1,), 3, dtype=torch.int32, device="cuda")
    w16 = torch.zeros(members * off, dtype=torch.bfloat16, device="cuda")
    ref = [t.clone() for t in (w, w16, m1, m2)]
    w16t = torch.zeros_like(w16)
    s = int(torch.cuda.current_stream().cuda_stream)
    native.check(lib.oafdtd_mlp_adam(ref[0].data_ptr(), ref[1].data_ptr(), grad.data_ptr(), ref[2].data_ptr(),
                                     ref[3].data_ptr(), members * off, lr.data_ptr(), 0.9, 0.999, 1e-8,
                                     step.data_ptr(), s), "adam")
    table = (C.c_int64 * (4 * len(layers)))(*[v for q in layers for v in q])
    native.check(lib.oafdtd_mlp_adam_net(w.data_ptr(), w16.data_ptr(), w16t.data_ptr(), grad.data_ptr(),
                                         m1.data_ptr(), m2.data_ptr(), len(layers), table, members, off,
                                         lr.data_ptr(), 0.9, 0.999, 1e-8, step.data_ptr(), s), "adam_net")
    for have, want in zip((w, w16, m1, m2), ref):
        assert torch.equal(have, want)
    for k in range(members):
        for wo, a, b, _ in layers:
            at = slice(k * off + wo, k * off + wo + a * b)
            assert torch.equal(w16t[at].view(b, a), w16[at].view(a, b).T)


@pytest.mark.parametrize("m,n,groups", [(8, 8, 1), (24, 136, 3), (256, 752, 2), (5, 9, 2)])
def test_loss_gradient_and_its_transpose(m, n, groups):
    # columns 128 at a time: less, a remainder, several; (5, 9) takes the separate kernels
    native, lib = _lib()
    gen = torch.Generator("cuda").manual_seed(2)
    y, t = (torch.randn(groups * m, n, generator=gen, device="cuda") for _ in range(2))
    g32, ref32 = torch.zeros_like(y), torch.zeros_like(y)
    g16, ref16 = (torch.zeros_like(y, dtype=torch.bfloat16) for _ in range(2))
    g16t = torch.zeros(groups, n, m, dtype=torch.bfloat16, device="cuda")
    loss, ref_loss = (torch.zeros(groups * m, device="cuda") for _ in range(2))
    s = int(torch.cuda.current_stream().cuda_stream)
    native.check(lib.oafdtd_mlp_mse_grad(y.data_ptr(), t.data_ptr(), groups * m, n, ref32.data_ptr(),
                                         ref16.data_ptr(), ref_loss.data_ptr(), groups, s), "mse_grad")
    native.check(lib.oafdtd_mlp_mse_grad_t(y.data_ptr(), t.data_ptr(), groups * m, n, g32.data_ptr(), g16.data_ptr(),
                                           g16t.data_ptr(), loss.data_ptr(), groups, s), "mse_grad_t")
    assert torch.equal(g32, ref32) and torch.equal(g16, ref16)
    assert torch.equal(g16t, ref16.view(groups, m, n).transpose(1, 2))
    # a sum of n squares in another order: (n + 1) roundings each, of 2^-24
    assert torch.all((loss - ref_loss).abs() <= 2 * (n + 1) * 2.0**-24 * ref_loss)


@pytest.mark.parametrize("n_in,n_out,rows,groups", [(8, 8, 1, 1), (24, 200, 40, 3), (264, 752, 256, 2)])
def test_a_batch_is_its_gathered_rows(n_in, n_out, rows, groups):
    native, lib = _lib()
    gen = torch.Generator("cuda").manual_seed(3)
    x, t = (torch.randn(97, c, generator=gen, device="cuda") for c in (n_in, n_out))
    idx = torch.randint(97, (groups, rows), generator=gen, device="cuda", dtype=torch.int32)
    x16 = torch.zeros(groups, rows, n_in, dtype=torch.bfloat16, device="cuda")
    x16t = torch.zeros(groups, n_in, rows, dtype=torch.bfloat16, device="cuda")
    t32 = torch.zeros(groups, rows, n_out, device="cuda")
    step = torch.full((1,), 6, dtype=torch.int32, device="cuda")
    s = int(torch.cuda.current_stream().cuda_stream)
    native.check(lib.oafdtd_mlp_batch(x.data_ptr(), n_in, t.data_ptr(), n_out, idx.data_ptr(), rows, groups,
                                      x16.data_ptr(), x16t.data_ptr(), t32.data_ptr(), step.data_ptr(), s), "batch")
    assert torch.equal(x16, x[idx.long()].bfloat16()) and torch.equal(x16t, x16.transpose(1, 2))
    assert torch.equal(t32, t[idx.long()]) and step.item() == 7


@pytest.mark.parametrize("rows,chunk,members,act", [(1, 4096, 1, "tanh"), (37, 4096, 3, "relu"), (200, 64, 2, "tanh")])
def test_prediction_is_the_layers_one_by_one(rows, chunk, members, act):
    # one row; rows off every tile; chunks with a remainder, written into their place among the members
    from open_analysis_gb300.surrogate import Mlp

    net = Mlp([7, 40, 136, 24], 8, seed=5, members=members, act=act)
    x = torch.randn(rows, 7, generator=torch.Generator().manual_seed(4)).numpy()
    have = net.predict_device(x, chunk)
    want = torch.empty_like(have)
    for a in range(0, rows, chunk):
        xc = torch.from_numpy(net.pad(x[a : a + chunk])).cuda().bfloat16()
        m = xc.shape[0]
        x16 = xc.expand(members, m, -1).contiguous()
        acts = [torch.empty((members, m, b), dtype=torch.bfloat16, device="cuda") for b in net.sizes[1:-1]]
        y = torch.empty((members, m, net.sizes[-1]), device="cuda")
        net._forward(x16.data_ptr(), acts, y.data_ptr(), m, net._stream())
        want[:, a : a + m] = y
    assert torch.equal(have, want)
    one = net.predict_device(x[0], chunk)  # a vector stands for as many equal rows as it is wide, padded
    assert one.shape[1] == net.sizes[0] and torch.equal(one[:, :1], net.predict_device(x[:1], chunk))


@pytest.mark.parametrize("shapes", [
    [(2, 72, 136, 40)],
    [(8, 512, 512, 256), (8, 8, 512, 256), (8, 512, 1024, 256), (1, 130, 72, 520)],  # a K of its own, ragged tiles
    [(1, 64, 72, 64)] * 3 + [(1, 20, 24, 12)] + [(3, 136, 200, 88)] * 9,  # one for the general kernels; two launches
])
def test_a_list_of_products_is_its_products(shapes):
    native, lib = _lib()
    gen = torch.Generator("cuda").manual_seed(6)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = int(torch.cuda.current_stream().cuda_stream)
    keep, items = [], []
    for g, m, n, k in shapes:
        a, b = (torch.randn(g, r, k, generator=gen, device="cuda").bfloat16() for r in (m, n))
        c, want = (torch.full((g, m, n), 7.0, device="cuda") for _ in range(2))
        keep.append((a, b, c, want))
        items.append(native.Gemm(a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, k, k, n, g, m * k, n * k, m * n))
        native.check(lib.oafdtd_mlp_gemm_tn(a.data_ptr(), b.data_ptr(), want.data_ptr(), None, None, None, None, m, n, k,
                                            k, k, n, m, 0, 0.0, g, m * k, n * k, m * n, 0, 0, status.data_ptr(), s), "tn")
    native.check(lib.oafdtd_mlp_gemm_list((native.Gemm * len(items))(*items), len(items), status.data_ptr(), s), "list")
    for _, _, c, want in keep:
        assert torch.equal(c, want)
    assert status.item() == 0
