"""Host and device memory that the surrogate's calls hand over: when it may be reused, how much is held."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _net(members: int, batch: int = 32):  # type: ignore[no-untyped-def]
    from open_analysis_gb300.surrogate import Mlp

    return Mlp([8, 64, 64, 16], members=members, batch=batch, seed=5)


@pytest.mark.parametrize("rows", [1, 128, 129, 512, 513, 700])
def test_inputs_may_be_reused_when_predict_returns(rows: int) -> None:
    """Pinned inputs overwritten as soon as ``oafdtd_mlp_predict`` has returned, behind a stream that is
    still busy (some 50 ms): the prediction is of what they held at the call. Eight columns: up to 1024
    and 4096 values as launch parameters, a copy above."""
    from open_analysis_gb300 import native

    net = _net(2)
    x = np.random.default_rng(1).standard_normal((rows, 8)).astype(np.float32)
    want = net.predict_device(x).clone()
    lib, layers = net.lib, len(net.layout)
    work = torch.empty(int(lib.oafdtd_mlp_predict_bytes(rows, layers, net._layers, 2)), dtype=torch.uint8, device="cuda")
    out = torch.zeros_like(want)
    pinned = torch.from_numpy(x).pin_memory()
    s = torch.cuda.current_stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)
    native.check(lib.oafdtd_mlp_predict(pinned.data_ptr(), rows, net.p32.data_ptr(), net.p16T.data_ptr(), layers,
                                        net._layers, 2, net.n_params, net.act, work.data_ptr(), out.data_ptr(),
                                        rows * net.sizes[-1], net.status.data_ptr(), int(s.cuda_stream)), "predict")
    pinned.fill_(0.0)
    torch.cuda.synchronize()
    assert torch.equal(out, want)
