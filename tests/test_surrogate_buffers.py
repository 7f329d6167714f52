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


def test_queued_epochs_hold_a_bounded_number_of_shuffles() -> None:
    """Many epochs queued behind a busy stream (some 250 ms): the shuffles drawn ahead of the training
    stream do not pile up (each is 2 members x 65536 rows of 8 bytes here, 1 MB)."""
    net = _net(2, batch=65536)
    rng = np.random.default_rng(2)
    x, t = rng.standard_normal((66000, 8)), rng.standard_normal((66000, 16))
    net.prepare(x, t)
    net.run_epoch(1e-3)
    torch.cuda.synchronize()
    before = torch.cuda.memory_stats()["active_bytes.all.current"]
    with torch.cuda.stream(net.stream):
        torch.cuda._sleep(500_000_000)
    for _ in range(40):
        net.run_epoch(1e-3)
    held = torch.cuda.memory_stats()["active_bytes.all.current"] - before
    torch.cuda.synchronize()
    assert held <= 4 * 2 * 65536 * 8, held


def test_epochs_draw_the_shuffles_of_one_seed() -> None:
    """Networks of one seed and data train alike, queued or waited for epoch by epoch, with all rows and
    with row subsets: an epoch's shuffle is not overwritten before its steps have read it."""
    rng = np.random.default_rng(3)
    x, t = rng.standard_normal((300, 8)), rng.standard_normal((300, 16))
    for rows in (None, [np.arange(0, 300, 2), np.arange(100, 290)]):
        got = []
        for wait in (False, True):
            net = _net(2)
            net.prepare(x, t, rows=rows)
            for _ in range(12):
                net.run_epoch(1e-3)
                if wait:
                    torch.cuda.synchronize()
            torch.cuda.synchronize()
            got.append(net.p32.clone())
        assert torch.equal(got[0], got[1])
