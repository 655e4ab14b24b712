"""GPU: work queued on other streams than the handle's own, calls made while a
solve that returned early (forward_device) still runs, and its failures."""
from dataclasses import replace

import numpy as np
import pytest

from mittet_main_b200 import workloads as W
from mittet_main_b200.capi import FP32

pytestmark = pytest.mark.gpu


def case(nt=1500):
    return W.small_case(n=(40, 36, 32), ncpml=8, nt=nt, precision=FP32, seed=6)


@pytest.mark.parametrize("resident", [True, False])
def test_a_solve_in_flight_keeps_what_it_was_started_with(monkeypatch, resident):
    """The wavelet, receivers, frequencies and shots of the next solve are set
    while the last one runs; its spectra and fields are its own."""
    import torch

    if not resident:
        monkeypatch.setenv("MITTET_RESIDENT", "0")
    wl = case()
    out = torch.zeros((1, len(wl.receivers), len(wl.omega), 2), dtype=torch.float64, device="cuda")
    with W.make_solver(wl) as s:
        want, _ = s.forward(wl.nt)
        want_f = s.fields(0)
        assert np.abs(want).max() > 0
        for change in (lambda: s.set_wavelet(0.5 * wl.wavelet), lambda: s.set_receivers(wl.receivers[::-1]),
                       lambda: s.set_freqs(2.0 * wl.omega), lambda: s.set_shots([wl.shots[0]] * 2)):
            torch.cuda.synchronize()
            s.forward_device(wl.nt, out, torch.cuda.current_stream())
            change()
            torch.cuda.synchronize()
            got = out.cpu().numpy()
            assert np.array_equal(got[..., 0] + 1j * got[..., 1], want)
            s.set_wavelet(wl.wavelet)
            s.set_receivers(wl.receivers)
            s.set_freqs(wl.omega)
            s.set_shots(wl.shots)
        s.forward_device(wl.nt, out, torch.cuda.current_stream())
        assert np.array_equal(s.fields(0), want_f)  # read behind the solve


@pytest.mark.parametrize("own_stream", [False, True])
def test_a_device_model_is_read_after_the_work_that_writes_it(own_stream):
    import torch

    wl = case(nt=60)
    sig = torch.from_numpy(np.ascontiguousarray(wl.sigma)).cuda()
    late = torch.full_like(sig, 0.7)
    busy = torch.empty(1 << 28, dtype=torch.float32, device="cuda")
    with W.make_solver(wl) as s:
        want, _ = s.forward(wl.nt)
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.current_stream()):
            for _ in range(60):  # about 20 ms of writes before the model's
                busy.fill_(1.0)
            late.copy_(sig)
            s.set_model_device(late)
        got, _ = s.forward(wl.nt)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("stall,env", [("MITTET_RESIDENT_STALL", {}), ("MITTET_PERSIST_STALL", {"MITTET_PERSIST": "1"})])
def test_a_stalled_device_solve_leaves_nan(monkeypatch, stall, env):
    import torch

    wl = case(nt=150)
    out = torch.full((1, len(wl.receivers), len(wl.omega), 2), 7.0, dtype=torch.float64, device="cuda")
    with W.make_solver(wl) as s:
        want, _ = s.forward(wl.nt)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    monkeypatch.setenv(stall, "1")
    monkeypatch.setenv("MITTET_PERSIST_WAIT_MS", "20")
    with W.make_solver(wl) as s:
        s.forward_device(wl.nt, out, torch.cuda.current_stream())
        assert torch.isnan(out).all()
    monkeypatch.delenv(stall)
    monkeypatch.delenv("MITTET_PERSIST_WAIT_MS")
    with W.make_solver(wl) as s:
        s.forward_device(wl.nt, out, torch.cuda.current_stream())
    got = out.cpu().numpy()
    assert np.array_equal(got[..., 0] + 1j * got[..., 1], want)
