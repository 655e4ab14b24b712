"""GPU: calls that read a solve's buffers after the set-up has changed: they
size the buffers for the present set-up or ask for a forward."""
from dataclasses import replace

import numpy as np
import pytest

from mittet_main_b200 import workloads as W
from mittet_main_b200.capi import FP32, MittetError

pytestmark = pytest.mark.gpu


def test_kernel_timing_after_a_change_of_receivers_and_volume():
    wl = replace(W.small_case(n=(40, 36, 32), ncpml=8, nt=140, precision=FP32, seed=6), receivers=[(9, 9, 9, "ex")])
    many = [(1 + q % 40, 1 + q // 40, 16, ("ex", "hz")[q % 2]) for q in range(1000)]
    with W.make_solver(wl) as s:
        want, _ = s.forward(wl.nt)
        s.set_receivers(many)
        assert s.time_kernels(wl.nt)["e_phase"] > 0
        s.set_freqs(np.arange(1, 9) * 6.28)
        s.set_volume_dft("xyz")
        assert s.time_kernels(wl.nt)["volume_dft"] > 0
        s.set_wavelet(wl.wavelet[:100])
        with pytest.raises(MittetError) as ex:
            s.time_kernels(wl.nt)
        assert ex.value.name == "MITTET_ERR_STATE"
        s.set_volume_dft("")
        s.set_wavelet(wl.wavelet)
        s.set_receivers(wl.receivers)
        s.set_freqs(wl.omega)
        got, _ = s.forward(wl.nt)
    assert np.abs(want).max() > 0 and np.array_equal(got, want)


def test_volume_spectra_of_another_setup_are_refused():
    wl = W.small_case(n=(32, 30, 28), ncpml=6, nt=20, precision=FP32, seed=6)
    with W.make_solver(replace(wl, omega=wl.omega[:1], volume_dft="x")) as s:
        s.forward(wl.nt)
        assert s.volume_dft(0, "ex").shape[0] == 1
        s.set_freqs(wl.omega)
        with pytest.raises(MittetError) as ex:
            s.volume_dft(0, "ex")
        assert ex.value.name == "MITTET_ERR_STATE"
