"""Solves of fewer steps than the block that the stepped path times when it
chooses between its graph and the persistent launch.

The timed block writes traces and reads the wavelet like a solve, so it has to
stay within the solve's own nt.  Short solves on a new handle (nt of 1, of less
than a block, of one block and a few steps) must give what the resident time
loop gives, bit for bit, and so must a longer one after them on that handle.
"""
from dataclasses import replace

import numpy as np
import pytest

from mittet_main_b200 import workloads as W
from mittet_main_b200.capi import FP32, FP64, SRC_ELECTRIC, SRC_MAGNETIC
from mittet_main_b200.solver import Shot

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("persist", ["", "1"])
@pytest.mark.parametrize("prec", [FP32, FP64])
@pytest.mark.parametrize("nt", [1, 20, 131])
def test_short_solve_on_a_new_handle(monkeypatch, nt, prec, persist):
    wl = W.small_case(n=(40, 36, 32), ncpml=7, nt=150, precision=prec, seed=5)
    shots = [Shot(points=[(14, 12, 15, "ex", SRC_ELECTRIC, 1.0), (20, 20, 20, "hz", SRC_MAGNETIC, 1e-3)]),
             Shot(points=[(25, 20, 10, "ey", SRC_ELECTRIC, 0.5)])]
    long = replace(wl, shots=shots, wavelet=wl.wavelet[:151])
    short = replace(long, nt=nt, wavelet=wl.wavelet[:nt + 1])

    def solve(env):
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        out = []
        with W.make_solver(short) as s:
            out += [*s.forward(nt, want_traces=True), s.fields(0), s.fields(1)]
            path = s.launch_path()["persistent"], s.resident_ctas()
            s.set_wavelet(long.wavelet)
            out += s.forward(long.nt, want_traces=True)
        for k in env:
            monkeypatch.delenv(k)
        return path, out

    (_, ctas), want = solve({})
    stepped = {"MITTET_RESIDENT": "0", **({"MITTET_PERSIST": persist} if persist else {})}
    (persistent, none), got = solve(stepped)
    assert ctas > 0 and none == 0 and (persistent or not persist)
    assert np.abs(want[-1]).max() > 0
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
