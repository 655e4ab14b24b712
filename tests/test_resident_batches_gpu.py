"""Batches on the resident time loop: the length of a launch, and the double
precision batches that the stepped path takes."""
from dataclasses import replace

import numpy as np
import pytest

from mittet_main_b200 import workloads as W
from mittet_main_b200.capi import FP32, FP64, SRC_ELECTRIC, SRC_MAGNETIC
from mittet_main_b200.solver import Shot

pytestmark = pytest.mark.gpu


def test_a_launch_of_many_shots_is_cut_short():
    """1500 shots of 32^3 take about 1.5 ms a step: 600 steps are not one
    launch of most of a second, and the shots' traces are those of the same
    shots solved alone."""
    n, nt, ns = (32, 32, 32), 600, 1500
    wl = W.small_case(n=n, ncpml=8, nt=nt, precision=FP32, seed=2)
    shots = [Shot(points=[(8 + q % 16, 8 + q // 16 % 16, 12, ("ex", "ey")[q % 2], SRC_ELECTRIC, 1.0 + 0.01 * (q % 7)),
                          (10, 12, 8 + q % 16, "hz", SRC_MAGNETIC, 1e-3)]) for q in range(ns)]
    rec = [(x, 16, 16, c) for x in range(6, 27, 5) for c in ("ex", "hz")]
    wl = replace(wl, shots=shots, receivers=rec)
    with W.make_solver(wl) as s:
        _, td = s.forward(nt, want_traces=True)
        ctas, launches = s.resident_ctas(), s.launch_count()
    # beside the time loop: the finite check and the traces' transform
    assert ctas > 0 and launches - 2 >= 2
    some = [0, 1, 7, 700, ns - 1]
    with W.make_solver(replace(wl, shots=[shots[q] for q in some])) as s:
        _, alone = s.forward(nt, want_traces=True)
    assert np.abs(alone).max() > 0
    assert np.array_equal(td[some], alone)


# of an 80^3 grid the stepped path takes batches of 14 shots and more
@pytest.mark.parametrize("ns,stepped", [(1, False), (8, False), (17, True)])
def test_fp64_batches_on_both_sides_of_the_rule(monkeypatch, ns, stepped):
    n, nt = (80, 80, 80), 30
    wl = W.small_case(n=n, ncpml=10, nt=nt, precision=FP64, seed=2)
    shots = [Shot(points=[(20 + q, 40, 30, ("ex", "ey")[q % 2], SRC_ELECTRIC, 1.0),
                          (40, 20 + q, 20, "hz", SRC_MAGNETIC, 1e-3)]) for q in range(ns)]
    wl = replace(wl, shots=shots)

    def solve():
        with W.make_solver(wl) as s:
            spec, td = s.forward(nt, want_traces=True)
            return s.resident_ctas(), [spec, td, s.fields(ns - 1)]

    ctas, a = solve()
    assert (ctas == 0) == stepped
    monkeypatch.setenv("MITTET_RESIDENT", "1")
    ctas, b = solve()
    assert ctas > 0
    assert np.abs(b[1]).max() > 0
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
