"""GPU: a wait of the allocation-free solve's resident launch that gives up
leaves NaN in every spectrum; the next call solves as usual."""
import numpy as np
import pytest

from mittet_main_b200 import capi
from mittet_main_b200 import workloads as W
from mittet_main_b200.capi import FP32
from tests.test_zz_noalloc_resident import solve

pytestmark = pytest.mark.gpu


def test_noalloc_wait_timeout_is_nan_and_recovers(monkeypatch):
    wl = W.small_case(n=(40, 36, 32), ncpml=7, nt=30, precision=FP32, seed=4)
    lib = capi.load()
    want = solve(lib, wl)
    assert np.isfinite(want).all() and np.abs(want).max() > 0
    monkeypatch.setenv("MITTET_RESIDENT_STALL", "1")
    monkeypatch.setenv("MITTET_PERSIST_WAIT_MS", "20")
    assert np.isnan(solve(lib, wl)).all()
    monkeypatch.delenv("MITTET_RESIDENT_STALL")
    monkeypatch.delenv("MITTET_PERSIST_WAIT_MS")
    assert np.array_equal(solve(lib, wl), want)
