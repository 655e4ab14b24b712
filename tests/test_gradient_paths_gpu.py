"""GPU: the forward passes of a gradient on their three paths (resident launch,
stepped straight into the history slots, stepped and copied), and the adjoint
against differences of the misfit where the oracle has no adjoint."""
from dataclasses import replace

import numpy as np
import pytest

from mittet_main_b200 import workloads as W
from mittet_main_b200.capi import FLAVOR_NCVER0027, FLAVOR_SATAN_I, FP32, FP64, SRC_ELECTRIC
from mittet_main_b200.solver import Shot
from tests.conftest import rel_l2
from tests.test_adjoint_gpu import observed, oracle_gradient

pytestmark = pytest.mark.gpu

PATHS = {"resident": {}, "direct": {"MITTET_RESIDENT": "0"}, "copy": {"MITTET_RESIDENT": "0", "MITTET_GRAD_COPY": "1"}}


def gradient(monkeypatch, wl, obs, path, every):
    for k, v in PATHS[path].items():
        monkeypatch.setenv(k, v)
    with W.make_solver(wl) as s:
        out = s.gradient(wl.nt, obs, checkpoint_every=every)
    for k in PATHS[path]:
        monkeypatch.delenv(k)
    return out


def two_shots(n, prec, flavor, magnetic, seed=5, ncpml=6):
    wl = W.small_case(n=n, ncpml=ncpml, nt=60, precision=prec, flavor=flavor, magnetic=magnetic, seed=seed)
    return replace(wl, shots=[wl.shots[0], Shot(points=[(n[0] - 15, 12, 15, "ey", SRC_ELECTRIC, 0.8)])])


# segments of 25 (the last of 10), one step, and one for all
@pytest.mark.parametrize("every", [25, 1, 60])
@pytest.mark.parametrize("prec,flavor", [(FP32, FLAVOR_NCVER0027), (FP64, FLAVOR_SATAN_I)])
def test_three_forward_paths_give_the_same_bits(monkeypatch, prec, flavor, every):
    wl = two_shots((45, 34, 30), prec, flavor, False)
    obs = observed(wl)
    res = {p: gradient(monkeypatch, wl, obs, p, every) for p in PATHS}
    assert np.abs(res["copy"][1]).max() > 0
    for p in ("resident", "direct"):
        assert res[p][0] == pytest.approx(res["copy"][0], rel=1e-13)  # the misfit is an atomic reduction
        assert np.array_equal(res[p][1], res["copy"][1]), p


# FP32: as derived in test_adjoint_gpu
@pytest.mark.parametrize("prec,tol", [(FP64, 1e-10), (FP32, 1e-5)])
@pytest.mark.parametrize("path", ["direct", "copy"])
def test_stepped_gradient_matches_the_oracle(monkeypatch, path, prec, tol):
    wl = W.small_case(n=(39, 24, 25), ncpml=5, nt=60, precision=prec, seed=3)
    mu = wl.cp.mu0 * (1.0 + 0.2 * np.random.default_rng(4).random(wl.sigma.shape))
    wl.mu = mu
    obs = observed(wl)
    Jo, Go = oracle_gradient(wl, obs, mu)
    J, G = gradient(monkeypatch, wl, obs, path, 25)
    assert J == pytest.approx(Jo, rel=tol)
    assert rel_l2(G, Go) <= tol


# A central difference along one random direction, sigma changed by up to 1e-4
# of itself inside the frame: truncation (1e-4)^2 / 6 times a curvature of order
# 100, rounding 1e-13 / 1e-4 times a misfit of order 100 times its change: 1e-5
# is far above both.  The FP32 gradient as in test_adjoint_gpu.
@pytest.mark.parametrize("n,flavor,with_mu", [((45, 34, 30), FLAVOR_SATAN_I, False), ((70, 34, 30), FLAVOR_SATAN_I, True),
                                              ((45, 34, 30), FLAVOR_NCVER0027, True)])
def test_gradient_against_differences_of_the_misfit(n, flavor, with_mu):
    wl = two_shots(n, FP64, flavor, True)
    rng = np.random.default_rng(9)
    if with_mu:
        wl = replace(wl, mu=wl.cp.mu0 * (1.0 + 0.2 * rng.random(wl.sigma.shape)))
    with W.make_solver(wl) as s:
        spec, _ = s.forward(wl.nt)
    obs = spec * (1.0 + 0.5 * rng.normal(size=spec.shape))
    d = np.zeros(wl.sigma.shape)
    nc = wl.cp.ncpml
    d[nc:-nc, nc:-nc, nc:-nc] = rng.uniform(0.2, 1.0, size=d[nc:-nc, nc:-nc, nc:-nc].shape)
    d *= 1e-4 * wl.sigma
    J = []
    for sgn in (1.0, -1.0):
        with W.make_solver(replace(wl, sigma=wl.sigma + sgn * d)) as s:
            spec, _ = s.forward(wl.nt)
        J.append(0.5 * float(np.sum(np.abs(spec - obs) ** 2)))
    with W.make_solver(wl) as s:
        _, G = s.gradient(wl.nt, obs, checkpoint_every=25)
    fd = (J[0] - J[1]) / 2.0
    assert abs(float(np.sum(G * d)) - fd) <= 1e-5 * abs(fd)
    with W.make_solver(wl, FP32) as s:
        _, G32 = s.gradient(wl.nt, obs, checkpoint_every=25)
    assert rel_l2(G32, G) <= 1e-5
