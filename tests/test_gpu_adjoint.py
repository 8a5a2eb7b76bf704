"""Discrete adjoint of the runner loop against central finite differences.

J = mean torque over the second half of the run (fixed three IBM sweeps, no
early exit). The finite differences use the f64 forward through the public
runner (`run_impeller`), with the relative step 1e-4 on nu and Omega and a
step of 1e-6 cells along random marker-position directions (the linear IBM
kernel has kinks at integer positions; a small step keeps every marker on
one side of them). Markers that sit exactly on an integer coordinate are on
a kink, where J has no derivative, so the generated markers are moved by a
seeded jitter of at most 0.1 cell first. Tolerance: 1e-5 relative for the
f64 adjoint; the f32 adjoint agrees with the f64 gradient to 1e-3.
"""
import numpy as np
import pytest

import lbmflow_b200 as lb
from lbmflow_b200 import sweep

pytestmark = pytest.mark.gpu

STEPS, WIN, K = 48, 24, 16
CFG = lb.DirectForcingConfig(max_iterations=3, slip_tolerance=0.0)


def tank(T=20, u_tip=0.04, re=200.0):
    c = sweep.TankCase(T, u_tip, re)
    geo = dict(sweep.tank_geometry(T))
    rng = np.random.default_rng(7)
    geo["marker_pos"] = geo["marker_pos"] + rng.uniform(-0.1, 0.1, size=geo["marker_pos"].shape)
    return c, geo


def J_of(c, geo, storage, nu=None, omega=None, pos=None):
    g = lb.Solver(c.dims, lattice=19, collision="trt", storage=storage, nu=c.nu if nu is None else nu,
                  solid=geo["solid"])
    body = lb.RotatingBody(geo["center"], [0.0, 0.0, c.omega if omega is None else omega],
                           geo["marker_pos"] if pos is None else pos, geo["marker_w"])
    t = g.run_impeller(body, STEPS, CFG)["torque_lu"]
    g.close()
    return float(np.mean(t[WIN:]))


def adjoint(c, geo, storage):
    g = lb.Solver(c.dims, lattice=19, collision="trt", storage=storage, nu=c.nu, solid=geo["solid"])
    body = lb.RotatingBody(geo["center"], [0.0, 0.0, c.omega], geo["marker_pos"], geo["marker_w"])
    r = g.adjoint_torque(body, STEPS, WIN, K, CFG)
    g.close()
    return r


@pytest.fixture(scope="module")
def case():
    c, geo = tank()
    return c, geo, adjoint(c, geo, "f64")


def test_adjoint_forward_equals_runner(case):
    c, geo, r = case
    assert abs(r["J"] - J_of(c, geo, "f64")) <= 1e-14 * abs(r["J"])
    assert r["adjoint_ms"] > 0 and r["forward_ms"] > 0


def test_adjoint_dnu_matches_finite_difference(case):
    c, geo, r = case
    h = 1e-4 * c.nu
    fd = (J_of(c, geo, "f64", nu=c.nu + h) - J_of(c, geo, "f64", nu=c.nu - h)) / (2 * h)
    assert abs(r["dJ_dnu"] - fd) <= 1e-5 * abs(fd), (r["dJ_dnu"], fd)


def test_adjoint_domega_matches_finite_difference(case):
    c, geo, r = case
    h = 1e-4 * c.omega
    fd = (J_of(c, geo, "f64", omega=c.omega + h) - J_of(c, geo, "f64", omega=c.omega - h)) / (2 * h)
    assert abs(r["dJ_domega_z"] - fd) <= 1e-5 * abs(fd), (r["dJ_domega_z"], fd)


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_adjoint_dpos_matches_finite_difference(case, seed):
    c, geo, r = case
    rng = np.random.default_rng(seed)
    d = rng.normal(size=geo["marker_pos"].shape)
    d /= np.linalg.norm(d)
    h = 1e-6
    p0 = geo["marker_pos"]
    fd = (J_of(c, geo, "f64", pos=p0 + h * d) - J_of(c, geo, "f64", pos=p0 - h * d)) / (2 * h)
    ad = float(np.sum(r["dJ_dpos"] * d))
    assert abs(ad - fd) <= 1e-5 * max(abs(fd), 1e-12) + 1e-9, (ad, fd)


def test_adjoint_f32_tracks_f64(case):
    c, geo, r64 = case
    r32 = adjoint(c, geo, "f32")
    assert abs(r32["dJ_dnu"] - r64["dJ_dnu"]) <= 1e-3 * abs(r64["dJ_dnu"])
    assert abs(r32["dJ_domega_z"] - r64["dJ_domega_z"]) <= 1e-3 * abs(r64["dJ_domega_z"])
    g32, g64 = r32["dJ_dpos"], r64["dJ_dpos"]
    assert np.linalg.norm(g32 - g64) <= 1e-3 * np.linalg.norm(g64)


@pytest.mark.parametrize("warm", [0, 3])
@pytest.mark.parametrize("storage", ["f64", "f32"])
def test_adjoint_segments_as_graphs_equal_eager_ones(storage, warm):
    # 101 steps in segments of 16 (six replayed as graphs and an odd
    # remainder), of 26 (launched one by one) and in one: the same steps, so
    # the same sums up to the order of the atomic additions into f64
    # accumulators (at most 1e7 terms of one sign mix: 1e-12)
    c, geo = tank()
    got = []
    for every in (16, 26, 102):
        g = lb.Solver(c.dims, lattice=19, collision="trt", storage=storage, nu=c.nu, solid=geo["solid"])
        body = lb.RotatingBody(geo["center"], [0.0, 0.0, c.omega], geo["marker_pos"], geo["marker_w"])
        if warm:
            g.run_impeller(body, warm, CFG)
        r = g.adjoint_torque(body, 101, 37, every, CFG)
        got.append((r, g.stage_out()))
        g.close()
    (a, fa), rest = got[0], got[1:]
    for b, fb in rest:
        assert np.array_equal(a["torque"], b["torque"]) and a["J"] == b["J"]
        assert np.array_equal(fa, fb)
        for k in ("dJ_dnu", "dJ_domega_z"):
            assert abs(a[k] - b[k]) <= 1e-12 * abs(a[k]), k
        assert np.abs(a["dJ_dpos"] - b["dJ_dpos"]).max() <= 1e-12 * np.abs(a["dJ_dpos"]).max()


@pytest.mark.parametrize("nm", [500, 1700])
def test_adjoint_of_bodies_about_the_wide_line(nm):
    # on both sides of 4,096 slots (the cluster, and one kernel per phase): the
    # gradient along random marker directions and in the speed against central
    # differences of the f64 forward
    from test_gpu_ibm_cluster import dense_body
    solid, body = dense_body(38, nm)
    steps, win = 14, 4

    def run(omega_z, pos):
        g = lb.Solver((38,) * 3, lattice=19, storage="f64", nu=0.02, solid=solid)
        b = lb.RotatingBody(body.center, [0.0, 0.0, omega_z], pos, body.weights)
        t = g.run_impeller(b, steps, CFG)["torque_lu"]
        slots = int(np.count_nonzero(np.any(g.force_field().reshape(-1, 3) != 0.0, axis=1)))
        g.close()
        return float(np.mean(t[win:])), slots

    w, pos = body.omega[2], np.asarray(body.positions).reshape(-1, 3)
    g = lb.Solver((38,) * 3, lattice=19, storage="f64", nu=0.02, solid=solid)
    r = g.adjoint_torque(body, steps, win, 6, CFG)
    J, slots = run(w, pos)
    assert (slots > 4096) == (nm > 1000), slots
    assert abs(r["J"] - J) <= 1e-13 * abs(J)
    h = 1e-4 * w
    fd = (run(w + h, pos)[0] - run(w - h, pos)[0]) / (2 * h)
    assert abs(r["dJ_domega_z"] - fd) <= 1e-5 * abs(fd)
    d = np.random.default_rng(4).normal(size=pos.shape)
    d /= np.linalg.norm(d)
    fd = (run(w, pos + 1e-6 * d)[0] - run(w, pos - 1e-6 * d)[0]) / 2e-6
    ad = float(np.sum(r["dJ_dpos"].reshape(-1, 3) * d))
    assert abs(ad - fd) <= 1e-5 * max(abs(fd), 1e-12) + 1e-9, (ad, fd)


def test_adjoint_rejects_unsupported():
    c, geo = tank()
    g = lb.Solver(c.dims, lattice=27, collision="cm", storage="f32", nu=c.nu, solid=geo["solid"])
    body = lb.RotatingBody(geo["center"], [0.0, 0.0, c.omega], geo["marker_pos"], geo["marker_w"])
    with pytest.raises(lb.UnsupportedError):
        g.adjoint_torque(body, 8, 4, 4, CFG)
    g = lb.Solver(c.dims, lattice=19, storage="f32", nu=c.nu, solid=geo["solid"], smagorinsky_cs=0.1)
    with pytest.raises(lb.UnsupportedError):
        g.adjoint_torque(body, 8, 4, 4, CFG)
