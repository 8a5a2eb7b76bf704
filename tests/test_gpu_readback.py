"""Readback through pinned slots, rank selection, and the default sweep kind.

Sizes straddle the readback's chunks (65,536 cells for the moments, 2 MiB of
values in general); everything compared here is a copy or the same arithmetic,
so equality is exact unless stated.
"""
import numpy as np
import pytest

import lbmflow_b200 as lb
from cases import cavity, seeded_state

pytestmark = pytest.mark.gpu


def box(dims):
    solid = np.zeros(dims[::-1], np.uint8)
    solid[0] = solid[-1] = 1
    solid[:, 0] = solid[:, -1] = 1
    solid[:, :, 0] = solid[:, :, -1] = 1
    return solid.ravel()


@pytest.mark.parametrize("dims", [(3, 3, 3), (5, 4, 3), (64, 32, 32), (41, 40, 40), (49, 53, 61)])
@pytest.mark.parametrize("q", [19, 27])
def test_populations_and_moments_come_back(dims, q):
    solid = box(dims)
    g = lb.Solver(dims, lattice=q, storage="f64", nu=0.05, solid=solid)
    f = seeded_state(q, g.n, 3)
    g.stage_in(f)
    assert np.array_equal(g.stage_out(), f)
    rho, ux, uy, uz = g.read_moments()
    fl = solid == 0
    assert np.abs(rho[fl] - 1.0 - f[:, fl].sum(0)).max() <= 1e-14  # q eps times the largest term
    assert np.all(rho[~fl] == 1.0) and np.all(ux[~fl] == 0.0) and np.all(uz[~fl] == 0.0)
    # a second solver at the same time, and the solid values of init_with
    h = lb.Solver(dims, lattice=q, storage="f64", nu=0.05, solid=solid)
    r0 = np.full(g.n, 1.01)
    u0 = np.full((g.n, 3), 0.002)
    h.init_with(r0, u0)
    m = h.read_moments()
    assert np.all(m[0][~fl] == 1.01) and np.all(m[2][~fl] == 0.002)
    assert np.array_equal(g.read_moments()[0], rho)


@pytest.mark.parametrize("n,scale", [(3, 1e-3), (4, 1e-3), (24, 0.0), (24, 1e-3), (52, 1e-3)])
def test_percentiles_are_the_sorted_ranks(n, scale):
    dims, solid, wall_u, nu = cavity(n)
    g = lb.Solver(dims, lattice=19, storage="f64", nu=nu, solid=solid, wall_u=wall_u)
    f = seeded_state(19, g.n, n, scale=1.0) * scale
    f[:, solid != 0] = 0.0
    g.stage_in(f)
    gam, tau, _ = g.stress_summary(0.01, 0.001, 0.7, 0.5, 0.35)
    v = np.sort(g.stress_field(0.01, 0.001, 0.7)["gamma_dot"][solid == 0])
    k = v.size
    assert gam["count"] == tau["count"] == k
    assert gam["max"] == v[-1] and tau["max"] == 0.7 * v[-1]
    for name, p in (("p50", 0.5), ("p90", 0.9), ("p95", 0.95), ("p99", 0.99)):
        r = p * (k - 1)
        lo, hi = int(np.floor(r)), int(np.ceil(r))
        want = v[lo] if lo == hi or k == 1 else v[lo] * (1.0 - (r - lo)) + v[hi] * (r - lo)
        assert gam[name] == want, name
    assert gam["fraction_above_threshold"] == (v > 0.5).sum() / k
    assert tau["fraction_above_threshold"] == (0.7 * v > 0.35).sum() / k


@pytest.mark.parametrize("q,coll,storage,kind", [
    (27, "cm", "f16", "window"), (27, "cm", "bf16", "window"), (19, "trt", "f16", "lean"), (19, "trt", "bf16", "lean"),
    (27, "trt", "f16", "lean"), (19, "trt", "f32", "lean"), (27, "cm", "f32", "async"), (27, "cm", "f64", "async"),
    (19, "trt", "f64", "async")])
@pytest.mark.parametrize("dims", [(16, 16, 16), (127, 128, 129), (128, 128, 128), (128, 128, 160)])
def test_default_sweep_does_not_depend_on_the_grid(dims, q, coll, storage, kind):
    # two kinds round in different orders, so the size alone must not choose
    solid = box(dims)
    mk = lambda: lb.Solver(dims, lattice=q, collision=coll, storage=storage, nu=0.02, solid=solid,  # noqa: E731
                           free_slip_top=True)
    g, d = mk(), mk()
    assert g.sweep_kernel == kind
    d.set_sweep_kernel(kind)
    f = seeded_state(q, g.n, 7)
    f[:, solid != 0] = 0.0
    for s in (g, d):
        s.stage_in(f)
        s.run(3)
    assert all(np.array_equal(a, b) for a, b in zip(g.read_moments(), d.read_moments()))
    # a variant names that kind's budgets
    g.set_sweep_variant(*{"lean": (8, 7), "window": (3, 3), "async": (4, 4)}[kind])
    assert g.sweep_kernel == kind


def test_renewed_relaxation_field_replays_like_single_steps():
    from lbmflow_b200 import sweep
    out = []
    for split in (False, True):
        g, body = sweep.build_case(sweep.TankCase(28, 0.04, 200.0), les_cs=0.0)
        for _ in range(3):
            g.wale_update()
            for k in ([1] * 10 if split else [10]):
                g.run_impeller(body, k)
        out.append(g.stage_out())
    assert np.array_equal(out[0], out[1])


def test_work_arrays_of_a_very_large_grid_are_given_back():
    # 24 bytes a cell is 288 MB here, above what a solver keeps between calls
    import torch
    dims = (240, 240, 208)
    g = lb.Solver(dims, lattice=19, storage="f16", nu=0.02, solid=box(dims))
    g.set_omega_field(np.full(g.n, 1.8))
    g.read_moments()

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    before = free()
    for call in (g.wale_update, lambda: g.stress_field(0.01, 0.001, 0.7), g.velocity_gradient,
                 lambda: g.stress_summary(0.01, 0.001, 0.7)):
        call()
        assert free() >= before - (64 << 20)
