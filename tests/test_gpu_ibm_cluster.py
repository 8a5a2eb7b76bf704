"""Direct forcing as one cluster kernel: marker and slot counts at the edges.

The kernel works in chunks of 32 markers and slots, in one of two forms (up
to 4,096 entries, and above), and leaves its sweep loop early. Each count is
compared with the oracle on the same f64 populations: diagnostics to 1e-10
(sums of at most 1e5 terms, n eps = 2e-11), field to 1e-12 of its largest
value (the spread sums in the reference's marker order).
"""
import numpy as np
import pytest

import lbmflow_b200 as lb
from cases import cavity, seeded_state
from test_gpu_ibm import assert_diag_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nm", [1, 31, 32, 33, 1025, 4096, 4097, 9000])
@pytest.mark.parametrize("radius,tol", [(1, 1e-2), (2, 0.0)])
def test_marker_counts_match_oracle(nm, radius, tol):
    from oracle import oracle as o
    dims, solid, wall_u, nu = cavity(34)
    rng = np.random.default_rng(nm)
    pos = rng.uniform(0.6, 32.4, (nm, 3))  # some stencils reach the walls
    w = rng.uniform(0.2, 0.8, nm)
    body = lb.RotatingBody([16.5, 16.5, 16.5], [0.0, 0.001, 0.002], pos, w)
    g = lb.Solver(dims, lattice=19, storage="f64", nu=nu, solid=solid, wall_u=wall_u)
    c = o.OracleSolver(dims, q=19, real_bits=64, nu=nu, solid=solid, wall_u=wall_u)
    f = seeded_state(19, g.n, 5)
    f[:, solid != 0] = 0.0
    g.stage_in(f)
    c.stage_in(f)
    for _ in range(2):  # the second application sees the first one's field
        dg = g.apply_rotating_ibm(body, lb.DirectForcingConfig(3, tol, radius, 0.9))
        do = c.ibm_apply(body.positions, body.weights, body.center, body.omega, 3, tol, radius, 0.9)
        assert_diag_close(dg, do, 1e-10)
        fg, fc = g.force_field(), c.force_field()
        assert np.abs(fg - fc).max() <= 1e-12 * np.abs(fc).max()


def dense_body(n, nm):
    """nm markers scattered in a disc of a closed box of n cells: about 8 slots
    each while they are few."""
    solid = np.zeros((n, n, n), np.uint8)
    solid[0] = solid[-1] = 1
    solid[:, 0] = solid[:, -1] = 1
    solid[:, :, 0] = solid[:, :, -1] = 1
    rng = np.random.default_rng(nm)
    th, r = rng.uniform(0.0, 2.0 * np.pi, nm), rng.uniform(0.1 * n, 0.44 * n, nm)
    z = 0.5 * n + rng.uniform(-1.0, 1.0, nm) * min(0.44 * n, 0.5 + nm / (0.6 * n * n))
    pos = np.stack([0.5 * n + r * np.cos(th), 0.5 * n + r * np.sin(th), z], axis=1)
    return solid.ravel(), lb.RotatingBody([0.5 * n] * 3, [0.0, 0.0, 0.0007], pos, np.full(nm, 0.3))


@pytest.mark.parametrize("storage", ["f64", "f16"])
@pytest.mark.parametrize("nm", [400, 1500, 3000, 6000])
@pytest.mark.parametrize("tol", [1e-2, 0.0])
def test_both_forms_give_the_same_bits(nm, tol, storage):
    # a call on its own leaves the cluster for the full-chip kernels above 4,096
    # slots, one beside a sweep above 6,000 + cells / 200 (6,460 here): the loop
    # and the calls one by one then run different forms, and every form sums in
    # the same order
    solid, body = dense_body(45, nm)
    a, b, c = (lb.Solver((45,) * 3, lattice=19, storage=storage, nu=0.03, solid=solid) for _ in range(3))
    cfg = lb.DirectForcingConfig(3, tol, 1, 1.0)
    r = a.run_impeller(body, 21, cfg)
    tq, ff = [], []
    for k in range(21):
        b.clear_body_force_field()
        d = b.apply_rotating_ibm(body, cfg)
        b.run(1)
        e = c.runner_step(0, body, cfg)
        tq.append(-d.torque[2])
        ff.append(d.fluid_force)
        assert d.iterations == e.iterations == r["ibm_iterations"][k]
        for key in ("slip_max", "slip_rms", "momentum_error_rel"):
            assert getattr(d, key) == getattr(e, key), key
        assert np.array_equal(d.torque, e.torque) and np.array_equal(d.marker_force, e.marker_force)
    slots = int(np.count_nonzero(np.any(a.force_field().reshape(-1, 3) != 0.0, axis=1)))
    assert {400: slots < 4096, 1500: 4096 < slots < 6400}.get(nm, slots > 6500), slots
    assert np.array_equal(r["torque_lu"], np.array(tq)) and np.array_equal(r["fluid_force"], np.array(ff))
    assert np.array_equal(a.stage_out(), b.stage_out()) and np.array_equal(a.stage_out(), c.stage_out())


# CRC-32 of the force field after two calls from integer-made inputs, as a
# chain of kernels with plain divisions gave it.
FIELD_CRC = {(300, 1): 0xa94664c8, (300, 2): 0x0d310867, (5000, 1): 0xcbb8dd4d, (5000, 2): 0xfc32f19a}


@pytest.mark.parametrize("nm,radius", list(FIELD_CRC))
def test_force_field_keeps_its_rounding(nm, radius):
    import zlib
    solid = np.zeros((22, 20, 18), np.uint8)
    solid[0] = solid[-1] = 1
    solid[:, 0] = solid[:, -1] = 1
    solid[:, :, 0] = solid[:, :, -1] = 1
    solid = solid.ravel()

    def lcg(k, m):  # m numbers in [0, 1)
        i = np.arange(m, dtype=np.uint64) + np.uint64(k)
        return ((i * np.uint64(2654435761) >> np.uint64(13)) % np.uint64(262144)).astype(np.float64) / 262144.0

    g = lb.Solver((18, 20, 22), lattice=19, storage="f64", nu=0.03, solid=solid)
    f = 2e-3 * (lcg(5, 19 * g.n).reshape(19, g.n) - 0.5)
    f[:, solid != 0] = 0.0
    g.stage_in(f)
    pos = 0.7 + lcg(77, 3 * nm).reshape(nm, 3) * np.array([15.6, 17.6, 19.6])
    body = lb.RotatingBody([8.5, 9.5, 10.5], [0.001, 0.0, 0.003], pos, 0.25 + 0.5 * lcg(9, nm))
    for relax in (1.0, 0.9):
        g.apply_rotating_ibm(body, lb.DirectForcingConfig(4, 0.0, radius, relax))
    out = np.ascontiguousarray(g.force_field() + 0.0)
    assert np.isfinite(out).all() and zlib.crc32(out.tobytes()) == FIELD_CRC[nm, radius], hex(zlib.crc32(out.tobytes()))


@pytest.mark.parametrize("T,q,coll,storage,kind", [
    (32, 19, "trt", "f32", None), (32, 19, "trt", "f16", None), (32, 27, "cm", "f64", None),
    # above 4,096 slots (the form of 1,024 threads), beside each persistent sweep
    (112, 19, "trt", "f32", "pair"), (112, 19, "trt", "f16", "pair"), (112, 19, "trt", "f32", "lean"),
    (112, 27, "cm", "f32", "async"), (112, 27, "cm", "bf16", "window"), (112, 27, "cm", "f16", "pair")])
def test_runner_loop_repeats_bitwise(T, q, coll, storage, kind):
    # the phases of one call are ordered by cluster barriers only, and the
    # sweep runs beside it: a missing barrier or a shared slot shows as a
    # difference between two runs
    from lbmflow_b200 import sweep
    case = sweep.TankCase(T, 0.05, 600.0)
    geo = sweep.tank_geometry(T)
    body = lb.RotatingBody(geo["center"], [0.0, 0.0, case.omega], geo["marker_pos"], geo["marker_w"])
    ref = None
    for _ in range(4):
        g = lb.Solver(case.dims, lattice=q, collision=coll, storage=storage, nu=case.nu, solid=geo["solid"],
                      smagorinsky_cs=0.1)
        if kind:
            g.set_sweep_kernel(kind)
        r = g.run_impeller(body, 40)
        got = (r["torque_lu"], r["ibm_iterations"], g.stage_out())
        if T > 100:
            assert np.count_nonzero(np.any(g.force_field().reshape(-1, 3) != 0.0, axis=1)) > 4096
        g.close()
        if ref is not None:
            assert all(np.array_equal(a, b) for a, b in zip(ref, got))
        ref = got
