"""The straight-line quotients and square roots of the FP64 kernels.

They replace the compiler's division and square root where a row's operands
are in range and must round the same; outside that range the plain formulas
are used.  So the results are the CPU oracle's bit for bit whatever the
magnitudes of the state: ordinary, exactly zero, near underflow.
"""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "2d-dns-godunov-solver-_b200", "csrc")


def test_quotients_and_roots_round_as_ieee(tmp_path):
    """Random arguments over the whole range, significands next to powers of
    two, and arguments built to lie next to a midpoint of two doubles."""
    exe = str(tmp_path / "exact_math_check")
    subprocess.check_call(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                           "-fmad=false", "-I" + CSRC, os.path.join(HERE, "exact_math_check.cu"), "-o", exe])
    rows = [tuple(int(x) for x in r.split()) for r in subprocess.check_output([exe], text=True).splitlines()]
    assert len(rows) == 7 and all(n > 1000 for _, n in rows)
    assert [bad for bad, _ in rows] == [0] * 7


def _state(mesh, seed, wild):
    """Density and pressure around one (wild: over 12 decades), a velocity
    component of every magnitude: ordinary, exactly zero, down to denormals."""
    rng = np.random.default_rng(seed)
    n = mesh.nCells
    rho, p = 1.0 + 0.1 * rng.uniform(-1, 1, n), 0.7 * (1.0 + 0.1 * rng.uniform(-1, 1, n))
    u = 2.0 + 0.1 * rng.uniform(-1, 1, n)
    x = mesh.cell_mid_points[:, 0] - mesh.cell_mid_points[:, 0].min()
    v = np.where(rng.random(n) < 0.2, 0.0, rng.choice([-1.0, 1.0], n) * 10.0 ** (-330.0 * (x / x.max()) ** 1.5))
    if wild:
        rho, p = rho * 10.0 ** rng.uniform(-6, 6, n), p * 10.0 ** rng.uniform(-6, 6, n)
        u = np.where(rng.random(n) < 0.3, 0.0, u * 10.0 ** rng.uniform(-40, 3, n))
    return rho, u, v, p


@pytest.mark.parametrize("loop", ["cell", "tile"])
@pytest.mark.parametrize("flux,limiter,viscous", [
    ("ausm", "minmod", False), ("ausm", "venkat", False), ("ausm", "vanleer", False), ("ausm", "vanalbada", False),
    ("ausm", "none", False), ("roe", "minmod", False), ("ausm", "venkat", True), ("ausm", "minmod", True)])
def test_every_magnitude_steps_as_the_oracle(pkg, orc, loop, flux, limiter, viscous):
    if viscous:
        mesh, cfg, _ = pkg.cases.cylinder_case(33, mach=2.0, flux=flux, limiter=limiter)
        cfg = dict(cfg, mu_ref=1e-3, T_ref=300.0, thermo=dict(cfg["thermo"], RGAS=0.7 / 300.0))
    else:
        mesh, cfg, _ = pkg.cases.square_inviscid(33, flux=flux, limiter=limiter)
    cfg = dict(cfg, init_nodes=1, CFL=0.05)
    prims = _state(mesh, 3, wild=False)
    o = orc.Oracle(mesh, cfg, nthreads=2)
    o.init_fields(*prims)
    s = pkg.setupSolver(mesh, cfg, loop=loop)
    s.createFields2d(0, *prims)
    for _ in range(3):
        bad = o.step()["nonfinite"]
        try:
            s.propagate2d(1)
            assert not bad
        except pkg._native.NativeError as e:
            assert bad and e.code == -4
        g = s.get_state(0)
        assert np.array_equal(g["Ucons"], o.field("Uold"), equal_nan=True), (loop, flux, limiter)
        assert np.array_equal(g["prims"], o.prims(), equal_nan=True)
        assert np.array_equal(g["node_prims"], o.node_prims(), equal_nan=True)
        if bad:  # the next time step of a failed state is not defined
            break
    s.close()


@pytest.mark.parametrize("flux", ["ausm", "roe"])
@pytest.mark.parametrize("limiter", ["minmod", "venkat", "vanleer", "vanalbada"])
def test_wild_states_give_the_oracles_fluxes(pkg, orc, flux, limiter):
    """States over tens of decades, whose reconstructions are negative,
    infinite or NaN on many faces: the fluxes are the plain formulas'."""
    mesh, cfg, _ = pkg.cases.square_inviscid(33, flux=flux, limiter=limiter)
    cfg = dict(cfg, init_nodes=1)
    prims = _state(mesh, 5, wild=True)
    o = orc.Oracle(mesh, cfg, nthreads=2)
    o.init_fields(*prims)
    s = pkg.setupSolver(mesh, cfg)
    s.createFields2d(0, *prims)
    F, Un = s.calcOneStageMUSCLcpuFast(0, 1.0, 1e-6, 0.0)
    o.calc_one_stage(1.0, 1e-6, 0.0)
    assert np.array_equal(F, o.field("FLUXES"), equal_nan=True)
    assert np.array_equal(Un, o.field("Unew"), equal_nan=True)
    s.close()
