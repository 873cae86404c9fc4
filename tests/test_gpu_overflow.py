"""Viscous terms whose Green-Gauss quotients leave the range of doubles.

The FP64 path follows IEEE division there too: an edge sum over a small area
overflows to an infinity, not to NaN, in the first gradient and in the
Laplacian, as the CPU oracle has it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quads", [False, True])
@pytest.mark.parametrize("viscosity", ["constant", "sutherland", "reference"])
def test_overflowing_quotients_give_the_oracles_infinities(pkg, orc, viscosity, quads):
    mesh = pkg.mesh.structured_mesh(13, 13, 0.0, 1.0e-5, 0.0, 1.0e-5, quads=quads)
    g = 1.4
    cfg = {"thermo": dict(pkg.cases.AIR), "flux": "ausm", "limiter": "minmod", "viscosity": viscosity,
           "art_viscosity": 1, "mu_ref": 1e-3, "T_ref": 300.0, "Pr": 0.72, "dt_mode": 0, "dt": 1e-9, "CFL": 0.4,
           "init_nodes": 1, "bc": [{"tag": -1, "kind": "outflow"}, {"tag": -2, "kind": "outflow"},
                                   {"tag": -3, "kind": "outflow"}]}
    n = mesh.nCells
    infinite = 0
    # one cell so fast that its energy over an edge of 1e-6 (a quotient 1e6
    # times as large, or twice that often) passes 1.8e308
    for e in (146.0, 147.2, 148.0, 149.6, 151.0, 152.6):
        u = np.full(n, 2.0)
        u[n // 2] = 10.0 ** e
        prims = (np.full(n, 1.2), u, np.full(n, 0.1), np.full(n, 1.0e5 / g))
        o = orc.Oracle(mesh, cfg, nthreads=2)
        o.init_fields(*prims)
        o.calc_diff_term()
        s = pkg.setupSolver(mesh, cfg)
        s.createFields2d(0, *prims)
        D, ref = s.calcDiffTerm(0), np.array(o.field("Diff"))
        s.close()
        infinite += int(np.isinf(ref).sum())
        assert np.array_equal(D, ref, equal_nan=True), e
    assert infinite > 0  # (the case does what it is for)
