"""The kernels that a mesh's size, its face order or a case's constants choose.

Register budgets and node blocks that the defaults take only for some sizes,
the node passes and the step reduction of large mixed meshes, the gradient
passes of a mesh whose cells do not list their edges as a closed walk, and
cases out of the range of the straight-line quotients.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Ucons", "prims", "node_prims")


def _disturbed(mesh, seed, rho, u, p):
    r = np.random.default_rng(seed)
    n = mesh.nCells
    return (rho * (1.0 + 0.1 * r.uniform(-1, 1, n)), u * (1.0 + 0.1 * r.uniform(-1, 1, n)),
            0.1 * u * r.uniform(-1, 1, n), p * (1.0 + 0.1 * r.uniform(-1, 1, n)))


def _quad_box(pkg, flux="ausm", limiter="minmod", viscosity="none", n=33):
    mesh = pkg.mesh.structured_mesh(n, n - 4, 0.0, 1.0, 0.0, 0.8, quads=True, jitter=0.1, seed=4)
    cfg = {"thermo": dict(pkg.cases.AIR, RGAS=0.7 / 300.0), "flux": flux, "limiter": limiter, "viscosity": viscosity,
           "art_viscosity": int(viscosity != "none"), "mu_ref": 1e-3, "T_ref": 300.0, "Pr": 0.72, "dt_mode": 2,
           "CFL": 0.1, "init_nodes": 1, "bc": [{"tag": -1, "kind": "inflow", "rho": 1.0, "u": 2.0, "v": 0.0, "p": 0.7},
                                               {"tag": -2, "kind": "outflow"}, {"tag": -3, "kind": "slip"}]}
    return mesh, cfg, _disturbed(mesh, 7, 1.0, 2.0, 0.7)


def _run(pkg, mesh, cfg, prims, steps, **launch):
    s = pkg.setupSolver(mesh, cfg, **launch)
    s.createFields2d(0, *prims)
    s.propagate2d(steps)
    st, h = s.get_state(0), s.history(0)
    s.close()
    return st, h


def _against_oracle(pkg, orc, cases, steps, **launch):
    """One handle of (mesh, cfg, prims) cases, step by step beside an oracle
    each: the same bits, and a state that left the admissible set reported
    when the oracle's did (and not stepped further)."""
    s = pkg.solver.Solver([m for m, _, _ in cases], [c for _, c, _ in cases], pkg.solver.make_launch(**launch))
    oracles = []
    for i, (mesh, cfg, prims) in enumerate(cases):
        s.createFields2d(i, *prims)
        oracles.append(orc.Oracle(mesh, cfg, nthreads=2))
        oracles[-1].init_fields(*prims)
    for step in range(steps):
        bad = any([o.step()["nonfinite"] for o in oracles])
        try:
            s.propagate2d(1)
            assert not bad
        except pkg._native.NativeError as e:
            assert bad and e.code == -4
        for i, o in enumerate(oracles):
            g = s.get_state(i)
            assert np.array_equal(g["Ucons"], o.field("Uold"), equal_nan=True), (launch, step, i)
            assert np.array_equal(g["prims"], o.prims(), equal_nan=True), (launch, step, i)
            assert np.array_equal(g["node_prims"], o.node_prims(), equal_nan=True), (launch, step, i)
        if bad:
            break
    s.close()


# ------------------------------------------------------------ launch shapes


@pytest.mark.parametrize("loop", ["tile", "cell"])
@pytest.mark.parametrize("case", ["cylinder", "square roe", "quads", "quads viscous"])
def test_pinned_launch_shapes_agree(pkg, case, loop):
    """Every shape against a pinned one, none against the defaults, whose
    choice depends on the mesh."""
    if case == "cylinder":
        mesh, cfg, prims = pkg.cases.cylinder_case(97)
    elif case == "square roe":
        mesh, cfg, prims = pkg.cases.square_inviscid(65, flux="roe", limiter="vanalbada")
    else:
        mesh, cfg, prims = _quad_box(pkg, viscosity="sutherland" if "viscous" in case else "none")
    ref, href = _run(pkg, mesh, cfg, prims, 20, loop=loop, min_blocks=4, node_block=64)
    for min_blocks, node_block in ((2, 64), (3, 64), (2, 128), (3, 128), (3, 256), (4, 128)):
        got, hgot = _run(pkg, mesh, cfg, prims, 20, loop=loop, min_blocks=min_blocks, node_block=node_block)
        for k in FIELDS:
            assert np.array_equal(ref[k], got[k]), (min_blocks, node_block, k)
        assert href == hgot, (min_blocks, node_block)


# ------------------------------------------------------- large mixed meshes


@pytest.mark.parametrize("loop", ["tile", "cell"])
def test_large_mixed_mesh(pkg, loop):
    """A viscous mesh of 160,000 nodes (one thread a node in the gradient node
    pass) and five tile groups (the step reduction over groups): ten steps
    against the FP64 path, each step's density within the mixed path's
    rounding (relative L2 1e-6: ten steps of a few FP32 roundings, 6e-8
    each, times the CFL number), and the statistics against the fields."""
    mesh, cfg, prims = pkg.cases.cylinder_case(400)
    assert mesh.nNodes > 100000 and mesh.nCells > 4 * 65536
    f64, _ = _run(pkg, mesh, cfg, prims, 10)
    s = pkg.setupSolver(mesh, cfg, precision="mixed", loop=loop)
    s.createFields2d(0, *prims)
    s.propagate2d(9)
    before = s.get_state(0)
    st = s.propagate2d(1)[0]
    after = s.get_state(0)
    s.close()
    U, ref = after["Ucons"], f64["Ucons"]
    assert np.sqrt(((U[:, 0] - ref[:, 0]) ** 2).sum() / (ref[:, 0] ** 2).sum()) < 1e-6
    assert st["rhoMin"] == before["prims"][:, 0].min() and st["rhoMax"] == before["prims"][:, 0].max()
    # areas are held in FP32: 6e-8 each; the residual's sums in FP64
    A = mesh.cell_areas[:, None]
    scale = np.abs(U * A).sum(axis=0)
    assert np.all(np.abs(np.array(st["totals"]) - (U * A).sum(axis=0)) <= 1e-7 * scale)
    dU = U - before["Ucons"]
    assert np.allclose(st["residual"], (dU * dU).sum(axis=0), rtol=1e-9, atol=0)


# -------------------------------------------------- cells that are no walks


def _no_walks(mesh):
    """Every third quad lists its faces in the order 0, 2, 1, 3."""
    rows = np.arange(0, mesh.nCells, 3)
    new = {}
    for name in ("cell_stiffness", "cell_edges_Nx", "cell_edges_Ny", "cell_edges_length"):
        a = np.array(getattr(mesh, name))
        a[rows, 1], a[rows, 2] = a[rows, 2].copy(), a[rows, 1].copy()
        new[name] = np.asfortranarray(a)
    for name in ("cells2nodes", "node2cellL2up", "node2cellL2down"):
        a = np.array(getattr(mesh, name))
        x = a[rows, 2:4].copy()
        a[rows, 2:4], a[rows, 4:6] = a[rows, 4:6].copy(), x
        new[name] = np.asfortranarray(a)
    return dataclasses.replace(mesh, **new)


@pytest.mark.parametrize("limiter", ["minmod", "venkat"])
def test_faces_out_of_walking_order_f64(pkg, orc, limiter):
    mesh, cfg, prims = _quad_box(pkg, limiter=limiter, viscosity="sutherland")
    mesh = _no_walks(mesh)
    for loop in ("tile", "cell"):
        _against_oracle(pkg, orc, [(mesh, cfg, prims)], 5, loop=loop)
    o = orc.Oracle(mesh, cfg, nthreads=2)
    o.init_fields(*prims)
    o.calc_diff_term()
    s = pkg.setupSolver(mesh, cfg)
    s.createFields2d(0, *prims)
    assert np.array_equal(s.calcDiffTerm(0), o.field("Diff"))
    s.close()


@pytest.mark.parametrize("loop", ["tile", "cell"])
def test_faces_out_of_walking_order_mixed(pkg, orc, loop):
    """Within the mixed path's acceptance bound, as its other viscous runs."""
    mesh, cfg, prims = _quad_box(pkg, viscosity="sutherland")
    mesh = _no_walks(mesh)
    o = orc.Oracle(mesh, cfg, nthreads=2)
    o.init_fields(*prims)
    o.run(5)
    st, _ = _run(pkg, mesh, cfg, prims, 5, precision="mixed", loop=loop)
    d, ref = st["Ucons"] - o.field("Uold"), o.field("Uold")
    assert (np.sqrt((d * d).sum(axis=0)) / np.sqrt((ref * ref).sum(axis=0)))[[0, 1, 3]].max() < 1e-5


# ------------------------------- out of range of the straight-line quotients


@pytest.mark.parametrize("viscous", [False, True])
def test_cases_in_and_out_of_range_in_one_handle(pkg, orc, viscous):
    """gamma 1.004 is out of the range: its case steps by the plain formulas
    beside one that does not."""
    cases = []
    for k, gamma in enumerate((1.4, 1.004)):
        if viscous:
            mesh, cfg, _ = pkg.cases.cylinder_case(33 + 4 * k, mach=2.0)
            cfg = dict(cfg, mu_ref=1e-3, T_ref=300.0)
            prims = _disturbed(mesh, 9 + k, 1.0, 2.0, 0.7)
        else:
            mesh, cfg, prims = pkg.cases.square_inviscid(33 + 4 * k, seed=3 + k)
        cases.append((mesh, dict(cfg, CFL=0.05, init_nodes=1,
                                 thermo=dict(cfg["thermo"], Gamma=gamma, RGAS=0.7 / 300.0)), prims))
    for loop in ("tile", "cell"):
        for group in (cases, cases[::-1], cases[1:]):
            _against_oracle(pkg, orc, group, 4, loop=loop)


# --------------------------------------------- Roe with quads and viscosity


@pytest.mark.parametrize("loop", ["tile", "cell"])
@pytest.mark.parametrize("case", ["quads", "quads viscous", "cylinder"])
def test_roe_at_every_magnitude(pkg, orc, case, loop):
    """A velocity component from ordinary down to denormals and exact zero."""
    if case == "cylinder":
        mesh, cfg, _ = pkg.cases.cylinder_case(33, mach=2.0, flux="roe")
        cfg = dict(cfg, mu_ref=1e-3, T_ref=300.0, CFL=0.05, init_nodes=1,
                   thermo=dict(cfg["thermo"], RGAS=0.7 / 300.0))
    else:
        mesh, cfg, _ = _quad_box(pkg, flux="roe", viscosity="sutherland" if "viscous" in case else "none")
        cfg = dict(cfg, CFL=0.05)
    rho, u, v, p = _disturbed(mesh, 13, 1.0, 2.0, 0.7)
    r = np.random.default_rng(14)
    x = mesh.cell_mid_points[:, 0] - mesh.cell_mid_points[:, 0].min()
    v = np.where(r.random(mesh.nCells) < 0.2, 0.0, np.sign(v) * 10.0 ** (-330.0 * (x / x.max()) ** 1.5))
    _against_oracle(pkg, orc, [(mesh, cfg, (rho, u, v, p))], 3, loop=loop)
