"""Which cases take the straight-line quotients: not those with an area or
size whose significand is all ones, the method's exception, but a cell whose
lower 32 bits alone are set must not turn its whole mesh over to the slower
formulas (on 2.09M cells one mesh in a thousand has such a cell)."""
import dataclasses
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "2d-dns-godunov-solver-_b200", "csrc")


def test_cases_in_range(tmp_path):
    exe = str(tmp_path / "exact_case_check")
    subprocess.check_call(["/usr/local/cuda/bin/nvcc", "-O1", "-std=c++17", "-I" + CSRC,
                           os.path.join(HERE, "exact_case_check.cu"), "-o", exe])
    got = [int(x) for x in subprocess.check_output([exe], text=True).split()]
    assert got == [1, 1, 1, 1, 0, 0, 0, 0, 0, 0]


@pytest.mark.gpu
def test_low_word_of_ones_rounds_as_the_oracle(pkg, orc):
    mesh, cfg, _ = pkg.cases.cylinder_case(33, mach=2.0)
    r = np.random.default_rng(21)
    n = mesh.nCells

    def low_ones(a):
        return (np.ascontiguousarray(a).view(np.uint64) | np.uint64(0xffffffff)).view(np.float64)

    mesh = dataclasses.replace(mesh, cell_areas=low_ones(mesh.cell_areas), HX=low_ones(mesh.HX))
    rho, u, p = (c * (1.0 + 0.1 * r.uniform(-1, 1, n)) for c in (1.1766, 700.0, 101325.0))
    prims, cfg = (rho, u, 70.0 * r.uniform(-1, 1, n), p), dict(cfg, init_nodes=1, CFL=0.05)
    for loop in ("tile", "cell"):
        o = orc.Oracle(mesh, cfg, nthreads=2)
        o.init_fields(*prims)
        o.calc_diff_term()
        s = pkg.setupSolver(mesh, cfg, loop=loop)
        s.createFields2d(0, *prims)
        assert np.array_equal(s.calcDiffTerm(0), o.field("Diff"))
        o.run(3)
        s.propagate2d(3)
        assert np.array_equal(s.get_state(0)["Ucons"], o.field("Uold"))
        s.close()
