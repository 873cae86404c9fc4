"""gd2d_last_timing reports the call it follows: no time of a call that took
no step, none of a launch shape that is no longer in use."""
import pytest

pytestmark = pytest.mark.gpu


def test_cell_time_is_not_of_an_older_call(pkg):
    mesh, cfg, prims = pkg.cases.square_inviscid(41)
    s = pkg.setupSolver(mesh, cfg)
    s.createFields2d(0, *prims)
    for steps in (1, 3, 64, 65, 1):  # the graphs' steps, several left over, a single one
        s.propagate2d(steps)
        total, cell, launches = s.last_timing()
        assert 0.0 < cell <= total and launches == 2 * steps, steps
    s.propagate2d(0)
    assert s.last_timing() == (0.0, 0.0, 0)
    s.close()


def test_cell_time_is_not_of_another_launch_shape(pkg):
    mesh, cfg, prims = pkg.cases.square_inviscid(41)
    s = pkg.setupSolver(mesh, cfg)
    s.createFields2d(0, *prims)
    for _ in range(2):
        s.propagate2d(1)
    s.autotune(steps_per_trial=8)
    assert s.last_timing()[1] == 0.0  # none of the shape chosen was timed
    s.propagate2d(1)
    total, cell, _ = s.last_timing()
    assert 0.0 < cell <= total
    s.close()
