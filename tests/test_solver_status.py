"""A pressure solve that runs past 100 iterations stops the solver the way the
reference's does (vfsph_div / vfsph_incomp flag a crash, DFSPHCudaImpl.cu:449-503,
and DFSPHSolver::tick stops ticking, DFSPHSolver.cpp:339-406): tickNsteps fails
after that substep, later ticks fail at once, and with "stopOnNonConvergence": false
the run goes on to the requested substeps and reports the status at the end."""
import pytest

import vtp
from vtp import scenes

pytestmark = pytest.mark.gpu


def _unreachable(kind="DFSPH"):
    sc = scenes.dam_break(kind, 3000, seed=35)
    sc.config[kind]["Required"]["divFreeThreshold"] = 1e-12   # the residual never gets there
    return sc


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("n", [1, 3])
def test_solve_past_100_iterations_stops_the_solver(vtp_gpu, graphs, n):
    s = vtp.solver_from_scene(_unreachable(), extra={"useGraphs": graphs})
    s.strict = False    # the reference's API: tickNsteps returns false and logs the error
    assert s.initialize()
    assert not s.tickNsteps(n)
    assert "exceeded 100 iterations" in s.last_error
    assert s.stats()["steps_done"] == 1          # stopped after the first substep
    assert not s.tickNsteps(1) and "crashed" in s.last_error
    s.destroy()


def test_without_stop_the_run_reports_at_the_end(vtp_gpu):
    s = vtp.solver_from_scene(_unreachable(), extra={"stopOnNonConvergence": False})
    s.strict = False
    assert s.initialize()
    assert not s.tickNsteps(3)
    assert "solver status after tick" in s.last_error
    assert s.stats()["status_bits"] & (1 << 3)    # ST_NOT_CONVERGED
    s.destroy()


def test_one_call_frame_reports_the_stop(vtp_gpu):
    sc = _unreachable()
    s = vtp.solver_from_scene(sc)
    s.strict = False
    assert s.initialize()
    nf = sc.objects[0].n
    p, v = vtp.HostBuffer((nf, 3)), vtp.HostBuffer((nf, 3))
    s.get_state_range_ptr(0, nf, p.ptr, v.ptr)
    assert not s.step_state_range_ptr(0, nf, p.ptr, v.ptr, 2, p.ptr, v.ptr)
    assert "exceeded 100 iterations" in s.last_error and s.stats()["steps_done"] == 1
    p.free()
    v.free()
    s.destroy()


@pytest.mark.parametrize("kind", ["DFSPH", "IMM", "IMMCT"])
def test_host_driven_solves_start_from_the_solver_s_state(vtp_gpu, kind):
    """"deviceLoop": false runs the solves from the host, without graphs, from the state the caller has
    set: the same bits as the captured substeps."""
    import numpy as np
    sc = (scenes.dam_break("DFSPH", 5000, seed=3) if kind == "DFSPH" else scenes.layered_mixture(kind, 14, seed=3))
    rng = np.random.default_rng(1)
    fluid = np.concatenate([np.full(o.n, o.material == 0) for o in sc.objects])
    vel = np.where(fluid[:, None], 0.05 * rng.standard_normal((fluid.size, 3)), 0.0).astype(np.float32)
    got = []
    for extra in ({}, {"useGraphs": False}, {"deviceLoop": False}):
        s = vtp.solver_from_scene(sc, extra=extra)
        assert s.initialize(), s.last_error
        s.set_field("vel", vel)
        assert s.tickNsteps(3), s.last_error
        got.append([s.get_field("pos"), s.get_field("vel")] + ([s.get_field("vol_frac")] if kind != "DFSPH" else []))
        s.destroy()
    for other in got[1:]:
        for x, y in zip(got[0], other):
            assert np.array_equal(x, y)
