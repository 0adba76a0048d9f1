"""mg_mode = tolerance in Solver.run: the V-cycle loop is a conditional node of the captured iteration. It takes
the host loop's decisions: same cycles, residuals, fields and p' as outer_iteration, bit for bit, on grids with
and without streamed levels, with one cycle and many, at the cycle cap, from rest, and across changes of mode."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bit_equal, config_text, cuda_available, describe_diff, snapshot_config

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]


def _params(sgpu_mod, nx, ny, precision, **kw):
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re="600", momentum_solver="gs_multicolour", pressure_solver="mg",
               precision=precision, maxit="100", error_tolerance="0", mg_mode="tolerance", **kw)
    return sgpu_mod.params_from_config(config_text(cfg))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,kw", [(16, 16, {}), (33, 20, {}), (64, 96, {"pressure_tolerance": "1e-8"}),
                                      (160, 320, {"pressure_tolerance": "0.5"}),
                                      (300, 280, {"pressure_tolerance": "1e-9", "pressure_maxit": "4"})])
def test_run_equals_host_issued_iterations(sgpu_mod, precision, nx, ny, kw):
    p = _params(sgpu_mod, nx, ny, precision, **kw)
    fields = (0, 1, 2, sgpu_mod.F_PC)
    with sgpu_mod.Solver(p) as a, sgpu_mod.Solver(p) as b:
        for n in (1, 3, 2):  # the second and third run replay the graph
            _, log = a.run(n)
            rows = np.array([b.outer_iteration() for _ in range(n)])
            assert bit_equal(np.ascontiguousarray(log[:, 1:]), rows)
            assert a.last_solve_stats() == b.last_solve_stats()
            for f in fields:
                assert bit_equal(a.download(f), b.download(f)), f"field {f}: " + describe_diff(a.download(f), b.download(f))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_run_follows_changes_of_mode(sgpu_mod, precision):
    p = _params(sgpu_mod, 96, 64, precision)
    with sgpu_mod.Solver(p) as a, sgpu_mod.Solver(p) as b:
        for mode in ((False,), (True, 1e-3, 50), (True, 1e-6, 50), (True, 1e-6, 2), (False,)):
            a.set_mg_mode(*mode)
            b.set_mg_mode(*mode)
            _, log = a.run(2)
            rows = np.array([b.outer_iteration() for _ in range(2)])
            assert bit_equal(np.ascontiguousarray(log[:, 1:]), rows)
            for f in (0, 1, 2, sgpu_mod.F_PC):
                assert bit_equal(a.download(f), b.download(f)), f"{mode}, field {f}"


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solve_p_after_run_has_its_own_statistics(sgpu_mod, precision):
    """The statistics are those of the last p' solve, a per-phase one after a run included."""
    p = _params(sgpu_mod, 64, 96, precision, pressure_tolerance="1e-7")
    with sgpu_mod.Solver(p) as a, sgpu_mod.Solver(p) as b:
        a.run(2)
        for _ in range(2):
            b.outer_iteration()
        for s in (a, b):
            for f in (0, 1):
                s.upload(f, 1e3 * s.download(f))  # another solve than the run's last
            s.assemble_u(), s.assemble_v(), s.assemble_p()
            s.solve_p()
        assert a.last_solve_stats() == b.last_solve_stats()
        assert a.warm_start_stats() == b.warm_start_stats()
        assert bit_equal(a.download(sgpu_mod.F_PC), b.download(sgpu_mod.F_PC))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_launch_count_holds_every_cycle(sgpu_mod, precision):
    """sgpu_launch_count counts the kernels of each cycle of a captured solve, not those of one: the launches of a
    run grow with the cycles it does as those of host-issued iterations do."""
    def launches(cap, host):
        p = _params(sgpu_mod, 160, 96, precision, pressure_tolerance="1e-300", pressure_maxit=str(cap))
        with sgpu_mod.Solver(p) as s:
            s.run(2)  # builds the graph
            before = sgpu_mod.launch_count()
            if host:
                for _ in range(5):
                    s.outer_iteration()
            else:
                s.run(5)
            assert s.last_solve_stats()["mg_vcycles"] == cap
            return sgpu_mod.launch_count() - before
    run = [launches(c, False) for c in (1, 2, 5)]
    host = [launches(c, True) for c in (1, 2)]
    assert run[2] - run[1] == 3 * (run[1] - run[0])
    assert run[1] - run[0] >= host[1] - host[0] > 0


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", [(5, 1), (1, 1)])
def test_solves_of_no_cycle(sgpu_mod, precision, nx, ny):
    """One column of cells has no u cells, so the lid drives nothing: b is zero, the loop runs no cycle, and p' and
    the statistics are those of the host's early return, not the previous solve's."""
    p = _params(sgpu_mod, nx, ny, precision)
    with sgpu_mod.Solver(p) as a, sgpu_mod.Solver(p) as b:
        for n in (1, 2):
            _, log = a.run(n)
            rows = np.array([b.outer_iteration() for _ in range(n)])
            assert bit_equal(np.ascontiguousarray(log[:, 1:]), rows) and not rows[:, 2].any()
            assert a.last_solve_stats() == b.last_solve_stats()
            assert a.last_solve_stats()["mg_vcycles"] == 0
            for f in (0, 1, 2, sgpu_mod.F_PC):
                assert bit_equal(a.download(f), b.download(f)), f"field {f}"
        # a solve of no cycle after one of several: its p' is zero again
        for s in (a, b):
            s.upload(sgpu_mod.F_V, np.random.default_rng(2).standard_normal(s.shape))
        for n in (1, 1):
            _, log = a.run(n)
            assert bit_equal(np.ascontiguousarray(log[:, 1:]), np.array([b.outer_iteration()]))
            assert a.last_solve_stats() == b.last_solve_stats()
            assert bit_equal(a.download(sgpu_mod.F_PC), b.download(sgpu_mod.F_PC))
        for s in (a, b):
            for f in (0, 1, 2):
                s.upload(f, np.zeros(s.shape))
        _, log = a.run(1)
        assert bit_equal(np.ascontiguousarray(log[:, 1:]), np.array([b.outer_iteration()]))
        for f in (0, 1, 2, sgpu_mod.F_PC):
            assert bit_equal(a.download(f), b.download(f)), f"field {f}"
        assert not a.download(sgpu_mod.F_PC).any() and a.last_solve_stats()["mg_vcycles"] == 0


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_graphs_of_both_modes_side_by_side(sgpu_mod, precision):
    """Switching between the modes keeps each one's graph: runs of either between runs of the other, tolerances that
    change and come back, and host-issued iterations in between give the host's results, p' and statistics too."""
    p = _params(sgpu_mod, 64, 96, precision)
    plan = [(False,), (True, 1e-6, 50), (False,), (True, 1e-6, 50), (False, 1e-3, 7), (True, 1e-2, 50), (True, 1e-6, 50), (False,)]
    with sgpu_mod.Solver(p) as a, sgpu_mod.Solver(p) as b:
        for k, mode in enumerate(plan):
            a.set_mg_mode(*mode)
            b.set_mg_mode(*mode)
            for hosted in ((True, False) if k % 3 == 2 else (False,)):
                rows = np.array([b.outer_iteration() for _ in range(2)])
                log = np.array([a.outer_iteration() for _ in range(2)]) if hosted else np.ascontiguousarray(a.run(2)[1][:, 1:])
                assert bit_equal(log, rows), f"{k}: {mode}"
            got, want = a.last_solve_stats(), b.last_solve_stats()
            assert got == want, f"{k}: {mode}"
            for f in (0, 1, 2, sgpu_mod.F_PC):
                assert bit_equal(a.download(f), b.download(f)), f"{k}: {mode}, field {f}"
