"""Device-side failure detection, tested without a GPU fault.

The mixed mode's correction sweep waits on mbarriers for the record copies it issues. Every such wait
is bounded: one that runs out sets a device word, which sgpu_run and sgpu_batch_run report as
SGPU_E_TIMEOUT, instead of hanging the GPU. sgpu_selftest_bounded_wait runs that same wait helper
on an mbarrier that nothing ever completes. The wait must give up and say so, and the context must
stay usable: a solve right after it runs normally.
"""
from __future__ import annotations

import pytest

from conftest import config_text, cuda_available, snapshot_config


@pytest.mark.parametrize("polls", [1, 4096])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_bounded_wait_gives_up_and_reports(sgpu_mod, polls):
    assert sgpu_mod.selftest_bounded_wait(polls)


@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_context_usable_after_a_give_up(sgpu_mod):
    assert sgpu_mod.selftest_bounded_wait(4096)
    cfg = snapshot_config("short_16")
    cfg.update(N_cells_x="48", N_cells_y="48", momentum_solver="gs_multicolour", pressure_solver="mg",
               precision="mixed", maxit="5", error_tolerance="0")
    with sgpu_mod.Solver(sgpu_mod.params_from_config(config_text(cfg))) as s:
        res, log = s.run(5)
    assert res.iterations == 5 and log.shape[0] == 5


def test_selftest_rejects_bad_arguments(sgpu_mod):
    # checked before any device work, so this runs without a GPU
    for polls in (0, -3, (1 << 20) + 1):
        with pytest.raises(sgpu_mod.SgpuError, match="polls"):
            sgpu_mod.selftest_bounded_wait(polls)


@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
@pytest.mark.parametrize("call", ["solve_p", "outer_iteration", "run"])
@pytest.mark.parametrize("n,kw", [(40, {"pressure_solver": "cg"}), (300, {"pressure_solver": "mg"}),
                                  (48, {"pressure_solver": "mg", "precision": "mixed"})])
def test_every_solving_call_reports_a_give_up(sgpu_mod, n, kw, call):
    """A wait that gave up during a call is that call's error, whichever entry point it is; the call after it is a
    solver's that never had one."""
    cfg = snapshot_config("short_16")
    cfg.update(N_cells_x=str(n), N_cells_y=str(n), momentum_solver="gs_multicolour", maxit="9", error_tolerance="0", **kw)
    p = sgpu_mod.params_from_config(config_text(cfg))
    go = {"solve_p": lambda s: s.solve_p(), "outer_iteration": lambda s: s.outer_iteration(), "run": lambda s: s.run(1)}[call]
    with sgpu_mod.Solver(p) as a, sgpu_mod.Solver(p) as b:
        for s in (a, b):
            s.assemble_u(), s.assemble_v(), s.assemble_p()
        a.selftest_set_timeout()
        with pytest.raises(sgpu_mod.SgpuError) as e:
            go(a)
        assert e.value.code == sgpu_mod.E_TIMEOUT
        zero = a.download(0) * 0.0
        for s in (a, b):  # the same fields in both, whatever the failed call left
            for f in (0, 1, 2):
                s.upload(f, zero)
            s.assemble_u(), s.assemble_v(), s.assemble_p()
            go(s)
        for f in (0, 1, 2, sgpu_mod.F_PC):
            assert (a.download(f) == b.download(f)).all()


@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_no_bounded_wait_to_fail(sgpu_mod):
    cfg = snapshot_config("short_16")
    cfg.update(momentum_solver="jacobi", pressure_solver="jacobi")
    with sgpu_mod.Solver(sgpu_mod.params_from_config(config_text(cfg))) as s:
        with pytest.raises(sgpu_mod.SgpuError, match="no bounded waits"):
            s.selftest_set_timeout()
