"""Two FP64 red-black sweeps per pass from the symmetric operator: strips of 116 columns, segments of at least 20
rows, even and odd sweep counts of the red-black solver (the odd one's last sweep runs by itself), and other
multigrid sweep counts, which run on the general kernels. Bit for bit the oracle's."""
from __future__ import annotations

import pytest

from conftest import bit_equal, config_text, cuda_available, describe_diff, snapshot_config

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]


def _check(sgpu_mod, oracle_mod, nx, ny, its, **kw):
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re="700", momentum_solver="gs_multicolour", maxit=str(its),
               error_tolerance="0", **kw)
    p = sgpu_mod.params_from_config(config_text(cfg))
    o = oracle_mod.Oracle(p)
    _, _, olog = o.run(its)
    with sgpu_mod.Solver(p) as g:
        _, log = g.run(its)
        assert bit_equal(log, olog), describe_diff(log, olog)
        for f in (0, 1, 2, sgpu_mod.F_PC):
            assert bit_equal(g.download(f), o.get(f)), f"field {f}: " + describe_diff(g.download(f), o.get(f))


@pytest.mark.parametrize("nx,ny,sweeps", [(1, 3, 1), (2, 2, 2), (20, 116, 2), (21, 117, 3), (41, 232, 4), (19, 233, 5),
                                          (130, 349, 8), (349, 5, 6)])
def test_red_black_solver(sgpu_mod, oracle_mod, nx, ny, sweeps):
    _check(sgpu_mod, oracle_mod, nx, ny, 4, pressure_solver="gs_redblack", maxit_inner_p=str(sweeps))


@pytest.mark.parametrize("nx,ny,pre,post", [(256, 232, 2, 2), (168, 704, 2, 2), (328, 352, 2, 1), (256, 464, 3, 2),
                                            (360, 348, 2, 2), (2048, 20, 2, 2)])
def test_v_cycle(sgpu_mod, oracle_mod, nx, ny, pre, post):
    _check(sgpu_mod, oracle_mod, nx, ny, 3, pressure_solver="mg", mg_pre=str(pre), mg_post=str(post))


@pytest.mark.parametrize("nx,ny,sweeps", [(10400, 116, 2), (10300, 117, 3), (5200, 232, 4), (5170, 233, 5), (3450, 349, 8),
                                          (40, 30011, 6)])
def test_red_black_solver_in_two_sweep_passes(sgpu_mod, oracle_mod, nx, ny, sweeps):
    """The same at the size from which a single solve takes two sweeps a pass (smaller ones launch a colour each)."""
    assert nx * ny > 1200000
    _check(sgpu_mod, oracle_mod, nx, ny, 2, pressure_solver="gs_redblack", maxit_inner_p=str(sweeps))


@pytest.mark.parametrize("nx,ny,sweeps", [(1, 3, 1), (2, 2, 2), (20, 116, 2), (21, 117, 3), (41, 232, 4), (19, 233, 5),
                                          (130, 349, 8), (349, 5, 6)])
def test_red_black_solver_of_a_batch_cavity(sgpu_mod, oracle_mod, nx, ny, sweeps):
    """The cavities of a batch of more than eight take two sweeps a pass at any size."""
    cfg = dict(snapshot_config("short_16"))
    cfg.update(Re="700", momentum_solver="gs_multicolour", maxit="4", error_tolerance="0", pressure_solver="gs_redblack",
               maxit_inner_p=str(sweeps))
    big = sgpu_mod.params_from_config(config_text(dict(cfg, N_cells_x="400", N_cells_y="300")))
    p = sgpu_mod.params_from_config(config_text(dict(cfg, N_cells_x=str(nx), N_cells_y=str(ny))))
    o = oracle_mod.Oracle(p)
    o.run(4)
    with sgpu_mod.Batch([big] * 8 + [p]) as b:
        b.run(4)
        for f in (0, 1, 2, sgpu_mod.F_PC):
            assert bit_equal(b.download(8, f), o.get(f)), f"field {f}: " + describe_diff(b.download(8, f), o.get(f))
