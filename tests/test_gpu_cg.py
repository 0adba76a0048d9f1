"""Conjugate gradients for p' (solve_pc_cg, pressure.cpp:208-317) in one kernel and pass by pass: grids of one
CTA and of many, one row per CTA, chunk remainders, narrow and wide, the first size that takes the
pass-by-pass kernels; iteration caps and loose tolerances. Bit for bit the oracle's, iteration counts too."""
from __future__ import annotations

import pytest

from conftest import bit_equal, config_text, cuda_available, describe_diff, snapshot_config

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("nx,ny,kw", [
    (1, 5, {}), (5, 1, {}), (7, 9, {}), (20, 33, {}), (33, 64, {}), (64, 65, {}), (150, 128, {}), (149, 129, {}),
    (300, 257, {}), (3, 500, {}), (500, 3, {}), (40, 50, {"pressure_maxit": "3"}), (40, 50, {"pressure_tolerance": "0.5"}),
    (296, 300, {"pressure_maxit": "40"}), (1400, 1310, {"pressure_maxit": "2"})])
def test_cg_bit_for_bit(sgpu_mod, oracle_mod, nx, ny, kw):
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re="400", momentum_solver="gs_multicolour", pressure_solver="cg",
               maxit="2", error_tolerance="0", **kw)
    p = sgpu_mod.params_from_config(config_text(cfg))
    o = oracle_mod.Oracle(p)
    with sgpu_mod.Solver(p) as g:
        for _ in range(2):
            ro, rg = o.outer_iteration(), g.outer_iteration()
            assert rg == ro
            assert g.last_solve_stats()["cg_iterations"] == o.cg_last_iterations()
        for f in (0, 1, 2, sgpu_mod.F_PC):
            a, b = g.download(f), o.get(f)
            assert bit_equal(a, b), f"field {f}: " + describe_diff(a, b)


@pytest.mark.parametrize("grids", [((300, 257), (296, 300)), ((40, 50), (600, 500)), ((149, 129), (1400, 1310))])
def test_two_handles_in_two_threads(sgpu_mod, grids):
    """Solves of two handles at once, from two host threads: each one-kernel solve takes up to every SM, so one waits
    for the other's blocks to leave. The same bits as one after the other."""
    from concurrent.futures import ThreadPoolExecutor

    def solve(nx, ny):
        cfg = dict(snapshot_config("short_16"))
        cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re="400", momentum_solver="gs_multicolour", pressure_solver="cg",
                   maxit="3", error_tolerance="0", pressure_maxit="60")
        with sgpu_mod.Solver(sgpu_mod.params_from_config(config_text(cfg))) as g:
            _, log = g.run(3)
            return log, [g.download(f) for f in (0, 1, 2, sgpu_mod.F_PC)]

    alone = [solve(*g) for g in grids]
    with ThreadPoolExecutor(2) as ex:
        for _ in range(2):
            for (log, fields), (log1, fields1) in zip(ex.map(lambda g: solve(*g), grids), alone):
                assert bit_equal(log, log1)
                assert all(bit_equal(a, b) for a, b in zip(fields, fields1))
