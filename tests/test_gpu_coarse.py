"""The coarsest multigrid level's solve (coarse_solve, multigrid.cpp:120-140) on every route it takes.

Its size decides the route: a thread per cell pair inside the tail kernel, in a CTA of its own, in a
cluster of 8 or 16 CTAs, or the general one-CTA loop. FP64 must equal the oracle bit for bit, the
sweep count included (the residual vote may not stop a sweep early or late)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bit_equal, config_text, cuda_available, describe_diff, snapshot_config

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]

GRIDS = [
    (4, 4),      # one level of half a warp
    (40, 72),    # 5 x 9: one warp inside the tail
    (64, 192),   # 4 x 12 under streamed levels
    (31, 33),    # one CTA, several warps; odd rows and columns
    (66, 62),    # 33 x 31: more pairs than the tail's threads (general loop)
    (45, 45),    # one CTA near its 1024 threads
    (46, 45),    # just past them: 8 CTAs
    (150, 250),  # 75 x 125 below a streamed level: 8 CTAs of 9 and 10 rows
    (131, 133),  # 16 CTAs
    (7, 701),    # too few rows for a cluster (general loop)
    (9, 511),    # bands of one and two rows
]


def _cfg(nx, ny, **kw):
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re="400", momentum_solver="gs_multicolour",
               pressure_solver="mg", maxit="3", error_tolerance="0", **kw)
    return config_text(cfg)


@pytest.mark.parametrize("nx,ny", GRIDS)
def test_coarse_solve(sgpu_mod, oracle_mod, nx, ny):
    p = sgpu_mod.params_from_config(_cfg(nx, ny))
    o = oracle_mod.Oracle(p)
    _, _, olog = o.run(3)
    with sgpu_mod.Solver(p) as g:
        _, log = g.run(3)
        assert bit_equal(log, olog), describe_diff(log, olog)
        for f in (0, 1, 2, sgpu_mod.F_PC):
            assert bit_equal(g.download(f), o.get(f)), f"field {f}: " + describe_diff(g.download(f), o.get(f))
        assert g.last_solve_stats()["coarse_sweeps"] == o.mg_last_coarse_sweeps()


@pytest.mark.parametrize("nx,ny", [(4, 4), (31, 33), (45, 45), (46, 45), (131, 133), (7, 701), (9, 511)])
def test_coarse_solve_fp32(sgpu_mod, nx, ny):
    """The float solve on one-level grids against the same sweeps in numpy FP32. A sweep rounds a cell
    about four times by 2^-24 and does not amplify what it was given, so at most 200 sweeps stay
    within 200 * 4 * 2^-24 < 1e-4 of the largest |p'|; the coarse tolerance (1e-5 of ||b||) is part of
    both."""
    p = sgpu_mod.params_from_config(_cfg(nx, ny, precision="mixed"))
    with sgpu_mod.Solver(p) as g:
        g.run(1)
        r = (slice(p.H, p.H + nx), slice(p.H + 1, p.H + 1 + ny))
        e, w, n, s, b, pc = (g.download(f)[r] for f in (*range(sgpu_mod.F_AEP, sgpu_mod.F_ASP + 1),
                                                         sgpu_mod.F_B, sgpu_mod.F_PC))
    f4 = np.float32
    ap = (e + w + n + s).astype(f4)
    e, w, n, s = (a.astype(f4) for a in (e, w, n, s))
    b = (b - b.mean()).astype(f4)
    b = (b - b.mean(dtype=float)).astype(f4)
    x = np.zeros((nx + 2, ny + 2), f4)
    i, j = np.indices((nx, ny))
    flow = lambda: e * x[1:-1, 2:] + w * x[1:-1, :-2] + s * x[2:, 1:-1] + n * x[:-2, 1:-1]  # noqa: E731
    bn = np.linalg.norm(b.astype(float))
    for _ in range(200):
        for c in (0, 1):
            x[1:-1, 1:-1] = np.where((i + j) % 2 == c, (b + flow()) / ap, x[1:-1, 1:-1])
        if np.linalg.norm((b - (ap * x[1:-1, 1:-1] - flow())).astype(float)) < 1e-5 * bn:
            break
    x = x[1:-1, 1:-1].astype(float)
    x -= x.mean()
    assert np.max(np.abs(pc - x)) <= 1e-4 * np.max(np.abs(x))


@pytest.mark.parametrize("nx,ny", [(2, 2), (1, 60), (7, 8), (8, 8), (10, 6), (32, 1), (28, 28), (128, 64), (5, 12)])
def test_one_warp_solve(sgpu_mod, oracle_mod, nx, ny):
    """Coarsest levels of at most 32 cell pairs, which one warp solves: its vote is also the barrier between a
    colour's stores and the other colour's loads. Alone, inside the one-CTA tail and inside the cluster tail."""
    p = sgpu_mod.params_from_config(_cfg(nx, ny))
    o = oracle_mod.Oracle(p)
    _, _, olog = o.run(3)
    with sgpu_mod.Solver(p) as g:
        _, log = g.run(3)
        assert bit_equal(log, olog), describe_diff(log, olog)
        for f in (0, 1, 2, sgpu_mod.F_PC):
            assert bit_equal(g.download(f), o.get(f)), f"field {f}: " + describe_diff(g.download(f), o.get(f))
        assert g.last_solve_stats()["coarse_sweeps"] == o.mg_last_coarse_sweeps()


@pytest.mark.parametrize("nx,ny", [(52, 52), (56, 56), (60, 60), (64, 64), (80, 48), (62, 66)])
def test_tail_in_global_memory(sgpu_mod, oracle_mod, nx, ny):
    """FP64 tails that do not fit one CTA's shared memory form their coarse operators in global memory and read
    them back in the same kernel. Alone, and as the cavity of a batch that takes the batch shape."""
    p = sgpu_mod.params_from_config(_cfg(nx, ny))
    o = oracle_mod.Oracle(p)
    o.run(3)
    with sgpu_mod.Solver(p) as g, sgpu_mod.Batch([sgpu_mod.params_from_config(_cfg(128, 128))] * 8 + [p]) as b:
        g.run(3)
        b.run(3)
        for f in (0, 1, 2, sgpu_mod.F_PC):
            for got in (g.download(f), b.download(8, f)):
                assert bit_equal(got, o.get(f)), f"field {f}: " + describe_diff(got, o.get(f))


@pytest.mark.parametrize("nx,ny", [(8, 8), (31, 33), (32, 32), (46, 45), (128, 128)])
@pytest.mark.parametrize("scale", [1e-100, 1e-148, 1e-155, 1e-157, 1e-159, 1e-161])
def test_right_hand_sides_whose_squares_underflow(sgpu_mod, oracle_mod, nx, ny, scale):
    """The reference stops when the sum of squares is small, and squares of values below 1e-154 lose their digits
    or vanish: it then stops earlier than the residuals themselves would say. Same sweep counts, same bits."""
    p = sgpu_mod.params_from_config(_cfg(nx, ny))
    o = oracle_mod.Oracle(p)
    b = np.random.default_rng(nx).standard_normal((p.nrows, p.ncols)) * scale
    with sgpu_mod.Solver(p) as g:
        for s in (o, g):
            s.assemble_u(), s.assemble_v(), s.assemble_p()
        o.set(sgpu_mod.F_B, b)
        g.upload(sgpu_mod.F_B, b)
        o.solve_p()
        g.solve_p()
        assert g.last_solve_stats()["coarse_sweeps"] == o.mg_last_coarse_sweeps()
        assert bit_equal(g.download(sgpu_mod.F_PC), o.get(sgpu_mod.F_PC))


@pytest.mark.parametrize("nx,ny", [(46, 45), (131, 133), (150, 250), (128, 128)])
def test_without_clusters(sgpu_mod, oracle_mod, monkeypatch, nx, ny):
    """SGPU_MG_CLUSTER=0 (and a device without clusters): the coarsest levels of more pairs than one CTA has threads
    on the general loop, tails on one CTA. Bit for bit the oracle's, and other launches than with clusters."""
    p = sgpu_mod.params_from_config(_cfg(nx, ny))
    o = oracle_mod.Oracle(p)
    _, _, olog = o.run(2)
    seconds = []
    for on in ("1", "0"):
        monkeypatch.setenv("SGPU_MG_CLUSTER", on)
        with sgpu_mod.Solver(p) as g:
            _, log = g.run(2)
            assert bit_equal(log, olog), describe_diff(log, olog)
            for f in (0, 1, 2, sgpu_mod.F_PC):
                assert bit_equal(g.download(f), o.get(f)), f"field {f}: " + describe_diff(g.download(f), o.get(f))
            assert g.last_solve_stats()["coarse_sweeps"] == o.mg_last_coarse_sweeps()
            seconds.append(min(g.run(10)[0].seconds for _ in range(3)))
    if nx != 128:  # one CTA on global memory takes several times the cluster's time: the switch was heeded
        assert seconds[1] > 1.5 * seconds[0], seconds
