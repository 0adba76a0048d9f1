"""The FP64 red-black updates divide by AP through its inverse where the exponents allow it (2^-100 <= AP <
2^101, 2^-900 <= dividend < 2^901) and by a division elsewhere. Both must give the oracle's bits: Re moves AP
past either bound, velocities scaled down put the dividends below theirs."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bit_equal, config_text, cuda_available, describe_diff, snapshot_config

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("nx,ny", [(31, 33), (64, 64), (300, 260)])
@pytest.mark.parametrize("re,scale", [("1e-35", 1.0), ("1e33", 1e-30), ("400", 1e-273), ("400", 1e-290)])
def test_dividends_and_divisors_past_the_bounds(sgpu_mod, oracle_mod, nx, ny, re, scale):
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re=re, momentum_solver="gs_multicolour", pressure_solver="mg",
               maxit="2", error_tolerance="0")
    p = sgpu_mod.params_from_config(config_text(cfg))
    o = oracle_mod.Oracle(p)
    rng = np.random.default_rng(nx)
    with sgpu_mod.Solver(p) as g:
        for f in (0, 1, 2):
            v = rng.standard_normal(o.get(f).shape) * scale
            o.set(f, v)
            g.upload(f, v)
        _, _, olog = o.run(2)
        if not np.isfinite(olog).all():  # a diverging run is an error there
            with pytest.raises(sgpu_mod.SgpuError):
                g.run(2)
            return
        _, log = g.run(2)
        assert bit_equal(log, olog), describe_diff(log, olog)
        for f in (0, 1, 2, sgpu_mod.F_PC):
            assert bit_equal(g.download(f), o.get(f)), f"field {f}: " + describe_diff(g.download(f), o.get(f))


def test_quotient_over_all_exponents(sgpu_mod):
    """The quotient itself against the IEEE division: both sides of every bound (2^-900 and 2^901 for the dividend,
    2^-100 and 2^101 for AP), quotients that are subnormal, half way between two subnormal numbers or below them
    all, zeros of both signs, infinities, NaN, negative and zero AP."""
    rng = np.random.default_rng(17)

    def numbers(exponents, n):
        e = rng.choice(exponents, n)
        m = np.where(rng.random(n) < 0.3, rng.choice([1.0, 1.5, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52, 1.25], n),
                     1.0 + rng.random(n))
        with np.errstate(under="ignore", over="ignore"):
            return np.ldexp(m, e) * rng.choice([1.0, -1.0], n)

    n = 400_000
    edges_a = np.r_[-902:-896, 898:904, -1074:-1020]
    edges_p = np.r_[-103:-97, 98:104]
    parts = [(numbers(np.arange(-1080, 1024), n), np.abs(numbers(np.arange(-110, 112), n))),
             (numbers(edges_a, n), np.abs(numbers(edges_p, n))),
             (numbers(np.arange(-1074, -895), n), np.abs(numbers(np.arange(-100, 101), n))),
             (numbers(np.arange(-1074, 1024), n), numbers(np.arange(-1074, 1024), n))]
    k = np.arange(1.0, 2001.0)  # quotients (2 j + 1) 2^-1075 and their neighbours
    for e in (1, 7, 40):
        p = np.full(k.size, 2.0 ** e)
        parts.append((k * 2.0 ** -1074, p))
        parts.append((k * 3 * 2.0 ** -1073, 3 * p))
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0 ** -1022, 1.0, -1.0, 2.0 ** -900,
                        2.0 ** 901, 2.0 ** -100, 2.0 ** 101, np.finfo(float).max])
    parts.append(tuple(x.ravel() for x in np.meshgrid(special, special)))
    for a, p in parts:
        with np.errstate(all="ignore"):
            want = a / p
        got = sgpu_mod.selftest_quotient(a, p)
        same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
        bad = np.flatnonzero(~same)
        assert bad.size == 0, (bad.size, a[bad[:3]], p[bad[:3]], got[bad[:3]], want[bad[:3]])


@pytest.mark.parametrize("nx,ny,scheme", [(700, 40, "UDS"), (500, 130, "QUICK")])
def test_red_black_from_rest(sgpu_mod, oracle_mod, nx, ny, scheme):
    """A tall cavity from rest: ahead of what the sweeps have reached p' falls through all small exponents to zero."""
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re="400", convection_scheme=scheme, momentum_solver="gs_multicolour",
               pressure_solver="gs_redblack", maxit="13", error_tolerance="0")
    p = sgpu_mod.params_from_config(config_text(cfg))
    o = oracle_mod.Oracle(p)
    o.run(13)
    small = np.abs(o.get(sgpu_mod.F_PC))
    assert ((small > 0) & (small < 2.0 ** -900)).any() and ((small > 0) & (small < 2.0 ** -1022)).any()
    with sgpu_mod.Solver(p) as g:
        g.run(13)
        for f in (0, 1, 2, sgpu_mod.F_PC):
            assert bit_equal(g.download(f), o.get(f)), f"field {f}: " + describe_diff(g.download(f), o.get(f))
