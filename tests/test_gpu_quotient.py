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
