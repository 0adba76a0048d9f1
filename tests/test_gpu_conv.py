"""The network's convolution kernels at the edges of their tiles: images narrower than a 16-pixel run, no
multiple of it, wider than a column tile, of one row; one-level networks (two convolutions), so that no
rounding flip cascades. The bounds are those of the shallow-network test: a BF16 rounding of FP32 sums taken
in another order, 0.5% of the output and 1% of a gradient."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(np.asarray(b, np.float64)), 1e-30))


@pytest.mark.parametrize("n,h,w,base", [(1, 1, 1, 16), (3, 5, 7, 16), (1, 2, 270, 16), (2, 33, 256, 32),
                                        (1, 64, 17, 64), (1, 3, 300, 128), (2, 130, 66, 16)])
def test_convolutions_at_tile_edges(sgpu_mod, n, h, w, base):
    import cnn_oracle
    params = cnn_oracle.init_params(base, 1, seed=n + h + w + base)
    rng = np.random.default_rng(5)
    x = rng.normal(size=(n, h, w, 2)).astype(np.float32)
    t = rng.normal(size=(n, h, w)).astype(np.float32)
    with sgpu_mod.Cnn(base, 1) as net:
        net.set_params(params)
        out = net.forward(x)
        loss, g = net.loss_grad(x, t)
    o = cnn_oracle.UNetOracle(base, 1)
    rloss, rg, ref = o.loss_grad(params, x, t)
    assert rel_l2(out, ref) < 5e-3 and abs(loss - rloss) <= 1e-2 * abs(rloss)
    for (cin, cout, _), (wo, bo) in zip(o.convs, o.offs):
        assert rel_l2(g[wo:bo], rg[wo:bo]) < 1e-2
        assert rel_l2(g[bo:bo + cout], rg[bo:bo + cout]) < 1e-2


@pytest.mark.parametrize("n,h,w,base", [(1, 40, 50, 16), (2, 61, 9, 32), (1, 200, 130, 16), (5, 19, 35, 64)])
def test_epilogue_of_partly_live_warps(sgpu_mod, n, h, w, base):
    """Tiles of several blocks of 128 pixels in which some lanes of a warp have an output pixel and others do not
    (halo columns, columns and rows past the image), with the masked input gradient too. Bounds as above."""
    import cnn_oracle
    params = cnn_oracle.init_params(base, 1, seed=h + w)
    rng = np.random.default_rng(11)
    x = rng.normal(size=(n, h, w, 2)).astype(np.float32)
    t = rng.normal(size=(n, h, w)).astype(np.float32)
    with sgpu_mod.Cnn(base, 1) as net:
        net.set_params(params)
        out = net.forward(x)
        _, g = net.loss_grad(x, t)
    o = cnn_oracle.UNetOracle(base, 1)
    _, rg, ref = o.loss_grad(params, x, t)
    assert rel_l2(out, ref) < 5e-3
    for (cin, cout, _), (wo, bo) in zip(o.convs, o.offs):
        assert rel_l2(g[wo:bo], rg[wo:bo]) < 1e-2
        assert rel_l2(g[bo:bo + cout], rg[bo:bo + cout]) < 1e-2


@pytest.mark.parametrize("n,h,w", [(4, 64, 64), (1, 70, 187), (2, 250, 50)])
def test_wide_convolutions_in_channel_chunks(sgpu_mod, n, h, w):
    """128 to 128 channels, whose weights do not fit beside a tile: images large enough to come in 16 channels at a
    time. Bounds as above."""
    import cnn_oracle
    params = cnn_oracle.init_params(128, 1, seed=n + h + w)
    rng = np.random.default_rng(3)
    x = rng.normal(size=(n, h, w, 2)).astype(np.float32)
    t = rng.normal(size=(n, h, w)).astype(np.float32)
    with sgpu_mod.Cnn(128, 1) as net:
        net.set_params(params)
        out = net.forward(x)
        _, g = net.loss_grad(x, t)
    o = cnn_oracle.UNetOracle(128, 1)
    _, rg, ref = o.loss_grad(params, x, t)
    assert rel_l2(out, ref) < 5e-3
    for (cin, cout, _), (wo, bo) in zip(o.convs, o.offs):
        assert rel_l2(g[wo:bo], rg[wo:bo]) < 1e-2
        assert rel_l2(g[bo:bo + cout], rg[bo:bo + cout]) < 1e-2
