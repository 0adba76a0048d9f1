"""FP64 on small grids, where a component's assembly and sweeps run on one thread-block cluster: every
cluster size, bands of the fewest rows, ragged columns, both colour counts and sweep counts from one up,
and the first grid that does not fit. Bit for bit the oracle's."""
from __future__ import annotations

import pytest

from conftest import bit_equal, config_text, cuda_available, describe_diff, snapshot_config

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("nx,ny,scheme,order,inner", [
    (1, 3, "QUICK", 4, 4), (2, 2, "UDS", 2, 1), (3, 200, "QUICK", 2, 3), (49, 50, "QUICK", 4, 4),
    (51, 50, "QUICK", 4, 4), (50, 90, "QUICK", 2, 2), (96, 96, "UDS", 2, 4), (130, 101, "QUICK", 4, 5),
    (200, 199, "QUICK", 4, 4), (215, 215, "QUICK", 4, 4), (32, 1200, "QUICK", 4, 4), (250, 255, "UDS", 2, 4)])
def test_small_grids_bit_for_bit(sgpu_mod, oracle_mod, nx, ny, scheme, order, inner):
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re="700", convection_scheme=scheme, diffusion_order=str(order),
               momentum_solver="gs_multicolour", pressure_solver="gs_redblack", maxit="6", error_tolerance="0",
               maxit_inner_u=str(inner), maxit_inner_v=str(inner))
    p = sgpu_mod.params_from_config(config_text(cfg))
    o = oracle_mod.Oracle(p)
    _, _, olog = o.run(6)
    with sgpu_mod.Solver(p) as g:
        _, log = g.run(6)
        assert bit_equal(log, olog), describe_diff(log, olog)
        for f in (0, 1, 2, sgpu_mod.F_PC, sgpu_mod.CU[8], sgpu_mod.CV[8]):
            a, b = g.download(f), o.get(f)
            if f in (sgpu_mod.CU[8], sgpu_mod.CV[8]):  # AP: over the component's own cells
                r = ((slice(p.H, p.H + nx), slice(p.H + 1, p.H + ny)) if f == sgpu_mod.CU[8]
                     else (slice(p.H + 1, p.H + nx), slice(p.H + 1, p.H + ny + 1)))
                a, b = a[r].copy(), b[r].copy()
            assert bit_equal(a, b), f"field {f}: " + describe_diff(a, b)


@pytest.mark.parametrize("nx,ny,scheme,order", [(300, 520, "QUICK", 4), (530, 120, "QUICK", 2), (260, 300, "UDS", 2),
                                                (420, 210, "UDS", 4)])
def test_stored_and_recomputed_coefficients_same_bits(sgpu_mod, monkeypatch, nx, ny, scheme, order):
    """Grids past the cluster: sweeps from stored coefficients and sweeps that recompute them (a device
    without memory for the records), over several strips and segments and an odd sweep count."""
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re="700", convection_scheme=scheme, diffusion_order=str(order),
               momentum_solver="gs_multicolour", pressure_solver="mg", maxit="5", error_tolerance="0",
               maxit_inner_u="3", maxit_inner_v="4")
    out = []
    for on in ("1", "0"):
        monkeypatch.setenv("SGPU_MOM_RECORDS", on)
        with sgpu_mod.Solver(sgpu_mod.params_from_config(config_text(cfg))) as g:
            _, log = g.run(5)
            out.append([log] + [g.download(f) for f in (0, 1, 2, sgpu_mod.F_PC)])
    for a, b in zip(*out):
        assert bit_equal(a, b), describe_diff(a, b)


def test_coefficient_arrays_appear_with_the_per_phase_calls(sgpu_mod, oracle_mod):
    """The coefficient arrays are allocated when a per-phase call needs them: zero before, the oracle's after,
    and an iteration in between changes nothing about that."""
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x="250", N_cells_y="240", momentum_solver="gs_multicolour", pressure_solver="mg", maxit="2")
    p = sgpu_mod.params_from_config(config_text(cfg))
    o = oracle_mod.Oracle(p)
    with sgpu_mod.Solver(p) as g:
        g.run(2)
        o.run(2)
        assert not g.download(sgpu_mod.CU[0]).any() and not g.download(sgpu_mod.CV[7]).any()
        g.assemble_u()
        o.assemble_u()
        for f in sgpu_mod.CU:
            a, b = (x[p.H:p.H + 250, p.H:p.H + 241].copy() for x in (g.download(f), o.get(f)))
            assert bit_equal(a, b), f"field {f}: " + describe_diff(a, b)


def test_records_given_up_for_the_coefficient_arrays(sgpu_mod):
    """A device that has no memory left for the coefficient arrays of a per-phase call: the handle gives up its
    records (87 MB here) for them, accounts for both, and goes on with the same bits."""
    import torch
    n = 1024
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(n), N_cells_y=str(n), momentum_solver="gs_multicolour", pressure_solver="mg", maxit="9",
               error_tolerance="0")
    p = sgpu_mod.params_from_config(config_text(cfg))
    field = p.nrows * (-(-p.ncols // 32) * 32) * 8
    with sgpu_mod.Solver(p) as a, sgpu_mod.Solver(p) as b:
        for s in (a, b):
            s.run(1)
        b.assemble_u()
        before = a.memory_bytes()
        free = torch.cuda.mem_get_info()[0]
        hog = torch.empty(free - (100 << 20), dtype=torch.uint8, device="cuda")
        try:
            a.assemble_u()
            after = a.memory_bytes()
            a.run(2)
        finally:
            del hog
            torch.cuda.empty_cache()
        b.run(2)
        assert b.memory_bytes() == before + 16 * field
        assert before - 5 * 2 * field * 1.1 < after - 16 * field <= before - 5 * 2 * field
        for f in (0, 1, 2, sgpu_mod.F_PC, sgpu_mod.CU[0], sgpu_mod.CU[7]):
            assert bit_equal(a.download(f), b.download(f)), f"field {f}"


@pytest.mark.parametrize("nx,ny,scheme,order,inner", [(3, 200, "QUICK", 2, 3), (50, 90, "QUICK", 2, 2), (130, 101, "QUICK", 4, 5),
                                                      (96, 96, "UDS", 2, 4)])
def test_small_grids_without_the_cluster(sgpu_mod, oracle_mod, monkeypatch, nx, ny, scheme, order, inner):
    """What a device without such clusters runs, and SGPU_MOM_CLUSTER=0 selects: the sweeps from stored and from
    recomputed coefficients, on grids that otherwise run on the cluster."""
    cfg = dict(snapshot_config("short_16"))
    cfg.update(N_cells_x=str(nx), N_cells_y=str(ny), Re="700", convection_scheme=scheme, diffusion_order=str(order),
               momentum_solver="gs_multicolour", pressure_solver="gs_redblack", maxit="6", error_tolerance="0",
               maxit_inner_u=str(inner), maxit_inner_v=str(inner))
    p = sgpu_mod.params_from_config(config_text(cfg))
    o = oracle_mod.Oracle(p)
    _, _, olog = o.run(6)
    bytes_held = []
    for cluster, records in (("1", "1"), ("0", "1"), ("0", "0")):
        monkeypatch.setenv("SGPU_MOM_CLUSTER", cluster)
        monkeypatch.setenv("SGPU_MOM_RECORDS", records)
        with sgpu_mod.Solver(p) as g:
            _, log = g.run(6)
            assert bit_equal(log, olog), describe_diff(log, olog)
            for f in (0, 1, 2, sgpu_mod.F_PC):
                assert bit_equal(g.download(f), o.get(f)), f"field {f}: " + describe_diff(g.download(f), o.get(f))
            bytes_held.append(g.memory_bytes())
    assert bytes_held[0] == bytes_held[2] < bytes_held[1]  # the second one did take the records
