"""The sweep kernel's tiles, layers and adjoint against the plane-streaming kernel, and
the radial lookups of the pseudocharge kernels against the oracle, at the sizes where
they can go wrong.

The window edges are the smallest and largest of every tile (pairs of columns: windows
that start at odd and even columns of the halo'd block, the last pair half outside), for
fields with one and with three projectors per slot.  Both kernels sum in FP64 in another
order: a moment of order k carries about k^2 roundings of size 1e-16 (npl 16: 1e-13 with
room), the bounds 1e-12 of the spectral range.  LiH's Lanczos runs take up to 290 steps and
stop on a plateau of the smallest eigenvalue, where a node's bound follows the order of
every sum, so the bounds of two kernels agree only within the stop: 1e-6 Ha of about 35
Ha, 3e-8, and the moments ten times that.  FP32 Lanczos vectors round at 6e-8, and
the stop at 1e-3 Ha is met within that of each other.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def _params(kind, system, nloc, form=0, npl=16, **kw):
    d = dict(kind=kind, system=system, form=form, cells=2, per_cell=12 if nloc < 14 else 20, block="3x2x2",
             nloc=nloc, npl=npl, kt=5.0)
    d.update(kw)
    return d


def _both(p, seed=3, rows=0):
    """Outputs of the sweep kernel (`rows` of sqb_set_sweep_rows) and of the plane-streaming kernel on the same inputs."""
    from perf import cases
    from sqdft_b200 import sq

    s = cases.prepare(p, seed)
    with s["ctx"] as ctx:
        ctx.set_sweep_rows(rows)
        ctx.set_node_kernel(sq.SQB_KERNEL_SWEEP)
        a = cases.run(s)
        assert ctx.stats()["node_kernel"] == sq.SQB_KERNEL_SWEEP
        ctx.set_node_kernel(sq.SQB_KERNEL_PLANE)
        b = cases.run(s)
        assert ctx.stats()["node_kernel"] == sq.SQB_KERNEL_PLANE
        return a, b


def _check_tiles(system, nloc, rows=0, **kw):
    kw.setdefault("per_cell", 20 if system == "lih" or nloc > 13 else 12)
    for form in (0, 1, 2):
        a, b = _both(_params("sq", system, nloc, form, **kw), rows=rows)
        tol = 1e-6 if form == 1 else 3e-8 if system == "lih" else 1e-12
        for k in ("chi", "zee"):
            assert _rel(a[k], b[k]) <= tol, (form, k)
        assert _rel(a["rho_pj"], b["rho_pj"]) <= 10 * tol, form
    for form in (0, 1):
        a, b = _both(_params("forces", system, nloc, form, **kw), rows=rows)
        assert _rel(a, b) <= (1e-5 if form else 1e-11), form


@pytest.mark.parametrize("system", ["al", "lih"])
@pytest.mark.parametrize("nloc", [4, 9, 10, 13, 15, 16, 17, 19, 21])
def test_tiles_match_plane_kernel(system, nloc):
    _check_tiles(system, nloc)


@pytest.mark.parametrize("kind,form", [("sq", 0), ("sq", 1), ("sq", 2), ("forces", 0), ("forces", 1)])
def test_sweep_rows_leave_the_pair_tile_alone(kind, form):
    """Three rows per thread were up to seven times slower than the pair tile: rows = 3 is accepted
    and runs it, to the bit, where no node runs on the one-column tile."""
    a, _ = _both(_params(kind, "al", 9, form))
    b, _ = _both(_params(kind, "al", 9, form), rows=3)
    for x, y in zip(a.values(), b.values()) if kind == "sq" else [(a, b)]:
        assert np.array_equal(x, y)


@pytest.mark.parametrize("system", ["al", "lih"])
def test_many_nodes_per_cta(system):
    """512 nodes of 9^3 windows, more than resident CTAs: what a CTA carries from one node to the
    next, of the other parity or not."""
    _check_tiles(system, 4, block="8x8x8", per_cell=20)
    (gv, ga), (gv0, ga0) = _both(_params("vjp", system, 4, npl=20, per_cell=20, block="8x8x8"))
    assert _rel(gv, gv0) <= 1e-12
    assert _rel(ga, ga0) <= 1e-11


@pytest.mark.parametrize("system,nloc,npl", [("al", 4, 4), ("al", 9, 16), ("al", 10, 20), ("al", 15, 36),
                                             ("al", 17, 12), ("lih", 8, 20), ("lih", 16, 64), ("lih", 19, 16)])
def test_adjoint_matches_plane_kernel(system, nloc, npl):
    """Block remainders of the quadratic form (16 vectors, 8 at a time), one block and several."""
    (gv, ga), (gv0, ga0) = _both(_params("vjp", system, nloc, npl=npl, per_cell=20))
    assert _rel(gv, gv0) <= 1e-12
    assert _rel(ga, ga0) <= 1e-11


@pytest.mark.parametrize("left,kernel", [(8.0e9, 2), (3.6e9, 1)])
def test_adjoint_where_memory_is_short(left, kernel):
    """35^3 windows, npl 64, 150 nodes: 3.4 GB of vectors for 148 CTAs.  With 8 GB free fewer CTAs
    take a quarter of it; with 3.6 GB, where the vectors alone would fit but not the scratch
    beside them, the call runs on the plane-streaming kernel."""
    import torch

    from perf import cases
    from sqdft_b200 import sq

    p = _params("vjp", "al", 17, npl=64, per_cell=20, block="6x5x5")
    s = cases.prepare(p, 3)
    with s["ctx"] as ctx:
        ctx.set_node_kernel(sq.SQB_KERNEL_PLANE)
        gv0, ga0 = cases.run(s)
    s = cases.prepare(p, 3)
    with s["ctx"] as ctx:
        torch.cuda.empty_cache()
        held = torch.empty(int(torch.cuda.mem_get_info()[0] - left), dtype=torch.uint8, device="cuda")
        try:
            free = torch.cuda.mem_get_info()[0]
            gv, ga = cases.run(s)
            taken = free - torch.cuda.mem_get_info()[0]
        finally:
            del held
            torch.cuda.empty_cache()
        assert ctx.stats()["node_kernel"] == kernel
    # the vectors' quarter, or the plane-streaming kernel's checkpoints (1.44 GB); 0.65 GB of scratch and tables
    assert taken <= (left / 4 if kernel == sq.SQB_KERNEL_SWEEP else 1.45e9) + 0.75e9
    assert _rel(gv, gv0) <= 1e-12
    assert _rel(ga, ga0) <= 1e-11


def test_layers_of_displaced_lih_fit():
    """Displaced 64-atom LiH, where first fit in replica order needs five or six layers."""
    from perf import cases
    from sqdft_b200 import sq

    p = _params("sq", "lih", 16, per_cell=20, npl=16, block="6x5x4")
    for seed in (0, 1, 2):
        s = cases.prepare(p, seed)
        with s["ctx"] as ctx:
            a = cases.run(s)
            assert ctx.stats()["node_kernel"] == sq.SQB_KERNEL_SWEEP
            ctx.set_node_kernel(sq.SQB_KERNEL_PLANE)
            b = cases.run(s)
        assert _rel(a["rho_pj"], b["rho_pj"]) <= 3e-7


def _long_runs(p, seed, rows=0, tol=None):
    """FP64 step of the sweep kernel, its Lanczos counts, the nodes whose runs pass six window
    edges (which another kernel repeats), and the step of the plane-streaming kernel."""
    from perf import cases
    from sqdft_b200 import sq

    c = cases._case(p, seed)
    if tol:
        c.lanczos_tol = tol
    with sq.Context(c, precision=0) as ctx:
        ctx.nonlocal_projectors()
        ctx.set_veff(c.veff)
        ctx.set_sweep_rows(rows)
        a = ctx.lanczos_moments()
        assert ctx.stats()["node_kernel"] == sq.SQB_KERNEL_SWEEP
        ctx.set_graph(1)  # a plain run, the capture and a replay
        for _ in range(3):
            g = ctx.lanczos_moments()
            for k in a:
                assert np.array_equal(a[k], g[k]), k
        ctx.set_graph(0)
        ctx.set_node_kernel(sq.SQB_KERNEL_PLANE)
        b = ctx.lanczos_moments()
    return a, b, (a["lanczos_iters"] > 6 * c.nw).reshape(-1)


def test_long_lanczos_runs_keep_the_plane_kernel():
    """64-atom LiH, 33^3 windows, a seed at which one node's stop moves by a step when the sums
    change their order (the moments by 4e-8, Ci by 2e-7): nodes with long runs are the
    plane-streaming kernel's bit for bit, the others agree to rounding."""
    from perf import cases

    p = next(c for c in cases.listed() if c["name"] == "sq_fp64_w33_lih")
    a, b, long = _long_runs(p, 2)
    assert 0 < long.sum() < long.size
    assert np.array_equal(a["lanczos_iters"], b["lanczos_iters"])
    for k in ("chi", "zee", "rho_pj"):
        x, y = (np.asarray(v[k]).reshape(long.size, -1) for v in (a, b))
        assert np.array_equal(x[long], y[long]), k
        assert _rel(x, y) <= 1e-12, k
    s, g = cases.prepare(p, 2), cases.prepare(p, 2)
    with s["ctx"], g["ctx"]:
        g["ctx"].set_graph(2)
        x, y = cases.run(s), cases.run(g)
    for k in ("rho", "rho_pj", "Ci", "chi", "zee"):
        assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("per_cell,nloc,seed", [(14, 12, 2), (16, 14, 2), (12, 10, 2), (12, 10, 6)])
def test_long_lanczos_runs_keep_the_order_of_their_sums(per_cell, nloc, seed):
    """8-atom LiH under first-fit layers, at seeds where bounds move by 2e-9 to 5e-9 of the
    spectral range with the order of the sums: the bounds against those of the kernel whose order
    the one-column tile keeps (golden file), to a few roundings of the range."""
    from pathlib import Path

    ref = np.load(Path(__file__).parent / "golden" / "lih_bounds_first_fit.npz")
    a, _, long = _long_runs(_params("sq", "lih", nloc, cells=1, per_cell=per_cell, block="5x4x3", kt=9.0), seed)
    assert long.any()
    for k in ("chi", "zee"):
        assert _rel(np.asarray(a[k]).reshape(-1), ref[f"{per_cell}_{nloc}_{seed}_{k}"].reshape(-1)) <= 1e-13, k


@pytest.mark.parametrize("nloc,rows", [(n, r) for n in (10, 14, 15, 16, 19) for r in (0, 3) if r == 0 or n <= 16])
def test_one_column_tile_matches_plane_kernel(nloc, rows):
    """8-atom LiH, where first fit needs four layers, at a stop of 1e-12 Ha, which most runs reach
    late: windows with a warp per row group (up to 31 wide) and with packed columns (from 33 on),
    n mod 3 of 0, 1 and 2 (three rows cover up to 33).  The converged bounds agree to the stop and their roundings."""
    a, b, long = _long_runs(_params("sq", "lih", nloc, cells=1, per_cell=20), 3, rows, 1e-12)
    assert long.any()
    for k in ("chi", "zee"):
        assert _rel(a[k], b[k]) <= 1e-10, k
    assert _rel(a["rho_pj"], b["rho_pj"]) <= 1e-9


@pytest.mark.parametrize("grid_kind", ["uniform", "coarse", "octaves"])
def test_radial_lookup_on_other_grids(grid_kind):
    """Radial grids with many points per lookup bin, with many bins per point, and with
    points on the bins' edges: b and rho_at equal the oracle's bit for bit."""
    from oracle.pyoracle import LocalOracle
    from perf import cases
    from sqdft_b200 import sq

    p = dict(kind="local", system="al", form=0, cells=1, per_cell=10, block="9x8x10", nloc=1, npl=4, kt=10.0)
    grid, loc, _ = cases._local_inputs(p, 5)
    r = {"uniform": np.linspace(0.0, 40.0, 6001), "coarse": np.linspace(0.0, 40.0, 41),
         "octaves": np.concatenate([[0.0], 2.0 ** (np.arange(-14 * 8, 6 * 8) / 8)])}[grid_kind]
    a = 1.1
    uu = np.exp(-(r / a) ** 2)
    loc.tables = [np.stack([r, -3 * np.tanh(r), -3 / np.cosh(r) ** 2, uu, -2 * r / a ** 2 * uu]) for _ in loc.tables]
    with sq.LocalContext(grid, loc) as ctx:
        out = ctx.charge_density()
    ref = LocalOracle(grid, loc).charge_density()
    assert np.array_equal(out["b"], ref["b"])
    assert np.array_equal(out["rho_at"], ref["rho_at"])


def test_a_list_that_names_long_runs_more_than_once():
    """sqb_lanczos_moments_nodes with more entries than the block has nodes: the list of nodes to
    repeat holds them all."""
    from perf import cases
    from sqdft_b200 import sq

    c = cases._case(_params("sq", "lih", 12, cells=1, per_cell=14, block="5x4x3", kt=9.0), 2)
    with sq.Context(c, precision=0) as ctx:
        ctx.nonlocal_projectors()
        ctx.set_veff(c.veff)
        a = ctx.lanczos_moments()
        long = np.flatnonzero(a["lanczos_iters"].reshape(-1) > 6 * c.nw)
        nodes = np.concatenate([np.repeat(long, 70), np.arange(c.n_nodes)]).astype(np.int32)
        b = ctx.lanczos_moments_nodes(nodes)
    assert long.size and len(nodes) > c.n_nodes + 60
    for k in ("chi", "zee", "rho_pj", "lanczos_iters"):
        assert np.array_equal(np.asarray(a[k]).reshape(c.n_nodes, -1)[nodes], np.asarray(b[k]).reshape(len(nodes), -1)), k
