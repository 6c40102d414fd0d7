"""The task sweep at the edges of its walk: patches smaller than a warp, of
one warp and one cell more, and of several; every row count (nb 1, 3, 4) and
coupling count; both layouts of psi; the factor store and the factors built in
the sweep; and inputs that are not numbers. Against the oracle's sweep."""
import numpy as np
import pytest
import torch

import oracle as O
from ubolt_b200 import problem as P
from ubolt_b200 import transport as T

pytestmark = pytest.mark.gpu

MESHES = {
    "tri_dg1": (lambda r: P.box_tris(13, 11, jitter=0.2, rng=r), 1, 4),
    "tri_dg0": (lambda r: P.box_tris(13, 11, jitter=0.2, rng=r), 0, 4),
    "quad_dg1": (lambda r: P.box_quads(17, 15, jitter=0.3, rng=r), 1, 6),
    "tet_dg1": (lambda r: P.box_tets(4, 3, 4), 1, 2),
    "hex_dg1": (lambda r: P.box_hexes(7, 6, 5), 1, 2),
    "hex_dg0": (lambda r: P.box_hexes(7, 6, 5), 0, 4),
}


def dev(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


@pytest.mark.parametrize("patch", [1, 31, 32, 33, 65, 256])
@pytest.mark.parametrize("mesh", MESHES)
def test_task_sweep_at_patch_edges(mesh, patch):
    make, order, sn = MESHES[mesh]
    rng = np.random.default_rng(11)
    m = make(rng)
    g, q = P.build_geometry(m, order), P.lqn(m.dim, sn)
    st = rng.uniform(0.3, 3.0, g.n_cells)
    ss = st * 0.5
    ctx = T.Context(g, q)
    keep = (dev(st), dev(ss))
    ctx.set_group(*keep)
    sw = T.Sweep(ctx, patch)
    sw.set_kernel("tasks")
    op = O.Operator(g, q, st, ss)
    qv = rng.standard_normal(op.n)
    ref = op.sweep(qv)
    psi, psi32 = sw.apply(dev(qv)), sw.apply(dev(qv, torch.float32))
    assert sw.status()["n_lagged"] == 0
    assert np.abs(psi.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.abs(psi32.double().cpu().numpy() - ref).max() <= 1e-4 * np.abs(ref).max()
    # An isotropic source, in both layouts: the same bits
    phi = dev(rng.standard_normal(ctx.n_nodes))
    for dt in (torch.float64, torch.float32):
        row = sw.apply_iso(phi, torch.empty(ctx.n_rows, dtype=dt, device="cuda"))
        om = sw.apply_iso(phi, torch.empty(ctx.n_rows, dtype=dt, device="cuda"), ordinate_major=True)
        assert torch.equal(om.reshape(q.n_angles, ctx.n_nodes).T.reshape(-1), row)
    # The factors built in the sweep: the same bits as from the store
    sw.set_factor_limit(0)
    assert torch.equal(sw.apply(dev(qv)), psi) and torch.equal(sw.apply(dev(qv, torch.float32)), psi32)
    assert sw.status()["timeouts"] == 0
    ctx.close()


def test_task_sweep_of_nan_ends():
    """Every input a NaN of all ones, the word that marks a value not stored
    yet: every output is a NaN, and no wait gives up."""
    rng = np.random.default_rng(12)
    m = P.box_tris(24, 20, jitter=0.2, rng=rng)
    g, q = P.build_geometry(m, 1), P.lqn(2, 4)
    ctx = T.Context(g, q)
    keep = (dev(np.ones(g.n_cells)), dev(np.full(g.n_cells, 0.5)))
    ctx.set_group(*keep)
    sw = T.Sweep(ctx, 16)
    sw.set_kernel("tasks")
    for dt, it in ((torch.float64, torch.int64), (torch.float32, torch.int32)):
        ones = torch.full((ctx.n_rows,), -1, dtype=it, device="cuda").view(dt)
        assert bool(torch.isnan(sw.apply(ones)).all())
        assert sw.status()["timeouts"] == 0
    ctx.close()


@pytest.mark.parametrize("n, order, sn, wave", [
    ((10, 9, 11), 0, 4, True), ((16, 16, 16), 0, 2, True), ((17, 16, 16), 0, 2, False), ((10, 9, 11), 1, 4, False),
    ((16, 16, 16), 0, 6, False)])
def test_automatic_kernel(n, order, sn, wave):
    """Small DG0 boxes of hexahedra take the wave kernel, up to 4096 cells and
    2^17 cell-ordinates; ordinate-major output runs there too, and a choice made
    by the caller is kept."""
    rng = np.random.default_rng(14)
    m = P.box_hexes(*n)
    g, q = P.build_geometry(m, order), P.lqn(3, sn)
    st = rng.uniform(0.3, 3.0, g.n_cells)
    ctx = T.Context(g, q)
    keep = (dev(st), dev(0.5 * st))
    ctx.set_group(*keep)
    sw = T.Sweep(ctx)
    assert (sw.status()["kernel"] == T._lib.SWEEP_WAVE) == wave
    op = O.Operator(g, q, st, 0.5 * st)
    qv = rng.standard_normal(op.n)
    ref = op.sweep(qv)
    phi = dev(rng.standard_normal(ctx.n_nodes))

    def check():
        assert np.abs(sw.apply(dev(qv)).cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
        for dt, tol in ((torch.float64, 1e-12), (torch.float32, 1e-4)):
            row = sw.apply_iso(phi, torch.empty(ctx.n_rows, dtype=dt, device="cuda"))
            om = sw.apply_iso(phi, torch.empty(ctx.n_rows, dtype=dt, device="cuda"), ordinate_major=True)
            om = om.reshape(q.n_angles, ctx.n_nodes).T.reshape(-1)
            assert float((om - row).abs().max()) <= tol * float(row.abs().max())
        assert sw.status()["timeouts"] == 0

    check()
    sw.set_kernel("tasks")
    assert sw.status()["kernel"] == T._lib.SWEEP_TASKS
    check()
    sw.set_kernel("auto")
    assert (sw.status()["kernel"] == T._lib.SWEEP_WAVE) == wave
    check()
    if wave:
        sw.set_kernel("wave")
        with pytest.raises(T._lib.UboltError):
            sw.apply_iso(phi, torch.empty(ctx.n_rows, dtype=torch.float64, device="cuda"), ordinate_major=True)
    # A whole solve and its adjoint, with the wave kernel's rows
    b = dev(rng.uniform(0.1, 1.0, op.n))
    for solve, mult in (("solve", T.TransportOperator(ctx).mult), ("solve_adjoint", T.TransportOperator(ctx).mult_transpose)):
        x, s = getattr(T.TransportSolver(ctx, rtol=1e-10), solve)(b)
        assert float(torch.linalg.norm(b - mult(x))) <= 1.01e-10 * float(torch.linalg.norm(b))
    ctx.close()
