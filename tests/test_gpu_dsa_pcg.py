"""The DSA's inner solve in one launch, where its layout changes: a few cells,
one per thread with the matrix in shared memory, one per thread without, and
more cells than threads. Against the same iteration in NumPy on the assembled
matrix (whose entries tests/test_dsa.py checks against the oracle)."""
import numpy as np
import pytest
import torch

from ubolt_b200 import problem as P
from ubolt_b200 import transport as T

pytestmark = pytest.mark.gpu

CASES = {
    "one_block": (lambda r: P.box_tris(5, 3, jitter=0.2, rng=r), 1),
    "blocks_and_a_rest": (lambda r: P.box_quads(45, 31, jitter=0.2, rng=r), 1),
    "dg0": (lambda r: P.box_hexes(12, 11, 7), 0),
    "tets_kept": (lambda r: P.box_tets(12, 12, 11, jitter=0.2, rng=r), 1),
    "hexes_past_shared_memory": (lambda r: P.box_hexes(35, 34, 34), 1),
    "more_cells_than_threads": (lambda r: P.box_tris(220, 190, jitter=0.2, rng=r), 1),
}


@pytest.mark.parametrize("case", CASES)
def test_inner_solve_matches_numpy(case):
    make, order = CASES[case]
    rng = np.random.default_rng(3)
    m = make(rng)
    g, q = P.build_geometry(m, order), P.lqn(m.dim, 2)
    st = rng.uniform(0.5, 3.0, g.n_cells)
    ss = st * rng.uniform(0.3, 0.9, g.n_cells)
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(ss, device="cuda"))
    ctx.set_group(*keep)
    its = 6
    dsa = T.DSAPrecon(ctx, inner_iterations=its)
    dsa.set_group()
    D, nb, A = dsa.matrix(), g.n_basis, q.n_angles
    x = rng.standard_normal(ctx.n_rows)
    rhs = np.repeat(g.volume, nb) * (x.reshape(-1, A) @ q.w)
    rows = np.arange(g.n_cells * nb).reshape(-1, nb)
    blocks = np.stack([np.asarray(D[rows[:, i], rows[:, j]]).ravel() for i in range(nb) for j in range(nb)],
                      axis=1).reshape(-1, nb, nb)
    jac = np.linalg.inv(blocks)
    apply_j = lambda v: np.einsum("cij,cj->ci", jac, v.reshape(-1, nb)).ravel()
    u, r = np.zeros_like(rhs), rhs.copy()
    z = apply_j(r)
    p, rho = z.copy(), r @ z
    for _ in range(its):
        s = D @ p
        alpha = rho / (p @ s)
        u, r = u + alpha * p, r - alpha * s
        z = apply_j(r)
        new = r @ z
        p, rho = z + new / rho * p, new
    ref = np.repeat(u / q.sum_weights, A)
    y = dsa.apply(torch.tensor(x, device="cuda")).cpu().numpy()
    # Six iterations amplify rounding by far less than 1e5
    assert np.linalg.norm(y - ref) <= 1e-11 * np.linalg.norm(ref)
    v = dsa.spmv(torch.tensor(rhs, device="cuda")).cpu().numpy()
    assert np.linalg.norm(v - D @ rhs) <= 1e-13 * np.linalg.norm(D @ rhs)
    ctx.close()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("case", ["one_block", "blocks_and_a_rest", "dg0"])
def test_spmv_of_an_infinite_boundary_value(case, bad):
    """A value that is not finite reaches the rows that have an entry for it,
    and a face without a neighbour adds nothing."""
    make, order = CASES[case]
    rng = np.random.default_rng(4)
    m = make(rng)
    g, q = P.build_geometry(m, order), P.lqn(m.dim, 2)
    st = rng.uniform(0.5, 3.0, g.n_cells)
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(0.5 * st, device="cuda"))
    ctx.set_group(*keep)
    dsa = T.DSAPrecon(ctx)
    dsa.set_group()
    u = rng.standard_normal(ctx.n_nodes)
    u[0] = u[-1] = bad  # a corner cell's first, another's last
    with np.errstate(invalid="ignore"):
        want = dsa.matrix() @ u
    got = dsa.spmv(torch.tensor(u, device="cuda")).cpu().numpy()
    assert np.isinf(want).any() or np.isnan(bad)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    assert np.array_equal(np.sign(got[np.isinf(want)]), np.sign(want[np.isinf(want)]))
    assert np.abs(got[ok] - want[ok]).max() <= 1e-13 * np.abs(want[ok]).max()
    ctx.close()


@pytest.mark.parametrize("name, make", [
    ("tri", lambda r: P.box_tris(160, 153, jitter=0.2, rng=r)), ("tri_more", lambda r: P.box_tris(161, 154, jitter=0.2, rng=r)),
    ("quad_more", lambda r: P.box_quads(231, 221, jitter=0.2, rng=r)),
    ("tet_more", lambda r: P.box_tets(21, 20, 20, jitter=0.2, rng=r)), ("hex_more", lambda r: P.box_hexes(38, 37, 36))])
def test_spmv_by_rows_and_by_cells(name, make):
    """Either side of the mesh size (49152 cells) at which the multiply changes from a
    thread per row to a thread per cell."""
    rng = np.random.default_rng(6)
    g, q = P.build_geometry(make(rng), 1), P.lqn(3 if name[0] in "h" or name[:3] == "tet" else 2, 2)
    assert (g.n_cells > 49152) == name.endswith("_more")
    st = rng.uniform(0.5, 3.0, g.n_cells)
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(0.5 * st, device="cuda"))
    ctx.set_group(*keep)
    dsa = T.DSAPrecon(ctx)
    dsa.set_group()
    u = rng.standard_normal(ctx.n_nodes)
    want = dsa.matrix() @ u
    got = dsa.spmv(torch.tensor(u, device="cuda")).cpu().numpy()
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
    ctx.close()


@pytest.mark.parametrize("nx, ny", [(40, 31), (300, 280), (400, 390)])
def test_vertex_inner_solve_matches_numpy(nx, ny):
    """The CG-SUPG vertices' inner solve: one per thread, and more than the
    threads of one block per SM and of two. Against the oracle's matrix."""
    import cg as OC
    rng = np.random.default_rng(8)
    m = P.box_quads(nx, ny, jitter=0.2, rng=rng)
    g, q = P.build_cg_geometry(m), P.lqn(2, 2)
    st = rng.uniform(0.5, 3.0, g.n_elements)
    ss = st * rng.uniform(0.3, 0.9, g.n_elements)
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(ss, device="cuda"))
    ctx.set_group(*keep)
    its = 6
    dsa = T.DSAPrecon(ctx, inner_iterations=its)
    dsa.set_group()
    ref = OC.Problem(m, q, st, ss)
    D = ref.dsa_matrix()[0]
    x = rng.standard_normal(ctx.n_rows)
    rhs = ref.dsa_restrict(x)
    jac = 1.0 / D.diagonal()
    u, r = np.zeros_like(rhs), rhs.copy()
    z = jac * r
    p, rho = z.copy(), r @ z
    for _ in range(its):
        s = D @ p
        alpha = rho / (p @ s)
        u, r = u + alpha * p, r - alpha * s
        z = jac * r
        new = r @ z
        p, rho = z + new / rho * p, new
    want = ref.dsa_prolong(u)
    y = dsa.apply(torch.tensor(x, device="cuda")).cpu().numpy()
    # Six iterations amplify rounding by far less than 1e5
    assert np.linalg.norm(y - want) <= 1e-11 * np.linalg.norm(want)
    ctx.close()
