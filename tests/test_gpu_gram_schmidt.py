"""The compressed basis's Gram-Schmidt step where its launch changes: more basis
vectors than a chunk of dots (8) and than a warp (32), up to the longest
restart, on one block, several, and more nodes than threads. Solves that need
many steps, forward and adjoint, against the full-basis solve, repeated for
equal bits (every block must work with the same scalars)."""
import numpy as np
import pytest
import torch

from ubolt_b200 import problem as P
from ubolt_b200 import transport as T

pytestmark = pytest.mark.gpu

# Meshes of one block of 512 nodes, of 36 blocks, and of more nodes than the
# largest grid's threads (2 x 148 blocks of 512)
MESHES = {
    "one_block": lambda r: P.box_tris(9, 9, jitter=0.2, rng=r),
    "many_blocks": lambda r: P.box_tris(64, 48, jitter=0.2, rng=r),
    "more_nodes_than_threads": lambda r: P.box_tris(172, 160, jitter=0.2, rng=r),
}


def diffusive(mesh):
    """A thick medium that scatters almost all: the spectrum is spread out."""
    rng = np.random.default_rng(21)
    m = MESHES[mesh](rng)
    g, q = P.build_geometry(m, 1), P.lqn(2, 2)
    st = 10.0 ** rng.uniform(0.0, 2.5, g.n_cells)
    ss = st * (1.0 - 10.0 ** rng.uniform(-5.0, -2.0, g.n_cells))
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(ss, device="cuda"))
    ctx.set_group(*keep)
    b = torch.tensor(rng.standard_normal(ctx.n_rows), device="cuda")
    return ctx, keep, b


@pytest.mark.parametrize("restart", [1, 8, 9, 33, 200])
@pytest.mark.parametrize("mesh", MESHES)
def test_long_bases_match_the_full_basis(mesh, restart):
    ctx, keep, b = diffusive(mesh)
    rtol = 1e-9
    # Restarts of one vector converge slowly: compare after a fixed number of steps
    max_it = 400 if restart >= 33 else 3 * restart
    op = T.TransportOperator(ctx)
    solves = {}
    for krylov in ("auto", "full"):
        solver = T.TransportSolver(ctx, rtol=rtol, restart=restart, max_it=max_it, krylov=krylov)
        for adjoint in (False, True):
            run = solver.solve_adjoint if adjoint else solver.solve
            xs = []
            for _ in range(6 if krylov == "auto" else 1):
                x = torch.zeros_like(b)
                try:
                    run(b, x)
                except T._lib.UboltError as e:
                    assert e.status == 5 and restart < 33  # not converged: the fixed number of steps
                xs.append(x)
            assert all(torch.equal(x, xs[0]) for x in xs[1:])
            r = b - (op.mult_transpose(xs[0]) if adjoint else op.mult(xs[0]))
            solves[krylov, adjoint] = xs[0], float(torch.linalg.norm(r) / torch.linalg.norm(b))
    for adjoint in (False, True):
        x1, r1 = solves["auto", adjoint]
        x2, r2 = solves["full", adjoint]
        if restart >= 33:
            assert r1 <= 1.01 * rtol and r2 <= 1.01 * rtol
        else:
            # The same Krylov space: the same minimal residual, up to rounding
            assert abs(r1 - r2) <= 1e-8 * r2
    ctx.close()


def test_the_solves_above_need_long_bases():
    ctx, keep, b = diffusive("many_blocks")
    x, s = T.TransportSolver(ctx, rtol=1e-9, restart=200, max_it=400).solve(b)
    assert s["krylov"] == 2 and s["iterations"] > 33
    ctx.close()


@pytest.mark.parametrize("block", [0, 7, 35])
def test_a_wait_that_gives_up_fails_the_solve(block):
    """Whichever block's wait runs out, the solve reports it, and the next
    one is as before."""
    ctx, keep, b = diffusive("many_blocks")
    solver = T.TransportSolver(ctx, rtol=1e-9, restart=200, max_it=400)
    ref, s = solver.solve(b)
    T._lib.check(T.lib.ubolt_solve_test_wait(ctx.handle, 2000, block))
    with pytest.raises(T._lib.UboltError) as e:
        solver.solve(b)
    assert e.value.status == 6  # UBOLT_ERR_TIMEOUT
    T._lib.check(T.lib.ubolt_solve_test_wait(ctx.handle, 1 << 24, -1))
    x, s2 = solver.solve(b)
    assert torch.equal(x, ref) and s2["iterations"] == s["iterations"]
    ctx.close()
