"""The element-block solves: cells that do not fill the last block, ordinate
counts above a block's threads, vectors off a 16-byte boundary, blocks that
need a row swap, and singular blocks. Against the oracle's inverted blocks."""
import numpy as np
import pytest
import torch

import oracle as O
from ubolt_b200 import problem as P
from ubolt_b200 import transport as T

pytestmark = pytest.mark.gpu

MESHES = {
    "tri": lambda r: P.box_tris(11, 7, jitter=0.3, rng=r),
    "quad": lambda r: P.box_quads(9, 7, jitter=0.3, rng=r),
    "tet": lambda r: P.box_tets(3, 2, 3, jitter=0.2, rng=r),
    "hex": lambda r: P.box_hexes(3, 5, 3),
}


def offset_copy(a, off):
    """A copy of a whose first element is `off` elements past an aligned address."""
    t = torch.empty(len(a) + 8, dtype=a.dtype, device="cuda")[off:off + len(a)]
    t.copy_(a)
    return t


@pytest.mark.parametrize("sn", [2, 6, 18])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("shape", MESHES)
def test_block_apply_matches_oracle(shape, order, sn):
    rng = np.random.default_rng(5)
    m = MESHES[shape](rng)
    g, q = P.build_geometry(m, order), P.lqn(m.dim, sn)
    # Thin to thick: at small sigma_t the streaming terms put the largest
    # entry of a column off the diagonal
    st = 10.0 ** rng.uniform(-3.0, 2.0, g.n_cells)
    ss = st * 0.5
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(ss, device="cuda"))
    ctx.set_group(*keep)
    op = O.Operator(g, q, st, ss)
    inv, _ = op.block_inverse()
    x = rng.standard_normal(op.n)
    ref = op.block_apply(inv, x)
    block = T.ElementBlockInverse(ctx)
    for off in (0, 1):
        y = block.apply(offset_copy(torch.tensor(x, device="cuda"), off), offset_copy(torch.zeros(op.n, dtype=torch.float64), off))
        assert np.abs(y.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
        y32 = block.apply(offset_copy(torch.tensor(x, dtype=torch.float32, device="cuda"), off),
                          offset_copy(torch.zeros(op.n, dtype=torch.float32), off))
        assert np.abs(y32.double().cpu().numpy() - ref).max() <= 1e-4 * np.abs(ref).max()
    # The transposed blocks: <B^{-T} u, B v> = <u, v> with B v from the forward solve
    u = torch.tensor(rng.standard_normal(op.n), device="cuda")
    lhs = torch.dot(block.apply_transpose(u), torch.tensor(x, device="cuda"))
    rhs = torch.dot(u, torch.tensor(ref, device="cuda"))
    assert abs(float(lhs - rhs)) <= 1e-11 * float(torch.linalg.norm(u)) * np.linalg.norm(ref)
    ctx.close()


def test_singular_block_gives_zero():
    """DG0 with no removal and no outflow cannot be: sigma_t = minus the
    outflow of one ordinate makes that cell's block exactly zero there."""
    m = P.box_quads(6, 5)
    g, q = P.build_geometry(m, 0), P.lqn(2, 2)
    nA = g.face_nA.reshape(g.n_cells, 4, 3)
    out = np.maximum(nA[7] @ q.omega[0], 0.0)
    st = np.ones(g.n_cells)
    st[7] = -(out.sum() / g.volume[7])
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(0.0 * st, device="cuda"))
    ctx.set_group(*keep)
    x = torch.ones(ctx.n_rows, dtype=torch.float64, device="cuda")
    y = T.ElementBlockInverse(ctx).apply(x).reshape(g.n_cells, q.n_angles)
    inv = T.ElementBlockInverse(ctx).inverse().reshape(g.n_cells, q.n_angles)
    # Where the inverted block is stored as zero, the solve gives zero
    assert torch.equal(y == 0.0, inv == 0.0)
    ctx.close()
