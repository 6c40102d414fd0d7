"""The DG1 applies on tets and hexes with more cells than the resident blocks
hold, so that a block walks its cells in rounds and the last round is ragged.
Against the oracle's matrix."""
import numpy as np
import pytest
import torch

import oracle as O
from ubolt_b200 import problem as P
from ubolt_b200 import transport as T

pytestmark = pytest.mark.gpu

# S8 has 80 ordinates: 20 threads a cell in FP32, so 148 SMs of 512 threads
# hold at most 3,789 cells at once (FP64: half)
MESHES = {
    "tet": lambda r: P.box_tets(9, 9, 9, jitter=0.2, rng=r),
    "hex": lambda r: P.box_hexes(16, 17, 15),
}
TOL = {torch.float64: 1e-13, torch.float32: 2e-5}


@pytest.mark.parametrize("reflect", [False, True])
@pytest.mark.parametrize("shape", MESHES)
def test_applies_in_rounds_match_oracle(shape, reflect):
    rng = np.random.default_rng(3)
    m = MESHES[shape](rng)
    g = P.build_geometry(m, 1, side_bc=[1, 0, 0, 1, 0, 0] if reflect else None)
    q = P.lqn(3, 8)
    st = rng.uniform(0.5, 2.0, g.n_cells)
    ss = st * rng.uniform(0.2, 0.9, g.n_cells)
    op = O.Operator(g, q, st, ss)
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(ss, device="cuda"))
    ctx.set_group(*keep)
    A = T.TransportOperator(ctx)
    for dtype, tol in TOL.items():
        xd = torch.tensor(rng.standard_normal(op.n), dtype=dtype, device="cuda")
        x = xd.double().cpu().numpy()
        nodes = x.reshape(-1, q.n_angles)
        st_t = np.repeat(ss, g.n_basis)[:, None] * (q.w / q.sum_weights)[None, :] * nodes.sum(axis=1)[:, None]
        for got, ref in ((A.mult(xd), op.apply(x)),
                         (A.mult_unscattered(xd), op.apply(x, scatter=False)),
                         (A.mult_transpose(xd), op.L.T @ x - st_t.ravel())):
            assert np.abs(got.double().cpu().numpy() - ref).max() < tol * np.abs(ref).max()
    ctx.close()
