"""The CG-SUPG multiply where its blocks change: stars that fill more than one
chunk, few ordinates per vertex, an ordinate count above a block's threads, and
vectors off a 16-byte boundary. Against the oracle."""
import numpy as np
import pytest
import torch

from ubolt_b200 import problem as P
from ubolt_b200 import transport as T

import cg as OC

pytestmark = pytest.mark.gpu

CASES = {
    "tri_s2": (lambda r: P.box_tris(7, 5, jitter=0.2, rng=r), 2),
    "quad_s18": (lambda r: P.box_quads(6, 5, jitter=0.2, rng=r), 18),
    "tet_s2": (lambda r: P.box_tets(3, 4, 3, jitter=0.1, rng=r), 2),
    "tet_s8": (lambda r: P.box_tets(3, 3, 3, jitter=0.1, rng=r), 8),
    "hex_s2": (lambda r: P.box_hexes(5, 4, 5), 2),
    "hex_s12": (lambda r: P.box_hexes(3, 2, 3), 12),
}


def offset_copy(a, off):
    t = torch.empty(len(a) + 8, dtype=a.dtype, device="cuda")[off:off + len(a)]
    t.copy_(a)
    return t


@pytest.mark.parametrize("case", CASES)
def test_cg_apply_matches_oracle(case):
    make, sn = CASES[case]
    rng = np.random.default_rng(9)
    m = make(rng)
    g, q = P.build_cg_geometry(m), P.lqn(m.dim, sn)
    st = rng.uniform(0.2, 4.0, g.n_elements)
    ss = st * rng.uniform(0.2, 0.9, g.n_elements)
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(ss, device="cuda"))
    ctx.set_group(*keep)
    ref_op = OC.Problem(m, q, st, ss)
    matrices = {True: ref_op.matrix(), False: ref_op.supg_matrix()}
    op = T.TransportOperator(ctx)
    x = rng.standard_normal(ctx.n_rows)
    for scatter, mult in ((True, op.mult), (False, op.mult_unscattered)):
        ref = matrices[scatter] @ x
        for off in (0, 1):
            y = mult(offset_copy(torch.tensor(x, device="cuda"), off), offset_copy(torch.zeros(ctx.n_rows, dtype=torch.float64), off))
            assert np.abs(y.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
            y32 = mult(offset_copy(torch.tensor(x, dtype=torch.float32, device="cuda"), off),
                       offset_copy(torch.zeros(ctx.n_rows, dtype=torch.float32), off))
            assert np.abs(y32.double().cpu().numpy() - ref).max() <= 1e-4 * np.abs(ref).max()
    ctx.close()
