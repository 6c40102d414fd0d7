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


def fan(n_side):
    """The unit box cut into 4 n_side triangles around its centre: one vertex
    whose star is all of them."""
    t = np.arange(n_side) / n_side
    ring = np.concatenate([np.stack([t, 0 * t], 1), np.stack([0 * t + 1, t], 1), np.stack([1 - t, 0 * t + 1], 1),
                           np.stack([0 * t, 1 - t], 1)])
    n = len(ring)
    i = np.arange(n)
    cells = np.stack([np.full(n, n), i, (i + 1) % n], axis=1).astype(np.int64)
    return P.Mesh(2, P.TRI, np.concatenate([ring, [[0.5, 0.5]]]), cells, ())


MORE = {
    # A star of 400 entries: more than a chunk in either precision, with few
    # ordinates, with a block's worth, and with more (the chunks staged again for
    # each of a block's rounds)
    "fan_s2": (lambda r: fan(100), 2),
    "fan_s8": (lambda r: fan(100), 8),
    "fan_s18": (lambda r: fan(100), 18),
    # Enough vertices for runs of ordinates where 128 threads hold several
    "quad_runs_s8": (lambda r: P.box_quads(75, 70, jitter=0.2, rng=r), 8),
    "tri_runs_s4": (lambda r: P.box_tris(115, 110, jitter=0.2, rng=r), 4),
    "tet_runs_s8": (lambda r: P.box_tets(12, 12, 11, jitter=0.1, rng=r), 8),
    "hex_runs_s6": (lambda r: P.box_hexes(15, 14, 15), 6),
    # S2 on 98304 rows and more: a thread per row on triangles, tetrahedra and
    # hexahedra in FP64
    "tri_rows_s2": (lambda r: P.box_tris(160, 155, jitter=0.2, rng=r), 2),
    "tet_rows_s2": (lambda r: P.box_tets(23, 22, 22, jitter=0.1, rng=r), 2),
    "hex_rows_s2": (lambda r: P.box_hexes(23, 22, 22), 2),
    "quad_rows_s2": (lambda r: P.box_quads(160, 155, jitter=0.2, rng=r), 2),
}


@pytest.mark.parametrize("case", MORE)
def test_cg_apply_at_its_launch_limits(case):
    make, sn = MORE[case]
    rng = np.random.default_rng(10)
    m = make(rng)
    g, q = P.build_cg_geometry(m), P.lqn(m.dim, sn)
    st = rng.uniform(0.2, 4.0, g.n_elements)
    ss = st * rng.uniform(0.2, 0.9, g.n_elements)
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(ss, device="cuda"))
    ctx.set_group(*keep)
    oracle = OC.Problem(m, q, st, ss)
    op = T.TransportOperator(ctx)
    x = rng.standard_normal(ctx.n_rows)
    for A, mult in ((oracle.matrix(), op.mult), (oracle.supg_matrix(), op.mult_unscattered)):
        want = A @ x
        for off in (0, 1):
            y = mult(offset_copy(torch.tensor(x, device="cuda"), off), offset_copy(torch.zeros(ctx.n_rows, dtype=torch.float64), off))
            assert np.abs(y.cpu().numpy() - want).max() <= 1e-12 * np.abs(want).max()
            y32 = mult(offset_copy(torch.tensor(x, dtype=torch.float32, device="cuda"), off),
                       offset_copy(torch.zeros(ctx.n_rows, dtype=torch.float32), off))
            assert np.abs(y32.double().cpu().numpy() - want).max() <= 1e-4 * np.abs(want).max()
    ctx.close()
