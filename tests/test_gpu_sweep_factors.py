"""The factor store against the factors a sweep forms as it goes, over the shapes
of the kernel that fills it: the class records staged in shared memory or too
large for it, a warp per task or per 32 positions of one, several blocks per
patch. The same arithmetic either way: equal bits."""
import numpy as np
import pytest
import torch

from ubolt_b200 import problem as P
from ubolt_b200 import transport as T

pytestmark = pytest.mark.gpu

CASES = {
    # Few tasks: a warp per 32 positions
    "quad_few": (lambda r: P.box_quads(21, 19, jitter=0.2, rng=r), 0, 2, 0),
    "tri_few": (lambda r: P.box_tris(11, 9, jitter=0.2, rng=r), 1, 2, 100),
    "hex_few": (lambda r: P.box_hexes(7, 6, 5), 1, 2, 0),
    # More: a warp per task, patches shared by several blocks
    "tri": (lambda r: P.box_tris(48, 45, jitter=0.2, rng=r), 1, 8, 0),
    "quad": (lambda r: P.box_quads(61, 47, jitter=0.2, rng=r), 1, 8, 0),
    "tet": (lambda r: P.box_tets(9, 8, 9, jitter=0.1, rng=r), 1, 4, 0),
    "tet_dg0": (lambda r: P.box_tets(9, 8, 9, jitter=0.1, rng=r), 0, 8, 0),
    "hex": (lambda r: P.box_hexes(12, 11, 13), 1, 6, 0),
    # Records of a patch past shared memory (FP64)
    "hex_unstaged": (lambda r: P.box_hexes(12, 11, 13), 1, 4, 250),
}


@pytest.mark.parametrize("case", CASES)
def test_store_equals_factors_formed_in_the_sweep(case):
    make, order, sn, patch = CASES[case]
    rng = np.random.default_rng(31)
    m = make(rng)
    g, q = P.build_geometry(m, order), P.lqn(m.dim, sn)
    st = rng.uniform(0.3, 3.0, g.n_cells)
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(0.5 * st, device="cuda"))
    ctx.set_group(*keep)
    sw = T.Sweep(ctx, patch)
    sw.set_kernel("tasks")
    x = torch.tensor(rng.standard_normal(ctx.n_rows), device="cuda")
    stored = [sw.apply(x), sw.apply(x.float())]
    assert sw.status()["factor_bytes"] > 0
    sw.set_factor_limit(0)
    formed = [sw.apply(x), sw.apply(x.float())]
    assert sw.status()["factor_bytes"] == 0
    assert all(torch.equal(a, b) for a, b in zip(stored, formed))
    assert sw.status()["timeouts"] == 0 and bool(torch.isfinite(stored[0]).all())
    ctx.close()
