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


@pytest.mark.parametrize("case", ["dg0", "few_rows", "scratch"])
def test_scratch_vector_is_held_only_where_a_sweep_uses_it(case):
    """Row vectors pass through a scratch vector from two rows per cell and 8 MB
    on; nothing is held for others. A limit below either store leaves it alone."""
    m = P.box_quads(*{"dg0": (600, 500), "few_rows": (160, 150), "scratch": (256, 250)}[case])
    g, q = P.build_geometry(m, 0 if case == "dg0" else 1), P.lqn(2, 4)
    ctx = T.Context(g, q)
    sw = T.Sweep(ctx, factor_limit=0)
    vec = 8 * ctx.n_rows
    before = torch.cuda.mem_get_info()[0]
    sw.set_factor_limit(vec)
    assert sw.status()["factor_bytes"] == 0
    held = before - torch.cuda.mem_get_info()[0]
    # (the allocator's pages: 2 MB)
    assert abs(held - (vec if case == "scratch" else 0)) <= 4 << 20
    assert vec > (8 << 20 if case != "few_rows" else 6 << 20)
    ctx.close()


SCRATCH = {
    # nb > 1 and 8 MB (FP32) and more, more than 64 ordinates in equal parts (80: two
    # of 40, 180: three of 60) and in uneven ones (288: four of 58 and one of 56), node
    # counts that are no multiple of 64
    "quad_s12": (lambda r: P.box_quads(97, 89, jitter=0.2, rng=r), 12),
    "tri_s18": (lambda r: P.box_tris(51, 47, jitter=0.2, rng=r), 18),
    "hex_s16": (lambda r: P.box_hexes(13, 13, 13), 16),
    "tet_s8": (lambda r: P.box_tets(11, 11, 11, jitter=0.1, rng=r), 8),
    "hex_s8": (lambda r: P.box_hexes(21, 19, 17), 8),
    "hex_s10": (lambda r: P.box_hexes(19, 17, 15), 10),
}


@pytest.mark.parametrize("case", SCRATCH)
def test_row_sweeps_through_the_scratch_vector(case):
    """Bit for bit the direct sweep of rows (no store and no scratch vector)."""
    make, sn = SCRATCH[case]
    rng = np.random.default_rng(32)
    m = make(rng)
    g, q = P.build_geometry(m, 1), P.lqn(m.dim, sn)
    st = rng.uniform(0.3, 3.0, g.n_cells)
    ctx = T.Context(g, q)
    assert 4 * ctx.n_rows >= 8 << 20 and ctx.n_nodes % 64 != 0
    keep = (torch.tensor(st, device="cuda"), torch.tensor(0.5 * st, device="cuda"))
    ctx.set_group(*keep)
    sw = T.Sweep(ctx)
    x = torch.tensor(rng.standard_normal(ctx.n_rows), device="cuda")
    keep_x = x.clone()
    through = [sw.apply(x), sw.apply(x.float())]
    sw.set_factor_limit(0)
    direct = [sw.apply(x), sw.apply(x.float())]
    assert all(torch.equal(a, b) for a, b in zip(through, direct)) and torch.equal(x, keep_x)
    assert sw.status()["timeouts"] == 0 and bool(torch.isfinite(direct[0]).all())
    ctx.close()
