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


def exact_box(sn=4):
    """A DG0 box whose side lengths are powers of two, so that a block,
    (|Ox| hy + |Oy| hx) / V + sigma_t, rounds twice and in one way only. With
    it the streaming part of every (cell, ordinate), in FP64 and in FP32."""
    m = P.box_quads(16, 8, 2.0, 4.0)
    g, q = P.build_geometry(m, 0), P.lqn(2, sn)
    hx, hy = 2.0 / 16, 4.0 / 8
    s64 = (np.abs(q.omega[:, 0]) * hy + np.abs(q.omega[:, 1]) * hx) / (hx * hy)
    o = np.abs(q.omega.astype(np.float32))
    s32 = (o[:, 0] * np.float32(hy) + o[:, 1] * np.float32(hx)) / np.float32(hx * hy)
    return g, q, s64, s32


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_dg0_quotient_is_the_division(dtype, off):
    """y = x / block, bit for bit, over the whole range of x: subnormal and
    zero numerators, quotients at the edge of overflow, infinities, NaN."""
    g, q, s64, s32 = exact_box()
    rng = np.random.default_rng(17)
    f = np.finfo(dtype)
    # As the library rounds them: sigma_t is given in FP64 and cast
    st = (10.0 ** rng.uniform(-2.0, 2.0, g.n_cells)).astype(dtype)
    b = ((s64 if dtype == np.float64 else s32)[None, :] + st[:, None]).astype(dtype).ravel()
    ctx = T.Context(g, q)
    keep = (torch.tensor(st.astype(np.float64), device="cuda"), torch.zeros(g.n_cells, dtype=torch.float64, device="cuda"))
    ctx.set_group(*keep)
    n = len(b)
    assert ctx.n_rows == n
    block = T.ElementBlockInverse(ctx)
    with np.errstate(all="ignore"):
        signs = rng.choice([-1.0, 1.0], n).astype(dtype)
        edge = np.where(b < 1, f.max * b, f.max)  # quotients next to the largest number
        for x in (signs * 2.0 ** rng.uniform(f.minexp, f.maxexp - 1, n), rng.standard_normal(n),
                  rng.integers(-9, 9, n) * f.smallest_subnormal, signs * f.smallest_normal * b,
                  edge, np.nextafter(edge, dtype(0)), np.nextafter(np.nextafter(edge, dtype(0)), dtype(0)),
                  rng.choice([0.0, -0.0, np.inf, -np.inf, np.nan], n)):
            x = np.asarray(x, dtype=dtype)
            want = x / b
            y = block.apply(offset_copy(torch.tensor(x, device="cuda"), off),
                            offset_copy(torch.zeros(n, dtype=torch.float64 if dtype == np.float64 else torch.float32), off))
            y = y.cpu().numpy()
            assert np.array_equal(np.isnan(y), np.isnan(want))
            ok = ~np.isnan(want)
            assert np.array_equal(y[ok], want[ok]) and np.array_equal(np.signbit(y[ok]), np.signbit(want[ok]))
    ctx.close()


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_zero_pivot_gives_zero(dtype, off):
    """sigma_t exactly minus the streaming part of one ordinate: that block is
    zero, and so is its row; every other row is the quotient."""
    g, q, s64, s32 = exact_box()
    s = s64 if dtype == np.float64 else s32
    st = np.ones(g.n_cells)
    st[7] = -np.float64(s[0])
    b = (s[None, :] + st.astype(dtype)[:, None]).astype(dtype)
    ctx = T.Context(g, q)
    keep = (torch.tensor(st, device="cuda"), torch.tensor(0.0 * st, device="cuda"))
    ctx.set_group(*keep)
    t = torch.float64 if dtype == np.float64 else torch.float32
    block = T.ElementBlockInverse(ctx)
    y = block.apply(offset_copy(torch.ones(ctx.n_rows, dtype=t, device="cuda"), off),
                    offset_copy(torch.full((ctx.n_rows,), 5.0, dtype=t), off)).cpu().numpy().reshape(b.shape)
    assert b[7, 0] == 0 and y[7, 0] == 0
    with np.errstate(divide="ignore"):
        assert np.array_equal(y[b != 0], (dtype(1) / b)[b != 0])
    if dtype == np.float64:
        inv = block.inverse().cpu().numpy().reshape(b.shape)
        assert inv[7, 0] == 0 and np.array_equal(inv == 0, b == 0)
    ctx.close()


@pytest.mark.parametrize("off", [0, 1])
def test_dg1_zero_pivot_gives_zero(off):
    """A box so large that the face terms, of the size of 1 / h, underflow in
    FP32 with nothing removed: columns of zeros, so every row is zero."""
    h = 2.0 ** 80
    m = P.box_quads(5, 3, 5 * h, 3 * h)
    g, q = P.build_geometry(m, 1), P.lqn(2, 4)
    assert np.float32(np.abs(g.face_own).max() * np.abs(g.face_nA).max()) != 0  # in FP64 the block is regular
    ctx = T.Context(g, q)
    zero = torch.zeros(g.n_cells, dtype=torch.float64, device="cuda")
    ctx.set_group(zero, zero)
    y = T.ElementBlockInverse(ctx).apply(offset_copy(torch.ones(ctx.n_rows, dtype=torch.float32, device="cuda"), off),
                                         offset_copy(torch.full((ctx.n_rows,), 5.0, dtype=torch.float32), off))
    assert bool((y == 0).all())
    ctx.close()


@pytest.mark.parametrize("sn", [4, 8, 12, 16])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("shape", MESHES)
def test_block_shapes_match_oracle(shape, order, sn):
    """Ordinate counts that make blocks of 96 to 160 threads, of one cell to
    dozens, and a cell walked in rounds."""
    test_block_apply_matches_oracle(shape, order, sn)
