"""p123's product over assembled rows against the oracle's element-by-element
one: 16-bit and 32-bit columns, and the element products that meshes with
too many neighbours keep."""
import numpy as np
import pytest

import parafem_gb300 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def box(nx, ny, nz, shuffle):
    """A distorted box; with `shuffle` its nodes are numbered at random."""
    prob = P.box8_problem(nx, ny, nz)
    rng = np.random.default_rng(4)
    g_num, nn = prob["g_num"], prob["nn"]
    coords = np.zeros((nn, 3))
    for e in range(g_num.shape[0]):
        coords[g_num[e] - 1] = prob["g_coord"][e].T
    coords += rng.uniform(-0.1, 0.1, coords.shape)
    if shuffle:
        new = rng.permutation(nn)
        g_num = (new[g_num - 1] + 1).astype(np.int32)
        coords = coords[np.argsort(new)]
    return g_num, coords


def fan(m):
    """m bricks around a common edge, whose nodes have 4 m + 2 neighbours."""
    t = 2.0 * np.pi * np.arange(m) / m
    ring = np.stack([np.cos(t), np.sin(t)], axis=1)
    mid = 1.3 * np.stack([np.cos(t + np.pi / m), np.sin(t + np.pi / m)], axis=1)
    flat = np.vstack([[[0.0, 0.0]], ring, mid])
    coords = np.vstack([np.column_stack([flat, np.full(len(flat), z)]) for z in (0.0, 1.0)])
    n = len(flat)
    sect = np.arange(m)
    quad = np.stack([0 * sect, 1 + sect, 1 + m + sect, 1 + (sect + 1) % m], axis=1)   # counter-clockwise from the axis
    # SHAPE_DER's order: (x-, z-), (x-, z+), (x+, z+), (x+, z-) at y-, then at y+
    a, b, c, d = quad.T
    g_num = np.stack([a, a + n, b + n, b, d, d + n, c + n, c], axis=1) + 1
    return g_num.astype(np.int32), coords


def check(g_num, coords, seed=1):
    nn = coords.shape[0]
    rng = np.random.default_rng(seed)
    free = np.ones(nn, np.int32)
    free[rng.integers(0, nn, max(nn // 9, 1))] = 0
    g_g, neq = P.number_equations1(g_num, free)
    g_coord = np.ascontiguousarray(coords[g_num - 1].transpose(0, 2, 1))
    kc = O.form_storkc(g_coord, 8, 2.0, 1.0, 3.0)
    x = rng.standard_normal(neq)
    with P.Solver() as s:
        s.setup_scalar8(g_num, g_g, g_coord, nn, neq)
        s.form_storkc(8, 2.0, 1.0, 3.0)
        u = s.ebe_matvec(x, 64)
        r = O.ebe_matvec8(g_g, kc, x)
        y, it, rel = s.solve(r, 1e-12, 20000, P.MODE_FP64_RES)
        fixed = np.unique(rng.integers(1, neq + 1, 3)).astype(np.int32)
        s.set_fixed(fixed, 1e20)
        store = s.get_diag()[fixed - 1]
        uf = s.ebe_matvec(x, 64)
    full = np.concatenate([[0.0], np.abs(x)])
    mag = np.zeros(neq + 1)
    np.add.at(mag, g_g, np.einsum("eji,ej->ei", np.abs(kc), full[g_g]))
    # storkc itself agrees to 1e-13 of its largest entry; rows of fewer than 128 terms lose less than 2^-45 more
    bound = 2.0 ** -45 * mag[1:] + 128 * 1e-13 * np.abs(kc).max() * np.abs(x).max()
    assert np.all(np.abs(u - r) <= bound)
    assert rel <= 1e-11 and np.linalg.norm(y - x) <= 1e-7 * np.linalg.norm(x)
    assert np.array_equal(uf[fixed - 1], x[fixed - 1] * store)
    rest = np.setdiff1d(np.arange(neq), fixed - 1)
    assert np.array_equal(uf[rest], u[rest])


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 5), (11, 7, 9), (33, 2, 31)])
@pytest.mark.parametrize("shuffle", [False, True])
def test_rows_of_small_boxes(shape, shuffle):
    check(*box(*shape, shuffle))


def test_rows_with_32_bit_columns():
    check(*box(41, 41, 41, True))        # 74,088 nodes numbered at random: offsets beyond 16 bits


@pytest.mark.parametrize("m", [5, 15, 16, 24])   # 22, 62, 66 and 98 neighbours: rows up to 64, element products beyond
def test_fans_of_bricks(m):
    check(*fan(m))


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 2, 7), (3, 31, 30), (31, 31, 31), (33, 29, 40)])
def test_rows_streamed_through_shared_memory(shape):
    """One slice of 32 rows, a ragged last one, fewer and more slices than warps, and iterations above and below
    30,000 slots."""
    check(*box(*shape, False))


@pytest.mark.parametrize("shape,shuffle", [((5, 4, 3), False), ((11, 7, 9), True), ((33, 29, 40), False), ((41, 41, 41), True),
                                           ((260, 256, 2), False), ((256, 2, 260), False), ((2, 260, 256), False)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_a_value_that_is_not_finite_reaches_its_neighbours_only(shape, shuffle, bad):
    """Boundary rows are shorter than their slice, and padded.  In a layer of 67,077 nodes the last layer's rows have
    no column within 16 bits of those of the layer before, with which they share a slice."""
    g_num, coords = box(*shape, shuffle)
    nn = coords.shape[0]
    g_g, neq = P.number_equations1(g_num, np.ones(nn, np.int32))
    g_coord = np.ascontiguousarray(coords[g_num - 1].transpose(0, 2, 1))
    x = np.random.default_rng(6).standard_normal(neq)
    with P.Solver() as s:
        s.setup_scalar8(g_num, g_g, g_coord, nn, neq)
        s.form_storkc(8, 2.0, 1.0, 3.0)
        u = s.ebe_matvec(x, 64)
        row = int(np.diff(np.unique(g_num[0]))[1]) + 1      # nodes from row to row: the last layer's slice-mates reach these
        for q in [0, neq // 2] + [max(neq - 1 - i, 1) for i in list(range(9)) + list(range(max(row - 4, 0), row + 9))]:
            xb = x.copy()
            xb[q] = bad
            ub = s.ebe_matvec(xb, 64)
            near = np.unique(g_g[(g_g == q + 1).any(axis=1)]) - 1
            far = np.setdiff1d(np.arange(neq), near)
            assert not np.isfinite(ub[near]).any() and np.array_equal(ub[far], u[far])
