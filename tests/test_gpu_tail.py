"""The iteration tail (node sums, updates and finish in one launch) of meshes
that the resident kernel does not take: against the C restatement of p121's
PCG, at the sizes where its slots per thread and its range end."""
import numpy as np
import pytest

import parafem_gb300 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def solver(prob, shared=False):
    s = P.Solver()
    s.setup(prob["g_num"], prob["g_g"], prob["g_coord"], prob["nn"], prob["neq"])
    s.set_material(100.0, 0.3)
    if shared:
        s.set_shared_km(s.form_km(1, 27))
    else:
        s.form_storkm(27)
    return s


@pytest.mark.parametrize("shape", [(30, 28, 29), (31, 30, 37)])
@pytest.mark.parametrize("limit", [1, 3, 12])
def test_early_iterates_match_the_oracle(shape, limit):
    """The same operations in another summation order: a few hundred ulp after 12 iterations."""
    prob = P.cube_problem(*shape)
    km = O.form_storkm(prob["g_coord"], 27, 100.0, 0.3)
    dg = O.diag(prob["g_g"], km, prob["neq"])
    with solver(prob) as s:
        for mode, test in ((P.MODE_P121, 0), (P.MODE_FP64_RES, 1)):
            _, ref, _ = O.pcg(prob["g_g"], km, dg, prob["r"], 0.0, limit, test)
            x, it, _ = s.solve(prob["r"], 0.0, limit, mode)
            assert it == limit
            assert np.abs(x - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("shape", [(30, 28, 29), (33, 36, 31)])
def test_modes_agree(shape):
    prob = P.cube_problem(*shape)
    with solver(prob) as s:
        ref, it, rel = s.solve(prob["r"], 1e-12, 20000, P.MODE_FP64_RES)
        assert rel <= 1e-11
        assert np.linalg.norm(prob["r"] - s.ebe_matvec(ref, 64)) <= 2e-11 * np.linalg.norm(prob["r"])
        y, jt, _ = s.solve(prob["r"], 1e-12, 20000, P.MODE_FP64_RES)
        assert it == jt and np.array_equal(ref, y)          # bitwise reproducible
        for mode in (P.MODE_MIXED, P.MODE_MIXED16, P.MODE_MIXED_RESTART):
            x, _, rel = s.solve(prob["r"], 1e-9, 20000, mode)
            assert rel <= 1e-9
            assert np.linalg.norm(x - ref) <= 1e-7 * np.linalg.norm(ref)
        x, _, _ = s.solve(prob["r"], 1e-11, 20000, P.MODE_P121)
        assert np.linalg.norm(x - ref) <= 1e-7 * np.linalg.norm(ref)


# 152 SMs: up to 311,296 freedoms are two per thread, 4,046,848 the most that the tail takes
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 2), (12, 11, 10), (29, 29, 28), (30, 28, 29), (68, 68, 70), (70, 69, 70)])
def test_one_element_matrix_for_all(shape):
    prob = P.cube_problem(*shape)
    with solver(prob, shared=True) as s:
        x, it, rel = s.solve(prob["r"], 1e-9, 20000, P.MODE_MIXED)
        assert rel <= 1e-9
        assert np.linalg.norm(prob["r"] - s.ebe_matvec(x, 64)) <= 2e-9 * np.linalg.norm(prob["r"])
        if shape[0] > 60:
            ref, _, _ = s.solve(prob["r"], 1e-9, 20000, P.MODE_FP64_RES)
            assert np.linalg.norm(prob["r"] - s.ebe_matvec(ref, 64)) <= 2e-9 * np.linalg.norm(prob["r"])


@pytest.mark.parametrize("graphs", [True, False])
def test_graphs_and_switches_make_no_difference(graphs):
    prob = P.cube_problem(30, 29, 29)
    out = []
    for persistent in (True, False):
        with solver(prob) as s:
            s.set_graphs(graphs)
            s.set_persistent(persistent)
            out.append(s.solve(prob["r"], 0.0, 45, P.MODE_P121)[0])
            out.append(s.solve(prob["r"], 0.0, 45, P.MODE_FP64_RES)[0])
            assert s.solve(prob["r"], 1e-6, 20000, P.MODE_MIXED)[2] <= 1e-6
    assert np.array_equal(out[0], out[2]) and np.array_equal(out[1], out[3])
    # the two modes differ in their stopping test only
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * np.abs(out[0]).max()


def test_forced_products_change_the_iterates_by_rounding_only():
    """14 warps leave shares of p.u for the tail, 12 do not; a solve in between changes nothing."""
    prob = P.cube_problem(30, 29, 29)
    with solver(prob) as s:
        a = s.solve(prob["r"], 1e-9, 20000, P.MODE_MIXED)
        s.set_tuning(1)
        b = s.solve(prob["r"], 1e-9, 20000, P.MODE_MIXED)
        s.set_tuning(0)
        c = s.solve(prob["r"], 1e-9, 20000, P.MODE_MIXED)
    assert b[2] <= 1e-9 and a[1] == c[1]
    assert np.array_equal(a[0], c[0])
    assert np.linalg.norm(a[0] - b[0]) <= 1e-7 * np.linalg.norm(a[0])


@pytest.mark.parametrize("shared", [True, False])
def test_beyond_the_tail_persistent_and_separate_kernels_agree(shared):
    """4.3 million freedoms: more than the tail takes."""
    prob = P.cube_problem(71, 70, 71)
    out = []
    with solver(prob, shared) as s:
        for persistent in (True, False):
            s.set_persistent(persistent)
            out.append([s.solve(prob["r"], 0.0, 11, m)[0] for m in (P.MODE_P121, P.MODE_FP64_RES)])
            if shared:
                out[-1].append(s.solve(prob["r"], 0.1, 200, P.MODE_MIXED)[0])
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [20, 22])
def test_elasticity_on_8_node_bricks(n):
    """27,783 freedoms (separate updates) and 36,501 (the tail behind the product of the 8-node bricks)."""
    prob = P.box8_problem(n, n, n)
    g_num, nn = prob["g_num"], prob["nn"]
    z = np.zeros(nn)
    for e in range(g_num.shape[0]):
        z[g_num[e] - 1] = prob["g_coord"][e][2]
    free = np.repeat((z > z.min() + 1e-9)[:, None], 3, axis=1)
    eq = np.where(free, np.cumsum(free.ravel(), dtype=np.int32).reshape(nn, 3), 0).astype(np.int32)
    neq = int(free.sum())
    g_g = eq[g_num - 1].reshape(-1, 24)
    r = np.zeros(neq)
    top = np.flatnonzero(z > z.max() - 1e-9)
    r[eq[top, 2] - 1] = -1.0 / top.size
    r[eq[top, 0] - 1] = 0.3 / top.size
    with P.Solver() as s:
        s.setup_solid8(g_num, g_g, prob["g_coord"], nn, neq)
        s.set_material(100.0, 0.3)
        s.form_storkm(8)
        x, _, rel = s.solve(r, 1e-11, 20000, P.MODE_FP64_RES)
        assert rel <= 1e-10
        assert np.linalg.norm(r - s.ebe_matvec(x, 64)) <= 1e-10 * np.linalg.norm(r)
        y, _, _ = s.solve(r, 1e-11, 20000, P.MODE_P121)
        assert np.linalg.norm(y - x) <= 1e-7 * np.linalg.norm(x)


@pytest.fixture(scope="module")
def beyond():
    """4.3 million freedoms, one storkm per element: the separate kernels, as the largest workloads run."""
    prob = P.cube_problem(71, 70, 71)
    with solver(prob) as s:
        yield prob, s


@pytest.mark.parametrize("mode", [P.MODE_MIXED, P.MODE_MIXED16])
def test_beyond_the_tail_mixed_solves_converge(beyond, mode):
    prob, s = beyond
    x, it, rel = s.solve(prob["r"], 1e-6, 20000, mode)
    assert it > 100 and rel <= 1e-6
    assert np.linalg.norm(prob["r"] - s.ebe_matvec(x, 64)) <= 1.01e-6 * np.linalg.norm(prob["r"])
    y, jt, _ = s.solve(prob["r"], 1e-6, 20000, mode)
    assert it == jt and np.array_equal(x, y)


@pytest.mark.parametrize("mode", [P.MODE_P121, P.MODE_FP64_RES])
def test_beyond_the_tail_graphs_and_persistent_kernels_give_the_same_iterates(beyond, mode):
    """45 iterations: 4, 8, 16 and 17 to a read of the state, 40 of them replayed from graphs where those are on."""
    prob, s = beyond
    out = []
    for graphs, persistent in ((True, False), (False, False), (True, True)):
        s.set_graphs(graphs)
        s.set_persistent(persistent)
        x, it, rel = s.solve(prob["r"], 0.0, 45, mode)
        assert it == 45
        true = np.linalg.norm(prob["r"] - s.ebe_matvec(x, 64)) / np.linalg.norm(prob["r"])
        assert abs(rel - true) <= 1e-9 * true
        out.append(x)
    s.set_graphs(True)
    s.set_persistent(False)
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


def test_beyond_the_tail_persistent_kernels_run_mixed_solves(beyond):
    prob, s = beyond
    ref = s.solve(prob["r"], 0.01, 20000, P.MODE_MIXED)
    s.set_persistent(True)
    x, it, rel = s.solve(prob["r"], 0.01, 20000, P.MODE_MIXED)
    s.set_persistent(False)
    assert it == ref[1] and rel == ref[2] and np.array_equal(x, ref[0])


def test_beyond_the_tail_8_node_bricks():
    """160^3 bricks of p123: 4,173,281 freedoms."""
    prob = P.box8_problem(160, 160, 160)
    r = np.random.default_rng(8).standard_normal(prob["neq"])
    with P.Solver() as s:
        s.setup_scalar8(prob["g_num"], prob["g_g"], prob["g_coord"], prob["nn"], prob["neq"])
        s.form_storkc(8, 1.0, 1.0, 1.0)
        x, it, rel = s.solve(r, 1e-8, 20000, P.MODE_FP64_RES)
        assert it > 30 and rel <= 2e-8
        assert np.linalg.norm(r - s.ebe_matvec(x, 64)) <= 2e-8 * np.linalg.norm(r)
        s.set_graphs(False)
        y, jt, _ = s.solve(r, 1e-8, 20000, P.MODE_FP64_RES)
        assert it == jt and np.array_equal(x, y)
