"""Small meshes, whose PCG runs as one resident kernel: against the C
restatement of p121's PCG, at the sizes where its element ring, its slots per
thread and its launches of 2000 iterations change."""
import threading

import numpy as np
import pytest

import parafem_gb300 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def solver(prob, material=(100.0, 0.3), nip=27):
    s = P.Solver()
    s.setup(prob["g_num"], prob["g_g"], prob["g_coord"], prob["nn"], prob["neq"])
    s.set_material(*material)
    s.form_storkm(nip)
    return s


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 4), (17, 1, 9), (9, 8, 7)])
@pytest.mark.parametrize("limit", [1, 2, 13])
def test_early_iterates_match_the_oracle(shape, limit):
    """The same operations in another summation order: a few hundred ulp after 13 iterations."""
    prob = P.cube_problem(*shape)
    km = O.form_storkm(prob["g_coord"], 27, 100.0, 0.3)
    dg = O.diag(prob["g_g"], km, prob["neq"])
    with solver(prob) as s:
        for mode, test in ((P.MODE_P121, 0), (P.MODE_FP64_RES, 1)):
            _, ref, _ = O.pcg(prob["g_g"], km, dg, prob["r"], 0.0, limit, test)
            x, it, _ = s.solve(prob["r"], 0.0, limit, mode)
            assert it == limit
            assert np.abs(x - ref).max() <= 1e-12 * np.abs(ref).max()


# 152 SMs: 14, 28 and 48 records of FP64, FP32 and FP16 per SM stay in shared
# memory (2,128, 4,256 and 7,296 elements); 77,824 slots are one per thread
@pytest.mark.parametrize("shape", [(13, 13, 12), (13, 13, 13), (16, 16, 16), (17, 16, 16), (20, 19, 18), (18, 18, 20), (19, 19, 21)])
def test_modes_agree_where_the_ring_and_the_slots_change(shape):
    prob = P.cube_problem(*shape)
    with solver(prob) as s:
        ref, _, rel = s.solve(prob["r"], 1e-12, 20000, P.MODE_FP64_RES)
        assert rel <= 1e-11
        u = s.ebe_matvec(ref, 64)
        assert np.linalg.norm(prob["r"] - u) <= 2e-11 * np.linalg.norm(prob["r"])
        for mode in (P.MODE_MIXED, P.MODE_MIXED16, P.MODE_MIXED_RESTART):
            x, _, rel = s.solve(prob["r"], 1e-9, 20000, mode)
            assert rel <= 1e-9
            assert np.linalg.norm(x - ref) <= 1e-7 * np.linalg.norm(ref)
        x, _, _ = s.solve(prob["r"], 1e-11, 20000, P.MODE_P121)
        assert np.linalg.norm(x - ref) <= 1e-7 * np.linalg.norm(ref)


def test_the_largest_resident_mesh_and_the_next_agree():
    """28 x 28 x 28 (311,296 slots hold it) and 30 x 29 x 29 (separate kernels): one field, two meshes of it."""
    for shape in ((28, 28, 28), (30, 29, 29)):
        prob = P.cube_problem(*shape)
        with solver(prob) as s:
            x, it, rel = s.solve(prob["r"], 1e-10, 20000, P.MODE_FP64_RES)
            y, jt, rel2 = s.solve(prob["r"], 1e-10, 20000, P.MODE_FP64_RES)
            assert it == jt and np.array_equal(x, y)          # bitwise reproducible
            assert rel <= 2e-10
            assert np.linalg.norm(prob["r"] - s.ebe_matvec(x, 64)) <= 2e-10 * np.linalg.norm(prob["r"])


def test_runs_longer_than_one_launch():
    """A heterogeneous bar needs 11,000 iterations (the C restatement: 11,368): the run goes on from launch to launch."""
    prob = P.cube_problem(2, 2, 60)
    e, v = P.random_material(240, 5, 1.0, 1000.0, 0.2, 0.35)
    with solver(prob, (e, v)) as s:
        x, it, rel = s.solve(prob["r"], 1e-9, 20000, P.MODE_FP64_RES)
        assert 10000 < it < 13000 and rel <= 2e-9
        assert s.solve(prob["r"], 0.0, 4321, P.MODE_FP64_RES)[1] == 4321
        z, kt, _ = s.solve(prob["r"], 1e-9, 40000, P.MODE_MIXED)
        assert kt > 2000
        assert np.linalg.norm(z - x) <= 1e-5 * np.linalg.norm(x)


def test_breakdown_is_reported():
    prob = P.cube_problem(3, 3, 3)
    r = prob["r"].copy()
    r[0] = np.nan
    with solver(prob) as s:
        for mode in (P.MODE_P121, P.MODE_FP64_RES):
            with pytest.raises(P.PfError, match="breakdown"):
                s.solve(r, 1e-8, 100, mode)
        x, it, rel = s.solve(prob["r"], 1e-10, 5000, P.MODE_FP64_RES)
        assert rel <= 1e-9


@pytest.mark.parametrize("mode", [P.MODE_P121, P.MODE_FP64_RES])
def test_a_negative_tolerance_is_never_met(mode):
    """The run ends at its limit, in the resident kernel, behind the products of 20- and of 8-node bricks."""
    for shape in ((3, 3, 3), (30, 29, 28)):
        prob = P.cube_problem(*shape)
        with solver(prob) as s:
            assert s.solve(prob["r"], -1.0, 9, mode)[1] == 9
    prob = P.box8_problem(32, 32, 32)
    with P.Solver() as s:
        s.setup_scalar8(prob["g_num"], prob["g_g"], prob["g_coord"], prob["nn"], prob["neq"])
        s.form_storkc(8, 1.0, 1.0, 1.0)
        assert s.solve(np.ones(prob["neq"]), -1.0, 9, mode)[1] == 9


def test_contexts_in_threads_leave_each_other_alone():
    """Resident runs of half the SMs side by side, of all of them one after the other, and iterations with the tail
    and products in between: every solve bitwise as alone."""
    jobs = [((3, 3, 3), P.MODE_P121), ((6, 6, 6), P.MODE_P121), ((6, 6, 6), P.MODE_MIXED), ((8, 8, 8), P.MODE_MIXED16),
            ((12, 11, 10), P.MODE_P121), ((30, 28, 29), P.MODE_MIXED)]
    probs = [P.cube_problem(*shape) for shape, _ in jobs]
    solvers = [solver(prob) for prob in probs]
    alone = [s.solve(q["r"], 1e-8, 20000, m) for s, q, (_, m) in zip(solvers, probs, jobs)]
    bad = []

    def run(i):
        for _ in range(8):
            x, it, _ = solvers[i].solve(probs[i]["r"], 1e-8, 20000, jobs[i][1])
            if it != alone[i][1] or not np.array_equal(x, alone[i][0]):
                bad.append(i)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s in solvers:
        s.close()
    assert not bad


def test_an_exchange_that_nothing_completes_runs_out():
    """The check runs the exchange and the bulk-copy wait, both to their limit; the context goes on."""
    prob = P.cube_problem(3, 3, 3)
    with solver(prob) as s:
        x, it, _ = s.solve(prob["r"], 1e-10, 5000, P.MODE_FP64_RES)
        before = s.launches()
        rc, msg = s.check_wait_timeout(64)
        assert rc != 0 and "code 2" in msg and s.launches() - before == 2
        y, jt, _ = s.solve(prob["r"], 1e-10, 5000, P.MODE_FP64_RES)
        assert it == jt and np.array_equal(x, y)
