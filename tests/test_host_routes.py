"""The host code that chooses and prepares the kernels, without a GPU: the
library's object files linked against a stand-in for the CUDA runtime
(fake_cudart.cpp) that keeps a log of the launches and can refuse
allocations and launches."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import parafem_gb300 as P
from parafem_gb300 import _build, pfgpu


@pytest.fixture(scope="session")
def fake_lib(tmp_path_factory):
    lib = _build.build()
    objs = [os.path.join(_build.OUT, os.path.splitext(s)[0] + ".o") for s in _build.CUDA_SOURCES + _build.CXX_SOURCES]
    if not all(os.path.exists(o) and os.path.getmtime(o) <= os.path.getmtime(lib) for o in objs):
        _build.build(force=True)
    out = str(tmp_path_factory.mktemp("fake"))
    cuda = os.path.join(os.path.dirname(os.path.dirname(_build.nvcc())), "include")
    so = os.path.join(out, "libpfgpu_fake.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", cuda,
                           os.path.join(os.path.dirname(__file__), "fake_cudart.cpp")] + objs + ["-o", so])
    L = ctypes.CDLL(so)
    for name, args in pfgpu._SIGS.items():
        getattr(L, name).argtypes = args
        getattr(L, name).restype = ctypes.c_int
    L.fake_used.restype = ctypes.c_longlong
    L.fake_limit.argtypes = L.fake_refuse_size.argtypes = [ctypes.c_longlong]
    L.fake_log.restype = ctypes.c_char_p
    return L


@pytest.fixture
def fake(fake_lib, monkeypatch):
    fake_lib.fake_reset()
    monkeypatch.setattr(pfgpu, "_lib", fake_lib)
    yield fake_lib
    fake_lib.fake_reset()


def kernels(fake):
    """(name, blocks) of the launches since the log was cleared."""
    return [tuple(line.rsplit(" ", 1)) for line in fake.fake_log().decode().splitlines() if " " in line]


def launched(fake, part):
    return sum(part in name for name, _ in kernels(fake))


def solver(n):
    prob = P.cube_problem(n, n, n)
    s = P.Solver()
    s.setup(prob["g_num"], prob["g_g"], prob["g_coord"], prob["nn"], prob["neq"])
    s.set_material(100.0, 0.3)
    return s, prob["r"]


@pytest.mark.parametrize("mode", [P.MODE_P121, P.MODE_FP64_RES])
def test_a_full_device_leaves_no_launch_on_freed_records(fake, mode):
    """A solve may give the fixed-point records back when an allocation fails.  No kernel may then be launched on
    them: the run takes the records, or the products that do without."""
    s, r = solver(3)
    s.form_storkm(8)
    fake.fake_limit(fake.fake_used())          # the device is full
    fake.fake_clear_log()
    s.solve(r, 1e-8, 3, mode)
    assert fake.fake_stale() == 0
    assert launched(fake, "k_pcg_resident") == 1
    s.close()


@pytest.mark.parametrize("mode", [P.MODE_P121, P.MODE_FP64_RES, P.MODE_MIXED, P.MODE_MIXED_RESTART, P.MODE_MIXED16])
def test_a_wait_that_runs_out_in_the_final_residual_fails_that_solve(fake, mode):
    """The products of the true residual wait for bulk copies; when one runs out they leave old results behind.  (Ten
    iterations, all in the resident kernel: the only k_elem_fix of the call is the residual's.)"""
    s, r = solver(3)
    s.form_storkm(8)
    fake.fake_poke(b"k_elem_fix", 6, 0, 2)
    with pytest.raises(P.PfError, match="wait timed out"):
        s.solve(r, 1e-8, 10, mode)
    fake.fake_clear_rules()
    s.solve(r, 1e-8, 10, mode)                 # reported once, not against a later call
    s.close()


def test_a_wait_that_runs_out_in_a_block_residual_fails_that_solve(fake):
    s, r = solver(3)
    s.form_storkm(8)
    rk = np.repeat(r[:, None], 8, axis=1)
    any_flag = 6 * 128 * 8 + 3 * 128 * 4       # of MState: every case wants a residual after the first update
    fake.fake_poke(b"k_mr_update1", 2, any_flag, 1)
    fake.fake_poke(b"k_mr_elem_fix", 6, 0, 2)
    with pytest.raises(P.PfError, match="wait timed out"):
        s.solve_multi(rk, 1e-8, 10, 32)
    fake.fake_clear_rules()
    fake.fake_poke(b"k_mr_update1", 2, any_flag, 1)
    s.solve_multi(rk, 1e-8, 10, 32)
    s.close()


COOPERATIVE_LAUNCH_TOO_LARGE, LAUNCH_OUT_OF_RESOURCES, NOT_SUPPORTED = 720, 701, 801


@pytest.mark.parametrize("error", [COOPERATIVE_LAUNCH_TOO_LARGE, LAUNCH_OUT_OF_RESOURCES, NOT_SUPPORTED])
@pytest.mark.parametrize("n,mode", [(3, P.MODE_P121), (3, P.MODE_MIXED), (29, P.MODE_FP64_RES), (29, P.MODE_MIXED)])
def test_where_all_sms_are_refused_the_separate_kernels_run(fake, error, n, mode):
    """3^3 elements would take the resident kernel, 29^3 the iteration tail."""
    s, r = solver(n)
    s.form_storkm(8)
    fake.fake_coop_error(error)
    fake.fake_clear_log()
    s.solve(r, 1e-8, 7, mode)
    names = [k for k, _ in kernels(fake)]
    assert not any("k_pcg_resident" in k or "k_pcg_tail" in k for k in names)
    # FP64: and one product for the residual; mixed: its one residual too
    assert launched(fake, "k_elem") == 8 and launched(fake, "k_scatter") == 8
    assert launched(fake, "k_pcg_update1") == 7 and launched(fake, "k_pcg_update2") == 7
    fake.fake_clear_log()
    s.solve(r, 1e-8, 20, mode)                 # and in graphs, from the fifth iteration on
    assert launched(fake, "captured") > 0 and launched(fake, "k_pcg_tail") == 0
    s.close()


def test_where_all_sms_are_refused_8_node_meshes_run_on(fake):
    prob = P.box8_problem(31, 31, 31)          # 32,768 slots: the iteration tail
    s = P.Solver()
    s.setup_scalar8(prob["g_num"], prob["g_g"], prob["g_coord"], prob["nn"], prob["neq"])
    s.form_storkc(8, 1.0, 1.0, 1.0)
    for error, tails in ((0, 7), (COOPERATIVE_LAUNCH_TOO_LARGE, 0)):
        fake.fake_coop_error(error)
        fake.fake_clear_log()
        s.solve(np.ones(prob["neq"]), 1e-8, 7, P.MODE_P121)
        assert launched(fake, "k_pcg_tail") == tails and launched(fake, "k_pcg_update2") == 7 - tails
    s.close()


def test_other_errors_of_a_cooperative_launch_are_reported(fake):
    s, r = solver(3)
    s.form_storkm(8)
    fake.fake_coop_error(719)                  # a launch failure
    with pytest.raises(P.PfError, match="cooperative launch"):
        s.solve(r, 1e-8, 7, P.MODE_P121)
    s.close()


RECORD = 14784                                 # bytes of one matrix's fixed-point record


@pytest.mark.parametrize("n", [3, 29])
def test_one_matrix_without_memory_for_its_record_takes_the_fma_products(fake, n):
    s, r = solver(n)
    fake.fake_refuse_size(RECORD)
    s.set_shared_km(np.eye(60))
    fake.fake_clear_log()
    s.solve(r, 1e-8, 3, P.MODE_FP64_RES)
    s.ebe_matvec(r, 64)
    assert launched(fake, "k_elem_shared64") == 5 and launched(fake, "_fix") == 0
    fake.fake_refuse_size(-1)
    s.set_shared_km(np.eye(60))
    fake.fake_clear_log()
    s.ebe_matvec(r, 64)
    assert launched(fake, "k_elem_shared_fix") == 1
    s.close()


def scalar8(fake, n=9):
    """p123's bricks; the stand-in's first slice of rows is 27 wide, so that rows are assembled."""
    prob = P.box8_problem(n, n, n)
    s = P.Solver()
    s.setup_scalar8(prob["g_num"], prob["g_g"], prob["g_coord"], prob["nn"], prob["neq"])
    fake.fake_poke(b"k_rows_width", 4, 0, 27)
    return s, np.ones(prob["neq"])


MEMORY_ALLOCATION, LAUNCH_FAILURE = 2, 719


@pytest.mark.parametrize("kernel", [b"k_rows_width", b"k_rows_fill"])
def test_rows_that_could_not_be_assembled_are_not_used(fake, kernel):
    s, r = scalar8(fake)
    s.form_storkc(8, 1.0, 1.0, 1.0)
    fake.fake_clear_log()
    s.ebe_matvec(r, 64)
    assert launched(fake, "k_row_") == 1 and launched(fake, "k_elem8") == 0
    fake.fake_fail(kernel, MEMORY_ALLOCATION)      # the element products instead
    s.form_storkc(8, 1.0, 1.0, 1.0)
    fake.fake_clear_log()
    s.ebe_matvec(r, 64)
    assert launched(fake, "k_row_") == 0 and launched(fake, "k_elem8") == 1
    fake.fake_reset()
    fake.fake_poke(b"k_rows_width", 4, 0, 27)
    fake.fake_fail(kernel, LAUNCH_FAILURE)         # an error, and no half-filled rows for later calls
    with pytest.raises(P.PfError):
        s.form_storkc(8, 1.0, 1.0, 1.0)
    fake.fake_clear_log()
    s.ebe_matvec(r, 64)
    assert launched(fake, "k_row_") == 0
    s.close()


def test_records_and_rows_give_way_to_later_allocations(fake):
    """On a device that the records or rows have filled, what a context allocates later finds their memory."""
    s, r = solver(3)
    for later in (lambda: s.set_material(np.full(27, 100.0), np.full(27, 0.3)), lambda: s.form_km(1, 8),
                  lambda: s.set_shared_km(np.eye(60))):
        s.form_storkm(8)
        fake.fake_clear_log()
        s.ebe_matvec(r, 64)
        assert launched(fake, "k_elem_fix") == 1
        fake.fake_limit(fake.fake_used())
        later()
        fake.fake_limit(-1)
    s.close()
    s, r = scalar8(fake)
    s.form_storkc(8, 1.0, 1.0, 1.0)
    fake.fake_limit(fake.fake_used())
    s.set_fixed([1, 2], 1e20)
    fake.fake_clear_log()
    s.ebe_matvec(r, 64)
    assert launched(fake, "k_row_") == 0 and launched(fake, "k_elem8") == 1
    s.close()


def names(fake):
    return {k.replace("captured ", "") for k, _ in kernels(fake)}


@pytest.mark.parametrize("n,prec,mode", [(3, 64, P.MODE_FP64_RES), (29, 64, P.MODE_FP64_RES), (29, 32, P.MODE_MIXED)])
def test_iterations_are_timed_with_the_kernels_of_a_solve(fake, n, prec, mode):
    s, r = solver(n)
    s.form_storkm(8)
    fake.fake_clear_log()
    s.solve(r, 1e-8, 20, mode)
    solve = {k for k in names(fake) if "k_pcg_resident" in k or "k_pcg_tail" in k or "k_elem" in k}
    before = s.launches()
    fake.fake_clear_log()
    s.bench_iterations(prec, 20)
    assert any("k_pcg_resident" in k or "k_pcg_tail" in k for k in solve)
    assert {k for k in solve if "k_pcg" in k} <= names(fake)
    # the launches of the timed iterations alone are counted: the initialisation's and theirs
    assert s.launches() - before == (2 + 1 if n == 3 else 2 + 2 * 20)
    s.close()


@pytest.mark.parametrize("n,mode,blocks", [(6, P.MODE_P121, 76), (7, P.MODE_P121, 152), (9, P.MODE_MIXED, 76), (10, P.MODE_MIXED, 152),
                                           (8, P.MODE_MIXED16, 76), (9, P.MODE_MIXED16, 152)])
def test_the_smallest_runs_take_half_the_sms(fake, n, mode, blocks):
    """Two of them go side by side (the stand-in has 152 SMs)."""
    s, r = solver(n)
    s.form_storkm(8)
    fake.fake_clear_log()
    s.solve(r, 1e-8, 3, mode)
    assert {int(b) for k, b in kernels(fake) if "k_pcg_resident" in k} == {blocks}
    s.close()


def test_a_grid_wide_wait_that_runs_out_fails_that_solve(fake):
    s, r = solver(29)
    s.form_storkm(8)
    fake.fake_poke(b"k_elem_fix", 6, 0, 3)     # the error word as k_pcg_tail leaves it
    with pytest.raises(P.PfError, match=r"grid-wide wait timed out \(code 3\)"):
        s.solve(r, 1e-8, 3, P.MODE_FP64_RES)
    fake.fake_clear_rules()
    s.solve(r, 1e-8, 3, P.MODE_FP64_RES)
    s.close()
