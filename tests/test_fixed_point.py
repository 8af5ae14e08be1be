"""FP64 element products in 64-bit fixed point: the record layout and walk on
the CPU, and the GPU products against extended precision."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

import parafem_gb300 as P
from parafem_gb300 import _build


# ---------------------------------------------------------------------------
# the record and the warp's walk, restated
EXP, D0, D11, D15, CHUNK0, CHUNK = 0, 128, 608, 848, 5184, 4800      # byte offsets and chunk sizes
RECORD = CHUNK0 + 2 * CHUNK


def row_off(s, h):
    """Byte offset in the record of row h of block diagonal s = 1..15."""
    if s == 15:
        return D15 + 240 * h
    if s > 10:
        return D15 + 480 + 960 * (14 - s) + 480 * h
    return (CHUNK0 if s > 5 else CHUNK0 + CHUNK) + 960 * ((10 - s) % 5) + 480 * h


def word_entry(w):
    """Entry (i, k) of 8-byte word w of a record, None for the exponents and the padding."""
    if w < D0 // 8:
        return None
    if w < D11 // 8:
        v = w - D0 // 8
        return v - v % 2, v
    if w < D15 // 8:
        return (2 * (w - D11 // 8) + 1,) * 2
    w14 = D15 // 8 + 60
    if w < w14:
        v = w - D15 // 8
        lane = (v % 30) // 2
        return 2 * lane + v // 30, 2 * (lane + 15) + v % 2
    first = w < CHUNK0 // 8
    v = w - (w14 if first else CHUNK0 // 8)
    s, r = (14 if first else 10) - v // 120, v % 120
    if first and s < 11:
        return None
    lane = (r % 60) // 2
    return 2 * lane + r // 60, 2 * ((lane + s) % 30) + r % 2


def test_record_holds_every_entry_of_a_symmetric_matrix_once():
    got = [word_entry(w) for w in range(RECORD // 8)]
    got = [tuple(sorted(g)) for g in got if g]
    assert sorted(got) == sorted((i, k) for i in range(60) for k in range(i, 60))


def walk(rec, p):
    """The product by the lanes' walk: sums handed to the next lane at every block diagonal from 15 down."""
    f = np.zeros((30, 2))
    t = np.zeros((30, 2))
    own = p.reshape(30, 2)
    for lane in range(30):
        at = D0 // 8 + 2 * lane
        k00, k01 = rec[at], rec[at + 1]
        f[lane] += np.array([[k00, k01], [k01, rec[D11 // 8 + lane]]]) @ own[lane]
    for s in range(15, 0, -1):
        t = np.roll(t, 1, axis=0)                        # lane l takes the sums of lane l - 1
        for lane in range(30 if s < 15 else 15):
            rows = [row_off(s, h) // 8 + 2 * lane for h in (0, 1)]
            k = np.array([rec[at:at + 2] for at in rows])
            f[lane] += k @ own[(lane + s) % 30]
            t[lane] += k.T @ own[lane]
    return (f + np.roll(t, 1, axis=0)).ravel()


def test_walk_gives_the_product():
    rng = np.random.default_rng(0)
    a = rng.integers(-50, 50, (60, 60)).astype(float)
    k = a + a.T
    p = rng.integers(-50, 50, 60).astype(float)
    rec = np.array([k[word_entry(w)] if word_entry(w) else np.nan for w in range(RECORD // 8)])
    assert np.array_equal(walk(rec, p), k @ p)           # small whole numbers: exact in any order


def split(v):
    low = ((v + (1 << 28)) % (1 << 29)) - (1 << 28)
    return (v - low) >> 29, low


@pytest.mark.parametrize("v", [0, 1, -1, (1 << 28) - 1, 1 << 28, -(1 << 28), -(1 << 28) - 1, (1 << 57) - 1, 1 << 57, -(1 << 57)])
def test_words_stay_in_32_bits_and_sums_in_63(v):
    high, low = split(v)
    assert high * (1 << 29) + low == v
    assert abs(high) <= 1 << 28 and abs(low) <= 1 << 28
    assert 60 * (1 << 28) ** 2 < 1 << 63 and 60 * 2 * (1 << 28) ** 2 < 1 << 63


# ---------------------------------------------------------------------------
def mesh(nx, ny, nz, amp, size=(1.0, 1.0, 1.0)):
    g_num, g_coord, nn = P.mesh_cube(nx, ny, nz)
    rng = np.random.default_rng(5)
    coords = np.zeros((nn, 3))
    for e in range(g_num.shape[0]):
        coords[g_num[e] - 1] = g_coord[e].T
    coords = (coords + rng.uniform(-amp, amp, (nn, 3))) * np.array(size)
    fix = P.cube_restraints(nx, ny, nz, 1, nn)
    g_g, neq = P.number_equations(g_num, fix)
    return g_num, np.ascontiguousarray(coords[g_num - 1].transpose(0, 2, 1)), nn, g_g, neq


def reference(km, g_g, p):
    """K p in extended precision; per row the sum of |K_ij p_j|, and the sum over its elements of
    sqrt(K_ii) max_j sqrt(K_jj) |p_j|, the size of the element's scaled product."""
    full = np.concatenate([[0], p.astype(np.longdouble)])
    pe = full[g_g]
    ue = np.einsum("eji,ej->ei", km.astype(np.longdouble), pe)
    me = np.einsum("eji,ej->ei", np.abs(km).astype(np.longdouble), np.abs(pe))
    root = np.sqrt(np.abs(np.einsum("eii->ei", km)))
    se = root * (root * np.abs(pe)).max(axis=1, keepdims=True)
    out = [np.zeros(p.size + 1, np.longdouble) for _ in range(3)]
    for o, v in zip(out, (ue, me, se)):
        np.add.at(o, g_g, v)
    return [o[1:] for o in out]


SHAPES = [((3, 2, 3), 0.08, (1, 1, 1)), ((1, 1, 1), 0.0, (1, 1, 1)), ((5, 4, 2), 0.05, (100.0, 1.0, 0.02)), ((9, 1, 7), 0.0, (1e-3, 1e-3, 2e-3))]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,amp,size", SHAPES)
@pytest.mark.parametrize("field", ["random", "smooth", "graded", "sparse", "tiny"])
def test_products_against_extended_precision(shape, amp, size, field):
    """Per row and element, in units of 2^(-s_i) and the largest |p_j| 2^(-s_j)
    rounded up to a power of two: entries of K' and p' lose 2^-58 each and the
    low x low products 2^-58, 60 terms of each: below 2^-50.  Those units are
    below eight times sqrt(K_ii) max_j sqrt(K_jj) |p_j|, hence 2^-47 of `size`;
    up to eight elements' results are then rounded and summed in FP64 (2^-49
    of the sum of |K_ij p_j|).  As a whole the error stays below that of a sum
    of FP64 FMA, about half an ulp of the sum of |K_ij p_j|."""
    g_num, g_coord, nn, g_g, neq = mesh(*shape, amp, size)
    nels = g_num.shape[0]
    e, v = P.random_material(nels, 3, 1.0, 1000.0, 0.2, 0.35)
    rng = np.random.default_rng(11)
    p = {"random": rng.standard_normal(neq), "smooth": 1.0 + 1e-6 * rng.standard_normal(neq),
         "graded": rng.standard_normal(neq) * np.exp(-6.0 * rng.random(neq)),
         "sparse": np.where(rng.random(neq) < 0.03, rng.standard_normal(neq), 0.0),
         "tiny": 1e-300 * rng.standard_normal(neq)}[field]
    with P.Solver() as s:
        s.setup(g_num, g_g, g_coord, nn, neq)
        s.set_material(e, v)
        s.form_storkm(27)
        u = s.ebe_matvec(p, 64)
        km = s.get_storkm()
    ref, mag, big = reference(km, g_g, p)
    err = np.abs(u - ref)
    assert np.all(err <= 2.0 ** -47 * big + 2.0 ** -49 * mag + 1e-320)
    assert np.linalg.norm(err.astype(float)) <= 2.0 ** -53 * np.linalg.norm(mag.astype(float)) + 1e-320


@pytest.mark.gpu
def test_asymmetric_and_indefinite_matrices_take_the_fma_products():
    """pf_set_storkm accepts any matrix with a diagonal; the records hold symmetric, positive ones only."""
    g_num, g_coord, nn, g_g, neq = mesh(2, 3, 2, 0.0)
    rng = np.random.default_rng(2)
    p = rng.standard_normal(neq)
    for kind in ("asymmetric", "indefinite"):
        a = rng.standard_normal((g_num.shape[0], 60, 60))
        km = a if kind == "asymmetric" else a + a.transpose(0, 2, 1)
        with P.Solver() as s:
            s.setup(g_num, g_g, g_coord, nn, neq)
            s.set_storkm(km)
            u = s.ebe_matvec(p, 64)
        ref, mag, _ = reference(km, g_g, p)
        assert np.all(np.abs(u - ref) <= 2.0 ** -44 * mag)


@pytest.mark.gpu
def test_non_finite_values_stay_non_finite():
    g_num, g_coord, nn, g_g, neq = mesh(2, 2, 2, 0.0)
    with P.Solver() as s:
        s.setup(g_num, g_g, g_coord, nn, neq)
        s.set_material(100.0, 0.3)
        s.form_storkm(27)
        for bad in (np.nan, np.inf, -np.inf):
            p = np.ones(neq)
            p[neq // 2] = bad
            u = s.ebe_matvec(p, 64)
            assert not np.isfinite(u[neq // 2])
        assert not s.ebe_matvec(np.zeros(neq), 64).any()


def wide_fields(neq, rng):
    """Values of very different size inside an element: most rows' terms are small beside the element's largest."""
    one = np.zeros(neq)
    one[neq // 2] = 1.0
    return {"one": one, "one over noise": np.where(one > 0, 1.0, 1e-9 * rng.standard_normal(neq)),
            "few": np.where(rng.random(neq) < 0.03, rng.standard_normal(neq), 0.0),
            "20 decades": rng.standard_normal(neq) * 10.0 ** (-20.0 * rng.random(neq))}


@pytest.mark.gpu
@pytest.mark.parametrize("shape,amp,size", SHAPES)
@pytest.mark.parametrize("how", ["storkm", "one matrix", "cases"])
def test_every_row_is_as_accurate_as_by_fma(shape, amp, size, how):
    """In fixed point a row is off by 180 x 2^-58 of the scaled units (test_products_against_extended_precision), and
    only rows with a term of 2^-5 or more are left so: 2^-45.5 of the sum of their |K_ij p_j|, or twice that, since
    terms are compared by their high words.  The others are off by what 60 FP64 FMA leave, 2^-47, and the sums over
    the elements by 2^-49 of it: below 2^-43."""
    g_num, g_coord, nn, g_g, neq = mesh(*shape, 0.0 if how == "one matrix" else amp, size)
    nels = g_num.shape[0]
    fields = wide_fields(neq, np.random.default_rng(12))
    with P.Solver() as s:
        s.setup(g_num, g_g, g_coord, nn, neq)
        if how == "one matrix":
            s.set_material(100.0, 0.3)
            one = s.form_km(1, 27)
            s.set_shared_km(one)
            km = np.repeat(np.asarray(one).reshape(1, 60, 60), nels, axis=0)
        else:
            s.set_material(*P.random_material(nels, 3, 1.0, 1000.0, 0.2, 0.35))
            s.form_storkm(27)
            km = s.get_storkm()
        if how == "cases":
            u = s.ebe_matvec_multi(np.stack(2 * list(fields.values()), axis=1), 64)
            us = [u[:, j] for j in range(len(fields))]
        else:
            us = [s.ebe_matvec(p, 64) for p in fields.values()]
    for p, u in zip(fields.values(), us):
        ref, mag, _ = reference(km, g_g, p)
        assert np.all(np.abs(u - ref) <= 2.0 ** -43 * mag)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_infinities_and_nan_reach_the_rows_that_they_reach_by_fma(bad):
    g_num, g_coord, nn, g_g, neq = mesh(3, 2, 3, 0.08)
    rng = np.random.default_rng(3)
    p = rng.standard_normal(neq)
    p[neq // 2] = bad
    with P.Solver() as s:
        s.setup(g_num, g_g, g_coord, nn, neq)
        s.set_material(100.0, 0.3)
        s.form_storkm(27)
        km = s.get_storkm()
        u = s.ebe_matvec(p, 64)
        uk = s.ebe_matvec_multi(np.repeat(p[:, None], 8, axis=1), 64)[:, 5]
    with np.errstate(invalid="ignore"):
        ref = reference(km, g_g, p)[0]
    for got in (u, uk):
        assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isfinite(got), np.isfinite(ref))
        assert np.array_equal(np.sign(got[np.isinf(ref)]), np.sign(ref[np.isinf(ref)]))


# ---------------------------------------------------------------------------
# the library's own helpers, on the host
@pytest.fixture(scope="module")
def helpers(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fix") / "fix_host.so")
    subprocess.check_call([_build.nvcc()] + _build.ARCH + ["-O1", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", _build.INCLUDE,
                           "-I", _build.SRC, os.path.join(os.path.dirname(__file__), "fix_host.cu"), "-o", so])
    L = ctypes.CDLL(so)
    L.fix_scale.argtypes = [ctypes.c_double]
    L.fix_size.argtypes = [ctypes.c_double, ctypes.c_int, ctypes.c_int]
    L.fix_entry.argtypes = [ctypes.c_double] + 3 * [ctypes.c_int] + 2 * [ctypes.POINTER(ctypes.c_int)]
    return L


def words(L, k, si, sk, extra):
    h, l = ctypes.c_int(), ctypes.c_int()
    ok = L.fix_entry(k, si, sk, extra, ctypes.byref(h), ctypes.byref(l))
    return ok, h.value, l.value


def test_offsets_are_the_restated_ones(helpers):
    assert helpers.record_bytes() == RECORD
    assert all(helpers.row_off(s, h) == row_off(s, h) for s in range(1, 16) for h in (0, 1))


@pytest.mark.parametrize("k", [1.0, 0.25, 0.2500001, 0.9999999, 2.0, 3.999, 4.0, 1e-300, 1e300, 5e-308, 1.7e308, 123.456])
def test_scaled_diagonal_lies_between_a_quarter_and_one(helpers, k):
    s = helpers.fix_scale(k)
    assert 0.25 <= Fraction(k) * Fraction(4) ** s < 1


@pytest.mark.parametrize("extra", [0, 2])
def test_words_hold_the_rounded_entry(helpers, extra):
    """K' in 57 + extra bits to half a unit, the high word within 2^(28 + extra), the low one within 2^28."""
    rng = np.random.default_rng(9)
    vals = np.concatenate([rng.uniform(-1, 1, 200) * 2.0 ** rng.integers(-80, 1, 200), [1 - 2.0 ** -53, -1 + 2.0 ** -53, 0.0, 2.0 ** -59, 2.0 ** -60]])
    for k in vals:
        for si, sk in ((0, 0), (300, -290), (-512, 512)):
            ks = float(np.ldexp(k, -si - sk))
            ok, h, l = words(helpers, ks, si, sk, extra)
            exact = Fraction(ks) * Fraction(2) ** (si + sk + 57 + extra)
            assert ok and abs(h) <= 1 << (28 + extra) and -(1 << 28) <= l < 1 << 28
            assert abs((h << 29) + l - exact) <= Fraction(1, 2)
    for k in (1.0, -1.5, np.inf, -np.inf, np.nan):
        assert not words(helpers, k, 0, 0, extra)[0]


@pytest.mark.parametrize("top", [3.9749, 3.9751])
def test_row_sums_leave_63_bits_on_both_sides_of_the_rule_for_two_more_bits(helpers, top):
    """k_pack_storkm adds fix_size over 15 entries per quarter row and gives an element two more bits when every
    quarter stays below 15.9 / 4.  Then the sums of |h| |h'| and of the two mixed products over 60 entries, h' up to
    2^28 and low words up to 2^28, stay below 2^63."""
    k = top / 15
    quarter = 15 * helpers.fix_size(k, 0, 0)
    wide = quarter >= int(15.9 / 4 * (1 << 20))
    assert wide == (top > 3.975)
    # the least quarter row that may still have the two bits, in real entries: each fix_size is an entry rounded up
    extra = 0 if wide else 2
    _, h, l = words(helpers, k, 0, 0, extra)
    full = 60 if not wide else 60 * (1 / k)             # up to |K'| = 1 everywhere
    assert full * abs(h) * (1 << 28) < 1 << 63
    assert full * abs(h) * (1 << 28) + 60 * (1 << 28) * (1 << 28) < 1 << 63


@pytest.mark.gpu
@pytest.mark.parametrize("c", [0.2649, 0.2651, 0.999])
@pytest.mark.parametrize("how", ["storkm", "one matrix", "cases"])
def test_products_at_the_largest_sums(c, how):
    """|K'_ij| = c everywhere and p_j at full scale with the signs of the row: 0.2649 has row sums of 15.894, the most
    that two more bits are given for, 0.2651 is just beyond, 0.999 the most without.  A sum beyond 63 bits would be
    off by 2^64 units.  Bound as in test_products_against_extended_precision; sqrt(K_ii) max sqrt(K_jj) |p_j| is c."""
    rng = np.random.default_rng(17)
    sign = rng.choice([-1.0, 1.0], 60)
    f = 1.0 - 1e-7 * rng.random((60, 60))
    km = c * sign[:, None] * sign[None, :] * np.minimum(f, f.T)
    g_num, g_coord, nn = P.mesh_cube(1, 1, 1)
    g_g = np.zeros((1, 60), np.int32)
    for a in range(20):
        g_g[0, 3 * a:3 * a + 3] = 3 * (g_num[0, a] - 1) + np.arange(1, 4)
    p = np.zeros(60)
    p[g_g[0] - 1] = sign * (1.0 - 1e-9 * rng.random(60))
    with P.Solver() as s:
        s.setup(g_num, g_g, g_coord, nn, 60)
        if how == "one matrix":
            s.set_shared_km(km)
        else:
            s.set_storkm(km[None])
        u = s.ebe_matvec_multi(np.repeat(p[:, None], 8, axis=1), 64)[:, 3] if how == "cases" else s.ebe_matvec(p, 64)
    ref, mag, big = reference(km[None], g_g, p)
    assert np.abs(ref).min() > 59.9 * c
    assert np.all(np.abs(u - ref) <= 2.0 ** -47 * big + 2.0 ** -49 * mag)
