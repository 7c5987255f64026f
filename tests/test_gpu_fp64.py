"""FP64 evaluation kernels at the sizes where their work division changes:
chunks of 256 targets, lanes by powers of two, segments of the interaction
lists, every degree, the symmetric pairs' leaf range, and arguments outside
the kernels' short forms.  Against the CPU oracle (a restatement of the
reference in FP64) or the same sums in numpy, at the FP64 parity bar."""
import numpy as np
import pytest

import barytree_b200 as B
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _cube(seed, n):
    rng = np.random.default_rng(seed)
    return (*(rng.uniform(-1, 1, n) for _ in range(3)), rng.uniform(-1, 1, n))


def _direct(t, s, q, kernel, kp):
    d2 = sum((a[:, None] - b[None, :]) ** 2 for a, b in zip(t, s))
    if kernel == 3:
        return (1.0 / np.sqrt(d2 + kp * kp)) @ q
    with np.errstate(divide="ignore"):
        k = np.exp(-kp * np.sqrt(d2)) / np.sqrt(d2) if kernel == 2 else 1.0 / np.sqrt(d2)
    return np.where(d2 > 0, k, 0.0) @ q


@pytest.mark.parametrize("kernel,kp", [(1, 0.0), (2, 0.7), (3, 1e-2)])
@pytest.mark.parametrize("nt", [1, 2, 3, 31, 33, 64, 65, 127, 128, 129, 255, 256, 257, 700])
def test_direct_sum_at_every_lane_split(kernel, kp, nt):
    x, y, z, q = _cube(nt, 3001)
    t = [x[:nt], y[:nt], z[:nt]]                    # targets among the sources: skipped pairs
    ref = _direct(t, (x, y, z), q, kernel, kp)
    assert _rel(B.direct(*t, x, y, z, q, kernel, kp), ref) <= TOL


@pytest.mark.parametrize("ctype", [1, 2, 3])
@pytest.mark.parametrize("degree", range(1, 13))
def test_every_degree(ctype, degree):
    x, y, z, q = _cube(degree, 5000)
    kernel, kp = (degree % 3) + 1, 0.3
    kw = dict(compute_type=ctype, degree=degree, theta=0.8, max_source_leaf=150, max_target_leaf=90)
    ref = O.treecode(x, y, z, None, x, y, z, q, None, kernel, [kp], 1, 1, ctype, 0.8, degree, 150, 90, 1.0, -1.0, 0)
    assert _rel(B.treecode(x, y, z, x, y, z, q, kernel=kernel, kernel_param=kp, **kw), ref) <= TOL


@pytest.mark.parametrize("kernel,kp", [(1, 0.0), (2, 0.7), (3, 1e-2)])
@pytest.mark.parametrize("ctype,sleaf,tleaf", [(1, 3, 3), (1, 10, 10), (1, 70, 10), (2, 10, 40), (3, 10, 10), (1, 40, 130)])
def test_source_nodes_smaller_than_a_group_of_four_per_thread(kernel, kp, ctype, sleaf, tleaf):
    x, y, z, q = _cube(sleaf + tleaf, 3000)
    kw = dict(compute_type=ctype, degree=3, theta=0.7, max_source_leaf=sleaf, max_target_leaf=tleaf)
    ref = O.treecode(x, y, z, None, x, y, z, q, None, kernel, [kp], 1, 1, ctype, 0.7, 3, sleaf, tleaf, 1.0, -1.0, 0)
    assert _rel(B.treecode(x, y, z, x, y, z, q, kernel=kernel, kernel_param=kp, **kw), ref) <= TOL


@pytest.mark.parametrize("kernel,kp", [(1, 0.0), (2, 0.7), (3, 1e-2)])
@pytest.mark.parametrize("n,leaf", [(4200, 600), (6000, 800), (9000, 1200), (14000, 2048)])
def test_symmetric_pairs(kernel, kp, n, leaf):
    """Leaves of 512 to 2048 particles in pairs; the rest direction by direction."""
    x, y, z, q = _cube(n, n)
    kw = dict(kernel=kernel, kernel_param=kp, degree=6, theta=0.7, max_source_leaf=leaf, max_target_leaf=leaf)
    sym, rep = B.treecode(x, y, z, x, y, z, q, return_report=True, **kw)
    off = B.treecode(x, y, z, x, y, z, q, symmetry=B.SYMMETRY_OFF, **kw)
    assert rep["sym_ptwise"] > 0
    assert _rel(sym, off) <= 1e-13
    assert np.array_equal(sym, B.treecode(x, y, z, x.copy(), y.copy(), z.copy(), q, **kw))
    # beside a system with targets of its own: the same bits as alone
    other = _cube(n + 1, 3000)
    systems = [(*other[:3], x, y, z, q), (x, y, z, x, y, z, q)]
    assert np.array_equal(B.treecode_batch(systems, **kw)[1], sym)
    assert np.array_equal(B.treecode_batch(systems, tree_build=B.TREE_HOST, **kw)[1], sym)


@pytest.mark.parametrize("approx", [1, 2])
def test_few_items_and_many_items_give_the_same_bits(approx):
    """A system evaluated alone (a block per list segment) and inside a batch
    with enough work items for one block per item."""
    rng = np.random.default_rng(7)
    one = _cube(1, 20000)
    big = tuple(rng.uniform(-1, 1, 1_300_000) for _ in range(4))
    kw = dict(approximation=approx, degree=3, theta=0.9, max_source_leaf=500, max_target_leaf=500,
              size_check=1.0 if approx == 1 else 4.0)
    sys_of = lambda p: (*p[:3], *p[:3], p[3])  # noqa: E731
    alone = B.treecode(*sys_of(one), **kw)
    assert np.array_equal(B.treecode_batch([sys_of(one), sys_of(big)], **kw)[0], alone)


@pytest.mark.parametrize("ctype", [1, 2, 3])
@pytest.mark.parametrize("approx", [1, 2])
def test_exponentials_that_all_underflow_sum_to_zero(ctype, approx):
    """Clouds four apart at kappa = 200: every exp(-kappa r) is zero in FP64."""
    if (ctype, approx) == (3, 2):
        pytest.skip("cluster-cluster Hermite is not provided")
    x, y, z, q = _cube(6, 4000)
    kw = dict(kernel=2, kernel_param=200.0, compute_type=ctype, approximation=approx, degree=4, theta=0.7,
              max_source_leaf=100, max_target_leaf=100, size_check=1.0 if approx == 1 else 4.0)
    assert np.all(B.treecode(x + 6.0, y, z, x, y, z, q, **kw) == 0.0)
    assert np.all(B.direct(x + 6.0, y, z, x, y, z, q, 2, 200.0) == 0.0)
    # subtraction: the correction alone is left
    tq = np.abs(q)
    c = 4.0 * np.pi / 200.0 / 200.0
    ss = B.direct(x + 6.0, y, z, x, y, z, q, 2, 200.0, singularity=B.Singularity.SUBTRACTION, target_q=tq,
                  source_w=np.ones_like(q))
    assert np.array_equal(ss, c * tq)


@pytest.mark.parametrize("ctype,approx", [(1, 1), (1, 2), (2, 1), (3, 1)])
def test_range_of_exponentials_does_not_change_a_system(ctype, approx):
    """A system within the short exponential's range keeps its bits in a batch
    beside one beyond it (which runs the whole batch on the other kernels)."""
    one, wide = _cube(8, 9000), _cube(9, 3000)
    sys_of = lambda p, s: (*(a * s for a in p[:3]), *(a * s for a in p[:3]), p[3])  # noqa: E731
    kw = dict(kernel=2, kernel_param=50.0, compute_type=ctype, approximation=approx, degree=5, theta=0.8,
              max_source_leaf=1200, max_target_leaf=1200, size_check=1.0 if approx == 1 else 4.0)
    alone = B.treecode(*sys_of(one, 1.0), **kw)                  # 50 * 2 sqrt(3) = 173
    pots = B.treecode_batch([sys_of(one, 1.0), sys_of(wide, 20.0)], **kw)
    assert np.array_equal(pots[0], alone)
    x, y, z, q = sys_of(wide, 20.0)[3:]
    assert _rel(pots[1], _direct((x, y, z), (x, y, z), q, 2, 50.0)) <= 1e-8


def test_growing_exponential_takes_the_short_forms():
    """kappa < 0: the same kernels and pairs as a decaying one, at about their
    time (the library's exp in every sum took four times as long)."""
    x, y, z, q = _cube(5, 60000)
    kw = dict(kernel=2, degree=6, theta=0.7, max_source_leaf=1000, max_target_leaf=1000)
    ms = {}
    for kp in (0.5, -0.5):
        best = []
        for _ in range(4):
            _, rep = B.treecode(x, y, z, x, y, z, q, kernel_param=kp, return_report=True, **kw)
            assert rep["sym_ptwise"] > 0
            best.append(rep["ms_eval_kernel"])
        ms[kp] = min(best[1:])
    assert ms[-0.5] <= 2.0 * ms[0.5], ms
    near = dict(kw, theta=1e-9, max_source_leaf=800, max_target_leaf=800)      # every pair of leaves direct
    p = [a[:6000] for a in (x, y, z, q)]
    got, rep = B.treecode(*p[:3], *p, kernel_param=-0.5, return_report=True, **near)
    assert rep["sym_ptwise"] > 0
    assert _rel(got, _direct(p[:3], p[:3], p[3], 2, -0.5)) <= TOL


@pytest.mark.parametrize("kernel,kp,scale", [(1, 0.0, 1e160), (1, 0.0, 1e-160), (3, 0.0, 1e-160), (2, -0.4, 1.0),
                                              (2, 900.0, 1.0), (2, 0.0, 1.0), (2, 1e-3, 1e160), (2, -400.0, 1.0)])
def test_arguments_outside_the_short_forms(kernel, kp, scale):
    """Squares that overflow or underflow, a growing exponential, one that
    underflows: what the library functions give, term by term.  Leaves of
    about 750 particles, so that the pair kernel meets them too."""
    x, y, z, q = _cube(3, 6000)
    x, y, z = x * scale, y * scale, z * scale
    with np.errstate(all="ignore"):
        d2 = sum((a[:, None] - a[None, :]) ** 2 for a in (x, y, z))
        if kernel == 2:
            r = np.sqrt(d2)
            ref = np.where(r > np.finfo(float).tiny, np.exp(-kp * r) / r, 0.0) @ q
        elif kernel == 3:
            ref = (1.0 / np.sqrt(d2)) @ q
        else:
            ref = np.where(d2 > np.finfo(float).tiny, 1.0 / np.sqrt(d2), 0.0) @ q
    got = [B.direct(x, y, z, x, y, z, q, kernel, kp)]
    kw = dict(kernel=kernel, kernel_param=kp, degree=3, max_source_leaf=800, max_target_leaf=800, theta=1e-9)
    pot, rep = B.treecode(x, y, z, x, y, z, q, return_report=True, **kw)            # near field only, pairs
    assert rep["sym_ptwise"] > 0
    got.append(pot)
    got.append(B.treecode(x, y, z, x, y, z, q, symmetry=B.SYMMETRY_OFF, **kw))
    for g in got:
        ok = np.isfinite(ref)
        assert np.array_equal(np.isfinite(g), ok)
        top = np.max(np.abs(ref[ok]), initial=0.0)            # (the squares of the norm overflow at 1e300)
        if top > 0:
            assert _rel(g[ok] / top, ref[ok] / top) <= 1e-12
        else:
            assert np.all(g[ok] == ref[ok])


def test_charge_that_is_not_finite_goes_through_the_pairs():
    """A NaN charge reaches every potential but its own particle's (the pair
    with itself is skipped), through the pair kernel's second route."""
    x, y, z, q = _cube(4, 6000)
    q[1234] = np.nan
    ref = _direct((x[1234:1235], y[1234:1235], z[1234:1235]), tuple(np.delete(a, 1234) for a in (x, y, z)),
                  np.delete(q, 1234), 1, 0.0)
    pot, rep = B.treecode(x, y, z, x, y, z, q, degree=3, max_source_leaf=800, max_target_leaf=800, theta=1e-9,
                          return_report=True)
    assert rep["sym_ptwise"] > 0
    assert np.array_equal(np.flatnonzero(~np.isnan(pot)), [1234])
    assert abs(pot[1234] - ref[0]) <= TOL * abs(ref[0])


# The short forms themselves, one kernel value per target: a unit charge at
# the origin and targets on the x axis, so that r^2 is r * r rounded once and
# the sum is the value.  Against extended precision (64 bits of mantissa).
U = 2.0 ** -53


def _values(r, kernel, kp):
    o = np.zeros(1)
    return B.direct(r, np.zeros_like(r), np.zeros_like(r), o, o, o, np.ones(1), kernel, kp)


def _radii(lo, hi, n):
    """Both exponent parities, and mantissas spread by an odd step."""
    return np.exp(np.linspace(np.log(lo), np.log(hi), n))


def test_reciprocal_root_to_the_last_place():
    """rsqrt_n: the estimate's error e leaves (5/16)|e|^3 < 2^-64 after the
    step, and the last rounding half a unit, at most 2^-53 of the value."""
    r = np.concatenate([_radii(1e-153, 1e153, 200_001), _radii(0.5, 8.0, 100_001)])
    r2 = r * r
    exact = 1.0 / np.sqrt(r2.astype(np.longdouble))
    assert np.max(np.abs(_values(r, 1, 0.0) - exact) / exact) <= 1.01 * U
    # eps^2 in the square: one rounding more, halved by the root
    r = _radii(1e-6, 1e3, 100_001).astype(np.float32).astype(np.float64)      # r * r exact
    for eps in (1e-3, 2.0):
        exact = 1.0 / np.sqrt(r.astype(np.longdouble) ** 2 + np.longdouble(eps * eps))
        assert np.max(np.abs(_values(r, 3, eps) - exact) / exact) <= 1.52 * U


@pytest.mark.parametrize("kappa", [0.0, 1e-9, 0.37, 1.0, 64.0, -0.37, -1.0, -64.0])
def test_exponential_to_the_last_places(kappa):
    """rsqrt_sqrt_n and exp64 in the Yukawa value: half a unit each for 1/r, for
    the table entry plus polynomial (truncated below 0.36 of 2^-53) and for the
    product, and the rounding of r times the exponent; every table entry, down
    to 2^-1021, zero below 2^-1022 and, growing, up to the overflow."""
    top = 700.0 / abs(kappa) if kappa else 1e100
    r = np.concatenate([_radii(1e-12 * top, top, 200_001), np.linspace(0.001, 1.0, 100_001) * min(top, 1e3)])
    s = np.sqrt((r * r).astype(np.longdouble))
    exact = np.exp(-np.longdouble(kappa) * s) / s
    normal = exact >= 2.0 ** -1021                          # (as doubles are rounded to 53 bits)
    err = np.abs(_values(r, 2, kappa) - exact)[normal] / exact[normal]
    r = r[normal]
    assert np.max(err / (3.5 + 1.1 * np.abs(kappa) * r)) <= U
    if kappa > 0:
        far = np.linspace(1022.01, 4000.0, 1001) * np.log(2.0) / kappa
        assert np.all(_values(far, 2, kappa) == 0.0)
    if kappa < 0:
        far = np.linspace(1024.01, 4000.0, 1001) * np.log(2.0) / -kappa
        assert np.all(np.isposinf(_values(far, 2, kappa)))
