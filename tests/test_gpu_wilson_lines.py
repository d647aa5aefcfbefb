"""All planar loops in the time-line gauge against the single-loop kernel
(which multiplies each loop's links up), where the two could part: loop
extents at the edges of the kernel's blocks of T, time extents split into
windows, several chunks of lines, links off SU(N), time lines that have no
inverse."""
import numpy as np
import pytest

import qcdgpu_b200 as Q

pytestmark = pytest.mark.gpu


def lattice(group, size, precision, sweeps=2, **kw):
    L = Q.Lattice(Q.default_config(group=group, size=size, precision=precision, start=Q.START_HOT,
                                   prng=Q.PRNG_PHILOX, beta=5.8 if group == 3 else 2.4, randseries=11, **kw))
    L.seed()
    L.init(Q.START_HOT)
    L.sweep(sweeps)
    return L


def check(L, Rmax, Tmax, loops, fp64=True):
    W = L.wilson_all(Rmax, Tmax, fp64_products=fp64)
    V = float(L.info().sites)
    for R, T in loops:
        w = L.wilson_sum(R, T)
        # FP64 products of up to R + T links with growing time lines: 1e-15 a factor on traces of size N,
        # as random errors of 3 V terms
        assert abs(W[R - 1, T - 1] - w) <= 1e-14 * 3 * V * L.cfg.group, (R, T, W[R - 1, T - 1], w)
    return W


@pytest.mark.parametrize("group,size,precision,rt", [
    (3, (2, 2, 2, 2), 1, (2, 2)),            # the column kernel: the smallest, the last below each limit
    (3, (8, 8, 8, 8), 1, (4, 6)),
    (3, (8, 6, 8, 12), 1, (3, 5)),
    (3, (8, 6, 8, 12), 1, (4, 4)),           # the gauge: T = 4, 5, 8, 9, 16, the edges of the blocks of T
    (2, (12, 10, 8, 10), 1, (4, 5)),
    (3, (8, 8, 8, 8), 0, (8, 8)),            # the halo is as long as the lattice
    (2, (6, 6, 6, 18), 0, (3, 9)),
    (3, (4, 4, 4, 16), 1, (4, 16)),
    (2, (10, 10, 10, 66), 1, (10, 3)),       # time extents split into windows, the last one ragged
    (3, (2, 2, 2, 150), 0, (2, 16)),
    (3, (24, 24, 24, 22), 0, (6, 3)),        # several chunks of lines, breaking inside a direction
    (3, (10, 10, 10, 6), 1, (6, 4)),         # short time extents: the column kernel, then the gauge
    (3, (10, 10, 10, 6), 1, (6, 6)),
])
def test_loops_equal_the_single_loops(group, size, precision, rt):
    L = lattice(group, size, precision)
    R, T = rt
    check(L, R, T, [(1, 1), (R, 1), (1, T), (R, T), (R, max(1, T - 1)), (max(1, R - 1), T)])
    check(L, 1, 1, [(1, 1)])
    L.close()


def test_repeated_calls_of_other_extents_share_the_scratch():
    """a larger call between two equal ones leaves the second the first's bits"""
    L = lattice(3, (6, 6, 8, 10), 0)
    a, b = L.wilson_all(3, 2), L.wilson_all(5, 5)
    L.wilson_all(6, 10)
    assert np.array_equal(L.wilson_all(3, 2), a) and np.array_equal(L.wilson_all(5, 5), b)
    L.close()


@pytest.mark.parametrize("group,size,precision", [(3, (24, 24, 24, 22), 1), (3, (20, 18, 22, 14), 0), (2, (6, 10, 8, 12), 1)])
def test_loops_do_not_depend_on_where_the_scratch_lies(group, size, precision):
    """the same bits in a context that has moved no table, and in one that has (the scratch then holds both parts,
    the first one, or all there is)"""
    A, B = lattice(group, size, precision, sweeps=1), lattice(group, size, precision, sweeps=1)
    t = B.download()
    a, b = A.wilson_all(5, 6), B.wilson_all(5, 6)
    assert np.array_equal(a, b) and np.array_equal(B.wilson_all(5, 6), a)
    assert np.array_equal(A.download(), t) and np.array_equal(A.wilson_all(5, 6), a)
    A.close()
    B.close()


@pytest.mark.parametrize("twist", [(0.0, 0.0), (0.4, 0.9)])
def test_links_off_su3(twist):
    """rows scaled by up to 3 %: the loops are products of the stored links,
    whatever their departure from SU(3)"""
    L = lattice(3, (6, 4, 6, 8), 1, phi=twist[0], omega=twist[1])      # 4 x 8 loops: the gauge
    t = L.download()
    L.upload(t * (1 + 0.01 * np.random.default_rng(3).standard_normal(t.size).clip(-3, 3)))
    check(L, 4, 8, [(1, 1), (4, 8), (2, 5), (3, 1)])
    L.close()


@pytest.mark.parametrize("size,loops", [((4, 4, 4, 64), (4, 8)), ((4, 4, 4, 150), (4, 10)), ((8, 6, 8, 16), (4, 6))])
def test_time_lines_near_singular_with_unit_determinant(size, loops):
    """row 1 of every link times s, row 2 over s, s = e^(+-0.4): determinants stay 1 while a time line grows
    singular to rounding (its condition to 1e8 at N4 = 64), so no loop may be taken through its inverse"""
    L = lattice(3, size, 1)
    t = L.download().reshape(12, -1, 4)
    g = np.exp(0.4 * np.random.default_rng(5).choice([-1.0, 1.0], size=(4,) + t.shape[1:2]))
    t[0:8, :, :3] *= np.tile(g, (2, 1))[:, :, None]      # row 1: x, y, z of planes 0-3 (real), 4-7 (imaginary)
    t[0:8, :, 3] /= np.tile(g, (2, 1))                   # row 2: w there, and planes 8-11
    t[8:12] /= g[:, :, None]
    L.upload(t.ravel())
    R, T = loops
    W = L.wilson_all(R, T)
    V = float(L.info().sites)
    for r, u in [(1, 1), (1, T), (2, 2), (R, T)]:
        n = 2 * (r + u)
        # n factors of norm e^0.4, some 8 roundings a product, traces of size 3 of 3 V loops, twice (both sides)
        tol = 2 * 3 * V * 3 * n * 8 * 1.2e-16 * np.exp(0.4 * n)
        assert abs(W[r - 1, u - 1] - L.wilson_sum(r, u)) <= tol, (r, u, W[r - 1, u - 1], L.wilson_sum(r, u), tol)
    L.close()


def test_time_lines_without_an_inverse_take_the_general_path():
    """a field of zeros (a context that was never started) has sums 0"""
    L = Q.Lattice(Q.default_config(group=3, size=(6, 6, 6, 6), precision=0, prng=Q.PRNG_PHILOX))
    assert np.all(L.wilson_all(5, 5) == 0.0) and np.all(L.wilson_all(5, 5, fp64_products=False) == 0.0)
    L.seed()
    L.init(Q.START_COLD)
    assert np.all(L.wilson_all(6, 6) == 3 * 3 * 6 ** 4)
    L.close()
