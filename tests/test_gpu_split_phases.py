"""The small-lattice phase kernel (a link's staple terms over six or three
warps, shape 0) against the one-thread-per-link kernels (shape 1), link by
link: blocks that are not full, the sizes on both sides of each limit, long
reject chains (random quads beyond the precomputed ones), several hits, the
RANLUX stream, and the graph's early launches against single phases (and
that large lattices, whose phases follow one another, equal them too)."""
import numpy as np
import pytest

import qcdgpu_b200 as Q

pytestmark = pytest.mark.gpu


def chain(shape, sweeps, **kw):
    L = Q.Lattice(Q.default_config(start=Q.START_HOT, randseries=7, reunit_every=2, **kw))
    L.seed()
    L.init(Q.START_HOT)
    L.set_shapes(shape, shape)
    L.sweep(sweeps)
    out = L.download()
    L.close()
    return out


@pytest.mark.parametrize("group", [3, 2])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("size", [(2, 2, 2, 2), (4, 2, 6, 2), (6, 6, 6, 6), (10, 10, 10, 8), (12, 12, 12, 8),
                                  (16, 16, 16, 8), (16, 16, 16, 14), (20, 20, 20, 14)])
def test_split_phases_give_the_same_chain(group, precision, size):
    kw = dict(group=group, precision=precision, size=size, beta=5.9 if group == 3 else 2.3, n_or=2, prng=Q.PRNG_PHILOX)
    assert np.array_equal(chain(0, 3, **kw), chain(1, 3, **kw))


@pytest.mark.parametrize("group,precision", [(3, 0), (3, 1), (2, 0), (2, 1)])
@pytest.mark.parametrize("prng", [Q.PRNG_PHILOX, Q.PRNG_RANLUX])
def test_split_phases_rejects_and_hits(group, precision, prng):
    """strong coupling (most first tries rejected, so the quads run past the
    table and some draws keep the link) and two hits per subgroup"""
    kw = dict(group=group, precision=precision, size=(6, 4, 6, 8), beta=0.3, nhit=3, nhitpar=2, n_or=1, prng=prng,
              prng_instances=512)
    assert np.array_equal(chain(0, 2, **kw), chain(1, 2, **kw))


@pytest.mark.parametrize("prng", [Q.PRNG_PHILOX, Q.PRNG_RANLUX])
def test_graph_sweeps_equal_single_phases(prng):
    """the graph launches phases early (their random numbers under the phase
    before); phase by phase there is nothing to overlap"""
    kw = dict(group=3, precision=0, size=(8, 8, 8, 8), beta=5.9, prng=prng, prng_instances=2048)
    L = Q.Lattice(Q.default_config(start=Q.START_HOT, randseries=7, reunit_every=2, **kw))
    L.seed()
    L.init(Q.START_HOT)
    for _ in range(2):
        for p in (1, 0):
            for d in range(4):
                if prng == Q.PRNG_RANLUX:
                    L.produce()
                L.phase(p, d)
    L.reunitarize()
    assert np.array_equal(L.download(), chain(0, 2, **kw))
    L.close()


def single_phases(L, n_or, ranlux):
    """two sweeps by single phase launches, none of them in a graph"""
    for _ in range(2):
        for kind in [Q.HEATBATH] + [Q.OVERRELAX] * n_or:
            for p in (1, 0):
                for d in range(4):
                    if ranlux and kind == Q.HEATBATH:
                        L.produce()
                    L.phase(p, d, kind)
    L.reunitarize()


@pytest.mark.parametrize("group,precision", [(3, 0), (3, 1), (2, 0), (2, 1)])
@pytest.mark.parametrize("size", [(24, 24, 24, 6), (20, 20, 20, 20), (24, 24, 24, 20)])
@pytest.mark.parametrize("mode", ["philox", "twisted", "ranlux"])
def test_every_shape_in_the_graph_equals_single_phases(group, precision, size, mode):
    """a phase reads links that the phase before wrote: whatever a graph lets
    overlap, the chain is that of launches one after another, for every shape
    and on both sides of 2^17 links a phase"""
    kw = dict(group=group, precision=precision, size=size, beta=5.9 if group == 3 else 2.3, n_or=1, nhit=4,
              prng=Q.PRNG_RANLUX if mode == "ranlux" else Q.PRNG_PHILOX, prng_instances=16384, start=Q.START_HOT,
              randseries=7, reunit_every=2)
    if mode == "twisted":
        kw.update(phi=0.4, omega=0.9)
    L = Q.Lattice(Q.default_config(**kw))

    def begin():
        L.seed()
        L.init(Q.START_HOT)

    begin()
    start = L.download()
    L.set_shapes(1, 1)
    single_phases(L, 1, mode == "ranlux")
    want = L.download()
    assert not np.array_equal(want, start)
    L.close()
    for look in ([True, False] if mode == "ranlux" else [True]):
        for shape in [0] if mode == "twisted" else [0, 3] if mode == "ranlux" else range(Q.TUNE_SHAPES):
            L = Q.Lattice(Q.default_config(**kw))
            L.set_prng_lookahead(look)
            begin()
            L.set_shapes(shape, shape)
            L.sweep(2)
            assert np.array_equal(L.download(), want), (look, shape)
            L.close()


@pytest.mark.parametrize("group,precision", [(3, 0), (3, 1), (2, 0), (2, 1)])
def test_the_tuner_times_small_lattices_as_the_sweep_runs_them(group, precision):
    """at 8^4 a phase takes less than a launch by the host, in either form.  In the graph the split heatbath takes
    0.49 (SU(3) FP64) to 0.75 (SU(3) FP32: 6.9 to 9.2 us) of the other's time, 0.77 with the graph's start (some
    4 us over 8 phases) in both; 0.85 leaves a tenth for the spread of the least of three.  (The overrelaxations lie
    closer, 2.1 to 2.3 us for SU(2) FP32, so their order is left open.)"""
    kw = dict(group=group, precision=precision, size=(8, 8, 8, 8), beta=5.9 if group == 3 else 2.3, n_or=2,
              prng=Q.PRNG_PHILOX)
    L = Q.Lattice(Q.default_config(start=Q.START_HOT, randseries=7, reunit_every=2, **kw))
    L.seed()
    L.init(Q.START_HOT)
    t = L.tune()
    assert t[0][0] < 0.85 * t[1][0] and L.shapes()[0] == 0, t
    L.sweep(3)
    assert np.array_equal(L.download(), chain(1, 3, **kw))
    L.close()
