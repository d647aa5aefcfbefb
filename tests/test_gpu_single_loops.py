"""The single Wilson loop with the lines shared in a block (time extents that
fill its threads) against products of the links taken in numpy, at the edges
of its blocks: columns that do not divide the block or the lattice, a full
column a block, extents handed to the general kernel; and the one-pass
profiles against the separate ones."""
import numpy as np
import pytest

import _oracle as O
import qcdgpu_b200 as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,size,precision,loops", [
    (3, (2, 2, 2, 2), 1, [(1, 1), (2, 1), (1, 2), (2, 2)]),  # 64 columns a block, 8 in the lattice
    (3, (8, 4, 10, 6), 0, [(8, 1), (7, 2), (6, 1), (4, 6)]), # 21 columns of 6: two threads idle, the last block ragged
    (2, (8, 6, 4, 18), 1, [(8, 2), (7, 1), (4, 7)]),         # 7 columns of 18
    (3, (8, 2, 2, 128), 0, [(8, 2), (8, 128)]),              # one column a block
    (2, (6, 4, 2, 96), 0, [(6, 1)]),                         # the least filled blocks that are taken
    (3, (6, 4, 2, 90), 0, [(6, 1)]),                         # the general kernel: a column fills too little
    (3, (6, 4, 2, 130), 1, [(6, 1), (2, 129)]),              # the general kernel: a column longer than a block
])
@pytest.mark.parametrize("twist", [(0.0, 0.0), (0.4, 0.9)])
def test_single_loops_match_the_oracle(group, size, precision, loops, twist):
    L = Q.Lattice(Q.default_config(group=group, size=size, precision=precision, start=Q.START_HOT, prng=Q.PRNG_PHILOX,
                                   beta=5.8 if group == 3 else 2.4, phi=twist[0], omega=twist[1]))
    L.seed()
    L.init(Q.START_HOT)
    t = L.download()
    c = O.make_cfg(group=group, dims=size, precision=precision, beta=5.8, nhit=10, row_align=64, gid_mode=False,
                   phi=twist[0], omega=twist[1])
    for R, T in loops:
        w, ow = L.wilson_sum(R, T), O.wilson(c, t, R, T)
        # 2 (R + T) FP64 factors a loop, 3 V loops of size up to N
        assert abs(w - ow) <= 1e-15 * 2 * (R + T) * 3 * O.volume(c) * group, (R, T, w, ow)
    L.close()


@pytest.mark.parametrize("size", [(2, 2, 2, 2), (6, 4, 10, 6), (34, 4, 6, 2), (4, 34, 2, 16), (16, 16, 36, 6)])
def test_one_pass_profiles_equal_the_separate_ones(size):
    L = Q.Lattice(Q.default_config(group=3, size=size, precision=0, start=Q.START_HOT, prng=Q.PRNG_PHILOX, beta=5.8))
    L.seed()
    L.init(Q.START_HOT)
    tot, prof = L.measure_all()
    assert tot == tuple(L.plaquette_sums()) + tuple(L.action_sums())
    assert all(np.array_equal(prof[a], L.action_profile(a)) for a in range(3))
    tot, prof = L.measure_all(polyakov=True)
    assert tot == tuple(L.polyakov_sums())
    assert all(np.array_equal(prof[a], L.polyakov_profile(a)) for a in range(3))
    L.close()
