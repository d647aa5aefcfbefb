"""Reference-layout link tables in and out through the bounded staging
buffer: whole planes at a time, several pieces, and pieces of one plane
(a plane larger than the buffer), with and without padding rows."""
import numpy as np
import pytest

import qcdgpu_b200 as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,size,precision,align", [
    (2, (2, 2, 2, 2), 0, 64),            # one piece, mostly padding
    (3, (6, 4, 10, 6), 1, 96),           # rows padded past V
    (3, (24, 24, 24, 24), 1, 64),        # 127 MB: six planes at a time
    (2, (64, 64, 32, 34), 0, 128),       # planes of 71 MB: pieces of one plane
])
def test_table_pieces_hold_the_field_site_by_site(group, size, precision, align):
    """the closed-form start is a function of the site index, so every piece
    shows whether its sites are where the table has them (suncl.cl:190-347;
    SU(2): the first component as stored, SU(3): the ratio of two components
    of row 1, which the row's normalisation keeps); a table put back gives
    the same field (observables and table bit for bit), padding is zero"""
    cfg = Q.default_config(group=group, size=size, precision=precision, start=Q.START_GID, prng=Q.PRNG_PHILOX,
                           row_align=align)
    L = Q.Lattice(cfg)
    L.init(Q.START_GID)
    i = L.info()
    V, rows = i.sites, i.rowsize
    assert rows % align == 0 and rows >= V
    a = L.download()
    t = a.reshape(-1, rows, 4)
    assert not t[:, V:].any()
    s = np.arange(V, dtype=np.float64)
    tol = 1e-12 if precision else 2e-6           # a few roundings of values below 1
    for mu in range(4):
        o = 0.001 * (mu + 1)
        f1 = np.sin((o + 10.0 / V) * s) / 2.0
        if group == 2:
            assert np.max(np.abs(t[mu, :V, 0] - f1)) < tol
        else:
            f2 = np.sin((o - 18.0 / V) * s) / 4.0
            assert np.max(np.abs(t[mu, :V, 0] * f2 - t[mu, :V, 1] * f1)) < tol
    K = Q.Lattice(cfg)
    K.upload(a)
    assert K.plaquette_sums() == L.plaquette_sums()
    assert np.array_equal(K.download(), a)
    L.close()
    K.close()
