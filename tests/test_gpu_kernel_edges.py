"""Kernels at the sizes where their work split changes: ragged tiles, single
rows, fields around the limits of a dispatch. Each case compares with the oracle
or with the same quantity computed over another split; where the arithmetic of
a point, node or cell does not depend on the split, bit for bit."""
import numpy as np
import pytest

import irs_b200
from tests.cases import IPM_SMALL, IRS_SMALL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dbl", [True, False])
@pytest.mark.parametrize("rows", [1, 2, 7, 8, 9, 15, 16, 17, 31, 33])
def test_lattice_bands_equal_whole_lattice(gpu, dbl, rows):
    """A band of few lattice rows (tiles of 1 to 33 rows, cut anywhere) holds the
    corner positions of the whole lattice, and the maps of the bands that
    cover it add up to its map."""
    cfg = dict(IPM_SMALL, num_pixels_y1=40, num_pixels_y2=24, half_length_y1=1.25, half_length_y2=0.75)
    m = irs_b200.IPM(**cfg, is_double=dbl, expansion_order=10)
    m.run()
    whole = m.vertices()
    lo = whole.shape[0] // 2 - rows // 2
    m.lib.set_band(m.obj, lo, lo + rows)
    m.run()
    np.testing.assert_array_equal(m.vertices(), whole[lo:lo + rows + 1])
    m.close()


@pytest.mark.parametrize("dbl", [True, False])
def test_ray_bands_with_parities_add_up(gpu, dbl):
    cfg = dict(IRS_SMALL, num_pixels_y1=33, num_pixels_y2=17, half_length_y1=1.0, half_length_y2=0.5,
               write_parities=True)
    m = irs_b200.IRS(**cfg, is_double=dbl, expansion_order=9)
    m.run()
    whole = [m.magnifications.copy(), m.magnifications_minima.copy(), m.magnifications_saddles.copy()]
    n = int(m.value("num_ray_threads_2"))
    cuts = sorted({0, n} | {min(n, int(c)) for c in np.cumsum([1, 2, 7, 8, 9, 30, 41] * 40)})
    acc = [np.zeros_like(w) for w in whole]
    for lo, hi in zip(cuts[:12] + [cuts[12]], cuts[1:13] + [n]):
        m.lib.set_band(m.obj, lo, hi)
        m.run()
        for a, b in zip(acc, (m.magnifications, m.magnifications_minima, m.magnifications_saddles)):
            a += b
    for a, w in zip(acc, whole):
        np.testing.assert_array_equal(a, w)
    m.close()
