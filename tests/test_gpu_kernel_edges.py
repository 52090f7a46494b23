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
    corner positions of the whole lattice, and the fixed-point maps of the bands
    that cover it (that one, those before it and after it) add up to its map."""
    cfg = dict(IPM_SMALL, num_pixels_y1=40, num_pixels_y2=24, half_length_y1=1.25, half_length_y2=0.75)
    m = irs_b200.IPM(**cfg, is_double=dbl, expansion_order=10)
    m.run()
    whole, total = m.vertices(), m.fixed_maps()
    assert total.any()
    n = whole.shape[0] - 1  # rows of cells
    lo = n // 2 - rows // 2
    acc = np.zeros_like(total)
    for a, b in ((0, lo), (lo, lo + rows), (lo + rows, n)):
        m.lib.set_band(m.obj, a, b)
        m.run()
        np.testing.assert_array_equal(m.vertices(), whole[a:b + 1])
        acc += m.fixed_maps()
    np.testing.assert_array_equal(acc, total)
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


@pytest.mark.parametrize("centre", [(0.0, 0.0), (0.35, -0.2), (-6.0, 4.0)])
@pytest.mark.parametrize("npix,half", [((1, 1), (0.5, 0.5)), ((1, 64), (0.02, 1.28)), ((57, 3), (1.14, 0.06))])
def test_rays_at_the_edges_of_small_maps(gpu, centre, npix, half):
    """Most rays miss these maps. With the approximate sheet they are dropped on
    the FP32 value of their position, with the exact sheet every ray is decided
    in FP64. Inside the field's circle, where all rays of the lattice are, the
    two sheets are the same -kappa_star z, so the counts agree ray for ray."""
    cfg = dict(IRS_SMALL, num_pixels_y1=npix[0], num_pixels_y2=npix[1], half_length_y1=half[0], half_length_y2=half[1],
               center_y1=centre[0], center_y2=centre[1], num_rays_y=400)
    maps = []
    for approx in (True, False):
        m = irs_b200.IRS(**cfg, approx=approx, expansion_order=10)
        m.run()
        assert (abs(m.value("center_x1")) + m.value("half_length_x1")) ** 2 + (
            abs(m.value("center_x2")) + m.value("half_length_x2")) ** 2 < (
            m.value("corner_x1") ** 2 + m.value("corner_x2") ** 2)
        maps.append(m.magnifications.copy())
        m.close()
    assert maps[0].sum() > 0
    np.testing.assert_array_equal(maps[0], maps[1])


@pytest.mark.parametrize("n,nphi,nb", [(1, 40, 2), (2, 12, 3), (3, 8, 4), (33, 8, 2)])
def test_critical_curves_of_few_stars_match_oracle(gpu, tmp_path, n, nphi, nb):
    """Fields of fewer roots than a CTA has warps, one phi step per side, several
    branches: the sets of critical-curve points at every phi agree with the
    oracle's to its expansion error."""
    from scipy.optimize import linear_sum_assignment

    from oracle import ccf_ref
    from tests.test_gpu_ccf import as_complex, star_field, write_stars
    stars, rad = star_field(n, kstar=0.3, seed=40 + n)
    write_stars(str(tmp_path / "s.bin"), stars, rad)
    c = irs_b200.CCF(kappa_tot=0.45, shear=0.25, starfile=str(tmp_path / "s.bin"), num_phi=nphi, num_branches=nb)
    c.run()
    assert c.value("max_error") < 1e-8
    L = ccf_ref.Lens(stars, 0.45, 0.25, c.kappa_star, 1.0, 1, rad)
    z = ccf_ref.critical_curves(L, ccf_ref.initial_roots(stars, c.num_roots, nphi, nb, rad), nphi, nb)
    ref, got = ccf_ref.outputs(L, z, nb)[0], as_complex(c.critical_curves)
    assert ref.shape == got.shape
    for b in range(nb):
        rows = np.arange(b, ref.shape[0], nb)
        for k in range(ref.shape[1]):
            d = np.abs(ref[rows, k][:, None] - got[rows, k][None, :])
            i, j = linear_sum_assignment(d)
            assert d[i, j].max() < 1e-7
    c.close()


@pytest.mark.parametrize("n", [31, 256, 257, 4096, 4097])
def test_critical_curves_on_both_sides_of_the_shared_positions(gpu, tmp_path, n):
    """Star positions are held in shared memory up to 4096 stars, read in steps
    of 8 x 32: every root of every phi solves the directly summed equation
    dw/dzbar* = dw/dz e^{-i phi} (1/mu there is the stop's bound 1e-9 plus the
    expansion's error, together below 1e-8), and no two roots are the same."""
    from oracle import ccf_ref
    from tests.test_gpu_ccf import as_complex, star_field, write_stars
    stars, rad = star_field(n, kstar=0.3, seed=7 + n)
    write_stars(str(tmp_path / "s.bin"), stars, rad)
    c = irs_b200.CCF(kappa_tot=0.45, shear=0.25, starfile=str(tmp_path / "s.bin"), num_phi=4, num_branches=1)
    c.run()
    got = as_complex(c.critical_curves)  # (roots, phi)
    L = ccf_ref.Lens(stars, 0.45, 0.25, c.kappa_star, 1.0, 1, rad)
    assert got.shape[0] == 2 * n
    cell = 1e-7 * c.value("expansion_order") / (1.1 * rad / 2.0 ** c.value("tree_levels"))
    for z in got.T:
        for part in np.array_split(z, max(1, 2 * n // 512)):
            _, dwdz, dwdzb, d2 = L.fields(part)
            inv_mu = np.abs(dwdz) ** 2 - np.abs(dwdzb) ** 2
            assert np.all(np.abs(inv_mu) < 2e-9 * (1 + np.abs(dwdzb) * np.abs(d2)) + 2 * cell * np.abs(dwdzb))
        assert np.unique(z).size == z.size
    c.close()


@pytest.mark.parametrize("index", [11, 17])
def test_batch_mass_sums_of_large_fields(gpu, index):
    """Kroupa fields of 3.8e5 and 7.6e5 float masses: the sums of m are exact in
    any order; the sum of m^2 of the larger one passes the last bit of its
    smallest terms on the way and is finished star by star. The corner, hence
    the map, is the single run's bit for bit."""
    from irs_b200.batch import random_realizations
    kw = random_realizations(24, num_pixels=32, half_length=12.0)[0][index]
    b = irs_b200.BatchIPM([kw], expansion_order=10)
    b.run()
    s = irs_b200.IPM(**kw, expansion_order=10)
    s.run()
    assert int(b.value("num_stars", 0)) == s.num_stars > 3e5
    np.testing.assert_array_equal(b.maps[0], s.magnifications)
    b.close()
    s.close()


@pytest.mark.parametrize("over", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("npix", [(1, 1), (3, 2), (32, 31), (33, 5), (127, 9), (128, 8), (129, 7)])
def test_crossing_maps_around_the_column_step(gpu, npix, over):
    """Maps whose rows end inside, at and past a step of 128 fine columns, in
    every oversampling the pooled kernel takes (0 to 3) and one it does not,
    against the oracle's counts."""
    from oracle import pyoracle as po
    rng = np.random.default_rng(npix[0] + 7 * over)
    t = -np.linspace(0, 2 * np.pi, 41)
    c = (rng.normal(0, 1, (60, 1)) + 1j * rng.normal(0, 1, (60, 1))
         + rng.uniform(0.1, 1, (60, 1)) * (np.cos(t) ** 3 + 1j * np.sin(t) ** 3))
    c[:, -1] = c[:, 0]
    n = irs_b200.NCC(half_length_y1=1.5, half_length_y2=1.2, num_pixels_y1=npix[0], num_pixels_y2=npix[1],
                     over_sample=over)
    n.set_caustics(c)
    n.run()
    ref, err = po.ncc(c, (0, 0), (1.5, 1.2), npix, over)
    assert err == n.value("errors")
    np.testing.assert_array_equal(n.num_caustic_crossings, ref)
    assert (n.value("min_num"), n.value("max_num")) == (ref.min(), ref.max())
    n.close()


def _corner_lattice(kind, rng):
    j, i = np.meshgrid(np.arange(31.0), np.arange(41.0), indexing="ij")
    x, y = (i - 20) * 1.1, (j - 15) * 1.1
    if kind == "horizontal":  # edges along rows, many of them on pixel lines
        return np.stack([x * 0.7, np.floor(y * 3) / 3], -1)
    if kind == "slivers":  # nearly vertical edges, rows snapped to lines
        yy = np.where(rng.random(y.shape) < 0.3, np.floor(y), y)
        return np.stack([x * 0.01 + rng.normal(0, 1e-7, x.shape), yy], -1)
    if kind == "just_past_lines":
        yy = np.floor(y) + np.where(rng.random(y.shape) < 0.5, 1e-9, 0.0)
        return np.stack([np.floor(x) + np.where(rng.random(x.shape) < 0.3, -1e-12, 0.0), yy], -1)
    if kind == "point_lens":  # cells stretched over many pixels around a lens
        r2 = x * x + y * y + 0.01
        return np.stack([x - 30 * x / r2, y - 30 * y / r2], -1)
    if kind == "far":  # beyond the range of int, not finite (x below 2^31: the oracle takes columns as int)
        v = np.stack([x, y], -1)
        pick = rng.random(x.shape)
        for k, (axis, val) in enumerate([(0, 2.0e9), (1, -3.0e9), (1, 5.0e9), (1, 1e18), (0, -1e300), (1, np.inf),
                                         (0, -np.inf), (1, np.nan), (1, 2147483648.0), (1, -2147483649.0)]):
            v[(pick >= 0.01 * k) & (pick < 0.01 * (k + 1)), axis] = val
        return v
    if kind == "fine":  # most triangles inside one pixel
        return np.stack([x * 0.04 + 0.013 * y, y * 0.05 - 0.01 * x], -1)
    return np.stack([x, y], -1) + rng.normal(0, 3.0, x.shape + (2,))  # "tangled"


@pytest.mark.parametrize("dbl", [False, True])
@pytest.mark.parametrize("kind", ["horizontal", "slivers", "just_past_lines", "point_lens", "far", "fine", "tangled"])
def test_deposition_of_awkward_cells(gpu, dbl, kind):
    """Fixed-point maps bit for bit against the oracle's."""
    import ctypes

    import torch

    import irs_b200._lib as L
    from oracle import pyoracle as po
    T, tdt = (ctypes.c_double, torch.float64) if dbl else (ctypes.c_float, torch.float32)
    f = L.load("ipm", dbl).ipm_deposit_noalloc
    f.argtypes = [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_longlong, T, ctypes.c_int, ctypes.c_int,
                  ctypes.c_void_p, ctypes.c_void_p]
    f.restype = ctypes.c_int
    npx, npy, factor = 37, 29, 0.61
    v = np.ascontiguousarray(_corner_lattice(kind, np.random.default_rng(11)) + np.array([npx / 2, npy / 2]))
    d_v = torch.from_numpy(v).to("cuda")
    d_map = torch.full((npy, npx), -1.0, dtype=tdt, device="cuda")
    assert f(d_v.data_ptr(), v.shape[1] - 1, v.shape[0] - 1, factor, npx, npy, d_map.data_ptr(),
             torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    q = po.ipm_deposit_fixed(v, factor if dbl else np.float32(factor), (npx, npy), single=not dbl)
    got = d_map.cpu().numpy()
    np.testing.assert_array_equal(got, (q.astype(np.float64) * 2.0 ** -32).astype(got.dtype))
    assert q.any()


@pytest.mark.parametrize("dbl", [False, True])
@pytest.mark.parametrize("ncx,ncy", [(31, 1), (33, 3), (64, 148), (1000, 301), (3000, 1700)])
def test_deposition_order_covers_every_cell_once(gpu, dbl, ncx, ncy):
    """Lattices of fewer cells than a warp, of one chunk per warp, and of more
    chunks than one wave or one grid of warps holds: every cell deposits its
    area exactly once, in a pixel of its own."""
    import ctypes

    import torch

    import irs_b200._lib as L
    T, tdt = (ctypes.c_double, torch.float64) if dbl else (ctypes.c_float, torch.float32)
    f = L.load("ipm", dbl).ipm_deposit_noalloc
    f.argtypes = [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_longlong, T, ctypes.c_int, ctypes.c_int,
                  ctypes.c_void_p, ctypes.c_void_p]
    f.restype = ctypes.c_int
    # cell (i, j) is pixel (i, j): its two triangles of half a pixel deposit factor each, and
    # 2 * 0.5 is exact in the map's fixed point
    i, j = torch.arange(ncx + 1, device="cuda").double(), torch.arange(ncy + 1, device="cuda").double()
    v = torch.stack([i[None, :].expand(ncy + 1, -1), j[:, None].expand(-1, ncx + 1)], -1).contiguous()
    d_map = torch.full((ncy, ncx), -1.0, dtype=tdt, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    rows = min(1024, 2 ** 20 // ncx)  # the most that a map of this entry point holds
    for lo in range(0, ncy, rows):
        hi = min(ncy, lo + rows)
        # all cells of the lattice each time; those of other rows lie off the map
        w = torch.stack([v[..., 0], v[..., 1] - lo], -1).contiguous()
        assert f(w.data_ptr(), ncx, ncy, 0.5, ncx, hi - lo, d_map[lo:hi].data_ptr(), stream) == 0
    torch.cuda.synchronize()
    assert bool((d_map == 1.0).all())


def test_batched_deposition_order_covers_every_cell_once(gpu):
    """The batched form takes blocks of 8 chunks, 32 of them per 32 x 32-cell tile
    here, more blocks than a grid has warps: an adaptive map at level 1 holds what the plain form
    deposits from the same corners, bit for bit."""
    kw = dict(IPM_SMALL, half_length_y1=64.0, half_length_y2=64.0, num_pixels_y1=2048, num_pixels_y2=2048)
    a = irs_b200.AdaptiveIPM(**kw, policy="uniform", level=1, audit_fraction=0.0)
    a.run()
    assert a.value("cells_base") > 2 ** 5 * 8 * 148 * 256 * 2
    m = irs_b200.IPM(**kw)
    m.run()
    np.testing.assert_array_equal(a.magnifications, m.magnifications)
    a.close()
    m.close()


def test_new_objects_take_no_pinned_memory_for_their_status(gpu):
    """Page-locked memory takes about a millisecond to get, more than the whole run
    of a small object: the first run of critical curves or of an adaptive map
    takes none, that of a map only what its pixels come back in."""
    import gc

    def pinned(make):
        gc.collect()
        m = make()
        before = m.value("pinned_bytes")
        m.run()
        got = m.value("pinned_bytes") - before
        m.close()
        return got

    lens, size = dict(kappa_tot=0.3, shear=0.3, kappa_star=0.27), dict(num_pixels_y1=32, num_pixels_y2=24)
    assert pinned(lambda: irs_b200.CCF(**lens, num_stars=3, num_phi=8, random_seed=5)) == 0
    ipm, irs = (dict(kw, **size, write_histograms=1) for kw in (IPM_SMALL, IRS_SMALL))
    assert pinned(lambda: irs_b200.AdaptiveIPM(**ipm)) == 0
    assert pinned(lambda: irs_b200.IPM(**ipm)) == 4 * 32 * 24
    assert pinned(lambda: irs_b200.IRS(**irs)) == 4 * 32 * 24


def test_status_words_of_an_object_that_runs_often_are_pinned(gpu):
    """They are fetched twice a run and pinned, one page, after 128 fetches; the
    map stays the same."""
    import gc
    gc.collect()
    m = irs_b200.IPM(**dict(IPM_SMALL, num_pixels_y1=32, num_pixels_y2=24))
    m.run()
    first, held = m.magnifications.copy(), m.value("pinned_bytes")
    for _ in range(63):
        m.run()
    assert m.value("pinned_bytes") == held
    m.run()
    assert m.value("pinned_bytes") == held + 4096
    np.testing.assert_array_equal(m.magnifications, first)
    m.close()
