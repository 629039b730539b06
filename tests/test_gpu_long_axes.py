"""Grids with long axes: more points than the kernels' shared copy of the axes
holds (they then read the resident ones), and more than the neighbour key of an
evaluation tells apart (columns are then compared one by one)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLUX_TOL = 1e-5


def _grid(n_teff, n_px, seed):
    from pasta_b200 import pasta as P
    teffs, ms, loggs = 4000.0 + 2.0 * np.arange(n_teff), np.array([-0.5, 0.0, 0.5]), np.array([3.5, 4.0, 4.5])
    labels = np.array([[t, m, g] for t in teffs for m in ms for g in loggs])
    rng = np.random.default_rng(seed)
    spectra = rng.integers(20000, 60000, (len(labels), n_px)).astype(np.uint16)
    wl = P.WlGrid(np.log10(4100.0), 2e-5, n_px, log=True)
    return P, labels, spectra, wl, P.InMemInterpolator.from_arrays(labels, spectra, None, wl)


@pytest.mark.parametrize("n_teff", [339, 340, 350, 1200])
def test_axes_around_the_size_of_the_shared_copy(n_teff):
    """1,024 values are 339 temperatures, their limits and 3 + 3 points of the other axes."""
    import oracle as O
    P, labels, spectra, wl, interp = _grid(n_teff, 640, n_teff)
    og = O.Grid(labels, spectra, None, O.WL_LOGSPACE, np.log10(4100.0), 2e-5)
    top = 4000.0 + 2.0 * (n_teff - 1)
    lab = np.array([[4000.0, -0.5, 3.5], [4001.3, 0.2, 4.1], [top, 0.5, 4.5], [top - 0.7, 0.0, 3.9], [0.5 * (4000.0 + top) + 0.9, 0.1, 4.0]])
    got = interp.interpolate_bulk(lab)
    for g, l in zip(got, lab):
        ref = og.interpolate(*l, O.F32)
        assert np.abs(g - ref).max() <= FLUX_TOL * np.abs(ref).max()
    # the swarm's clamps read the same axes
    obs = 10.0 ** (np.log10(4100.0) + 2e-5 * np.linspace(30.0, 600.0, 400))
    disp, cont = P.FixedResolutionDispersion(obs, 85000.0, wl), P.ConstantContinuum()
    flux, var = interp.produce_model(disp, *lab[4], 5.0, 0.0), np.full(400, 1e-4, np.float32)
    fitter = interp.get_fitter(disp, cont, P.PSOSettings(10, 8), (0.0, 20.0), (-2.0, 2.0))
    batched, plain = (fitter.fit(interp, flux, var, seed=5, mode=mode) for mode in (0, 1))
    assert batched.label.as_list() == plain.label.as_list()
    assert batched.chi2 == plain.chi2


def test_axes_longer_than_the_neighbour_key():
    """Labels whose cubes differ by 16,384 temperatures, and by one, in one segment: each as by itself."""
    P, labels, spectra, wl, interp = _grid(16384 + 40, 192, 1)
    t = np.array([4000.0 + 2.0 * k + 0.7 for k in (1, 2, 5, 5, 30)])
    t = np.concatenate([t, t + 2.0 * 16384])
    lab = np.array([[x, m, 4.1] for x in t for m in (0.1, 0.2, -0.3)] * 2)
    together = interp.interpolate_bulk(lab)
    for l, row in zip(lab, together):
        np.testing.assert_array_equal(row, interp.interpolate(*l))
    assert not np.array_equal(together[0], together[15])
    # and merged across segments
    many = np.tile(lab, (8, 1))[np.random.default_rng(0).permutation(8 * len(lab))]
    for l, row in zip(many[:200:7], interp.interpolate_bulk(many)[:200:7]):
        np.testing.assert_array_equal(row, interp.interpolate(*l))
