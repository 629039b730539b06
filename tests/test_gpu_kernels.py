"""Edges of single kernels: tile remainders, the smallest sizes, and the rules
that choose between two forms of a kernel.  An evaluation's result never
depends on the batch it is in, so the forms are compared bit for bit; values
are compared with plain numpy in double precision (chi2 relative 1e-5, the
tolerance of the other chi2 tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHI2_TOL = 1e-5


@pytest.fixture(scope="module")
def env():
    from pasta_b200 import pasta as P
    from pasta_b200 import synth as S
    spec = S.config0_grid(n_px=4000)
    labels, spectra, factors = S.make_grid(spec)
    wl = P.WlGrid(spec.log_first, spec.log_step, spec.n_px, log=True)
    interp = P.InMemInterpolator.from_arrays(labels, spectra, factors, wl)
    star = S.make_star(spec, [7130.0, 0.07, 4.02, 50.0, 20.0], 3001, 100.0, 85000.0, seed=3)
    return dict(P=P, S=S, spec=spec, interp=interp, wl=wl, star=star)


def _near(star, n, seed):
    rng = np.random.default_rng(seed)
    lab = star.label + rng.uniform(-1.0, 1.0, (n, 5)) * [300.0, 0.2, 0.2, 30.0, 20.0]
    return lab


def _chunk_chi2(wl, flux, var, model, chunks, degree, overlap=0.2):
    """chi2 of the blended chunk polynomials of flux / model, in double."""
    n = len(wl)
    edge = lambda i: min(max(i / chunks * (wl[-1] - wl[0]) + wl[0], wl[0]), wl[-1])  # noqa: E731
    start = [0 if c == 0 else int(np.searchsorted(wl, edge(c - overlap), "right")) for c in range(chunks)]
    stop = [n if c == chunks - 1 else int(np.searchsorted(wl, edge(c + 1 + overlap), "left")) for c in range(chunks)]
    y, cont, prev = flux / model, np.zeros(n), None
    for c, (a, b) in enumerate(zip(start, stop)):
        x = (wl[a:b] - wl[a]) / (wl[b - 1] - wl[a]) * 2.0 - 1.0
        q, _ = np.linalg.qr(np.polynomial.legendre.legvander(x, degree))
        fit = np.zeros(n)
        fit[a:b] = q @ (q.T @ y[a:b])
        lo = a if c == 0 else stop[c - 1]
        cont[lo:b] = fit[lo:b]
        if c:
            t = (wl[a:lo] - wl[lo - 1]) / (wl[a] - wl[lo - 1])
            f = np.sin(t * np.pi / 2.0) ** 2
            cont[a:lo] = prev[a:lo] * f + fit[a:lo] * (1.0 - f)
        prev = fit
    r = (flux - cont * model)[50:n - 50]
    return float((r * r / var[50:n - 50]).sum() / (n - 100))


@pytest.mark.parametrize("n,chunks,degree", [(300, 2, 0), (301, 2, 3), (640, 3, 5), (1023, 5, 8), (1025, 4, 7), (2049, 9, 4),
                                             (4097, 12, 2), (5003, 8, 5), (9001, 17, 9), (3001, 6, 15)])
@pytest.mark.parametrize("scale", [1.0, 1e-18])
def test_chunk_fit_edges(env, n, chunks, degree, scale):
    """Pixel counts around the kernel's blocks of 64, 128 and 256 pixels, fewer and more chunks than warps, and
    (scale 1e-18) variances around 1e-40, below the normal range, where the fast reciprocal does not hold.  The
    rounding of such a variance is at most 0.5 * 2^-149 / 4e-41 = 2e-5 of it."""
    P = env["P"]
    rng = np.random.default_rng(n)
    wl = np.geomspace(4100.0, 4900.0, n)
    model = (0.7 + 0.3 * np.cos(wl / 3.0)).astype(np.float32)
    sigma = 0.01
    x = np.linspace(-1.0, 1.0, n)
    flux = (model * (1.0 + 0.2 * x - 0.1 * x * x) + sigma * rng.standard_normal(n)) * scale
    flux, var = flux.astype(np.float32), np.full(n, (sigma * scale) ** 2, np.float64)
    var32 = var.astype(np.float32)
    got = P.ChunkContinuumFitter(wl, chunks, degree, 0.2).fit_and_return_chi2(model, flux, var32)
    ref = _chunk_chi2(wl, flux.astype(np.float64), var, model.astype(np.float64), chunks, degree)
    assert abs(got - ref) <= (CHI2_TOL + (2e-5 if scale < 1.0 else 0.0)) * ref


@pytest.mark.parametrize("chunks,degree", [(5, 8), (8, 5), (2, 1), (11, 3)])
def test_chunk_fit_pairs_match_single_evaluations(env, chunks, degree):
    """A large batch works pairs of evaluations (an odd number of them here), a small one each alone."""
    P, star, interp = env["P"], env["star"], env["interp"]
    disp = P.FixedResolutionDispersion(star.wl, 85000.0, env["wl"])
    cont = P.ChunkContinuumFitter(star.wl, chunks, degree, 0.2)
    fitter = interp.get_fitter(disp, cont, P.PSOSettings(8, 2), (0.0, 300.0), (-150.0, 150.0))
    lab = _near(star, 1301, 5)
    lab[[3, 10, 11, 1300], 0] = 1e5  # labels outside the grid, alone and as a pair
    both = np.array(fitter.chi2(interp, star.flux, star.var, lab))
    assert np.isnan(both[[3, 10, 11, 1300]]).all()
    for a in (0, 9, 512, 1288):
        alone = np.array(fitter.chi2(interp, star.flux, star.var, lab[a:a + 13]))
        np.testing.assert_array_equal(both[a:a + 13], alone)


@pytest.mark.parametrize("n_obs", [1, 37, 129, 1024, 1025, 3800])
@pytest.mark.parametrize("vsini,rv", [(20.0, 0.0), (150.0, -0.0), (299.0, 0.0), (60.0, -40.0)])
def test_resampling_of_broadening_blocks(env, n_obs, vsini, rv):
    """The resampling inside the broadening kernel: observed pixels from the very first grid pixel (float index 0) on,
    fewer than a round of the kernel's threads, exact rounds, one more; against the oracle in double."""
    import oracle as O
    P, S, spec, interp = env["P"], env["S"], env["spec"], env["interp"]
    wl_grid = spec.wl()
    first = wl_grid[0] if rv == 0.0 else wl_grid[0] * 1.01
    wl = np.geomspace(first, wl_grid[3800], n_obs)
    wl[0] = first
    labels, spectra, factors = S.make_grid(spec)
    og = O.Grid(labels, spectra, factors, O.WL_LOGSPACE, spec.log_first, spec.log_step)
    rng = np.random.default_rng(n_obs)
    flux = (1.0 + 0.1 * rng.standard_normal(n_obs)).astype(np.float32)
    var = np.full(n_obs, 0.01, np.float32)
    ones = np.ones(n_obs, np.float32)
    lab = np.array([[7130.0, 0.07, 4.02, vsini, rv]])
    disp, cont = P.FixedResolutionDispersion(wl, 85000.0, env["wl"]), P.FixedContinuum(ones)
    fitter = interp.get_fitter(disp, cont, P.PSOSettings(8, 2), (0.0, 300.0), (-150.0, 150.0))
    keep = interp.direct_max
    try:
        interp.direct_max = 0  # the FFT path
        got = fitter.chi2(interp, flux, var, lab)[0]
    finally:
        interp.direct_max = keep
    od, oc = O.Disp(og, O.DISP_FIXED, wl, 85000.0), O.Cont(O.CONT_FIXED, continuum=ones)
    ref, st = O.chi2(og, od, oc, flux, var, lab, O.F64)
    assert st[0] == 0
    assert abs(got - ref[0]) <= CHI2_TOL * ref[0]


def _contracted(star, n, seed):
    rng = np.random.default_rng(seed)
    return star.label + rng.uniform(-1.0, 1.0, (n, 5)) * [20.0, 0.004, 0.01, 5.0, 1.0]


@pytest.mark.parametrize("members", [8, 17, 64])
def test_tensor_core_groups_alone_and_among_many(env, members):
    """One tensor-core group is cut into items of two tiles, hundreds of groups into whole slabs; every pixel is the same."""
    P, star, interp = env["P"], env["star"], env["interp"]
    disp = P.FixedResolutionDispersion(star.wl, 85000.0, env["wl"])
    keep = interp.tc_min
    try:
        interp.tc_min = 8
        lab = _contracted(star, 64 * 640, 8)
        lab[members:64] = _near(star, 64 - members, 9)  # the first segment's group has `members` evaluations
        fitter = interp.get_fitter(disp, P.ConstantContinuum(), P.PSOSettings(8, 2), (0.0, 300.0), (-150.0, 150.0))
        many = np.array(fitter.chi2(interp, star.flux, star.var, lab))
        few = np.array(fitter.chi2(interp, star.flux, star.var, lab[:64]))
    finally:
        interp.tc_min = keep
    np.testing.assert_array_equal(many[:64], few)


def test_groups_at_grid_edges(env):
    """Evaluations of one segment whose cubes lie at the grid's edges and nodes (two or three neighbours on an axis):
    together, in any group, as one at a time."""
    P, spec, interp = env["P"], env["spec"], env["interp"]
    rng = np.random.default_rng(12)

    def axis(v):
        return rng.choice(np.concatenate([v[[0, 1, -2, -1]], v[[0, 0, -2, -2]] + rng.uniform(0.2, 0.8, 4) * np.diff(v)[[0, 0, -1, -1]]]))
    lab = np.array([[axis(spec.teffs), axis(spec.ms), axis(spec.loggs)] for _ in range(150)])
    lab[100:] = lab[rng.integers(0, 100, 50)]  # shared cubes
    together = interp.interpolate_bulk(lab)
    for i in list(range(0, 150, 7)) + [149]:
        np.testing.assert_array_equal(together[i], interp.interpolate(*lab[i]))


@pytest.mark.parametrize("n", [1, 300, 349, 350, 1100])
def test_results_copied_in_parts(env, n):
    """Model rows copied out through the staging buffer's halves of 4 MB (349 rows of 3,001 pixels just fit one):
    less than a half, a half, one row more, several."""
    P, star, interp = env["P"], env["star"], env["interp"]
    disp = P.FixedResolutionDispersion(star.wl, 85000.0, env["wl"])
    lab = _near(star, n, 31)
    many = interp.produce_model_bulk(disp, lab)
    for i in {0, n // 2, n - 1, min(n - 1, 348), min(n - 1, 349)}:
        np.testing.assert_array_equal(many[i], interp.produce_model(disp, *lab[i]))


def test_calls_from_several_threads(env):
    """Calls of several threads on one grid share the scratch memory and the staging buffer; every result is its own."""
    import threading
    P, star, interp = env["P"], env["star"], env["interp"]
    disp = P.FixedResolutionDispersion(star.wl, 85000.0, env["wl"])
    fitter = interp.get_fitter(disp, P.ChunkContinuumFitter(star.wl, 5, 8, 0.2), P.PSOSettings(8, 2), (0.0, 300.0),
                               (-150.0, 150.0))
    labs = [_near(star, 20 + 37 * k, k) for k in range(6)]
    want = [(np.array(fitter.chi2(interp, star.flux, star.var, lab)), interp.produce_model_bulk(disp, lab)) for lab in labs]
    bad = []

    def work(k):
        for _ in range(10):
            c, m = np.array(fitter.chi2(interp, star.flux, star.var, labs[k])), interp.produce_model_bulk(disp, labs[k])
            if not (np.array_equal(c, want[k][0]) and np.array_equal(m, want[k][1])):
                bad.append(k)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("kind", ["none", "unsorted"])
@pytest.mark.parametrize("n", [1, 70])
def test_evaluations_resampled_after_the_broadening(env, kind, n):
    """Stars whose evaluations k_broaden leaves to the later resampling (no instrument profile with vsini 0 among the
    labels, or unsorted pixels), in one segment and in two, against the oracle in double."""
    import oracle as O
    P, S, spec, interp, star = env["P"], env["S"], env["spec"], env["interp"], env["star"]
    order = np.arange(len(star.wl))
    if kind == "unsorted":
        order = np.random.default_rng(4).permutation(len(order))
    wl, flux, var = star.wl[order], star.flux[order], star.var[order]
    ones = np.ones(len(wl), np.float32)
    lab = _near(star, n, 77)
    lab[::3, 3] = 0.0
    labels, spectra, factors = S.make_grid(spec)
    og = O.Grid(labels, spectra, factors, O.WL_LOGSPACE, spec.log_first, spec.log_step)
    if kind == "none":
        disp, od = P.NoConvolutionDispersion(wl, env["wl"]), O.Disp(og, O.DISP_NONE, wl)
    else:
        disp, od = P.FixedResolutionDispersion(wl, 85000.0, env["wl"]), O.Disp(og, O.DISP_FIXED, wl, 85000.0)
    fitter = interp.get_fitter(disp, P.FixedContinuum(ones), P.PSOSettings(8, 2), (0.0, 300.0), (-150.0, 150.0))
    got = np.array(fitter.chi2(interp, flux, var, lab))
    ref, st = O.chi2(og, od, O.Cont(O.CONT_FIXED, continuum=ones), flux, var, lab, O.F64)
    assert (st == 0).all()
    np.testing.assert_allclose(got, ref, rtol=CHI2_TOL)


@pytest.mark.parametrize("resolution", [20000.0, 40000.0, 60000.0, 85000.0, 200000.0])
@pytest.mark.parametrize("vsini,rv", [(0.0, 0.0), (60.0, 0.0), (299.0, 20.0)])
def test_per_pixel_instrument_kernels(env, resolution, vsini, rv):
    """Per-pixel instrument kernels of several widths in the broadening blocks, over the whole grid (both ends pass
    through, the last block stands alone or half empty), against the oracle in single precision (1e-5 of the maximum)."""
    import oracle as O
    P, S, spec, interp = env["P"], env["S"], env["spec"], env["interp"]
    wl = spec.wl()[:-1] if rv == 0.0 else np.geomspace(spec.wl()[0] * 1.001, spec.wl()[-2] * 0.999, 3001)
    sig = (wl / (resolution * np.linspace(1.0, 1.5, len(wl))) / 2.355).astype(np.float32)
    labels, spectra, factors = S.make_grid(spec)
    og = O.Grid(labels, spectra, factors, O.WL_LOGSPACE, spec.log_first, spec.log_step)
    lab = [7130.0, 0.07, 4.02, vsini, rv]
    keep = interp.direct_max
    try:
        interp.direct_max = 0  # the FFT path
        got = interp.produce_model(P.VariableResolutionDispersion(wl, sig, env["wl"]), *lab)
    finally:
        interp.direct_max = keep
    ref = O.Disp(og, O.DISP_VARIABLE, wl, disp=sig).produce_model(lab, O.F32)
    assert np.abs(got.astype(np.float64) - ref).max() <= 1e-5 * np.abs(ref).max()
