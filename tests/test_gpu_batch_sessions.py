"""A stepped batch of fits and other calls on its grid in between: larger
batches, longer spectra and servers move the grid's workspace, which the
batch's captured step works in.  Results are those of the batch left alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _env():
    from pasta_b200 import pasta as P
    from pasta_b200 import synth as S
    spec = S.config0_grid(n_px=4000)
    labels, spectra, factors = S.make_grid(spec)
    wl = P.WlGrid(spec.log_first, spec.log_step, spec.n_px, log=True)
    interp = P.InMemInterpolator.from_arrays(labels, spectra, factors, wl)
    stars = [S.make_star(spec, [7100.0 + 40.0 * i, 0.05, 4.0, 50.0, 20.0], 3000, 100.0, 85000.0, seed=i) for i in range(3)]
    return P, S, spec, interp, wl, stars


def _batch(P, interp, wl, stars):
    disp = [P.FixedResolutionDispersion(s.wl, 85000.0, wl) for s in stars]
    cont = [P.ChunkContinuumFitter(s.wl, 4, 5, 0.2) for s in stars]
    return P.BatchFit(interp, disp, cont, P.PSOSettings(12, 6), [s.flux for s in stars], [s.var for s in stars],
                      (0.0, 300.0), (-150.0, 150.0), seeds=[1, 2, 3])


def _result(b):
    return [(status, list(r.label.as_list()), r.chi2, list(r.continuum_params)) for status, r in b.finish()]


def _more_labels(P, S, spec, interp, wl, star):
    lab = star.label + np.random.default_rng(1).uniform(-1.0, 1.0, (900, 5)) * [300.0, 0.2, 0.2, 30.0, 20.0]
    interp.produce_model_bulk(P.FixedResolutionDispersion(star.wl, 85000.0, wl), lab)


def _longer_spectrum(P, S, spec, interp, wl, star):
    s = S.make_star(spec, [7130.0, 0.07, 4.02, 50.0, 20.0], 9000, 100.0, 85000.0, seed=9)
    interp.produce_model(P.FixedResolutionDispersion(s.wl, 85000.0, wl), 7130.0, 0.07, 4.02, 50.0, 20.0)


@pytest.mark.parametrize("other", [_more_labels, _longer_spectrum])
def test_calls_between_the_steps_of_a_batch(other):
    P, S, spec, interp, wl, stars = _env()
    b = _batch(P, interp, wl, stars)
    b.step(7)
    want = _result(b)
    P, S, spec, interp, wl, stars = _env()  # a grid of its own: a workspace no larger than the batch's
    b = _batch(P, interp, wl, stars)
    for k in range(7):
        if k in (2, 5):
            other(P, S, spec, interp, wl, stars[0])
        b.step(1)
    assert _result(b) == want
    assert all(r[0] == 0 for r in want)
