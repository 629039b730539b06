"""Served fits of stars with linear-model continua, alone and among chunk and
constant ones, in more slots than one with the slots used again: label, chi2
and continuum parameters are those of the fit alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    from pasta_b200 import pasta as P
    from pasta_b200 import synth as S
    spec = S.config0_grid(n_px=4000)
    labels, spectra, factors = S.make_grid(spec)
    wl = P.WlGrid(spec.log_first, spec.log_step, spec.n_px, log=True)
    return P, S, spec, P.InMemInterpolator.from_arrays(labels, spectra, factors, wl), wl


def _stars(env, kinds):
    P, S, spec, interp, wl = env
    out = []
    for i, (kind, lab) in enumerate(zip(kinds, S.random_labels(spec, len(kinds), seed=4, vsini=(10, 150), rv=(-60, 60)))):
        star = S.make_star(spec, lab, 2500 + 150 * i, 80.0, 85000.0, seed=60 + i)
        if kind == "chunk":
            cont = P.ChunkContinuumFitter(star.wl, 3 + i % 3, 4, 0.2)
        elif kind == "constant":
            cont = P.ConstantContinuum()
        else:
            cont = P.LinearModelContinuumFitter(S.legendre_design(star.wl, kind))
        out.append((star, P.FixedResolutionDispersion(star.wl, 85000.0, wl), cont))
    return out


@pytest.mark.parametrize("slots", [1, 3, 5])
@pytest.mark.parametrize("kinds", [(12, 12, 12, 12, 12, 12), (20, "chunk", 12, 12, "constant", 40), ("chunk", 12, 12, 70, "chunk", 16)])
def test_served_fits_of_linear_continua(env, slots, kinds):
    P, S, spec, interp, wl = env
    settings = P.PSOSettings(8, 5)
    stars = _stars(env, kinds)
    alone = [interp.get_fitter(d, c, settings, (0.0, 300.0), (-150.0, 150.0)).fit(interp, s.flux, s.var, seed=9)
             for s, d, c in stars]
    srv = P.Server(interp, max_slots=slots)
    ids = [srv.submit(d, c, settings, s.flux, s.var, (0.0, 300.0), (-150.0, 150.0), seed=9) for s, d, c in stars]
    done = {}
    for _ in range(100):
        srv.step()
        done.update({i: (status, r) for i, status, r in srv.poll()})
        if len(done) == len(ids):
            break
    for i, want in zip(ids, alone):
        status, got = done[i]
        assert status == 0
        assert got.label.as_list() == want.label.as_list()
        assert got.chi2 == want.chi2
        assert len(got.continuum_params) == len(want.continuum_params) > 0
        np.testing.assert_array_equal(got.continuum_params, want.continuum_params)
