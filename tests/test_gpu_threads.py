"""Calls of several threads on several grids of one device.  Calls are
serialised per grid, so these run at the same time on the device's one stream,
staging buffer and scratch pool, while fits and servers capture their graphs.
Every result is that of the call alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _env(n_px, seed):
    from pasta_b200 import pasta as P
    from pasta_b200 import synth as S
    spec = S.config0_grid(n_px=n_px)
    labels, spectra, factors = S.make_grid(spec)
    wl = P.WlGrid(spec.log_first, spec.log_step, spec.n_px, log=True)
    interp = P.InMemInterpolator.from_arrays(labels, spectra, factors, wl)
    star = S.make_star(spec, [7130.0, 0.07, 4.02, 50.0, 20.0], n_px * 3 // 4, 100.0, 85000.0, seed=seed)
    disp = P.FixedResolutionDispersion(star.wl, 85000.0, wl)
    fitter = interp.get_fitter(disp, P.ChunkContinuumFitter(star.wl, 4, 5, 0.2), P.PSOSettings(10, 6), (0.0, 300.0),
                               (-150.0, 150.0))
    return P, interp, star, disp, fitter


def _labels(star, n, seed):
    rng = np.random.default_rng(seed)
    return star.label + rng.uniform(-1.0, 1.0, (n, 5)) * [300.0, 0.2, 0.2, 30.0, 20.0]


def _fits(env):
    P, interp, star, disp, fitter = env
    out = []
    for seed in range(4):
        r = fitter.fit(interp, star.flux, star.var, seed=seed)
        out += [list(r.label.as_list()), r.chi2, list(r.continuum_params)]
    return out


def _served(env):
    P, interp, star, disp, fitter = env
    srv = P.Server(interp, max_slots=2)
    cont = P.ChunkContinuumFitter(star.wl, 4, 5, 0.2)
    ids = [srv.submit(disp, cont, P.PSOSettings(10, 4), star.flux, star.var, (0.0, 300.0), (-150.0, 150.0), seed=s)
           for s in range(4)]
    done = {}
    for _ in range(100):
        srv.step()
        done.update({i: (status, list(r.label.as_list()), r.chi2, list(r.continuum_params)) for i, status, r in srv.poll()})
        if len(done) == len(ids):
            break
    return [done[i] for i in ids]


def _models(env):
    """Results of 100 kB, and of 9 MB (several staged parts)."""
    P, interp, star, disp, fitter = env
    out = []
    for n in (9, 800):
        lab = _labels(star, n, n)
        out += [interp.produce_model_bulk(disp, lab), np.array(fitter.chi2(interp, star.flux, star.var, lab))]
    return out


def _same(a, b):
    if isinstance(a, np.ndarray):
        return np.array_equal(a, b)
    if isinstance(a, (list, tuple)):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    return a == b


def test_grids_of_one_device_in_several_threads():
    jobs = [(_env(4000, 3), _fits), (_env(4100, 4), _models), (_env(4200, 5), _served), (_env(3900, 6), _models)]
    want = [f(e) for e, f in jobs]
    bad = []

    def work(k):
        try:
            for _ in range(6):
                if not _same(jobs[k][1](jobs[k][0]), want[k]):
                    bad.append((k, "differs"))
        except Exception as e:  # noqa: BLE001
            bad.append((k, repr(e)))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
