"""The per-image reductions of the preparation (templates' edge mean and sigma, RMS over the valid
shells, window sums), split over several CTAs per image: window sizes with one part per image, with
a remainder and with the most parts, templates of odd sizes, windows that hang over the micrograph;
stage by stage against the FP64 oracle with the tolerance of the other stage tests."""
import numpy as np
import pytest

import gisspa
import oracle
from parity import half_spectrum, rel_err
from test_gpu_parity import stage

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,shape,tsize", [(32, (45, 80), (17, 13)), (48, (48, 48), (48, 48)),
                                           (336, (400, 371), (101, 64)), (1024, (1024, 1100), (255, 301))])
def test_prepared_templates_and_windows(L, shape, tsize):
    rng = np.random.default_rng(L)
    img = rng.standard_normal(shape).astype(np.float32)
    tmpl = rng.standard_normal((3, *tsize)).astype(np.float32) + np.float32(0.5)
    cfg = gisspa.Config.default(angpix=1.2, phistep=90.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=200.0,
                                diameter=min(tsize), window_size=L, overlap=L // 3, norm_type=1)
    ctf = gisspa.Ctf(1.4, 0.05, 25.0)
    s = gisspa.Searcher(cfg)
    s.set_templates(tmpl)
    assert rel_err(stage(s, 1, None, ctf, 0.0, (3, L, L), np.float32), oracle.prep_templates(cfg, ctf, tmpl).real) < 1e-4
    o = half_spectrum(oracle.window_spectra(cfg, oracle.prep_image(cfg, ctf, img)))
    g = stage(s, 3, img, ctf, 0.0, o.shape, np.complex64)
    assert rel_err(g, o) < 1e-4
