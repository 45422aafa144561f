"""norm_type=0 peaks with the row maximum checked before the chunk scan: windows of every row kernel,
a border that leaves a few pixels, none, or all of the window, against the FP64 oracle's picks."""
import numpy as np
import pytest

import gisspa
import oracle
from parity import check_template_picks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,diameter", [(256, 40.0), (256, 500.0), (320, 30.0), (512, 1030.0)])
def test_peaks(L, diameter):
    rng = np.random.default_rng(L)
    img = rng.standard_normal((720, 720)).astype(np.float32)
    tmpl = rng.standard_normal((3, 64, 64)).astype(np.float32)
    cfg = gisspa.Config.default(angpix=1.0, phistep=120.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=200.0,
                                diameter=diameter, threshold=2.0, window_size=L, overlap=L // 4, norm_type=0)
    ctf = gisspa.Ctf(1.5, 0.0, 0.0)
    s = gisspa.Searcher(cfg)
    s.set_templates(tmpl)
    g = s.search(img, ctf)
    o, m, _, _ = oracle.search(cfg, ctf, img, tmpl, want_margins=True)
    assert len(g) > 0 or len(o) == 0
    assert not check_template_picks(g, o, m, cfg.threshold)["failures"]
