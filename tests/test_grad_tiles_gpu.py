"""The score gradient's pixel tiles: masks smaller than a tile, of a few tiles, and cut by the
window (large diameters, shifts towards an edge), against the FP64 oracle's score and its central
differences, with the tolerances of the adjoint's own oracle test.  (Where a mask is cut by the
window, samples enter and leave the template as it turns: steps of 1e-6 pass none of them here.)"""
import numpy as np
import pytest

import gisspa
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("diameter,shift", [(2.0, (0.31, -0.23)), (30.0, (0.31, -0.23)), (30.0, (27.4, -25.7)),
                                            (120.0, (0.31, -0.23))])
def test_tiles(diameter, shift):
    L = 64
    rng = np.random.default_rng(int(diameter))
    img = rng.standard_normal((250, 256)).astype(np.float32)
    tmpl = rng.standard_normal((3, 40, 40)).astype(np.float32)
    cfg = gisspa.Config.default(angpix=2.0, phistep=45.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=200.0,
                                diameter=diameter, window_size=L, overlap=24, norm_type=1, threshold=0.5,
                                pick_mode=gisspa.PICK_TOPK, topk=3, exclusion_radius=5.0)
    ctf = gisspa.Ctf(1.4, 0.05, 25.0)
    s = gisspa.Searcher(cfg)
    s.set_templates(tmpl)
    picks = s.search(img, ctf)
    assert len(picks)
    _, st = oracle.search(cfg, ctf, img, tmpl, want_stats=True)
    ox, oy = oracle.window_offsets(256, L, cfg.overlap), oracle.window_offsets(250, L, cfg.overlap)
    img_pre = oracle.prep_image(cfg, ctf, img)
    prep = oracle.prep_templates(cfg, ctf, tmpl).real
    for p in picks[:2]:
        b = int(p["window"])
        off = (ox[b % len(ox)], oy[b // len(ox)])
        px, py = int(p["x"]) - off[0], int(p["y"]) - off[1]
        mu, sd = st[b, py, px]
        q0 = np.array([*shift, float(p["theta"]) + 1.7])

        def f(q):
            return oracle.pick_score(cfg, prep[int(p["template_id"])], img_pre, off, px, py, *q, mu, sd)

        fd = np.array([(f(q0 + d) - f(q0 - d)) / 2e-6 for d in 1e-6 * np.eye(3)])
        g = s.score_grad(p[None], q0[None].astype(np.float32), ctf)[0]
        ours = np.array([g["d_dx"], g["d_dy"], g["d_theta"]], np.float64)
        assert abs(float(g["score"]) - f(q0)) <= 1e-4 * abs(f(q0)) + 1e-5
        assert np.linalg.norm(ours - fd) < 1e-3 * max(np.linalg.norm(fd), 1e-6), (ours, fd)
