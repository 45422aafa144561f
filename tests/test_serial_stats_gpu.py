"""LoadImage statistics: the reference's running FP32 sums evaluated in parallel, against the
oracle's serial loop, on micrographs whose outlier bounds (integers, from those sums) decide which
pixels are replaced: sums that drift by their own rounding, that hover around zero, that stay zero
for a while or whose terms are exact ties; sizes around a chunk of 256 and a block of 4096 terms."""
import numpy as np
import pytest

import gisspa
import oracle
from parity import rel_err
from test_gpu_parity import stage

pytestmark = pytest.mark.gpu


def _image(kind, shape, rng):
    x = rng.standard_normal(shape, dtype=np.float32)
    if kind == "counts":
        x = np.round(20 + 4 * x).astype(np.float32)
    elif kind == "ties":
        x = np.round(3 * x).astype(np.float32)
    elif kind == "late":
        x[: shape[0] // 2] = 0
    elif kind == "alternating":
        x = np.where(np.arange(x.size) % 2, 1, -1).astype(np.float32).reshape(shape)
    # outliers on both sides of the bounds
    at = rng.integers(0, x.size, 40)
    x.reshape(-1)[at] += np.float32(x.std()) * rng.uniform(-9, 9, 40).astype(np.float32)
    return x


@pytest.mark.parametrize("shape", [(32, 32), (31, 33), (64, 64), (63, 65), (300, 211), (1024, 1024)])
@pytest.mark.parametrize("kind", ["noise", "counts", "ties", "late", "alternating"])
def test_serial_statistics_match_the_serial_loop(kind, shape):
    rng = np.random.default_rng(len(kind) + shape[1])
    img = _image(kind, shape, rng)
    cfg = gisspa.Config.default(angpix=1.0, phistep=90.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=200.0,
                                diameter=20.0, window_size=32, norm_type=1)
    ctf = gisspa.Ctf(1.5, 0.05, 20.0)
    s = gisspa.Searcher(cfg)
    s.set_templates(rng.standard_normal((1, 16, 16)).astype(np.float32))
    g = stage(s, 2, img, ctf, 0.0, img.shape, np.float32)
    assert rel_err(g, oracle.prep_image(cfg, ctf, img)) < 1e-4
