"""Sweep 1 with two templates per transform (window sizes 256, 320, 512, 1024) against the one-template
kernels that a fixed launch shape selects: per-pixel sums, sums of squares and best correlations
of one rank's sweep.  Template counts that leave the last pair half empty or a launch with fewer
pairs than shares per row, one window and several, every spectrum precision."""
import numpy as np
import pytest

import gisspa
import synth

pytestmark = pytest.mark.gpu

# Both paths hold the same stored spectra and FP32 transforms of 2 L^2 points: either's rounding is
# at most about log2(L^2) * 2^-24 = 1.2e-6 of the map's rms (L = 1024); ten times that bounds the
# difference of sums over a few dozen of them.
RTOL = 1e-5


def _state(cfg, tmpl, img, ctf):
    import torch
    s = gisspa.Searcher(cfg)
    s.set_templates(tmpl)
    info = s.shard_begin(img, ctf)
    s.shard_sweep(1, 0, info.n_angles)
    n = info.n_pixels
    s1 = torch.empty(n, device="cuda", dtype=torch.float64)
    s2 = torch.empty_like(s1)
    key = torch.empty(n, device="cuda", dtype=torch.int64)
    s.shard_export(s1.data_ptr(), s2.data_ptr(), key.data_ptr())
    s.close()
    k = key.cpu().numpy().view(np.uint64) ^ np.uint64(1 << 63)
    hi = (k >> np.uint64(32)).astype(np.uint32)
    best = np.where(hi & 0x80000000, hi & 0x7FFFFFFF, ~hi).astype(np.uint32).view(np.float32)
    return s1.cpu().numpy(), s2.cpu().numpy(), best.astype(np.float64), (~k & np.uint64(0xFFFFFFFF)).astype(np.int64)


@pytest.mark.parametrize("spec", [gisspa.SPEC_FP32, gisspa.SPEC_FP16, gisspa.SPEC_BF16])
@pytest.mark.parametrize("L,shape,nt", [(256, (256, 256), 1), (256, (500, 700), 7), (320, (320, 320), 2),
                                        (320, (500, 660), 5), (512, (512, 512), 9), (512, (512, 512), 3),
                                        (512, (900, 1300), 4), (1024, (1024, 1024), 3),
                                        (1024, (1900, 2700), 4)])
def test_paired_sweep_equals_the_one_template_sweep(L, shape, nt, spec):
    c = synth.make_case(shape=shape, n_particles=3, snr=0.5, n_templates=nt, tsize=L // 4, seed=L + nt, margin=L // 5)
    cfg = gisspa.Config.default(angpix=1.0, phistep=60.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=200.0,
                                diameter=L / 5, threshold=3.0, window_size=L, overlap=L // 4, norm_type=1,
                                pick_mode=gisspa.PICK_TOPK, topk=10, spectrum_precision=spec)
    ctf = gisspa.Ctf(c.defocus, c.dfdiff, c.dfang)
    a = _state(cfg, c.templates, c.image, ctf)
    b = _state(cfg.copy(template_batch=2, window_batch=2), c.templates, c.image, ctf)
    for x, y in zip(a[:3], b[:3]):
        assert np.linalg.norm(x - y) <= RTOL * np.linalg.norm(y)
    # where the two name another template-rotation, the best two correlations are within rounding
    other = a[3] != b[3]
    assert other.mean() < 1e-3
    assert np.all(np.abs(a[2] - b[2])[other] <= RTOL * np.abs(b[2]).max())
