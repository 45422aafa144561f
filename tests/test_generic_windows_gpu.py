"""Window sizes without hand-tuned kernels: every radix of the mixed-radix rows (2 to 16, alone and
in plans of several stages), and correlation maps, sums and chunk picks at window sizes whose rows
per CTA and templates per pass differ, against numpy and the FP64 oracle with the tolerances of the
tests of the other sizes."""
import numpy as np
import pytest

import gisspa
import oracle
from parity import check_chunk_picks, rel_err
from test_gpu_parity import stage

pytestmark = pytest.mark.gpu


def _searcher(L, **over):
    cfg = gisspa.Config.default(angpix=2.0, phistep=90.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=200.0,
                                diameter=24.0, window_size=L, overlap=L // 4, norm_type=1, **over)
    return cfg, gisspa.Searcher(cfg)


@pytest.mark.parametrize("n", [7, 10, 12, 14, 15, 28, 60, 90, 225, 343, 420, 1500, 3136, 8100])
@pytest.mark.parametrize("sign", [-1, 1])
def test_mixed_radix_rows(n, sign):
    torch = pytest.importorskip("torch")
    _, s = _searcher(64)
    rows = 1 + 5000 // n
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((rows, n)) + 1j * rng.standard_normal((rows, n))).astype(np.complex64)
    d = torch.from_numpy(x.copy()).cuda()
    assert gisspa.load().gisspa_debug_fft(s.h, d.data_ptr(), rows, n, sign) == 0
    ref = np.fft.fft(x.astype(np.complex128), axis=1) if sign < 0 else np.fft.ifft(x.astype(np.complex128), axis=1) * n
    err = np.linalg.norm(d.cpu().numpy() - ref) / np.linalg.norm(ref)
    assert err < 3e-6 * np.log2(n)  # as the other FFT rows


@pytest.mark.parametrize("L,nt", [(32, 1), (48, 33), (112, 5), (240, 3), (400, 2), (720, 2), (1008, 1), (2048, 1)])
@pytest.mark.parametrize("spec", [gisspa.SPEC_FP32, gisspa.SPEC_FP16])
def test_maps(L, nt, spec):
    torch = pytest.importorskip("torch")
    _, s = _searcher(L, spectrum_precision=spec)
    rng = np.random.default_rng(L)
    dt = np.complex64 if spec == gisspa.SPEC_FP32 else np.float16
    W = np.fft.fft2(rng.standard_normal((2, L, L))) / L
    T = np.fft.fft2(rng.standard_normal((nt, L, L))) / L
    dW = np.ascontiguousarray(np.swapaxes(W, 1, 2)[:, :L // 2 + 1].astype(np.complex64))
    dT = np.ascontiguousarray(np.swapaxes(T, 1, 2)[:, :L // 2 + 1].astype(np.complex64))
    if spec == gisspa.SPEC_FP16:  # the maps of the rounded spectra
        dT = np.ascontiguousarray(dT.view(np.float32).astype(np.float16))
        half = dT.astype(np.float32).view(np.complex64)
    else:
        half = dT
    out = torch.zeros((2, nt, L, L), dtype=torch.float32, device="cuda")
    gW, gT = torch.from_numpy(dW).cuda(), torch.from_numpy(dT).cuda()
    assert gisspa.load().gisspa_cc_maps(s.h, gW.data_ptr(), 2, gT.data_ptr(), nt, spec, out.data_ptr()) == 0
    g = out.cpu().numpy()
    for b in range(2):
        for n in range(nt):
            z = np.fft.ifft(dW[b].astype(np.complex128) * np.conj(half[n].astype(np.complex128)), axis=1)
            ref = np.fft.fftshift(np.fft.irfft(z.T, n=L, axis=1))
            assert rel_err(g[b, n], ref) < 1e-4, (b, n)


@pytest.mark.parametrize("L", [112, 240])
def test_statistics_and_picks(L):
    rng = np.random.default_rng(L)
    img = rng.standard_normal((2 * L, 2 * L - 9)).astype(np.float32)
    tmpl = rng.standard_normal((9, 40, 40)).astype(np.float32)
    cfg, s = _searcher(L, threshold=3.0)
    ctf = gisspa.Ctf(1.4, 0.05, 25.0)
    s.set_templates(tmpl)
    picks = s.search(img, ctf)
    _, st = oracle.search(cfg, ctf, img, tmpl, want_stats=True)
    ms = stage(s, 5, None, ctf, 0.0, (st.shape[0], L, L, 2), np.float32)
    assert np.abs(ms[..., 0] - st[..., 0]).max() <= 1e-4 * np.abs(st[..., 1]).max()
    assert rel_err(np.where(ms[..., 1] > 0, 1 / np.maximum(ms[..., 1], 1e-30), 0), st[..., 1]) < 1e-4
    o, m, near, nm = oracle.search(cfg, ctf, img, tmpl, want_margins=True)
    assert len(o) > 0
    assert not check_chunk_picks(picks, o, m, near, nm, cfg.threshold)["failures"]
