"""The slit convolution at the edges of its CTA and pass sizes (outputs per CTA,
taps per pass, the two groups' shares), against numpy in FP64.  Tolerance: 1e-5
of the peak, as in tests/test_gpu_slit.py."""
import numpy as np
import pytest

from radis_gb300 import slit as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 4, 9, 17, 511, 513, 1030])
@pytest.mark.parametrize("n", [1, 7, 300, 9729, 8 * 128 * 152, 8 * 128 * 152 + 1])
def test_slit_sizes(native_lib, n, m):
    rng = np.random.default_rng(n * 7919 + m)
    x = rng.uniform(0.0, 1.0, n).astype(np.float32)
    s = rng.uniform(0.0, 1.0, m).astype(np.float32)
    full = np.convolve(x.astype(np.float64), s.astype(np.float64)) if n * m < 1e8 else None
    if full is None:
        k = n + m
        full = np.fft.irfft(np.fft.rfft(x.astype(np.float64), k) * np.fft.rfft(s.astype(np.float64), k), k)
    ref = 0.25 * full[(m - 1) // 2:(m - 1) // 2 + n]
    for mode in ("same", "valid"):
        y = S.convolve_device(torch.from_numpy(x).cuda(), s, 0.25, mode=mode).cpu().numpy().astype(np.float64)
        la = min(n, m)
        bad = np.zeros(n, bool)
        if mode == "valid":
            bad[:(la - 1) // 2] = True
            bad[n - la // 2:] = True
        assert np.array_equal(np.isnan(y), bad)
        assert np.max(np.abs((y - ref)[~bad]), initial=0.0) <= 1e-5 * np.max(np.abs(ref))
