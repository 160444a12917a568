"""The FFT stage over transform lengths of every column length (8 to 1024) and
row plan kind, at odd and even numbers of points, against the oracle on the
same grid; the adjoint through the same kernels against the tangent.

Tolerance: 2e-5 of the peak: FP32 rounding of a transform grows to ~log2(N) x
6e-8 ~ 1.3e-6, and the scatter before it is held to 2e-5."""
import numpy as np
import pytest

from oracle import ldm_oracle as O
from radis_gb300 import _lib as L
from radis_gb300 import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
TOL = 2e-5


@pytest.fixture(scope="module")
def ctx(native_lib):
    c = L.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("layout", [1, 3])
@pytest.mark.parametrize("n_v", [17, 128, 501, 640, 1537, 2560, 5001, 20001, 61441, 153601, 409601, 1100001])
def test_spectrum_lengths(ctx, n_v, layout):
    vmin, dv, T, p, x = 2000.0, 0.002, 900.0, 0.5, 0.2
    lines = S.uniform_lines(min(max(n_v // 4, 40), 20_000), vmin, vmin + n_v * dv, seed=n_v)
    ln = L.Lines(ctx, lines, 28.0)
    plan = L.Plan(ln, vmin, dv, n_v, n_G=2, n_L=6, layout=layout)
    out, info = plan.synthesize_host(T, p, x)
    ref = O.synthesize(lines, T, p, x, vmin, dv, n_v, info.grid.axes(), info.grid.n_ft, molar_mass=28.0, fft_workers=8)
    gpu = out.astype(np.float64) * np.exp(info.log_scale)
    # unaligned device output: the same values
    buf = torch.zeros(n_v + 1, dtype=torch.float32, device="cuda")
    plan.synthesize_device(T, p, x, buf[1:].data_ptr(), 1)
    torch.cuda.synchronize()
    assert np.array_equal(buf[1:].cpu().numpy(), out)
    assert np.max(np.abs(gpu - ref)) <= TOL * np.max(np.abs(ref))
    # g . dA/dtheta from the adjoint and from the tangent
    g = torch.rand(n_v + 1, dtype=torch.float32, device="cuda")[1:]
    d = torch.empty((3, n_v), dtype=torch.float32, device="cuda")
    grad = plan.backward(T, p, x, g.data_ptr(), stream_ptr=1)
    jinfo = plan.jvp(T, p, x, d.data_ptr(), stream_ptr=1)
    torch.cuda.synchronize()
    dd = d.double() * np.exp(jinfo.log_scale)
    for q in range(3):
        assert abs(grad[q] - float(torch.dot(g.double(), dd[q]))) <= 2e-4 * float(torch.dot(g.double(), dd[q].abs()))
    plan.close()
    ln.close()
