"""Derivatives on skeleton rows where the spectrum itself takes merged rows:
against the same derivatives on node rows (layout 1), for sparse lists (the
tangent scattered straight into the skeleton rows) and dense ones (projected in a
pass).

Tolerance: 4e-5 of each derivative's peak, and of sum |g| |dA| for products,
twice the bound between two layouts of a spectrum (2e-5): a tangent's rows are
differences of rows of the spectrum's size."""
import numpy as np
import pytest

from radis_gb300 import _lib as L
from radis_gb300 import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(native_lib):
    c = L.Context(0)
    yield c
    c.close()


def derivatives(ctx, lines, mass, n_v, cond, g, layout):
    ln = L.Lines(ctx, lines, mass)
    plan = L.Plan(ln, 2000.0, 0.001, n_v, dxG=S.DXG_DEFAULT, dxL=S.DXL_DEFAULT, layout=layout)
    d = torch.zeros((3, n_v), dtype=torch.float32, device="cuda")
    info = plan.jvp(*cond, d.data_ptr(), stream_ptr=1)
    v = np.asarray(plan.backward(*cond, g.data_ptr(), stream_ptr=1))
    _, i = plan.synthesize_host(*cond)
    out = d.cpu().double().numpy() * np.exp(info.log_scale)
    plan.close()
    ln.close()
    return out, v, i.layout


@pytest.mark.parametrize("n_lines,n_v,mass,p", [
    (1, 1000, 28.0, 1.0), (777, 50_001, 28.0, 1.0), (4_000, 100_000, 28.0, 0.3), (400_000, 50_001, 28.0, 1.0),
    (3_000, 30_003, [2.0, 28.0, 60.0], 1.0)])
def test_derivative_rows(ctx, n_lines, n_v, mass, p):
    hi = 2000.0 + n_v * 0.001
    lines = S.uniform_lines(n_lines, 2000.0, hi, seed=n_v, delta=(-0.01, 0.01))
    if np.ndim(mass):
        lines["iso"] = np.random.default_rng(1).integers(0, 3, n_lines).astype(np.uint8)
        mass = np.array(mass)
    cond = (700.0, p, 0.1)
    g = torch.from_numpy(np.random.default_rng(2).normal(size=n_v).astype(np.float32)).cuda()
    a, va, layout = derivatives(ctx, lines, mass, n_v, cond, g, 0)
    b, vb, _ = derivatives(ctx, lines, mass, n_v, cond, g, 1)
    gh = np.abs(g.cpu().double().numpy())
    for q in range(3):
        assert np.max(np.abs(a[q] - b[q])) <= 4e-5 * np.max(np.abs(b[q])), (q, layout)
        assert abs(va[q] - vb[q]) <= 4e-5 * np.sum(gh * np.abs(b[q])), (q, layout)
