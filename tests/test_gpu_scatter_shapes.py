"""The scatter's tile shapes at the edges of their ranges, against the oracle's
LDM tensor: windows of fewer columns than SMs, one column more than a whole
round of tiles, copies of the tile (lists of many lines per column) and both
accumulator widths.

Tolerance: 2e-5 of the LDM's peak, the bound of the scatter at the default node
spacing (tests/test_gpu_parity.py)."""
import numpy as np
import pytest

from oracle import ldm_oracle as O
from radis_gb300 import _lib as L
from radis_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(native_lib):
    c = L.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("accumulator", [32, 64])
@pytest.mark.parametrize("n_v,per_col,shift", [(3, 300, False), (33, 1, True), (151, 40, True), (153, 40, False),
                                               (64 * 152 + 1, 6, True), (1025, 100, False)])
def test_scatter_tiles(ctx, n_v, per_col, shift, accumulator):
    vmin, dv, T, p, x = 2000.0, 0.005, 1200.0, 2.0, 0.2
    width = n_v * dv
    lines = S.uniform_lines(max(int(per_col * n_v), 64), vmin - 0.1 * width, vmin + 1.1 * width, seed=n_v,
                            delta=(-0.01, 0.01) if shift else None)
    ln = L.Lines(ctx, lines, 44.0)
    plan = L.Plan(ln, vmin, dv, n_v, dxG=S.DXG_DEFAULT, dxL=S.DXL_DEFAULT, accumulator=accumulator)
    ldm, info = plan.debug_ldm(T, p, x)
    kpos, lgG, lgL, Sl = O.line_quantities(lines, T, p, x, vmin, dv, molar_mass=44.0)
    ref = O.ldm_scatter(kpos, lgG, lgL, Sl * O.number_density(p, T, x), n_v, info.grid.axes())
    ref = np.transpose(ref, (1, 2, 0))
    gpu = ldm.astype(np.float64) * np.exp(info.log_scale)
    assert np.max(np.abs(gpu - ref)) <= 2e-5 * np.max(np.abs(ref))
    assert info.lines_in_window == np.sum((np.floor(kpos) >= 0) & (np.floor(kpos) + 1 < n_v))
    a, ia = plan.synthesize_host(T, p, x)   # the projecting flush where the grid takes it, twice: deterministic
    b, _ = plan.synthesize_host(T, p, x)
    assert ia.accum_bits == accumulator and np.array_equal(a, b)
    plan.close()
    ln.close()
