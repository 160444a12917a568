"""The Gaussian rows that a tile of the scatter holds, and the projection of
its columns to skeleton rows: windows of two rows up to all of them, odd
numbers of Lorentzian nodes, up to 30 skeleton rows, two and more copies of the
tile, tiles of one column, and windows of so many nodes that the projection's
coefficients (or 32 columns) no longer fit beside them.

Tolerances: the LDM within 2e-5 of its peak of the oracle's, on the grids with
a Gaussian spacing of at least 4e-3 (below, the FP32 fraction of a cell, 2^-24
of a log width over the spacing, is what the oracle's differs by); the spectrum from
skeleton rows within 2e-5 of its peak of the one from node rows (the
decomposition's 1e-8, the FP32 transforms of either and the TF32 split of
2^-22 per product add up to less)."""
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


# masses, n_v, dv, vmin, lines per column, n_G, n_L, accumulator, pressure shift
CASES = [
    ([44.0], 20_001, 0.01, 2000.0, 2, 8, 15, 32, False),          # two or three rows of eight
    ([2.0, 44.0, 90.0], 5_001, 0.01, 2000.0, 3, 10, 14, 32, True),   # most rows: masses far apart
    ([2.0, 44.0, 90.0], 5_001, 0.01, 2000.0, 3, 24, 9, 64, True),
    ([18.0], 3_001, 2.0, 10.0, 1, 40, 7, 32, False),              # steep Gaussian axis: wide windows at low v0
    ([44.0], 1_217, 0.01, 2000.0, 400, 6, 9, 32, False),          # dense: two copies
    ([44.0], 1_217, 0.01, 2000.0, 400, 6, 9, 64, False),          # dense: eight copies
    ([44.0], 100, 0.01, 2000.0, 20, 12, 56, 64, True),            # 672 nodes: no room for coefficients
    ([44.0], 100, 0.01, 2000.0, 300, 16, 63, 32, False),          # 1008 nodes, no room for copies
    ([44.0], 9_001, 0.01, 2000.0, 1, 13, 62, 64, True),           # 806 nodes of 64-bit sums: tiles of 28 columns
]


@pytest.mark.parametrize("masses,n_v,dv,vmin,per_col,n_G,n_L,accumulator,shift", CASES)
def test_scatter_windows(ctx, masses, n_v, dv, vmin, per_col, n_G, n_L, accumulator, shift):
    T, p, x = 1200.0, 0.5, 0.2
    width = n_v * dv
    lines = S.uniform_lines(max(int(per_col * n_v), 64), max(vmin - 0.1 * width, 0.5 * vmin), vmin + 1.1 * width, seed=n_v,
                            delta=(-0.01, 0.01) if shift else None)
    mass = np.array(masses)
    if len(masses) > 1:
        lines["iso"] = np.random.default_rng(n_v).integers(0, len(masses), len(lines["v0"])).astype(np.uint8)
    else:
        mass = masses[0]
    ln = L.Lines(ctx, lines, mass)
    kw = dict(n_G=n_G, n_L=n_L, accumulator=accumulator)
    plan = L.Plan(ln, vmin, dv, n_v, layout=1, **kw)
    ldm, info = plan.debug_ldm(T, p, x)
    kpos, lgG, lgL, Sl = O.line_quantities(lines, T, p, x, vmin, dv, molar_mass=mass)
    ref = O.ldm_scatter(kpos, lgG, lgL, Sl * O.number_density(p, T, x), n_v, info.grid.axes())
    ref = np.transpose(ref, (1, 2, 0))
    gpu = ldm.astype(np.float64) * np.exp(info.log_scale)
    if info.grid.axes()[1] >= 4e-3:
        assert np.max(np.abs(gpu - ref)) <= 2e-5 * np.max(np.abs(ref))
    a, ia = plan.synthesize_host(T, p, x)
    plan.close()
    skel = L.Plan(ln, vmin, dv, n_v, layout=3, **kw)
    b, ib = skel.synthesize_host(T, p, x)
    c, _ = skel.synthesize_host(T, p, x)
    skel.close()
    ln.close()
    assert ia.accum_bits == ib.accum_bits == accumulator and np.array_equal(b, c)
    assert np.max(np.abs(a - b)) <= 2e-5 * np.max(np.abs(a)), (ib.layout, ib.fft_rows)


@pytest.mark.parametrize("accumulator", [32, 64])
@pytest.mark.parametrize("columns", [[0], [15], [16, 17], [5, 700, 9_998], [9_999]])
def test_mostly_empty_columns(ctx, columns, accumulator):
    """A few lines in a window of empty columns: the projection leaves out the
    columns and nodes that hold nothing.  Skeleton against node rows, 2e-5 of
    the peak; nothing at all where the only line lies on the last column."""
    vmin, dv, n_v = 2000.0, 0.01, 10_000
    lines = S.uniform_lines(200, vmin + 200.0, vmin + 400.0, seed=3, s_lo=1e-21, s_hi=1e-20, el_mean=1.0)
    lines["v0"][:len(columns)] = vmin + dv * (np.array(columns) + 0.3)   # the others span the node axes
    ln = L.Lines(ctx, lines, 44.0)
    out = []
    for layout in (1, 3):
        plan = L.Plan(ln, vmin, dv, n_v, n_G=6, n_L=9, accumulator=accumulator, layout=layout)
        out.append(plan.synthesize_host(900.0, 0.5, 0.2))
        plan.close()
    ln.close()
    (a, _), (b, i) = out
    assert i.layout == 4 and (np.max(a) > 0) == (columns[0] + 1 < n_v)
    assert np.max(np.abs(a - b)) <= 2e-5 * np.max(np.abs(a))
