"""The field map against the reference quadrature and the direct sums, where it can go wrong:
cell edges and corners, the band's edge, outside the root square, remainders
of the kernel's chunks, and non-finite points."""

import ctypes

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from bem_b200 import _lib, engine  # noqa: E402
from bem_b200.tables import BemTables  # noqa: E402

import gpu_util as gu  # noqa: E402


def _direct(tab, pts):
    v = tab.view("adaptive", field_map=False)
    x, y, z = (torch.as_tensor(np.ascontiguousarray(pts[:, k]), device="cuda") for k in range(3))
    e = [torch.empty_like(x) for _ in range(3)]
    _lib.check(_lib.lib().spt_bem_field(x.data_ptr(), y.data_ptr(), z.data_ptr(), len(pts), ctypes.byref(v), 0,
                                        e[0].data_ptr(), e[1].data_ptr(), e[2].data_ptr(),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "spt_bem_field")
    return torch.stack(e, -1).cpu().numpy()


def _cells(tab):
    m, tag = tab.field_map()
    m = m[(tag & 0xFFFF) * _lib.MAP_UNIT:].cpu().numpy()
    rec = m[int(m[2]):int(m[3])].reshape(-1, _lib.MAP_REC)
    return rec[:, 0], rec[:, 1], 1.0 / rec[:, 2]


@pytest.mark.parametrize("fixture", ["bem_sphere", "bem_well", "bem_post", "sigma_c1", "sigma_c3"])
def test_map_matches_reference_quadrature_at_cell_edges(fixture):
    """Corners, edge midpoints and centres of cells of every size, a rounding
    error inside and outside: 2e-12 of the larger of the cell's field and the
    uniform one (the adaptive rule's 1e-12 bound, twice, as the samples are
    its sums with tighter thresholds; the truncation, 2e-14, is far below).
    Against the reference quadrature; points an edge leaves without a cell
    are the direct sums bit for bit (at their default thresholds those are
    themselves 3e-12 off it in places of the 3000-panel well)."""
    g = load_golden(fixture)
    tab = BemTables(g["profile"], g["sigma"], int(g["n_subdiv"]) if "n_subdiv" in g else 8)
    rc, zc, h = _cells(tab)
    rng = np.random.default_rng(1)
    pick = rng.choice(len(rc), min(len(rc), 400), replace=False)
    fr = np.array([-1, 1, -1, 1, 0, 0, -1, 1, 0]) * (1 + np.array([0, 0, 1, 1, 0, 0, 1, -1, 0]) * 1e-9)
    fz = np.array([-1, -1, 1, 1, 0, -1, 0, 0, 1]) * (1 - np.array([0, 1, 0, 1, 0, 1, 0, 0, -1]) * 1e-9)
    rho = np.abs(rc[pick, None] + h[pick, None] * fr)
    z = zc[pick, None] + h[pick, None] * fz
    ph = rng.uniform(0, 2 * np.pi, rho.shape)
    pts = np.stack([rho * np.cos(ph), rho * np.sin(ph), z], -1).reshape(-1, 3)
    got, ref = engine.bem_field(tab, pts, far_rule="adaptive").cpu().numpy(), engine.bem_field(tab, pts).cpu().numpy()
    norm = np.linalg.norm(ref, axis=-1).reshape(rho.shape).max(axis=1, keepdims=True)
    uniform = np.abs(float(g["E_gun"])) if "E_gun" in g else np.linalg.norm(ref, axis=-1).max()
    err = np.abs(got - ref).max(axis=-1).reshape(rho.shape)
    direct = np.all(got == _direct(tab, pts), axis=-1).reshape(rho.shape)
    assert direct[:, 4].mean() < 0.05  # the cells did take part: every centre (column 4) lies in one
    assert (err / np.maximum(norm, uniform))[~direct].max() < 2e-12


def test_chunks_and_band_leave_each_point_its_value():
    """A point's value does not depend on the points beside it or on their
    number (chunks of 8 to 256, a remainder in each), near the surface or in
    a cell; and other thresholds than the map's are the direct sums."""
    g = load_golden("sigma_c1")
    tab = BemTables(g["profile"], g["sigma"], 8)
    rng = np.random.default_rng(2)
    n = 5 * 148 * 2 * 8 + 3
    d, th = 10 ** rng.uniform(-10, -6, n), rng.uniform(0, 1.2, n)
    pts = np.stack([(50e-9 + d) * np.sin(th), np.zeros(n), 5e-6 + (50e-9 + d) * np.cos(th)], -1)
    whole = engine.bem_field(tab, pts, far_rule="adaptive")
    for a, b in ((0, 1), (1, 8), (8, 17), (100, 357), (357, 357 + 2369), (3000, n)):
        assert torch.equal(engine.bem_field(tab, pts[a:b], far_rule="adaptive"), whole[a:b])
    assert tab.view("adaptive").reserved >> 16 == _lib.MAP_TAG
    for kw in (dict(ratio4=9.0), dict(ratio2=200.0), dict(ratio_run=5.0), dict(cluster_kappa=0.0), dict(bounds=False)):
        assert tab.view("adaptive", **kw).reserved == 0
    assert tab.view("reference").reserved == 0


def test_points_without_a_cell():
    """Outside the root square, and non-finite: the direct path's results."""
    g = load_golden("bem_sphere")
    tab = BemTables(g["profile"], g["sigma"], int(g["n_subdiv"]))
    nan, inf = float("nan"), float("inf")
    pts = np.array([[1.0, 0, 0], [0, 0, -5.0], [0, 0, 7.0], [nan, 0, 0], [0, nan, 1e-6], [0, 0, nan], [inf, 0, 0],
                    [0, 0, inf], [0, 0, -inf]])
    np.testing.assert_array_equal(engine.bem_field(tab, pts, far_rule="adaptive").cpu().numpy(), _direct(tab, pts))


@pytest.mark.parametrize("fixture", ["bem_sphere", "bem_well", "bem_post", "sigma_c1", "sigma_c3"])
def test_radial_field_near_the_axis_keeps_its_digits(fixture):
    """E_rho from 1e-12 to 1e-6 of the surface's distance off the axis against
    the reference quadrature (whose near-axis terms are exact there): it falls
    with rho, and so does its error.  A cell's error is bounded by 2e-12 of
    the field, as at its edges, times rho / half-width; cells are at least a
    24th of their distance from the surface wide (one twice as wide that is 12
    half-widths away is taken), so 24 x 2e-12 x rho / distance."""
    g = load_golden(fixture)
    prof = g["profile"]
    tab = BemTables(prof, g["sigma"], int(g["n_subdiv"]) if "n_subdiv" in g else 8)
    assert tab.field_map() is not None
    scale = np.hypot(prof[:, 0], prof[:, 1] - prof[:, 1].mean()).max()
    d = scale * 10 ** np.linspace(-2.6, 0.8, 35)
    for f in (1e-12, 1e-9, 1e-7, 1e-6):
        pts = np.stack([f * d, np.zeros_like(d), prof[0, 1] + d], -1)  # every profile starts on the axis
        got, ref = engine.bem_field(tab, pts, far_rule="adaptive").cpu().numpy(), engine.bem_field(tab, pts).cpu().numpy()
        uniform = np.abs(float(g["E_gun"])) if "E_gun" in g else np.linalg.norm(ref, axis=-1).max()
        bound = 24 * 2e-12 * f * np.maximum(np.linalg.norm(ref, axis=-1), uniform)
        assert (np.abs(got[:, 0] - ref[:, 0]) <= bound).all()


def test_nan_points_are_near_no_panel():
    """A NaN coordinate is no panel's neighbour: one attempt of such a single
    electron beside a healthy one counts that one's near panels only (the sinh
    rule at 71 intervals a panel was what a NaN point cost), and a field call
    gives the finite points beside NaN ones their own values."""
    g = load_golden("trace_post")
    spec = dict(kind="post_bem", E_gun=float(g["E_gun"]), R=float(g["R"]), L=float(g["L"]), z0=float(g["z0"]),
                profile=g["profile"], sigma=g["sigma"], n_subdiv=int(g["n_subdiv"]), z_handoff=float(g["z_handoff"]),
                kill_z_below=0.0)
    geo = gu.device_geometry(spec)
    near = []
    for x in ([0.0, float("nan")], [0.0]):
        pos = np.array([[v, 1e-9, geo.L + geo.R + 1e-11] for v in x])
        n = len(pos)
        tr = engine.Tracer(geo, far_rule="adaptive")
        b = engine.GroupBatch(pos, np.zeros((n, 3)), np.zeros(n), np.full(n, gu.Q_E), np.full(n, gu.M_E), [1] * n)
        tr.launch(b, tr.params(1e-12, 1e-8, 1e-12, 1e-12, gu.CM, 1))
        near.append(tr.counter_dict()["near_pairs"])
    assert near[0] == near[1] > 0
    tab = geo.bem_tables("cuda")
    pts = np.stack([np.zeros(64), np.full(64, 1e-9), geo.L + geo.R * (1 + 10.0 ** np.linspace(-6, 1, 64))], -1)
    want = engine.bem_field(tab, pts, far_rule="adaptive").cpu().numpy()
    mixed = pts.copy()
    mixed[1::2, 0] = mixed[::4, 2] = np.nan
    got = engine.bem_field(tab, mixed, far_rule="adaptive").cpu().numpy()
    finite = np.isfinite(mixed).all(axis=-1)
    np.testing.assert_array_equal(got[finite], want[finite])
    assert np.isnan(got[~finite]).any(axis=-1).all()


def test_first_calls_do_without_cells_until_they_pay():
    """A fresh geometry's first calls read a map without cells (every point its
    own direct sum: the bits that a point near the surface has with cells too)
    and keep the 2e-12 bound; the call that reaches field_map.worth points has
    the cells, and then a point's value still does not depend on the points
    beside it or on their number."""
    from bem_b200 import field_map

    g = load_golden("bem_sphere")
    tab = BemTables(g["profile"], g["sigma"], int(g["n_subdiv"]))
    R = g["profile"][0, 1]
    rng = np.random.default_rng(3)
    n = field_map.worth(g["profile"])
    th, ph, d = rng.uniform(0, np.pi, n), rng.uniform(0, 2 * np.pi, n), 10 ** rng.uniform(-3, 1, n)
    pts = R * (1 + d)[:, None] * np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], -1)
    first = engine.bem_field(tab, pts[:2000], far_rule="adaptive")
    assert tab.view("adaptive", points=0).reserved >> 16 == _lib.MAP_TAG and not tab._map
    ref = engine.bem_field(tab, pts[:2000])
    scale = ref.norm(dim=1).clamp(min=abs(float(g["E_gun"])))
    assert ((first - ref).norm(dim=1) / scale).max() < 2e-12
    whole = engine.bem_field(tab, pts, far_rule="adaptive")
    rc, zc, h = _cells(tab)
    assert tab._map and len(rc) > 0
    # within two panel lengths of the surface no point has a cell
    near = torch.as_tensor(d[:2000] * R < np.linalg.norm(np.diff(g["profile"], axis=0), axis=1).min(), device="cuda")
    assert near.any() and torch.equal(whole[:2000][near], first[near])
    assert ((whole[:2000] - ref).norm(dim=1) / scale).max() < 2e-12
    for a, b in ((0, 1), (1, 8), (8, 17), (100, 357), (357, 357 + 2369), (3000, 40_003)):
        assert torch.equal(engine.bem_field(tab, pts[a:b], far_rule="adaptive"), whole[a:b])
    nan, inf = float("nan"), float("inf")
    out = np.array([[1.0, 0, 0], [0, 0, -5.0], [0, 0, 7.0], [nan, 0, 0], [0, nan, 1e-6], [0, 0, nan], [inf, 0, 0]])
    got = engine.bem_field(tab, out, far_rule="adaptive").cpu().numpy()
    assert np.array_equal(np.isnan(got).any(axis=-1), ~np.isfinite(out).all(axis=-1))
