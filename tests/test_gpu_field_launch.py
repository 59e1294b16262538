"""Field launches (spt_field.cu) where their work split can go wrong: point
counts that give 1 to 64 shares a point, panel counts and sub-panels that leave
remainders, masked and ragged groups, an offset table that starts above 0."""

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
from oracle import bem as ob  # noqa: E402

import gpu_util as gu  # noqa: E402


@pytest.mark.parametrize("n_subdiv", [1, 3, 8])
@pytest.mark.parametrize("panels", [5, 32, 33, 97, 600])
def test_reference_rule_at_every_share_count(panels, n_subdiv):
    """n points of a sphere's field, against the oracle: summation order only,
    ~sqrt(19200) roundings of terms some ten times the field, and the oracle's
    own: 1e-11 as the parity tests of this rule."""
    th = np.linspace(0, np.pi, panels + 1)
    prof = np.stack([np.sin(th), np.cos(th)], -1) * 1e-6
    prof[0, 0] = prof[-1, 0] = 0.0
    sig = 3e7 * np.cos(th)
    tab = BemTables(prof, sig, n_subdiv)
    rng = np.random.default_rng(panels)
    d, ang, ph = 10 ** rng.uniform(-2, 1, 9600), rng.uniform(0.01, np.pi, 9600), rng.uniform(0, 6.28, 9600)
    r = 1e-6 * (1 + d)
    pts = np.stack([r * np.sin(ang) * np.cos(ph), r * np.sin(ang) * np.sin(ph), r * np.cos(ang)], -1)
    ref = ob.field(pts[:40], prof, sig, n_subdiv)
    for n in (1, 2, 7, 40, 151, 1200, 9600):
        got = engine.bem_field(tab, pts[:n]).cpu().numpy()[:40]
        m = len(got)
        assert (np.abs(got - ref[:m]).max(axis=-1) / np.linalg.norm(ref[:m], axis=-1)).max() < 1e-11


def _geometry(kind):
    g = load_golden(dict(post="trace_post", well="trace_well")[kind])
    spec = dict(kind=kind + "_bem", E_gun=float(g["E_gun"]), R=float(g["R"]), profile=g["profile"], sigma=g["sigma"],
                n_subdiv=int(g["n_subdiv"]), z_handoff=float(g["z_handoff"]), kill_z_below=0.0)
    spec.update(dict(L=float(g["L"]), z0=float(g["z0"])) if kind == "post" else dict(H=float(g["H"])))
    return gu.device_geometry(spec)


@pytest.mark.parametrize("rule", ["reference", "adaptive"])
@pytest.mark.parametrize("kind", ["post", "well"])
def test_stage_of_ragged_groups_is_its_groups_alone(kind, rule):
    """Groups of 1, 2, 31, 33 and 256 in one call, with inactive particles,
    particles inside the conductor and above the handoff, against each group's
    own call (other shares a point: 1e-12 of each acceleration), and through
    an offset table that starts at the second group with n_particles left 0."""
    geo = _geometry(kind)
    sizes = [1, 2, 31, 33, 256]
    n = sum(sizes)
    rng = np.random.default_rng(4)
    R = geo.R
    top = geo.L if kind == "post" else 0.0
    pos = np.stack([rng.uniform(-R, R, n), rng.uniform(-R, R, n), top + R * 10 ** rng.uniform(-3, 0.5, n)], -1)
    pos[::7, 2] = -2.0 * R if kind == "well" else 0.5 * top       # inside the conductor (mostly)
    pos[::11, 2] = 1.1 * geo.z_handoff
    act = (rng.random(n) < 0.7).astype(np.uint8)
    q, m = np.full(n, gu.Q_E), np.full(n, gu.M_E)
    whole = engine.accel(geo, pos, act, q, m, sizes, gu.CM, 1e-12, far_rule=rule).cpu().numpy()
    assert np.all(whole[act == 0] == 0.0)
    off = np.concatenate([[0], np.cumsum(sizes)])
    for a, b in zip(off[:-1], off[1:]):
        one = engine.accel(geo, pos[a:b], act[a:b], q[a:b], m[a:b], [b - a], gu.CM, 1e-12, far_rule=rule).cpu().numpy()
        np.testing.assert_allclose(whole[a:b], one, rtol=0, atol=1e-12 * np.linalg.norm(one, axis=-1).max())
    t = lambda v, d=torch.float64: torch.as_tensor(np.ascontiguousarray(v), dtype=d, device="cuda")
    x, y, z, tq, tm = t(pos[:, 0]), t(pos[:, 1]), t(pos[:, 2]), t(q), t(m)
    ta, to = t(act, torch.uint8), t(off, torch.int64)
    out = torch.full((3, n), 7.0, dtype=torch.float64, device="cuda")
    a = _lib.SptAccelArgs()
    a.n_groups, a.max_group_size = len(sizes) - 1, 256
    a.group_offset = to.data_ptr() + 8
    a.x, a.y, a.z, a.active, a.charge, a.mass = (v.data_ptr() for v in (x, y, z, ta, tq, tm))
    a.charge_to_mass, a.coulomb_constant, a.plummer_radius = gu.CM, engine.COULOMB_CONSTANT, 1e-12
    a.ax, a.ay, a.az = (out[k].data_ptr() for k in range(3))
    view, s = geo.bem_tables("cuda").view(rule), geo.to_struct()
    _lib.check(_lib.lib().spt_accel(ctypes.byref(a), ctypes.byref(s), ctypes.byref(view),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "spt_accel")
    got = out.T.cpu().numpy()
    np.testing.assert_array_equal(got[:1], 7.0)
    np.testing.assert_allclose(got[1:], whole[1:], rtol=0, atol=1e-12 * np.linalg.norm(whole, axis=-1).max())
    # in place: the accelerations over the positions
    a.n_groups, a.n_particles, a.group_offset = len(sizes), n, to.data_ptr()
    a.ax, a.ay, a.az = a.x, a.y, a.z
    _lib.check(_lib.lib().spt_accel(ctypes.byref(a), ctypes.byref(s), ctypes.byref(view),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "spt_accel")
    got = torch.stack([x, y, z], -1).cpu().numpy()
    np.testing.assert_allclose(got, whole, rtol=0, atol=1e-12 * np.linalg.norm(whole, axis=-1).max())


def test_on_surface_offset_around_its_threshold():
    """Points 0 to a few 1e-8 panel lengths from a panel, both sides (the
    offset acts below 1e-9, the scan that skips it from 1e-8), with the run
    bounds and without (every segment scanned): the same bits."""
    g = load_golden("sigma_c1")
    prof = g["profile"]
    tab = BemTables(prof, g["sigma"], 8)
    rows = []
    for k in (3, 60, 99, 100, 500):
        t = prof[k + 1] - prof[k]
        L = np.hypot(*t)
        nrm = np.array([-t[1], t[0]]) / L
        for f in (0.0, 0.3e-9, 0.999e-9, 1.001e-9, 3e-9, 0.99e-8, 1.01e-8, 5e-8, 1e-3, 0.5):
            for u in (0.0, 0.4, 1.0):
                p = prof[k] + u * t + f * L * nrm
                rows += [[p[0], 0.0, p[1]], [0.6 * p[0], 0.8 * p[0], p[1]]]
    pts = np.array(rows)
    x, y, z = (torch.as_tensor(np.ascontiguousarray(pts[:, k]), device="cuda") for k in range(3))
    out = []
    for bounds in (True, False):
        view = tab.view("reference", bounds=bounds)
        e = [torch.empty_like(x) for _ in range(3)]
        _lib.check(_lib.lib().spt_bem_field(x.data_ptr(), y.data_ptr(), z.data_ptr(), len(pts), ctypes.byref(view), 0,
                                            e[0].data_ptr(), e[1].data_ptr(), e[2].data_ptr(),
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "spt_bem_field")
        out.append(torch.stack(e, -1).cpu().numpy())
    assert np.isfinite(out[0]).all()
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("rule", ["reference", "adaptive"])
@pytest.mark.parametrize("kind", ["post", "well"])
def test_stage_reads_no_field_that_was_not_written(kind, rule):
    """Outputs full of NaN on entry, particles on the edge of the valid region
    to the last bits, n_particles below the groups' total (it only sizes the
    launch): every acceleration is finite, and that of the one-launch form to
    1e-12 of the largest, edge points aside (there the two may differ in what
    they take for vacuum)."""
    geo = _geometry(kind)
    rng = np.random.default_rng(5)
    n, R = 512, geo.R
    top = geo.L if kind == "post" else 0.0
    ph = rng.uniform(0, 6.28, n)
    edge = np.arange(n) < n // 2
    rho = np.where(edge, R * (1 - 1e-6), R * rng.uniform(0.1, 0.9, n))
    pos = np.stack([rho * np.cos(ph), rho * np.sin(ph), np.full(n, top)], -1)
    pos[edge, 2] -= 0.5 * (geo.L if kind == "post" else geo.H)  # the post's and the well's wall
    pos[~edge, 2] += R * 10 ** rng.uniform(0.1, 0.5, (~edge).sum())
    pos[edge, 0] *= 1 + rng.integers(-3, 4, edge.sum()) * 2.0**-53
    t = lambda v, d=torch.float64: torch.as_tensor(np.ascontiguousarray(v), dtype=d, device="cuda")
    act, q, m, off = t(np.ones(n), torch.uint8), t(np.full(n, gu.Q_E)), t(np.full(n, gu.M_E)), t([0, 200, 300, n], torch.int64)
    view, s = geo.bem_tables("cuda").view(rule), geo.to_struct()

    def stage(n_particles, in_place=False):
        x = t(pos.T.copy())
        out = x if in_place else torch.full((3, n), float("nan"), dtype=torch.float64, device="cuda")
        a = _lib.SptAccelArgs()
        a.n_groups, a.max_group_size, a.n_particles, a.group_offset = 3, 256, n_particles, off.data_ptr()
        a.x, a.y, a.z = (x[k].data_ptr() for k in range(3))
        a.active, a.charge, a.mass = act.data_ptr(), q.data_ptr(), m.data_ptr()
        a.charge_to_mass, a.coulomb_constant, a.plummer_radius = gu.CM, engine.COULOMB_CONSTANT, 1e-12
        a.ax, a.ay, a.az = (out[k].data_ptr() for k in range(3))
        _lib.check(_lib.lib().spt_accel(ctypes.byref(a), ctypes.byref(s), ctypes.byref(view),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "spt_accel")
        return out.T.cpu().numpy()

    one = stage(n, in_place=True)
    scale = np.linalg.norm(one[~edge], axis=-1).max()
    for n_particles in (n, 0, 1, 100):
        got = stage(n_particles)
        assert np.isfinite(got).all()
        np.testing.assert_allclose(got[~edge], one[~edge], rtol=0, atol=1e-12 * scale)


def test_stage_takes_wider_and_deeper_rows():
    """Positions as rows of six (positions and velocities) and as [N, 3, 1]:
    the same accelerations, the latter in its shape."""
    geo = _geometry("post")
    rng = np.random.default_rng(6)
    pos = np.stack([*rng.normal(0, geo.R, (2, 5)), geo.L + geo.R * rng.uniform(1.1, 2, 5)], -1)
    run = lambda p: engine.accel(geo, p, np.ones(5, np.uint8), np.full(5, gu.Q_E), np.full(5, gu.M_E), [2, 3], gu.CM, 1e-12)
    want = run(pos)
    assert torch.equal(run(np.concatenate([pos, pos], 1)), want)
    assert torch.equal(run(pos[:, :, None]), want[:, None, :])


def test_threads_with_calls_of_different_sizes():
    """Two threads on their own streams, one asking for a few points at a time
    and one for many (different shared memory, clusters and splits), by both
    rules: every call succeeds with the values it has alone."""
    import threading

    geo = _geometry("post")
    tab = geo.bem_tables("cuda")
    assert tab.field_map() is not None  # with its cells from the start: their coming changes the last digits
    rng = np.random.default_rng(8)
    d, th = 10 ** rng.uniform(-3, 0.5, 6000), rng.uniform(0, 1.0, 6000)
    r = geo.R * (1 + d)
    pts = torch.as_tensor(np.stack([r * np.sin(th), np.zeros_like(r), geo.L + r * np.cos(th)], -1), device="cuda")
    want = {(n, rule): engine.bem_field(tab, pts[:n], far_rule=rule) for n in (1, 5, 6000) for rule in ("reference", "adaptive")}
    torch.cuda.synchronize()
    failed = []

    def work(sizes):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for k in range(600):
                    n, rule = sizes[k % len(sizes)], ("adaptive", "adaptive", "reference")[k % 3]
                    got = engine.bem_field(tab, pts[:n], far_rule=rule)
                    if k % 50 == 0 and not torch.equal(got, want[n, rule]):
                        failed.append((n, rule))
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(s,)) for s in ((1, 5), (6000,), (5, 6000))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[:3]
