"""spt_image_force where its split of a group over the CTA can go wrong: groups
of 1, 2, 3, 4 (8, 4, 2, 2 warps a particle), 5, 8, 9 and 33 (one), each alone
and all in one ragged batch, solution and geometry level, against the oracle
(1e-11 of the largest force, the bound of the entry point's parity tests)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from bem_b200 import geometry as bg  # noqa: E402
from bem_b200.constants import ELEMENTARY_CHARGE  # noqa: E402
from bem_b200.image_charge import ImageChargeSolution  # noqa: E402
from oracle import image_charge as oic  # noqa: E402

SIZES = (1, 2, 3, 4, 5, 8, 9, 33)


@pytest.mark.parametrize("n_max", [0, 1, 16, 20])
@pytest.mark.parametrize("level", ["solution", "geometry"])
def test_groups_of_every_split_match_one_by_one(level, n_max):
    geo = bg.HemisphericalTipBEMGeometry(-1e7, 50e-9, z0=3e-9, image_n_max=n_max, sigma=np.zeros(40))
    sol = geo.image_solution("cuda")
    rng = np.random.default_rng(n_max)
    n = sum(SIZES)
    th, ph = rng.uniform(0, 1.0, n), rng.uniform(0, 6.28, n)
    r = 50e-9 + 10 ** rng.uniform(-9.5, -6.5, n)
    pos = np.stack([r * np.sin(th) * np.cos(ph), r * np.sin(th) * np.sin(ph), r * np.cos(th)], -1)
    act = (rng.random(n) < 0.85).astype(np.uint8)
    t = lambda v, d=torch.float64: torch.as_tensor(np.ascontiguousarray(v), dtype=d, device="cuda")
    q = t(np.full(n, -ELEMENTARY_CHARGE))
    off = np.concatenate([[0], np.cumsum(SIZES)])
    g = geo.to_struct() if level == "geometry" else None
    whole = sol.force(t(pos), q, t(act, torch.uint8), t(off, torch.int64), max(SIZES), geometry=g).cpu().numpy()
    assert np.all(whole[act == 0] == 0.0)
    for a, b in zip(off[:-1], off[1:]):
        one = sol.force(t(pos[a:b]), q[a:b].contiguous(), t(act[a:b], torch.uint8), t([0, b - a], torch.int64),
                        int(b - a), geometry=g).cpu().numpy()
        # the same group, its right-hand sides perhaps in other partial sums
        np.testing.assert_allclose(whole[a:b], one, rtol=0, atol=1e-11 * max(np.abs(one).max(), 1e-300))
        ref = _oracle(geo, sol, pos[a:b], act[a:b], level)
        np.testing.assert_allclose(whole[a:b], ref, rtol=0, atol=1e-11 * max(np.abs(ref).max(), 1e-300))


def _oracle(geo, sol, pos, act, level):
    ref = oic.ImageSolution(sol.profile, sol.n_max, A=sol.A.cpu().numpy())
    p, q, a = pos[None], np.full((1, len(pos)), -ELEMENTARY_CHARGE), act[None].astype(bool)
    if level == "solution":
        return ref.image_force(p, q, a, sol.d_lo, sol.d_hi)[0]
    return np.where(a[0][:, None], oic.geometry_image_force(ref, p, q, a, geo.z0, geo.R, z_handoff=geo.z_handoff)[0], 0.0)


@pytest.mark.parametrize("level", ["solution", "geometry"])
def test_empty_groups_leave_the_others_as_they_are(level):
    """Empty groups first, last, between others and alone: the forces are, bit
    for bit, those of the batch without them (a group's sums depend on its own
    particles and the launch's largest size only), and nothing else is written."""
    geo = bg.HemisphericalTipBEMGeometry(-1e7, 50e-9, z0=3e-9, image_n_max=16, sigma=np.zeros(40))
    sol = geo.image_solution("cuda")
    rng = np.random.default_rng(7)
    sizes = [0, 0, 3, 0, 1, 0, 0, 9, 0]
    n = sum(sizes)
    th, ph = rng.uniform(0, 1.0, n), rng.uniform(0, 6.28, n)
    r = 50e-9 + 10 ** rng.uniform(-9.5, -6.5, n)
    t = lambda v, d=torch.float64: torch.as_tensor(np.ascontiguousarray(v), dtype=d, device="cuda")
    pos = t(np.stack([r * np.sin(th) * np.cos(ph), r * np.sin(th) * np.sin(ph), r * np.cos(th)], -1))
    q, act = t(np.full(n, -ELEMENTARY_CHARGE)), t(np.ones(n), torch.uint8)
    g = geo.to_struct() if level == "geometry" else None
    off = lambda s: t(np.concatenate([[0], np.cumsum(s)]), torch.int64)
    full = sol.force(pos, q, act, off([s for s in sizes if s]), 9, geometry=g)
    out = torch.full((3, n), 7.0, dtype=torch.float64, device="cuda")
    assert torch.equal(sol.force(pos, q, act, off(sizes), 9, geometry=g, out=out), full)
    assert torch.isfinite(full).all()
    out.fill_(7.0)
    sol.force(pos, q, act, off([0, 0]), 9, geometry=g, out=out)
    assert (out == 7.0).all()


@pytest.mark.parametrize("n_max", [16, 20, 40])
def test_scratch_to_the_last_byte_of_shared_memory(n_max):
    """A profile and a max_group_size whose scratch leaves 8 to 200 bytes of a
    CTA's 227 KiB: the launch takes it, and two electrons' forces are those of
    a launch for groups of two (other partial sums of the right-hand sides:
    1e-11 of the largest force)."""
    P, E = next((P, E) for P in range(40, 65) for E in range(1, 513)
                if 8 <= 227 * 1024 - 8 * (13 * E + 2 * (n_max + 1) * (E + P * (1 + 256 // P))) <= 200)
    th = np.linspace(0, 0.5 * np.pi, P)
    prof = np.stack([47e-9 * np.sin(th), 47e-9 * np.cos(th)], -1)
    sol = ImageChargeSolution(prof, n_max, 0.5e-9, 5e-9)
    t = lambda v, d=torch.float64: torch.as_tensor(np.ascontiguousarray(v), dtype=d, device="cuda")
    pos = t([[10e-9, 5e-9, 60e-9], [-20e-9, 3e-9, 80e-9]])
    args = (pos, t([-ELEMENTARY_CHARGE] * 2), t([1, 1], torch.uint8), t([0, 2], torch.int64))
    want = sol.force(*args, 2)
    assert (sol.force(*args, E) - want).abs().max() <= 1e-11 * want.abs().max()
