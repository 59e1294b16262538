"""The far sums' ring kernel across its branches, through one-panel fields:
points at both sides of p = d2 / D = 1e-3 (where the close-ring routine takes
over) and of rho^2 = 1e-10 (a^2 + z^2) (the near-axis expansion), against the
same Gauss nodes summed with the entry point spt_ring_field (the AGM run to
convergence)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from bem_b200 import engine  # noqa: E402
from bem_b200.tables import BemTables, far_nodes  # noqa: E402


@pytest.mark.parametrize("scale", [1e-12, 1e-6, 1.0, 1e6])
def test_ring_branches_match_converged_agm(scale):
    """One panel of length 0.02 a at radius a: relative to |E|, 16 roundings
    of the sum's 32 terms at each of the few operations that carry them, and
    for E_rho those of K - (...) E / d2, which cancels as a / rho towards
    the axis."""
    prof = np.array([[1.0, -0.01], [1.0, 0.01]]) * scale
    sig = np.array([1.0, 1.5]) / scale
    tab = BemTables(prof, sig, 8)
    # distances from the ring around p = 1e-3 (d = 0.0632 a), each side, and far away; the panel's own band excluded
    d = np.concatenate([0.0633 * (1 + np.array([-0.3, -1e-3, -1e-9, 1e-9, 1e-3, 0.3])), [0.1, 0.5, 1.5, 10.0, 1e3]])
    ang = np.linspace(0.1, 6.2, 13)
    dd, aa = (v.ravel() for v in np.meshgrid(d, ang))
    rho, z = np.abs(1.0 + dd * np.cos(aa)), dd * np.sin(aa)
    x = np.concatenate([1e-5 * np.array([0.5, 1 - 1e-6, 1 + 1e-6, 2.0]) * np.sqrt(1 + 0.3**2), [1e-3, 0.0]])
    rho, z = np.concatenate([rho, x]) * scale, np.concatenate([z, np.full(len(x), 0.3)]) * scale
    pts = np.stack([rho, np.zeros_like(rho), z], -1)
    got = engine.bem_field(tab, pts).cpu().numpy()
    rq, zq, aq, sq = far_nodes(prof, sig, 8)
    r, zz, a = (np.array(np.broadcast_to(v, (len(rho), len(rq)))).ravel() for v in (rho[:, None], z[:, None] - zq, rq))
    er, ez = (v.cpu().numpy().reshape(len(rho), -1) @ (aq * sq) for v in engine.ring_field(r, zz, a))
    norm = np.hypot(er, ez)
    eps = np.finfo(float).eps
    assert (np.abs(got[:, 2] - ez) / norm).max() < 16 * eps
    cancel = np.where(rho > 0, np.sqrt(scale**2 + z**2) / np.maximum(rho, 1e-300), 0.0) ** 2
    assert np.all(np.abs(got[:, 0] - er) / norm < 16 * eps * (1 + cancel))
    np.testing.assert_array_equal(got[:, 1], 0.0)
