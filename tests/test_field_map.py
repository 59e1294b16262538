"""Lookup tables of the field map (bem_b200/field_map.py): every point of a
cell finds it, points outside every cell find none (CPU; the walk below is
the device's map_find)."""

import numpy as np
import pytest

from bem_b200 import field_map as fm


def _find(tab, u, v):
    R, B = fm._lib.MAP_ROOT_BITS, fm._lib.MAP_BITS
    iu, iv, sh, low = int(u * 2**30), int(v * 2**30), 30 - R, (1 << B) - 1
    e = tab[((iv >> sh) << R) + (iu >> sh)]
    while e < -1 and sh >= B:
        sh -= B
        e = tab[(1 << 2 * R) + ((-2 - e) << 2 * B) + (((iv >> sh) & low) << B) + ((iu >> sh) & low)]
    return e if e >= -1 else -1


@pytest.mark.parametrize("depth", [1, 2, 3, 7, 8, 9, 13, 14, 18])
def test_link_tables_find_every_cell(depth):
    rng = np.random.default_rng(depth)
    i = j = np.zeros(1, dtype=np.int64)
    divided, cells = {}, []
    for level in range(depth + 1):
        split = np.ones(len(i), bool) if level == 0 else rng.random(len(i)) < (0.55 if level < depth else 0.0)
        for a, b in zip(i[~split], j[~split]):
            if rng.random() < 0.8:  # the rest: squares without a cell
                cells.append((level, a, b))
        i, j = i[split][:40], j[split][:40]
        if len(i) == 0:
            break
        divided[level] = (i, j)
        i, j = (np.concatenate([2 * i + a for a in (0, 1) for _ in (0, 1)]),
                np.concatenate([2 * j + b for _ in (0, 1) for b in (0, 1)]))
    level, ci, cj = (np.array(c, dtype=np.int64) for c in zip(*cells))
    tab = fm.link_tables((level, ci, cj, np.arange(len(cells))), divided)
    for k, (l, a, b) in enumerate(cells):
        for fu, fv in ((0.0, 0.0), (0.5, 0.5), (1 - 1e-4, 0.0), (0.3, 1 - 1e-4)):
            assert _find(tab, (a + fu) / 2.0**l, (b + fv) / 2.0**l) == k
    taken = {}
    for l, a, b in cells:
        taken.setdefault(l, set()).add((a, b))
    for u, v in rng.random((200, 2)):
        hit = any((int(u * 2**l), int(v * 2**l)) in s for l, s in taken.items())
        assert (_find(tab, u, v) >= 0) == hit


def test_power_coefficients_reproduce_the_samples():
    """Nodes -> Chebyshev -> powers, evaluated back at the nodes: the products
    of 12-term rows leave a few rounding errors of the largest value."""
    rng = np.random.default_rng(0)
    x = fm.NODES
    f = np.exp(x[:, None] * 0.7) * np.cos(x[None, :] + 0.2) + rng.normal(size=(fm.N, fm.N)) * 1e-15
    c = fm.DCT @ f @ fm.DCT.T
    p = fm.MONO.T @ c @ fm.MONO
    V = x[:, None] ** np.arange(fm.N)
    assert np.abs(V @ p @ V.T - f).max() < 1e-13


@pytest.fixture
def tables(monkeypatch):
    """The field map's bookkeeping of a 100-panel BemTables, sampling replaced
    by a count of the calls."""
    import types

    import torch

    from bem_b200.tables import BemTables

    t = BemTables.__new__(BemTables)
    t.clusters, t._map_worth = object(), fm.worth(np.zeros((101, 2)))
    t.seg = types.SimpleNamespace(device=torch.device("cuda"))
    t._map = t._bare = None
    t._map_points, t._map_lock = 0, __import__("threading").Lock()
    t.calls, t.capturing, t.memory = [], False, True

    def build(tab):
        t.calls.append("cells")
        if not t.memory:
            raise torch.cuda.OutOfMemoryError("no memory")
        return ("cells", 1)

    monkeypatch.setattr(fm, "build", build)
    monkeypatch.setattr(fm, "bare", lambda tab: t.calls.append("bare") or ("bare", 2))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: t.capturing)
    return t


def test_cells_are_sampled_when_the_points_asked_for_pay(tables):
    n = tables._map_worth
    assert n == fm.WORTH + 100 * fm.WORTH_PER_PANEL
    for k in (1, 33, n // 2, n - n // 2 - 35):
        assert tables.field_map(points=k)[0] == "bare"
    assert tables.calls == ["bare"]
    assert tables.field_map(points=1)[0] == "cells"
    assert tables.field_map(points=1)[0] == "cells" and tables.calls == ["bare", "cells"]


def test_a_kept_view_samples_the_cells_at_once(tables):
    assert tables.field_map()[0] == "cells" and tables.calls == ["cells"]


def test_nothing_is_built_under_capture(tables):
    tables.capturing = True
    assert tables.field_map() is None and tables.field_map(points=10**9) is None and tables.calls == []
    tables.capturing = False
    assert tables.field_map(points=1)[0] == "bare"
    tables.capturing = True
    assert tables.field_map(points=10**9)[0] == "bare" and tables.calls == ["bare"]


def test_lack_of_memory_is_tried_again_after_as_many_points(tables):
    n = tables._map_worth
    tables.memory = False
    assert tables.field_map(points=n)[0] == "bare" and tables.calls == ["cells", "bare"]
    assert tables.field_map(points=n - 1)[0] == "bare" and tables.calls == ["cells", "bare"]
    tables.memory = True
    assert tables.field_map(points=1)[0] == "cells"
