"""Host side of the field and stage calls (bem_b200/engine.py), on the CPU."""

import pytest

torch = pytest.importorskip("torch")

from bem_b200 import engine  # noqa: E402


@pytest.mark.parametrize("shape", [(4, 3), (4, 6), (4, 3, 1), (1, 3), (0, 3), (3, 5, 2)])
@pytest.mark.parametrize("strided", [False, True])
def test_columns_are_the_first_three(shape, strided):
    """Rows of three or more columns, a trailing dimension, no row at all, and
    strided rows: each column contiguous, as taken one by one."""
    p = torch.arange(2 * torch.Size(shape).numel(), dtype=torch.float64).reshape(2 * shape[0], *shape[1:])
    p = p[::2] if strided else p[: shape[0]]
    cols = engine._columns(p)
    assert len(cols) == 3
    for k, c in enumerate(cols):
        assert c.is_contiguous() and torch.equal(c, p[:, k])


@pytest.mark.parametrize("shape", [(4, 2), (4,)])
def test_fewer_than_three_columns_are_refused(shape):
    with pytest.raises((IndexError, ValueError)):
        x, y, z = engine._columns(torch.zeros(shape))
