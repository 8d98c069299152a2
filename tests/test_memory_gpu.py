"""Device memory that scenes keep: buffers that stay where they are between builds."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import wide_probe  # noqa: E402


@pytest.mark.parametrize("large,more", [(1000, 10), (1000, 1000), (1000, 5000)])
def test_buffers_of_one_allocation_stay_in_place(large, more):
    """A builder that builds triangles and boxes by turns allocates in the first turn alone."""
    assert wide_probe.lib().probe_reserve_moves(large, more, 4) == 0
