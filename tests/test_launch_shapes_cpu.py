"""Launch shapes that the native library computes on the host (no GPU needed)."""
import pytest

_C = pytest.importorskip("fluidmoe_b200._C")


@pytest.mark.parametrize("T", [1, 64, 1000, 4096, 18_944, 100_000])
@pytest.mark.parametrize("H", [8, 512, 4096])
def test_a_waiting_unpermute_leaves_room(T, H):
    """CTAs that poll for peers' rows: one for eight tokens, or one per SM, at most."""
    pieces = T * (H // 8)
    free, waiting = _C.unpermute_grid(T, H, 0), _C.unpermute_grid(T, H, 1)
    assert free == min(max(1, -(-pieces // 256)), 148 * 16)
    assert waiting == min(free, max(148, min(-(-T // 8), 148 * 16)))
