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


@pytest.mark.parametrize("s", [1, 128, 129, 4096, 32768])
@pytest.mark.parametrize("groups,per_group", [(1, 1), (1, 8), (8, 4), (2, 6), (1, 3), (16, 1)])
def test_head_split_divides_the_group(s, groups, per_group):
    """Query heads of a group over CTAs of the attention backward: equal shares, a power of two, none where every SM
    has more to do than the longest CTA."""
    from fluidmoe_b200.ops.flash import _head_split

    split = _head_split(s, 1, groups, per_group)
    assert split & (split - 1) == 0 and per_group % split == 0
    tiles = -(-s // 128)
    if tiles * per_group * 148 * 2 <= 3 * groups * per_group * tiles * (tiles + 1) // 2:
        assert split == 1


@pytest.mark.parametrize("T", [1, 500, 1535, 1536, 8192])
@pytest.mark.parametrize("H,E", [(1024, 8), (4096, 8), (2048, 64), (8, 1)])
def test_router_gradient_off_16_bytes_keeps_its_shares(T, H, E):
    """Rows that the tensor core does not take: two CTAs an SM, of at least 32 tokens each, whatever their number."""
    tiles = -(-H // 1024) * -(-E // (8 if E <= 8 else 16))
    assert _C.router_wgrad_splits(T, H, E, 0) == max(1, min(2 * 148 // tiles, -(-T // 32)))
    if T < 1536:
        assert _C.router_wgrad_splits(T, H, E, 1) == _C.router_wgrad_splits(T, H, E, 0)
