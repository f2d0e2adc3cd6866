"""The experts' sorted order against a plain count."""
import pytest
import torch

from test_kernels_gpu import DEV, ops  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,padded", [(64, False), (128, True)])
@pytest.mark.parametrize("P,E,n", [(1, 1, 1), (70, 31, 31), (1000, 32, 33), (5000, 33, 33), (3000, 256, 300),
                                   (64, 3, 1)])
def test_the_sorted_order(ops, P, E, n, tile, padded):  # noqa: F811
    """Every pair has a place of its own among its expert's rows, every tile belongs to the expert whose
    rows it holds; outputs E and above have no place."""
    ids = torch.randint(0, n, (P, 1), generator=torch.Generator().manual_seed(P + E)).int().to(DEV)
    place = torch.full((P,), -7, dtype=torch.int32, device=DEV)
    counts = torch.bincount(ids.flatten().cpu().long(), minlength=E)[:E]
    if padded:
        tiles = ops.moe_tc_tiles(P, E)
        tile_expert = torch.full((tiles,), -7, dtype=torch.int32, device=DEV)
        used = torch.zeros(1, dtype=torch.int32, device=DEV)
        ops.moe_group_padded(ids, E, place, tile_expert, used)
        starts = torch.cumsum((counts + tile - 1) // tile * tile, 0)
        starts = torch.cat([torch.zeros(1, dtype=torch.long), starts])[:E]
    else:
        tiles = ops.moe_max_tiles(P, E)
        tile_expert = torch.full((tiles,), -7, dtype=torch.int32, device=DEV)
        row0, order = torch.zeros_like(tile_expert), torch.full((P,), -7, dtype=torch.int32, device=DEV)
        offsets = torch.zeros(E + 1, dtype=torch.int32, device=DEV)
        ops.moe_group(ids, E, offsets, place, order, tile_expert, row0)
        starts = torch.cat([torch.zeros(1, dtype=torch.long), torch.cumsum(counts, 0)])
        assert offsets.cpu().tolist() == starts.tolist()
        starts = starts[:E]
    flat, at = ids.flatten().cpu().long(), place.cpu().long()
    assert bool((at[flat >= E] == -1).all())
    for e in range(E):
        assert sorted(at[flat == e].tolist()) == list(range(int(starts[e]), int(starts[e] + counts[e])))
    n_tiles = (counts + tile - 1) // tile
    want = [e for e in range(E) for _ in range(int(n_tiles[e]))]
    assert tile_expert.cpu().tolist() == want + [-1] * (tiles - len(want))
    if padded:
        assert used.item() == len(want)
    else:
        assert row0.cpu().tolist()[:len(want)] == [int(starts[e]) + tile * i for e in range(E)
                                                   for i in range(int(n_tiles[e]))]
        kept = order.cpu().long()[:int(counts.sum())]
        assert at[kept].tolist() == list(range(int(counts.sum())))


def test_the_most_experts(ops):  # noqa: F811
    """4,095 experts: the order's counts, places and starts fill the 48 KB a launch has without asking."""
    E, P = 4095, 700
    ids = torch.randint(0, E, (P, 1), generator=torch.Generator().manual_seed(1)).int().to(DEV)
    place, used = torch.full((P,), -7, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    tile_expert = torch.full((ops.moe_tc_tiles(P, E),), -7, dtype=torch.int32, device=DEV)
    ops.moe_group_padded(ids, E, place, tile_expert, used)
    want = sorted(set(ids.flatten().tolist()))           # (700 pairs: a tile of 128 rows each)
    assert used.item() == len(want) and tile_expert.tolist()[:len(want)] == want
    assert bool((tile_expert[len(want):] == -1).all())
    assert all(want[p // 128] == e for p, e in zip(place.tolist(), ids.flatten().tolist()))
