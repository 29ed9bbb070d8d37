"""The one-launch Morton sort, the pyramid of the sorted rows and the maps of all its levels against the step-by-step
functions they stand in for."""
import numpy as np
import pytest
import torch

from warpconvnet_b200 import IntCoords, Voxels, generate_kernel_map, morton_code
from warpconvnet_b200._native import check_device_status
from warpconvnet_b200.geometry.coords.ops.stride import unique_strided_rows
from warpconvnet_b200.geometry.coords.search.level_maps import LevelMaps, PyramidBuild

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _scene(n, sizes, span, seed, low=-40):
    g = torch.Generator().manual_seed(seed)
    coords = torch.randint(0, span, (n, 3), generator=g, dtype=torch.int64) + low
    offsets = torch.tensor([0] + sizes).cumsum(0)
    assert int(offsets[-1]) == n
    return coords.int().to(DEV), offsets


@pytest.mark.parametrize("n,sizes,span", [(1, [1], 5), (31, [31], 9), (2049, [2049], 64), (30000, [7000, 0, 22999, 1], 200),
                                          (400000, [150000, 250000], 3000), (5000, [2000, 3000], 1 << 22), (3000, [10] * 255 + [450], 30),
                                          (4000, [16] * 250, 1 << 21)])
@pytest.mark.parametrize("channels,dtype", [(3, torch.float16), (4, torch.float32), (40, torch.float16)])
def test_sort_equals_stable_argsort(n, sizes, span, channels, dtype):
    coords, offsets = _scene(n, sizes, span, n)
    feats = torch.randn(n, channels, generator=torch.Generator().manual_seed(1)).to(dtype).to(DEV)
    got = Voxels(coords, feats, offsets=offsets).sort()
    origin = torch.div(coords.min(0).values, 16, rounding_mode="floor") * 16
    codes = morton_code(coords, origin=origin.int())
    batch = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).to(DEV)
    by_code = torch.argsort(codes, stable=True)
    perm = by_code[torch.argsort(batch[by_code], stable=True)]
    assert torch.equal(got.extra_attributes["perm"], perm)
    assert torch.equal(got.extra_attributes["code"], codes)
    assert torch.equal(got.coordinate_tensor, coords[perm])
    assert torch.equal(got.batch_indexed_coordinates[:, 0].long(), batch[perm])
    assert torch.equal(got.feature_tensor, feats[perm])
    assert torch.equal(got.batched_coordinates.morton_origin, origin.int())
    check_device_status(DEV)


def _distinct(n, batches, span, seed):
    rng = np.random.default_rng(seed)
    parts = []
    for b in range(batches):
        cells = rng.choice(span ** 3, n, replace=False)
        parts.append(np.stack(np.unravel_index(cells, (span,) * 3), 1) - 13)
    return torch.from_numpy(np.concatenate(parts).astype(np.int32)).to(DEV), torch.arange(batches + 1) * n


@pytest.mark.parametrize("n,batches,span", [(1, 1, 4), (40, 2, 6), (900, 3, 20), (4097, 1, 40), (90000, 1, 90), (30000, 3, 60),
                                             (131073, 2, 120)])
def test_pyramid_and_level_maps_equal_level_by_level(n, batches, span):
    """Row counts below, at and above the tile order's windows, levels of a single row, several scenes."""
    coords, offsets = _distinct(n, batches, span, n)
    v = Voxels(coords, torch.zeros(len(coords), 1, device=DEV), offsets=offsets).sort()
    maps = LevelMaps(v.batched_coordinates)
    levels = maps.finish()
    assert levels is not None
    rows, offs = v.batch_indexed_coordinates, v.offsets
    for l in range(5):
        if l:
            rows, _, _, offs = unique_strided_rows(maps.rows[l - 1].contiguous(), (2, 2, 2), in_offsets=offs)
            assert torch.equal(maps.rows[l], rows) and torch.equal(levels[l - 1].offsets, offs)
            down = generate_kernel_map(maps.rows[l - 1].contiguous(), rows, (2, 2, 2), (2, 2, 2))
            assert torch.equal(maps.child[l - 1], down.neighbor_table(len(rows)))
        want = generate_kernel_map(rows, rows, (1, 1, 1), (3, 3, 3)).neighbor_table(len(rows))
        order = maps.order[l]
        if order is None:
            assert torch.equal(maps.nbr[l], want)
        else:
            assert torch.equal(torch.sort(order).values, torch.arange(len(rows), device=DEV, dtype=torch.int32))
            assert torch.equal(maps.nbr[l], want[:, order.long()])
    km = v.batched_coordinates._shared[("kmap", (3, 3, 3), (1, 1, 1))]
    assert torch.equal(km.neighbor_table(len(v)), generate_kernel_map(v.batch_indexed_coordinates.contiguous(), v.batch_indexed_coordinates.contiguous(),
                                                                      (1, 1, 1), (3, 3, 3)).neighbor_table(len(v)))
    check_device_status(DEV)


def test_repeated_voxels_and_huge_extents_are_not_usable():
    coords, offsets = _scene(3000, [3000], 8, 3)  # 512 cells: many repeats
    v = Voxels(coords, torch.zeros(3000, 1, device=DEV), offsets=offsets).sort()
    assert LevelMaps(v.batched_coordinates).finish() is None
    assert v.batched_coordinates._shared["morton_info"] is None
    coords, offsets = _scene(50, [50], 1 << 23, 4)
    v = Voxels(coords, torch.zeros(50, 1, device=DEV), offsets=offsets).sort()
    assert PyramidBuild(v.batched_coordinates).finish() is None
    check_device_status(DEV)


def test_large_pyramids_keep_no_more_than_their_rows(monkeypatch):
    from warpconvnet_b200.geometry.coords.search import level_maps
    from warpconvnet_b200.nn.functional.sparse_conv import strided_coordinates
    g = torch.Generator(device="cuda").manual_seed(0)
    n = 300000
    cell = torch.randperm(128 ** 3, generator=g, device="cuda")[:n].int()
    xyz = torch.stack([cell // (128 * 128), cell // 128 % 128, cell % 128], dim=1).int().contiguous()
    tables = []
    for limit in (n + 1, n):
        monkeypatch.setattr(level_maps, "TRIMMED_ROWS", limit)
        ic = Voxels(xyz, torch.zeros(n, 1, device="cuda"), offsets=torch.tensor([0, n])).sort().batched_coordinates
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        level, rows = ic, 0
        for _ in range(4):
            level = strided_coordinates(level, (2, 2, 2))
            rows += len(level)
        kept = torch.cuda.memory_allocated() - before
        assert kept > 80 * n if limit > n else kept < 20 * rows + (64 << 10)
        maps, _ = ic._shared["level_maps"]
        tables.append([maps.kmap(l, w).neighbor_table(maps.n[l if w == 3 else l + 1]).clone() for l in range(4) for w in (3, 2)])
    assert all(torch.equal(a, b) for a, b in zip(*tables))
    check_device_status(torch.device("cuda:0"))


def test_a_coordinate_set_keeps_its_own_tables_only():
    """The maps of a network's levels: the memory behind the tables of one coordinate set (neighbours and row order of its
    level, children of the next) is not that of another's."""
    coords, offsets = _scene(60000, [20000, 40000], 150, 5)
    key = torch.unique(torch.cat([torch.repeat_interleave(torch.arange(2), torch.tensor([20000, 40000]))[:, None], coords.cpu().long()], 1), dim=0)
    offsets = torch.tensor([0, int((key[:, 0] == 0).sum()), len(key)])
    v = Voxels(key[:, 1:].int().to(DEV), torch.zeros(len(key), 1, device=DEV), offsets=offsets).sort()
    maps = LevelMaps(v.batched_coordinates)
    assert maps.finish() is not None
    storages = []
    for l in range(1, 5):
        held = [maps.nbr[l]] + ([] if maps.order[l] is None else [maps.order[l]]) + ([maps.child[l]] if l < 4 else [])
        assert len({t.untyped_storage().data_ptr() for t in held}) == 1
        words = -(-maps.n[l] // 64) * 64, -(-maps.n[l + 1] // 64) * 64 if l < 4 else 0
        size = held[0].untyped_storage().nbytes()   # (beside the assertion, whose message would print the storage)
        assert size <= 4 * (28 * words[0] + 8 * words[1])
        storages.append(held[0].untyped_storage().data_ptr())
    storages += [maps.child[0].untyped_storage().data_ptr(), maps.nbr[0].untyped_storage().data_ptr()]
    assert len(set(storages)) == 6
    check_device_status(DEV)


def test_the_storages_of_large_pyramids_are_those_of_their_rows(monkeypatch):
    """What a pyramid keeps as the sum of the storages that are held (16 bytes of coordinates and 4 of first children a row):
    ``torch.cuda.memory_allocated`` also depends on which blocks the allocator has left."""
    from warpconvnet_b200.geometry.coords.search import level_maps
    from warpconvnet_b200.nn.functional.sparse_conv import strided_coordinates
    n = 300000
    cell = torch.randperm(128 ** 3, generator=torch.Generator().manual_seed(1))[:n].int()
    xyz = torch.stack([cell // (128 * 128), cell // 128 % 128, cell % 128], dim=1).contiguous().to(DEV)
    for limit in (n + 1, n):
        monkeypatch.setattr(level_maps, "TRIMMED_ROWS", limit)
        ic = Voxels(xyz, torch.zeros(n, 1, device=DEV), offsets=torch.tensor([0, n])).sort().batched_coordinates
        level, rows, held = ic, 0, []
        for _ in range(4):
            level = strided_coordinates(level, (2, 2, 2))
            rows += len(level)
            held.append(level._shared["bcoords"])
        maps, _ = ic._shared["level_maps"]
        first = maps.build.first
        held += list(first) if isinstance(first, list) else [first]
        assert maps.build.out is None
        kept = sum({t.untyped_storage().data_ptr(): t.untyped_storage().nbytes() for t in held}.values())
        assert kept >= 80 * n if limit > n else kept <= 20 * rows
    check_device_status(DEV)
