"""Coordinate pyramid and kernel maps of a natively sorted ``Voxels``, all levels at once.

An addition to the reference's structures, for coordinate sets that ``Voxels.sort`` has put in Morton order: the
coarser levels come from comparing neighbouring rows (:func:`morton_pyramid`), and the 3x3x3 maps in tile order with
the stride-2 child tables of a whole U-Net from one launch per stage (:class:`LevelMaps`).  The row counts are written
by the kernel into pinned memory; :meth:`PyramidBuild.finish` is the one point where the host waits, and it waits for
the small pyramid kernels only: whatever was enqueued behind them keeps the device busy meanwhile.
"""
from __future__ import annotations

import ctypes
from typing import List, Optional

import torch
from torch import Tensor

from ...._native import Level, check, device_status, lib, pinned_result, ptr, query_bytes, raise_for_status, stream_ptr
from ..integer import IntCoords
from .search_results import IntSearchResult

PYRAMID_LEVELS = 4
# The levels are written into buffers for as many rows as the finest one (their sizes are not known before): 80 bytes per
# fine row, of which a room's levels use about 7.  From this many rows on what is there is copied out; below it the eight
# copies are not worth the at most 168 MB that stay with the coordinates.
TRIMMED_ROWS = 1 << 21


class PyramidBuild:
    """The four stride-2 levels below a sorted coordinate set, enqueued on the current stream."""

    def __init__(self, ic: IntCoords):
        info = ic._shared["morton_info"]
        rows = ic._shared["bcoords"]
        dev = rows.device
        n = rows.shape[0]
        offsets = ic.offsets if ic.offsets.dtype == torch.int64 and ic.offsets.is_contiguous() else ic.offsets.to(torch.int64).contiguous()
        self.ic, self.rows, self.info, self.n, self.device = ic, rows, info, n, dev
        self.batches = len(offsets) - 1
        self.out = torch.empty((PYRAMID_LEVELS, n, 4), dtype=torch.int32, device=dev)
        self.first = torch.empty((PYRAMID_LEVELS, n), dtype=torch.int32, device=dev)
        self.counts = torch.empty(24, dtype=torch.int32, device=dev)
        ws = torch.empty(query_bytes("wcn_pyramid_workspace_bytes", n), dtype=torch.uint8, device=dev)

        def launch(host: Tensor) -> None:
            check(lib().wcn_pyramid(ptr(rows), n, ptr(info), ptr(offsets), self.batches, PYRAMID_LEVELS, ptr(self.out),
                                    ptr(self.first), ptr(self.counts), ptr(host), ptr(ws), ptr(device_status(dev)),
                                    stream_ptr(dev)), "wcn_pyramid")
        self.host, self._done = pinned_result(PYRAMID_LEVELS * (self.batches + 1) + 2, torch.int64, dev, launch)

    def finish(self) -> Optional[List[IntCoords]]:
        """Waits for the counts; the levels' coordinates, or None when the rows are not what the pyramid needs
        (repeated voxels, an extent of 2^21 or more)."""
        self._done.synchronize()
        host = self.host.tolist()
        self.host = self._done = None  # (an event cannot be copied, and coordinates that hold this object can)
        nb = self.batches + 1
        raise_for_status(host[-1], self.device)
        if not host[-2]:
            return None
        self.ic._shared.setdefault("facts", {})["distinct"] = True
        levels = []
        sizes = [host[(l + 1) * nb - 1] for l in range(PYRAMID_LEVELS)]
        outs = [self.out[l, :m] for l, m in enumerate(sizes)]
        if self.n >= TRIMMED_ROWS:
            outs = [o.clone() for o in outs]
            self.first = [self.first[l, :m].clone() for l, m in enumerate(sizes)]
        self.out = None
        for l in range(PYRAMID_LEVELS):
            offs = host[l * nb:(l + 1) * nb]
            rows = outs[l]
            c = object.__new__(IntCoords)
            c.offsets = torch.tensor(offs, dtype=torch.int64)
            c.offsets.__dict__["_wcn_tuple"] = tuple(offs)  # the form kernel-map cache keys want
            c.batched_tensor = rows[:, 1:]
            c.voxel_size = c.voxel_origin = c.tensor_stride = None
            c._shared = {"bcoords": rows, "morton_origin": self.counts[8 + 4 * l:11 + 4 * l], "facts": {"distinct": True}}
            levels.append(c)
        return levels


def link_levels(ic: IntCoords, levels: List[IntCoords]) -> None:
    """Leaves the levels where :func:`strided_coordinates` looks for them."""
    for c in levels:
        ic._shared[("strided", (2, 2, 2))] = c
        ic = c


def morton_pyramid(ic: IntCoords) -> bool:
    """Computes and links the stride-2 levels of a natively sorted set; False when it is none (or not usable)."""
    if ic._shared.get("morton_info") is None:
        return False
    return LevelMaps(ic, begin=False, small_window_rows=LAYER_SMALL_WINDOW_ROWS).attach()


# 3x3x3 tables of at least this many rows are put in tile order.
TILE_ORDER_ROWS = 1024
# Tables of up to this many rows are ordered in small windows: for the forward of a network, whose layers over so few rows
# are bound by latency (MinkUNet-34, limit 65536 against 4096: 20 000 voxels 1.006 against 1.021 ms, 60 000 1.156 / 1.157,
# 150 000 1.465 / 1.502, 300 000 1.907 / 1.915, 1 200 000 4.506 / 4.492; small windows throughout cost the last 3 %).
# Tables that layers ask for one by one (their gradients use them too) get the large windows: the fp32 layers of a 60 000-row
# room took 195 us in them and 216 in small ones.
SMALL_WINDOW_ROWS = 65536
LAYER_SMALL_WINDOW_ROWS = 4096


class LevelMaps:
    """Tables of levels 0..4: the constructor enqueues the pyramid and (``begin``) level 0, :meth:`finish` the other levels - or
    :meth:`attach` leaves this object with the levels' coordinates, whose tables :meth:`ensure` makes as layers ask."""

    def __init__(self, ic: IntCoords, tile_order_rows: int = TILE_ORDER_ROWS, begin: bool = True,
                 small_window_rows: int = SMALL_WINDOW_ROWS):
        self.build = PyramidBuild(ic)
        self.min_rows = tile_order_rows
        self.small_window_rows = small_window_rows
        n = self.build.n
        self.n = [n]
        self.rows = [self.build.rows]
        self.nbr, self.order, self.child, self._bricks = {}, {}, {}, {}
        if begin:
            self._enqueue(range(1))

    def _enqueue(self, which) -> None:
        b = self.build
        levels = (Level * len(which))()
        for slot, l in zip(levels, which):
            n = self.n[l]
            nbr = torch.empty((27, n), dtype=torch.int32, device=b.device)
            order = torch.empty(n, dtype=torch.int32, device=b.device) if n >= self.min_rows else None
            bricks = torch.empty(query_bytes("wcn_level_brick_bytes", n), dtype=torch.uint8, device=b.device)
            self.nbr[l], self.order[l], self._bricks[l] = nbr, order, bricks
            slot.rows, slot.n, slot.level = self.rows[l].data_ptr(), n, l
            slot.bricks, slot.order, slot.nbr = bricks.data_ptr(), ptr(order), nbr.data_ptr()
            if l:
                child = self.child[l - 1] = torch.empty((8, n), dtype=torch.int32, device=b.device)
                slot.child, slot.first_child = child.data_ptr(), b.first[l - 1].data_ptr()
                slot.rows_below, slot.n_below = self.rows[l - 1].data_ptr(), self.n[l - 1]
        check(lib().wcn_level_maps(ctypes.addressof(levels), len(which), ptr(b.info), ptr(b.counts),
                                   self.small_window_rows, stream_ptr(b.device)), "wcn_level_maps")

    def _levels(self) -> Optional[List[IntCoords]]:
        """The coordinates of levels 1..4, linked (None: not usable)."""
        b = self.build
        levels = b.finish()
        if levels is None:
            b.ic._shared["morton_info"] = None
            return None
        link_levels(b.ic, levels)
        for c in levels:
            self.rows.append(c._shared["bcoords"])
            self.n.append(self.rows[-1].shape[0])
        return levels

    def _window3(self, l: int) -> IntSearchResult:
        if self.order[l] is not None:
            return IntSearchResult.from_tiled_table(self.nbr[l], self.order[l], self.n[l], 13)
        return IntSearchResult.from_neighbor_table(self.nbr[l], self.n[l], None, 13)

    def _window2(self, l: int) -> IntSearchResult:
        return IntSearchResult.from_neighbor_table(self.child[l], self.n[l], None, None)

    def finish(self) -> Optional[List[IntCoords]]:
        """The coordinates of levels 1..4 (None: not usable); their maps are enqueued and every level's maps left with
        its coordinates, where layers of those geometries find them."""
        levels = self._levels()
        if levels is None:
            return None
        self._enqueue(range(1, PYRAMID_LEVELS + 1))
        self._bricks = None
        for l, c in enumerate([self.build.ic] + levels):
            c._shared[("kmap", (3, 3, 3), (1, 1, 1))] = self._window3(l)
            if l < PYRAMID_LEVELS:
                c._shared[("kmap", (2, 2, 2), (2, 2, 2))] = self._window2(l)
        return levels

    def attach(self) -> bool:
        """Levels linked, the maps made as layers ask for them (:meth:`kmap`); False: not usable."""
        levels = self._levels()
        if levels is None:
            return False
        self._bricks = {}
        for l, c in enumerate([self.build.ic] + levels):
            c._shared["level_maps"] = (self, l)
        self.build.ic = None  # (the coordinate sets hold this object, not the other way round)
        return True

    def kmap(self, l: int, window: int) -> Optional[IntSearchResult]:
        """The map of level ``l``: 3x3x3 onto itself or 2x2x2 onto the next level."""
        at = l if window == 3 else l + 1
        if at > PYRAMID_LEVELS:
            return None
        if at not in self.nbr:
            self._enqueue(range(at, at + 1))
            self._bricks = {}
        return self._window3(l) if window == 3 else self._window2(l)
