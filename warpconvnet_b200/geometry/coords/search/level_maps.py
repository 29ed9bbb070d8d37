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
        self.out_ptr = self.first_ptr = self.counted = None
        self.host, self._done = pinned_result(PYRAMID_LEVELS * (self.batches + 1) + 2, torch.int64, dev, launch)

    def sizes(self) -> Optional[List[int]]:
        """Waits for the counts; the levels' row counts, or None when the rows are not what the pyramid needs
        (repeated voxels, an extent of 2^21 or more)."""
        self._done.synchronize()
        host = self.counted = self.host.tolist()
        self.host = self._done = None  # (an event cannot be copied, and coordinates that hold this object can)
        nb = self.batches + 1
        raise_for_status(host[-1], self.device)
        if not host[-2]:
            return None
        sizes = [host[(l + 1) * nb - 1] for l in range(PYRAMID_LEVELS)]
        if self.n >= TRIMMED_ROWS:
            outs = [self.out[l, :m].clone() for l, m in enumerate(sizes)]
            self.first = [self.first[l, :m].clone() for l, m in enumerate(sizes)]
            self.out = outs
        # where each level's rows and first children start
        trimmed = isinstance(self.out, list)
        self.out_ptr = [self.out[l].data_ptr() if trimmed else self.out.data_ptr() + 16 * l * self.n for l in range(PYRAMID_LEVELS)]
        self.first_ptr = [self.first[l].data_ptr() if trimmed else self.first.data_ptr() + 4 * l * self.n for l in range(PYRAMID_LEVELS)]
        return sizes

    def finish(self) -> Optional[List[IntCoords]]:
        """The levels' coordinates, or None (see :meth:`sizes`)."""
        return None if self.sizes() is None else self.coordinates()

    def coordinates(self) -> List[IntCoords]:
        """The levels' coordinates, once their sizes are known."""
        host, nb = self.counted, self.batches + 1
        self.ic._shared.setdefault("facts", {})["distinct"] = True
        levels, outs = [], self.out
        self.out = self.counted = self.out_ptr = self.first_ptr = None   # (addresses would be wrong in a copy)
        for l in range(PYRAMID_LEVELS):
            offs = host[l * nb:(l + 1) * nb]
            rows = outs[l] if isinstance(outs, list) else outs[l, :offs[-1]]
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
        self.nbr, self.order, self.child, self._bricks = {}, {}, {}, None
        self.at, self._made = {}, []   # (nbr, order, child) addresses of a level; tables whose tensors have not been made
        if begin:
            self._enqueue(range(1))

    def _enqueue(self, which) -> None:
        """The maps of some levels: of one level as tensors of their own, of several in a piece of memory for each
        coordinate set (an allocation costs the host 2 us, a view as much), of which :meth:`_tensors` makes views: who keeps
        one set keeps its tables and no others.  The table of the children between two levels is the finer set's."""
        b, dev = self.build, self.build.device
        levels = (Level * len(which))()
        if len(which) == 1:
            l, n = which[0], self.n[which[0]]
            nbr = self.nbr[l] = torch.empty((27, n), dtype=torch.int32, device=dev)
            order = self.order[l] = torch.empty(n, dtype=torch.int32, device=dev) if n >= self.min_rows else None
            bricks = self._bricks = torch.empty(query_bytes("wcn_level_brick_bytes", n), dtype=torch.uint8, device=dev)
            child = None
            if l:
                child = self.child[l - 1] = torch.empty((8, n), dtype=torch.int32, device=dev)
            self.at[l] = (nbr.data_ptr(), ptr(order), ptr(child))
            brick_at = [bricks.data_ptr()]
        else:
            words, want, brick_at, bytes_ = {}, dict.fromkeys(range(max(which[0] - 1, 0), which[-1] + 1), 0), [], 0
            for l in which:
                n = self.n[l]
                words[l] = -(-n // 64) * 64   # every table starts on a 256-byte boundary
                want[l] += (28 if n >= self.min_rows else 27) * words[l]
                if l:
                    want[l - 1] += 8 * words[l]
                brick_at.append(bytes_)
                bytes_ += -(-query_bytes("wcn_level_brick_bytes", n) // 256) * 256
            memory = {l: torch.empty(w, dtype=torch.int32, device=dev) for l, w in want.items()}
            base, used = {l: m.data_ptr() for l, m in memory.items()}, dict.fromkeys(want, 0)
            bricks = self._bricks = torch.empty(bytes_, dtype=torch.uint8, device=dev)
            brick_at = [bricks.data_ptr() + v for v in brick_at]

            def take(l: int, rows: int, of: int) -> int:
                used[l] += rows * words[of]
                return used[l] - rows * words[of]

            for l in which:
                nbr, order = take(l, 27, l), take(l, 1, l) if self.n[l] >= self.min_rows else None
                child = take(l - 1, 8, l) if l else None
                self.at[l] = (base[l] + 4 * nbr, None if order is None else base[l] + 4 * order,
                              None if child is None else base[l - 1] + 4 * child)
                self._made.append((l, memory[l], nbr, order, memory.get(l - 1), child))
        for slot, l, brick in zip(levels, which, brick_at):
            slot.rows, slot.n, slot.level = self._row_ptr(l), self.n[l], l
            slot.nbr, slot.order, slot.child = self.at[l]
            slot.bricks = brick
            if l:
                slot.first_child = b.first_ptr[l - 1] if b.first_ptr else b.first[l - 1].data_ptr()
                slot.rows_below, slot.n_below = self._row_ptr(l - 1), self.n[l - 1]
        check(lib().wcn_level_maps(ctypes.addressof(levels), len(which), ptr(b.info), ptr(b.counts),
                                   self.small_window_rows, stream_ptr(dev)), "wcn_level_maps")

    def _row_ptr(self, l: int) -> int:
        return self.rows[l].data_ptr() if l < len(self.rows) else self.build.out_ptr[l - 1]

    def _tensors(self) -> None:
        """The tables that have been enqueued as tensors."""
        self.at = {}   # (addresses would be wrong in a copy)
        for l, memory, nbr, order, finer, child in self._made:
            n = self.n[l]
            self.nbr[l] = memory[nbr:nbr + 27 * n].view(27, n)
            self.order[l] = None if order is None else memory[order:order + n]
            if child is not None:
                self.child[l - 1] = finer[child:child + 8 * n].view(8, n)
        self._made = []

    def _sizes(self) -> bool:
        """Waits for the sizes of the levels; False: not usable."""
        sizes = self.build.sizes()
        if sizes is None:
            self.build.ic._shared["morton_info"] = None
            return False
        self.n += sizes
        return True

    def _levels(self) -> List[IntCoords]:
        """The coordinates of levels 1..4, linked."""
        levels = self.build.coordinates()
        link_levels(self.build.ic, levels)
        self.rows += [c._shared["bcoords"] for c in levels]
        return levels

    def _window3(self, l: int) -> IntSearchResult:
        if self.order[l] is not None:
            return IntSearchResult.from_tiled_table(self.nbr[l], self.order[l], self.n[l], 13)
        return IntSearchResult.from_neighbor_table(self.nbr[l], self.n[l], None, 13)

    def _window2(self, l: int) -> IntSearchResult:
        return IntSearchResult.from_neighbor_table(self.child[l], self.n[l], None, None)

    def launch(self) -> bool:
        """Waits for the sizes of the levels and enqueues the maps of levels 1..4 (False: not usable): their addresses are in
        ``at``.  :meth:`keep` does the rest, for which the device need not wait."""
        if not self._sizes():
            return False
        self._enqueue(range(1, PYRAMID_LEVELS + 1))
        self._bricks = None
        return True

    def finish(self) -> Optional[List[IntCoords]]:
        """:meth:`launch` and :meth:`keep` (None: not usable)."""
        return self.keep() if self.launch() else None

    def keep(self) -> List[IntCoords]:
        """The coordinates of levels 1..4, with every level's maps left with its coordinates, where layers of those
        geometries find them."""
        levels = self._levels()
        self._tensors()
        for l, c in enumerate([self.build.ic] + levels):
            c._shared[("kmap", (3, 3, 3), (1, 1, 1))] = self._window3(l)
            if l < PYRAMID_LEVELS:
                c._shared[("kmap", (2, 2, 2), (2, 2, 2))] = self._window2(l)
        return levels

    def attach(self) -> bool:
        """Levels linked, the maps made as layers ask for them (:meth:`kmap`); False: not usable."""
        if not self._sizes():
            return False
        levels = self._levels()
        self._bricks = None
        self._tensors()
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
            self._bricks = None
            self._tensors()
        return self._window3(l) if window == 3 else self._window2(l)
