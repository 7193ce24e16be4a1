"""CPU: the arithmetic of the even-share schedule of the persistent decode kernels, restated in Python and walked by the
library's own code.

The device code (anna_b200/csrc/balanced_schedule.cuh) lets every work unit derive its tile range, the slot of each
partial it writes and the number of partials each stream will receive from three numbers (tiles per row, units,
scratch capacity).  The properties the fused merge relies on are checked here for many ragged batches: every tile is
covered exactly once, slots of a stream are 0 .. partials-1 without gaps or repeats, and no stream needs more slots
than the scratch holds."""
from __future__ import annotations

import ctypes
import random

import pytest

from anna_b200 import _lib

TILE = 16


def share_of(total: int, units: int, max_tiles: int, capacity: int, min_tiles: int) -> int:
    share = (total + units - 1) // units
    share = max(share, min_tiles)
    return max(share, (max_tiles + capacity - 2) // (capacity - 1))


def segments(lengths: list[int], streams_per_row: int, units: int, capacity: int, min_tiles: int):
    """(unit, row, stream, first tile, tiles, slot, partials) for every piece, walking the line like the kernel."""
    tiles_row = [(n + TILE - 1) // TILE for n in lengths]
    prefix = [0]
    for n in tiles_row:
        prefix.append(prefix[-1] + n * streams_per_row)
    total = prefix[-1]
    if total == 0:
        return [], 0
    share = share_of(total, units, max(tiles_row), capacity, min_tiles)
    out = []
    for unit in range(units):
        pos, end = min(unit * share, total), min((unit + 1) * share, total)
        while pos < end:
            row = max(b for b in range(len(lengths)) if prefix[b] <= pos and tiles_row[b] > 0)
            n = tiles_row[row]
            stream = (pos - prefix[row]) // n
            tile = (pos - prefix[row]) - stream * n
            seg = min(n - tile, end - pos)
            stream_first = prefix[row] + stream * n
            first_unit = stream_first // share
            out.append((unit, row, stream, tile, seg, unit - first_unit,
                        (stream_first + n - 1) // share - first_unit + 1))
            pos += seg
    return out, share


@pytest.mark.parametrize("seed", range(12))
def test_even_share_covers_every_tile_once_with_dense_slots(seed):
    rng = random.Random(seed)
    batch = rng.choice([1, 2, 7, 32, 100])
    lengths = [rng.choice([0, 1, 15, 16, 17, rng.randint(1, 9000)]) for _ in range(batch)]
    if seed % 4 == 0:
        lengths[rng.randrange(batch)] = 40000          # one long row among short ones
    streams_per_row = rng.choice([1, 2, 8])
    units = rng.choice([4, 444, 1776])
    capacity = rng.choice([2, 3, 16, 64])
    min_tiles = rng.choice([1, 4])
    pieces, share = segments(lengths, streams_per_row, units, capacity, min_tiles)
    covered: dict[tuple[int, int], list[int]] = {}
    slots: dict[tuple[int, int], list[tuple[int, int]]] = {}
    for unit, row, stream, tile, seg, slot, partials in pieces:
        assert seg >= 1 and 0 <= slot < partials <= capacity
        covered.setdefault((row, stream), []).extend(range(tile, tile + seg))
        slots.setdefault((row, stream), []).append((slot, partials))
    for row, n in enumerate(lengths):
        tiles = (n + TILE - 1) // TILE
        for stream in range(streams_per_row):
            if tiles == 0:
                assert (row, stream) not in covered
                continue
            assert sorted(covered[(row, stream)]) == list(range(tiles))
            got = sorted(s for s, _ in slots[(row, stream)])
            partials = slots[(row, stream)][0][1]
            assert got == list(range(partials)) and all(p == partials for _, p in slots[(row, stream)])
    if pieces:
        work = {}
        for unit, *_rest in pieces:
            work[unit] = work.get(unit, 0) + _rest[3]
        assert max(work.values()) <= share


FUSED_MAX_CHUNKS = 512  # kFusedMaxChunks: weights per head that the fused merge stages in shared memory


@pytest.mark.parametrize("capacity", [600, 4096])
def test_even_share_never_exceeds_the_fused_merge_limit(capacity):
    """A caller may hand in a scratch larger than the fused merge can stage; the kernel clamps the capacity it gives
    to the schedule to 512, so one very long row beside short ones still gets at most 512 partials."""
    lengths = [512 * 1024] + [1] * 7           # ~586 partials with an unclamped capacity and 592 units
    pieces, _ = segments(lengths, 1, 592, min(capacity, FUSED_MAX_CHUNKS), 4)
    assert pieces
    assert max(partials for *_head, partials in pieces) <= FUSED_MAX_CHUNKS
    unclamped, _ = segments(lengths, 1, 592, capacity, 4)
    assert max(partials for *_head, partials in unclamped) > FUSED_MAX_CHUNKS  # the case the clamp is for


def walked(lengths: list[int], streams_per_row: int, units: int, capacity: int, *, tail: int = 0, min_tiles: int = 8,
           segment_tiles: int = 0, stream_tiles: int = 0) -> list[tuple[int, ...]]:
    """(unit, row, stream, first tile, end tile, slot, partials) of every segment, by the kernels' own arithmetic."""
    rows, count = (ctypes.c_int64 * len(lengths))(*lengths), ctypes.c_int()
    room = sum((n + TILE - 1) // TILE for n in lengths) * streams_per_row + 1
    out = (ctypes.c_int32 * (7 * room))()
    _lib.check(_lib.lib().anna_kv_selftest_even_shares(rows, len(lengths), streams_per_row, units, capacity, tail, min_tiles,
                                                       segment_tiles, stream_tiles, out, room, ctypes.byref(count)), "walk")
    assert count.value <= room
    return [tuple(out[7 * i:7 * i + 7]) for i in range(count.value)]


def random_batch(seed: int):
    rng = random.Random(100 + seed)
    lengths = [rng.choice([0, 1, 16, 17, rng.randint(1, 5000)]) for _ in range(rng.choice([1, 3, 16, 70]))]
    return lengths, rng.choice([1, 2, 8]), rng.choice([296, 444, 592]), rng.choice([2, 8, 65])


@pytest.mark.parametrize("seed", range(12))
def test_the_restatement_is_what_the_kernels_walk(seed):
    lengths, streams_per_row, units, capacity = random_batch(seed)
    restated, _ = segments(lengths, streams_per_row, units, capacity, 8)
    assert walked(lengths, streams_per_row, units, capacity) == [
        (unit, row, stream, tile, tile + seg, slot, partials) for unit, row, stream, tile, seg, slot, partials in restated]


@pytest.mark.parametrize("segment_tiles,stream_tiles,tail", [(0, 0, 0), (12, 0, 0), (20, 20, 0), (20, 20, 33)])
@pytest.mark.parametrize("seed", range(40))
def test_segments_cover_every_tile_once_and_number_the_partials(seed, segment_tiles, stream_tiles, tail):
    """Shares that cross streams (with and without the first segment's cost on the line) and pieces of single streams."""
    lengths, streams_per_row, units, capacity = random_batch(seed)
    made = walked(lengths, streams_per_row, units, capacity, tail=tail, segment_tiles=segment_tiles,
                  stream_tiles=stream_tiles)
    streams: dict[tuple[int, int], list[tuple[int, ...]]] = {}
    for unit, row, stream, first, end, slot, partials in made:
        assert 0 <= unit < units and first < end
        streams.setdefault((row, stream), []).append((first, end, slot, partials))
    tiles = [max(0, n - tail + TILE - 1) // TILE for n in lengths]
    assert set(streams) == {(row, s) for row, n in enumerate(tiles) if n for s in range(streams_per_row)}
    for (row, _), parts in streams.items():
        assert len(parts) <= capacity
        assert [p[0] for p in parts] == [0] + [p[1] for p in parts[:-1]] and parts[-1][1] == tiles[row]
        assert [p[2:] for p in parts] == [(slot, len(parts)) for slot in range(len(parts))]


@pytest.mark.parametrize("batch,low,high,streams_per_row,units", [(96, 129, 500, 8, 592), (64, 129, 1000, 8, 592),
                                                                  (64, 312, 2500, 8, 592), (300, 129, 1000, 2, 444)])
def test_short_streams_do_not_pile_up_in_one_unit(batch, low, high, streams_per_row, units):
    """A segment costs about 20 tiles beside its own.  No unit gets more than its share of tiles and segments together,
    plus one segment that begins inside a stream; counting tiles alone, some unit got several times that."""
    tail, cost, capacity = 128, 20, 2
    lengths = [low + (high - low) * i // (batch - 1) for i in range(batch)]
    tiles = [(n - tail + TILE - 1) // TILE for n in lengths]
    line = streams_per_row * sum(n + cost for n in tiles)
    share = max((line + units - 1) // units, 8, (max(tiles) + capacity - 2) // (capacity - 1))

    def worst(stream_tiles: int, segment_tiles: int) -> int:
        spent = [0] * units
        for unit, _, _, first, end, _, _ in walked(lengths, streams_per_row, units, capacity, tail=tail,
                                                   segment_tiles=segment_tiles, stream_tiles=stream_tiles):
            spent[unit] += end - first + cost
        return max(spent)

    assert worst(cost, cost) <= share + cost < worst(0, 0) / 1.5
