"""Host-side pieces of the KV path that need no GPU: run canonicalisation, batch and group packing."""
import struct

import pytest
import torch

from aboleth_b200.kv import copy as kvcopy


def test_block_pairs_merge_into_maximal_runs():
    runs = kvcopy.canonicalize_block_runs([4, 5, 6, 30, 31, 9], [20, 21, 22, 3, 4, 5])
    assert runs == [(4, 20, 3), (30, 3, 2), (9, 5, 1)]
    # source consecutive but destination not: no merge
    assert kvcopy.canonicalize_block_runs([1, 2, 3], [7, 9, 10]) == [(1, 7, 1), (2, 9, 2)]
    # a descending pair never merges, an empty transfer has no runs
    assert kvcopy.canonicalize_block_runs([5, 4], [1, 0]) == [(5, 1, 1), (4, 0, 1)]
    assert kvcopy.canonicalize_block_runs([], []) == []
    with pytest.raises(ValueError):
        kvcopy.canonicalize_block_runs([1, 2], [1])
    # every page is covered exactly once, in order
    src, dst = [8, 9, 2, 3, 4, 11], [0, 1, 2, 3, 4, 5]
    covered = [(s + i, d + i) for s, d, n in kvcopy.canonicalize_block_runs(src, dst) for i in range(n)]
    assert covered == list(zip(src, dst))


def test_batches_pack_as_four_little_endian_words():
    packed = kvcopy.pack_batches([(0x1000, 0x2000, 4096, 0x3000), (0x1100, 0x2100, 512, 0x3008)], "cpu")
    assert packed.dtype == torch.uint8 and packed.numel() == 64
    words = struct.unpack("<8Q", bytes(packed.tolist()))
    assert words == (0x1000, 0x2000, 4096, 0x3000, 0x1100, 0x2100, 512, 0x3008)


def test_batches_that_publish_one_cell_share_one_arrival_counter():
    """Three batches name cell A, one names cell B: two groups, and a group's target is the worker
    total of all its batches, so cell A is published by the last worker of its last batch."""
    cell_a, cell_b = 0x5000, 0x5008
    group_of, target, groups = kvcopy.pack_groups([cell_a, cell_b, cell_a, cell_a], workers=16, device="cpu")
    assert groups == 2
    assert group_of.tolist() == [0, 1, 0, 0] and target.tolist() == [48, 16]
    assert group_of.dtype == target.dtype == torch.int32
    # one cell per batch degenerates to the per-batch count
    group_of, target, groups = kvcopy.pack_groups([1, 2, 3], workers=4, device="cpu")
    assert groups == 3 and group_of.tolist() == [0, 1, 2] and target.tolist() == [4, 4, 4]


@pytest.mark.parametrize("src,dst,refused", [([7, 8], [0, 1], -4), ([6, 7, 8, 9], [0, 1, 2, 3], -4), ([8], [0], -4),
                                             ([-9], [0], -4), ([-1, 0, 8], [0, 1, 2], -4), ([0, 1], [-1, 0], -5),
                                             ([0, 1], [3, 4], -5),
                                             (list(range(7, -1, -1)) * 40 + [8], [1, 0] * 160 + [0], -3)])
def test_every_page_of_a_transfer_lies_inside_the_pool_and_the_slot(src, dst, refused):
    """A run that starts inside the pool of 8 pages (or the slot of 4) and leaves it is refused before anything is
    launched, as a run that starts outside is; more runs than one launch carries are left to the uploaded path."""
    import ctypes

    from aboleth_b200.ops._kernels import call_rc

    array, n = ctypes.c_longlong * len(src), len(src)
    runs = ctypes.c_int(0)
    rc = call_rc("ab_kv_push_pages", array(*src), array(*dst), n, 4096, 2, 8, 8 * 256, 256, 65536, 4 * 256, 131072, 8,
                 4, 1, 4096, 4096, 4, 256, ctypes.byref(runs), 0)
    assert rc == refused


def test_a_block_counted_from_the_end_is_not_followed_by_the_first():
    assert kvcopy.canonicalize_block_runs([-2, -1, 0, 1], [3, 4, 5, 6]) == [(-2, 3, 2), (0, 5, 2)]
    assert kvcopy.canonicalize_block_runs([4, 5], [-1, 0]) == [(4, -1, 1), (5, 0, 1)]


@pytest.mark.parametrize("pages", [list(range(8)), list(range(0, 600, 2))])   # one launch's arguments, and uploaded
def test_transfers_to_different_slots_share_no_arrival_counter(pages, monkeypatch):
    """Each transfer counts the arrivals of its readiness groups on counters of its own: several may be in flight, also
    on different streams, and a shared one would mix their counts."""
    import aboleth_b200 as ab
    from aboleth_b200.kv import CompiledKVTransferManager, KVPoolLayout

    used = []

    def push_pages(src, dst, *, arrivals, **_):
        used.append(arrivals)
        return 1 if len(src) == 8 else None

    monkeypatch.setattr(kvcopy, "push_pages", push_pages)
    monkeypatch.setattr(kvcopy, "push", lambda packed, arrivals, *a, **k: used.append(arrivals))
    with ab.World(0, 1, device="cpu") as world:
        world.connect_all("p2p")
        layout = KVPoolLayout(layers=9, blocks=600, page_bytes=16, slots=3, slot_pages=300)
        kv = CompiledKVTransferManager(world, layout)
        for slot in range(3):
            kv.start_transfer("r", consumer=0, src_blocks=pages, slot=slot, epoch=1)
        counters = {a.data_ptr() + 4 * i for a in used for i in range(a.numel())}
        assert all(a.numel() == kv.groups and a.is_contiguous() for a in used)
        assert len(counters) == 3 * kv.groups
        for slot in (-1, 3):
            with pytest.raises(IndexError):
                kv.start_transfer("r", consumer=0, src_blocks=pages, slot=slot, epoch=1)
