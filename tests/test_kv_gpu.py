"""KV page push on one GPU: a rank pushes page runs into its own slot storage."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_canonical_runs():
    from aboleth_b200.kv import canonicalize_block_runs

    assert canonicalize_block_runs([4, 5, 6, 9, 10, 2], [0, 1, 2, 3, 4, 7]) == [(4, 0, 3), (9, 3, 2), (2, 7, 1)]
    assert canonicalize_block_runs([1, 2], [5, 7]) == [(1, 5, 1), (2, 7, 1)]
    with pytest.raises(ValueError):
        canonicalize_block_runs([1], [1, 2])


def test_push_pages_publish_readiness_and_lifecycle():
    import aboleth_b200 as ab
    from aboleth_b200.kv import CompiledKVTransferManager, KVPoolLayout, TransferState

    torch.cuda.set_device(0)
    with ab.World(0, 1, device=0) as world:
        world.connect_all("p2p")
        layout = KVPoolLayout(layers=6, blocks=32, page_bytes=4096, slots=2, slot_pages=8)
        kv = CompiledKVTransferManager(world, layout)
        g = torch.Generator(device="cuda").manual_seed(0)
        kv.pool.copy_(torch.randint(0, 255, kv.pool.shape, generator=g, device="cuda", dtype=torch.uint8))
        record = kv.begin_step("req-1")
        assert record is not None and record.slot == 0 and record.epoch == 1
        blocks = [3, 4, 5, 17, 9, 10]
        launched = kv.start_transfer("req-1", consumer=0, src_blocks=blocks, slot=record.slot,
                                     epoch=record.epoch)
        assert launched == 6 * 3  # three runs per layer
        kv.wait_for_layer("req-1", 0, source=0)
        kv.wait_for_layer("req-1", 5, source=0)
        torch.cuda.synchronize()
        assert kv.status.tolist() == [0, 0]
        assert kv.poll("req-1", source=0) == TransferState.READY
        for layer in range(6):
            got = kv.slot_pages("req-1", layer)[: len(blocks)]
            assert torch.equal(got, kv.pool[layer, blocks])
        kv.release("req-1")
        # Slots are admission-controlled.
        assert kv.begin_step("a").slot == 0 and kv.begin_step("b").slot == 1 and kv.begin_step("c") is None
        kv.abort("a")
        assert kv.begin_step("c").slot == 0
        with pytest.raises(RuntimeError, match="not allowed"):
            kv.ledger.get("a").move(TransferState.READY)
        # A consumer whose producer never pushes gives up with status 1, it does not hang.
        from aboleth_b200.kv import copy as kvcopy
        kvcopy.wait_ready(kv.ready[0, 0, 0:1], 99, kv.status, timeout_ns=20_000_000)
        torch.cuda.synchronize()
        assert kv.status.tolist()[0] == 1 and kv.poll("c", source=0) == TransferState.FAILED


def test_engine_pull_runtime_on_one_device():
    """The decode side pulls remapped blocks of every layer; here both 'ranks' are one device, so the
    peer table is stood in by the local addresses (the kernels only see addresses)."""
    import aboleth_b200 as ab
    from aboleth_b200.integrations import VLLMKVPeerRuntime

    torch.cuda.set_device(0)

    class _Table:
        def __init__(self, caches):
            self.caches = caches

        def addresses(self, name):
            return [self.caches[name[3:]].data_ptr()] * 2

        def close(self):
            pass

    with ab.World(0, 1, device=0) as world:
        world.connect_all("p2p")
        runtime = VLLMKVPeerRuntime(rank=0, world_size=2, device=0, world=world)
        g = torch.Generator(device="cuda").manual_seed(5)
        layers = {f"layer{i}": torch.randint(0, 255, (64, 2, 16, 128), generator=g, device="cuda",
                                             dtype=torch.uint8) for i in range(6)}
        remote = {k: v.clone() for k, v in layers.items()}      # what the prefill rank holds
        world.exchange_regions = lambda regions, tag="": _Table(remote)
        runtime.register_kv_caches(layers, consumer_order=tuple(layers))
        assert runtime.plan.physicalization.direct_destination
        local_ids, remote_ids = [40, 41, 42, 7, 8, 60], [3, 4, 5, 20, 21, 9]
        before = {k: v.clone() for k, v in layers.items()}
        ticket = runtime.start_layered_pull_blocks(local_block_ids=local_ids, remote_block_ids=remote_ids,
                                                   remote_rank=1)
        assert set(ticket.layer_events) == set(layers)
        ticket.completion.synchronize()
        runtime.check()
        assert runtime.last_run_count == 3 and "generated_p2p" in runtime.last_physicalization
        for name, cache in layers.items():
            assert torch.equal(cache[local_ids], remote[name][remote_ids])
            untouched = [b for b in range(64) if b not in local_ids]
            assert torch.equal(cache[untouched], before[name][untouched])
        us = runtime.pull_blocks(local_block_ids=[0, 1], remote_block_ids=[62, 63], remote_rank=1)
        assert us > 0 and torch.equal(layers["layer3"][0:2], remote["layer3"][62:64])
        with pytest.raises(ValueError, match="outside the registered cache"):
            runtime.start_pull_blocks(local_block_ids=[64], remote_block_ids=[0], remote_rank=1)
        with pytest.raises(ValueError, match="other rank"):
            runtime.start_pull_blocks(local_block_ids=[1], remote_block_ids=[0], remote_rank=0)


def test_shared_readiness_cell_is_published_after_the_last_batch():
    """Eight batches of very different sizes publish ONE cell.  A consumer CTA of the same launch
    waits for the cell and sums the destinations at once: with one arrival counter per group the
    sum is the sources' sum every time; a counter per batch would publish after the smallest."""
    from aboleth_b200.kv import copy as kvcopy

    torch.cuda.set_device(0)
    g = torch.Generator(device="cuda").manual_seed(3)
    sizes = [4096, 8 << 20, 16384, 2 << 20, 256, 6 << 20, 65536, 1 << 20]
    workers = 16
    total = sum(sizes)
    src = torch.randint(1, 255, (total,), generator=g, device="cuda", dtype=torch.uint8)
    dst = torch.zeros(total, dtype=torch.uint8, device="cuda")
    cell = torch.zeros(1, dtype=torch.int64, device="cuda")
    observed = torch.zeros(1, dtype=torch.int64, device="cuda")
    status = torch.zeros(2, dtype=torch.int64, device="cuda")
    arrivals = torch.zeros(8, dtype=torch.int32, device="cuda")
    records, at = [], 0
    for s in sizes:
        records.append((src.data_ptr() + at, dst.data_ptr() + at, s, cell.data_ptr()))
        at += s
    batches = kvcopy.pack_batches(records, "cuda")
    group_of, group_target, groups = kvcopy.pack_groups([r[3] for r in records], workers, "cuda")
    assert groups == 1 and group_target.tolist() == [len(sizes) * workers]
    want = int(src.view(torch.int64).sum().item())
    for epoch in range(1, 201):
        dst.zero_()
        kvcopy.push_observed(batches, arrivals, len(sizes), epoch, workers=workers, threads=256,
                             status=status, cell=cell, observed=observed, group_of=group_of,
                             group_target=group_target)
        torch.cuda.synchronize()
        assert status.tolist() == [0, 0], (epoch, status.tolist())
        assert int(observed.item()) == want, epoch
        assert int(cell.item()) == epoch and arrivals.tolist() == [0] * 8
    assert torch.equal(dst, src)


@pytest.mark.parametrize("page_bytes,layers,blocks,src,dst", [
    (16, 1, 4, [3], [0]),                                                  # one page, one vector
    (4112, 5, 40, [7, 8, 9, 30, 31, 2, 39], None),                          # two groups, the second of one layer
    (40, 6, 24, [4, 5, 11, 20, 21, 22], [5, 6, 0, 1, 2, 3]),                # runs that are not 16-byte aligned
    (66560, 9, 70, list(range(64)), None),                                  # one long run: every CTA cuts it
    (256, 3, 700, [2 * i for i in range(300)], None),                       # more runs than one launch carries
    (1024, 2, 16, [-1, 0, 5], [2, 0, 1]),                                   # a page counted from the pool's end
    (1024, 2, 16, [14, -1, 0, 1, -3, -2], None),                            # ... with pages before and after it
    (256, 2, 700, [2 * i for i in range(280)] + [-2, -1, 0, 1], None),      # the same, uploaded
])
def test_push_of_page_runs_copies_every_byte_and_nothing_else(page_bytes, layers, blocks, src, dst):
    import aboleth_b200 as ab
    from aboleth_b200.kv import CompiledKVTransferManager, KVPoolLayout

    torch.cuda.set_device(0)
    with ab.World(0, 1, device=0) as world:
        world.connect_all("p2p")
        pages = len(src)
        kv = CompiledKVTransferManager(world, KVPoolLayout(layers=layers, blocks=blocks, page_bytes=page_bytes, slots=3,
                                                           slot_pages=pages + 1))
        g = torch.Generator(device="cuda").manual_seed(page_bytes)
        kv.pool.copy_(torch.randint(0, 255, kv.pool.shape, generator=g, device="cuda", dtype=torch.uint8))
        to = list(range(pages)) if dst is None else dst
        want = torch.full_like(kv.slots, 255)
        want[1][:, to] = kv.pool[:, src]
        for epoch in (1, 2):  # the arrival counters have to be zero again
            kv.slots.fill_(255)
            kv.start_transfer("r", consumer=0, src_blocks=src, slot=1, epoch=epoch, dst_pages=dst)
            torch.cuda.synchronize()
            assert torch.equal(kv.slots, want)
            assert kv.ready[1].flatten().tolist() == [epoch] * kv.groups and int(kv.ready[0].abs().sum()) == 0
            assert int(kv._arrivals.abs().sum()) == 0
        at = [s % blocks for s in src]
        runs = [(s, d) for i, (s, d) in enumerate(zip(at, to)) if i == 0 or (s, d) != (at[i - 1] + 1, to[i - 1] + 1)]
        off = any((kv.pool[n, s].data_ptr() | kv.slots[1, n, d].data_ptr()) & 15 for n in range(layers) for s, d in runs)
        assert (kv.status.tolist()[0] == 3) == off
        for bad in ([blocks], [-blocks - 1], [blocks - 1, blocks], [2 * i for i in range(280)] + [blocks - 1, blocks]):
            if len(bad) > pages + 1:
                continue
            with pytest.raises(IndexError):
                kv.start_transfer("r", consumer=0, src_blocks=bad, slot=1, epoch=3)
        with pytest.raises(ValueError):
            kv.start_transfer("r", consumer=0, src_blocks=[], slot=1, epoch=3)
        with pytest.raises(ValueError):
            kv.start_transfer("r", consumer=0, src_blocks=[0, 1], slot=1, epoch=3, dst_pages=[-1, 0])


def test_transfers_on_two_streams_publish_their_own_cells():
    """Transfers to two slots at the same time, each from a stream of its own, many times over: every cell shows its own
    transfer's epoch, every byte has arrived, and the counters are zero again."""
    import aboleth_b200 as ab
    from aboleth_b200.kv import CompiledKVTransferManager, KVPoolLayout

    torch.cuda.set_device(0)
    with ab.World(0, 1, device=0) as world:
        world.connect_all("p2p")
        layout = KVPoolLayout(layers=8, blocks=64, page_bytes=4096, slots=2, slot_pages=32)
        kv = CompiledKVTransferManager(world, layout)
        kv.pool.copy_(torch.randint(0, 255, kv.pool.shape, device="cuda", dtype=torch.uint8))
        pages = [list(range(32)), list(range(63, 31, -1))]
        streams = [torch.cuda.Stream() for _ in pages]
        torch.cuda.synchronize()
        for epoch in range(1, 21):
            for slot, stream in enumerate(streams):
                with torch.cuda.stream(stream):
                    kv.start_transfer("r", consumer=0, src_blocks=pages[slot], slot=slot, epoch=epoch)
        torch.cuda.synchronize()
        for slot in range(2):
            assert torch.equal(kv.slots[slot], kv.pool[:, pages[slot]])
        assert kv.ready.flatten().tolist() == [20] * kv.ready.numel() and int(kv._arrivals.abs().sum()) == 0
        assert kv.status.tolist()[0] == 0
