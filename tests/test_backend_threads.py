"""What two threads may do to one stored tensor, forced on the CPU by running the second
thread's step at the point where it hurts most: a container replaced while a description of it
is made, and a write settled, replaced or erased while another thread settles it."""
import torch

from neuzip_b200 import _lib, backend


class FakeEvent:
    def __init__(self, on_query=None):
        self.on_query = on_query

    def query(self):
        if self.on_query is not None:
            step, self.on_query = self.on_query, None
            step()
        return True

    def synchronize(self):
        self.query()


class FakeLibrary:
    """Header parsing and the single decode; notes the container every decode was given."""
    def __init__(self, total=64, words=100):
        self.total, self.words, self.seen = total, words, []

    def nz_parse_header(self, host, total, words):
        total._obj.value, words._obj.value = self.total, self.words
        return 0

    def nz_decompress_bf16_item(self, address, out, flags, precision, canon, status, stream):
        item = _lib.DecompressItem.from_address(address)
        self.seen.append((item.container, item.container_bytes, item.max_unit_words))
        return 0


def make(monkeypatch, on_query=None):
    monkeypatch.setattr(backend, "_stream", lambda: 0)
    be = backend._cuda.Manager_f7_n0()
    be._lib = FakeLibrary()
    be._hdr_base = [0]
    entry = backend._Entry(16, torch.bfloat16, 256, 0, torch.zeros(4096, dtype=torch.uint8),
                           torch.zeros(16, dtype=torch.uint8))
    entry.pending = (3, FakeEvent(on_query))
    be._cache["w"] = entry
    return be, entry


def described(entry):
    return entry.container.data_ptr(), entry.container.numel(), entry.max_unit_words


def test_description_published_after_the_container_was_replaced(monkeypatch):
    be, entry = make(monkeypatch)
    fill = be._set_normalizer

    def settled_by_another_thread(item, e):
        be._set_normalizer = fill
        be._settle(e, block=True)           # between reading the pointers and publishing them
        fill(item, e)

    be._set_normalizer = settled_by_another_thread
    out = torch.empty(16, dtype=torch.bfloat16)
    staging = entry.container
    be._decode(entry, out)
    # that call used the buffer it read, which its description kept alive
    assert be._lib.seen[0][0] == staging.data_ptr()
    assert entry.container is not staging
    for _ in range(2):
        be._decode(entry, out)
        assert be._lib.seen[-1] == described(entry)


def test_two_threads_settle_one_entry(monkeypatch):
    be, entry = make(monkeypatch)
    # the other thread settles while this one asks whether the header has arrived
    entry.pending[1].on_query = lambda: be._settle(entry, block=False)
    be._settle(entry, block=False)
    assert be._hdr_free == [3] and len(be._event_pool) == 1       # given back once
    assert entry.pending is None and entry.version == 1 and entry.container.numel() == 64


def test_replaced_while_settled(monkeypatch):
    be, entry = make(monkeypatch)
    entry.pending[1].on_query = lambda: be.erase("w")
    be._settle(entry, block=True)
    assert be._hdr_free == [3] and len(be._event_pool) == 1


def test_batch_bound_while_an_entry_is_settled(monkeypatch):
    be, entry = make(monkeypatch)
    pending = entry.pending
    entry.pending = None
    entry.stamp = 1 << 60                   # a fresh write: the batch runs the block it fills first
    fill = be._set_normalizer

    def settled_by_another_thread(item, e):
        if be._set_normalizer is not fill:
            be._set_normalizer = fill
            e.pending = pending
            be._settle(e, block=True)
        fill(item, e)

    class Out:                               # make_batch wants CUDA outputs
        dtype, is_cuda = torch.bfloat16, True
        numel = staticmethod(lambda: 16)
        data_ptr = staticmethod(lambda: 0)

    be._set_normalizer = settled_by_another_thread
    batch = be.make_batch(["w"], [Out()])
    seen = []

    def batched(items, count, precision, lane, canon, status, stream):
        seen.append((items[0].container, items[0].container_bytes, items[0].max_unit_words))
        return 0

    be._lib.nz_decompress_bf16_batch = batched
    be.run_batch(batch)
    assert seen[-1] == described(entry)
