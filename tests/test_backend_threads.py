"""What two threads may do to one stored tensor, forced on the CPU by running the second
thread's step at the point where it hurts most: a description of a container that is published
after the container has been replaced."""
import ctypes

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
