"""The cached per-bin sums of k N and N of power-of-two grids: another stream
waits for the one that writes them, callers get copies, and the number of
entries is bounded."""

import pytest
import torch

from pmwd_gb300 import spec_util as su


class _Tensor:
    def __init__(self, name, log):
        self.name, self.log = name, log

    def clone(self):
        self.log.append(('clone', self.name))
        return _Tensor(self.name + "'", self.log)

    def record_stream(self, stream):
        self.log.append(('record_stream', self.name, stream.name))


class _Event:
    def __init__(self, stream, log):
        self.stream, self.log, self.done = stream, log, False

    def query(self):
        return self.done


class _Stream:
    def __init__(self, name, log):
        self.name, self.log = name, log

    def record_event(self):
        self.log.append(('record_event', self.name))
        return _Event(self.name, self.log)

    def wait_event(self, event):
        self.log.append(('wait_event', self.name, event.stream))


def test_another_stream_waits_and_gets_copies():
    log = []
    a, b = _Stream('a', log), _Stream('b', log)
    cache = su._GeometryCache()
    assert cache.get('grid', b) is None and log == []
    cache.put('grid', (_Tensor('k', log), _Tensor('n', log)), a)
    # the copies are enqueued before the event that stands for them
    assert log == [('clone', 'k'), ('clone', 'n'), ('record_event', 'a')]
    log.clear()
    k, n = cache.get('grid', b)
    assert log[0] == ('wait_event', 'b', 'a')
    assert set(log[1:3]) == {('record_stream', "k'", 'b'), ('record_stream', "n'", 'b')}
    assert log[3:] == [('clone', "k'"), ('clone', "n'")]
    assert (k.name, n.name) == ("k''", "n''")
    # nothing to wait for once it is written, nothing to record on the writing stream itself
    cache.entries['grid'][1].done = True
    log.clear()
    cache.get('grid', a)
    assert log == [('clone', "k'"), ('clone', "n'")]


def test_entries_are_bounded_and_the_oldest_goes():
    log = []
    s = _Stream('s', log)
    cache = su._GeometryCache(size=3)
    for i in range(3):
        cache.put(i, (_Tensor(str(i), log),), s)
    assert cache.get(0, s) is not None   # used again: 1 is the oldest now
    cache.put(3, (_Tensor('3', log),), s)
    assert [cache.get(i, s) is None for i in range(4)] == [False, True, False, False]


@pytest.mark.gpu
def test_second_stream_gets_finished_sums(cuda):
    """The first call of a grid on a stream that is still busy, the second at once on another."""
    f = torch.randn((32, 64, 32), device=cuda)
    want = su.powspec(f, 1.0)
    torch.cuda.synchronize()
    su._GEOMETRY.clear()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(int(1e8))   # some 50 ms
        first = su.powspec(f, 1.0)
    with torch.cuda.stream(b):
        second = su.powspec(f, 1.0)
    torch.cuda.synchronize()
    for got in (first, second):
        for x, y in zip(got, want):
            # sums in another order of the same float64 terms, P of float32 products
            torch.testing.assert_close(x, y, rtol=1e-6, atol=0, equal_nan=True)   # empty bins: 0 / 0
        assert torch.equal(got[2], want[2])


@pytest.mark.gpu
def test_a_callers_change_stays_its_own(cuda):
    f = torch.randn((16, 32, 16), device=cuda)
    su._GEOMETRY.clear()
    want = su.powspec(f, 1.0)[2]
    keep = want.clone()
    want.zero_()
    for _ in range(2):
        got = su.powspec(f, 1.0)[2]
        assert torch.equal(got, keep)
        got.zero_()
