"""The sampler's host side with stand-ins for the device and its kernels: a kernel's or a copy's result is in its page-locked buffer
at once, the events wait for nothing, and what is looked at is whose buffer that is."""
import threading
from types import SimpleNamespace

import pytest
import torch

from nanoinfer_b200.sampling import SampleRow, SamplingParams
from nanoinfer_b200.sampling import sampler as sampler_module
from nanoinfer_b200.sampling.sampler import Sampler


class OnDevice(torch.Tensor):
    device = torch.device("cuda")


class FakeEvent:
    def record(self):
        pass

    def synchronize(self):
        pass


class FakeOps:
    """Every call's tokens are a number of its own, upward from 1."""
    sample_rows_most = 64

    def __init__(self):
        self.calls = 0

    def sample_rows(self, logits, rows, out):
        self.calls += 1
        out[:len(rows)] = self.calls

    def sample(self, logits, temperature, top_k, top_p, uniform, out):
        self.calls += 1
        out[:] = self.calls

    def argmax(self, logits, out):
        self.calls += 1
        out[:] = self.calls


@pytest.fixture()
def sampler(monkeypatch):
    def empty(*shape, device=None, **kw):
        t = torch.empty(*shape, **kw)
        return t if device is None else t.as_subclass(OnDevice)
    fake = SimpleNamespace(empty=empty, device=torch.device, int32=torch.int32, float32=torch.float32, Tensor=torch.Tensor,
                           cuda=SimpleNamespace(Event=FakeEvent))
    monkeypatch.setattr(sampler_module, "torch", fake)
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda self: self)
    return Sampler(FakeOps(), "cuda")


def logits(n):
    return torch.zeros(n, 16).as_subclass(OnDevice)


def rows(n, temperature=0.7):
    return [SampleRow(SamplingParams(temperature=temperature), None, i, seed=i) for i in range(n)]


@pytest.mark.parametrize("n", [1, 64, 65, 300])
def test_a_read_that_is_out_is_not_written_by_later_calls(sampler, n):
    for turn in range(3):           # the buffers come back and are used again
        first = sampler.ops.calls + 1
        out = [sampler.sample_async(logits(n), rows(n)) for _ in range(6)]
        for k in range(9):          # sampled, greedy, and of another size
            for m, t in ((n, 0.7), (n, 0.0), (2, 0.7), (90, 0.7)):
                expect = sampler.ops.calls + 1
                assert sampler.sample(logits(m), rows(m, t)) == [expect] * m
        for i, p in enumerate(out):
            assert p.wait() == [first + i] * n
            assert p.wait() == [first + i] * n


def test_threads_that_wait_have_buffers_of_their_own(sampler):
    both = threading.Barrier(2)
    plain = sampler.ops.sample_rows
    lock = threading.Lock()

    def sample_rows(logits, rows, out):
        with lock:
            plain(logits, rows, out)
            mine = int(out[0])
        both.wait(10)               # both calls' tokens are stored before either is read
        seen.append((mine, out))

    sampler.ops.sample_rows = sample_rows
    got, seen = [], []
    threads = [threading.Thread(target=lambda: got.append(sampler.sample(logits(3), rows(3)))) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(20)
    assert sorted(got) == [[1] * 3, [2] * 3]
    assert seen[0][1].data_ptr() != seen[1][1].data_ptr()
    assert len(sampler._free_tokens) == 2


def test_parameters_by_value_are_what_the_arrays_hold():
    kinds = [dict(temperature=1e-3, top_k=5), dict(temperature=3.3e38), dict(temperature=1e39, top_p=0.5), dict(temperature=float("inf"), top_p=2.0),
             dict(), dict(temperature=1.0, top_k=1 << 40), dict(temperature=1.0, top_k=-3, top_p=0.0)]
    by_value = Sampler._row_parameters([SampleRow(SamplingParams(**k), None, 3, seed=-1) for k in kinds])
    assert [r[:3] for r in by_value] == [(1e-3, 5, 1.0), (3.3e38, 0, 1.0), (float("inf"), 0, 0.5), (float("inf"), 0, 1.0), (1.0, 1, 1.0),
                                         (1.0, 0x7FFFFFFF, 1.0), (1.0, 0, 0.0)]
    arrays = Sampler(FakeOps(), "cpu")._device_parameters([SampleRow(SamplingParams(**k), None, 3, seed=-1) for k in kinds], "cpu")
    for row, *par in zip(by_value, *(a.tolist() for a in arrays)):         # the same beyond the rows that go by value
        assert torch.tensor(row[:3], dtype=torch.float32).tolist() == torch.tensor(par[:3], dtype=torch.float32).tolist()
    assert by_value[0][3:] == (0, (1 << 64) - 1, 3) and by_value[4][3:] == (1, 0, 0)
