"""partition_deposits_on_device fills buffers of torch's stream from the context's stream: the fills
and the work that the caller has queued on torch's stream come before the library's writes."""
import numpy as np
import pytest

import cmpmc_b200 as cm
from cmpmc_b200 import _ffi


def _deposits(n, seed):
    rng = np.random.default_rng(seed)
    dep = np.zeros(n, dtype=_ffi.DEPOSIT_DTYPE)
    dep["pos"] = rng.uniform(-0.01, 0.01, (n, 3))
    dep["edep_eV"] = 10.0 ** rng.uniform(1.0, 4.0, n)
    dep["is_nuclear_recoil"] = np.arange(n) % 2
    return dep, rng.integers(1, 1 << 63, size=(n, 4), dtype=np.uint64)


class _Tensor:
    def __init__(self, a):
        self.a = a

    def to(self, dev):
        return self

    def cpu(self):
        return self

    def numpy(self):
        return self.a

    def data_ptr(self):
        return self.a.ctypes.data


def test_every_call_waits_for_the_allocations(monkeypatch):
    """On the CPU with a recorded torch: a synchronize between each allocation and the call after."""
    import types
    log = []

    class Stream:
        def synchronize(self):
            log.append("sync")

    def zeros(n, dtype=None, device=None):
        log.append("alloc")
        return _Tensor(np.zeros(n, dtype=dtype))

    torch = types.SimpleNamespace(
        from_numpy=_Tensor, zeros=zeros, empty=zeros, int64=np.int64, uint8=np.uint8,
        device=lambda d: ("device", d),
        cuda=types.SimpleNamespace(current_stream=lambda d: log.append(d) or Stream()))

    def call(*args):
        log.append("call")
        return 4 if args[7] is None else 0  # CMPMC_ERR_CAPACITY: the sizing call

    monkeypatch.setitem(__import__("sys").modules, "torch", torch)
    monkeypatch.setattr(_ffi, "load", lambda: types.SimpleNamespace(cmpmc_gpu_partition_deposits=call))
    dep, states = _deposits(3, 1)
    cm.partition_deposits_on_device(types.SimpleNamespace(context=lambda d: 0), dep, states, device=1)
    assert log.count("call") == 2 and ("device", "cuda:1") in log
    clean = False  # a synchronize since the last allocation
    for what in log:
        if what == "call":
            assert clean, log
        clean = what == "sync" or (clean and what != "alloc")


@pytest.mark.gpu
@pytest.mark.parametrize("own_stream", [False, True])
def test_partition_beside_queued_work(ge_lattice, own_stream):
    import torch
    eng = cm.SimulationEngine(ge_lattice, cm.DetectorModel())
    dep, states = _deposits(257, 5)
    opts = cm.PartitionOptions(max_sampled_pairs=16, max_sampled_phonons=8)
    want = cm.partition_deposits_on_device(eng, dep, states, opts)
    stream = torch.cuda.Stream() if own_stream else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        a = torch.ones(1 << 26, device="cuda")
        for _ in range(200):  # some milliseconds of queued work
            a.mul_(1.0001)
        got = cm.partition_deposits_on_device(eng, dep, states, opts)
    torch.cuda.synchronize()
    for w, g in zip(want, got):
        assert w.tobytes() == g.tobytes()
