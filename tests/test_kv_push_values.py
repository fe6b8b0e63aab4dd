"""The values that a device KV container hands to its push kernel, which reads adjacent floats from one address."""
import contextlib
import types

import numpy as np
import pytest
import torch


class _Plane:
    """Stands in for the data plane: reads the values as the kernel does."""

    def __init__(self):
        self.read = None

    def push(self, b, rnd, *, with_gradient, values, stream):
        n = b.n
        self.values = values
        self.read = values.detach().as_strided((n,), (1,), values.storage_offset()) if n else None


class _Buffer:
    def __init__(self, n):
        self.n = n


def _container(n, k):
    from parameter_server_b200.parameter.kv import DeviceKVVector
    kv = DeviceKVVector.__new__(DeviceKVVector)
    kv.dev, kv.k, kv.stream, kv._round, kv.plane = torch.device("cpu"), k, None, 0, _Plane()
    kv._buffer = lambda keys: _Buffer(n * k)
    return kv


def _forms(n, k):
    m = torch.arange(4.0 * n * k).view(n * k, 4)
    yield "column", m[:, 1]
    yield "column as a matrix", m[:, 1:2]
    yield "every second", torch.arange(2.0 * n * k)[::2]
    yield "expanded scalar", torch.full((1,), 3.0).expand(n * k)
    yield "expanded row", torch.arange(float(k)).expand(n, k)
    yield "transposed", torch.arange(float(n * k)).view(k, n).t()
    yield "part of wider rows", torch.arange(float(n * (k + 3))).view(n, k + 3)[:, 1:1 + k]
    yield "behind an offset", torch.arange(n * k + 1.0)[1:]
    yield "double", torch.arange(n * k, dtype=torch.float64)[:]
    yield "needs a gradient", torch.arange(float(n * k), requires_grad=True)
    yield "imaginary parts of a conjugate", torch.complex(torch.zeros(n * k), torch.arange(float(n * k))).conj().imag
    yield "numpy column", np.arange(2.0 * n * k, dtype=np.float32).reshape(n * k, 2)[:, 1]


@pytest.mark.parametrize("n,k", [(1, 1), (7, 1), (5, 3), (4, 8)])
def test_push_hands_adjacent_floats_to_the_kernel(n, k):
    for name, values in _forms(n, k):
        kv = _container(n, k)
        kv._push_half(torch.arange(n), values)
        want = torch.as_tensor(values).detach().to(torch.float32).reshape(-1)
        assert torch.equal(kv.plane.read, want), name


@pytest.mark.parametrize("n,k", [(7, 1), (5, 3)])
def test_push_only_leaves_the_caller_its_values(monkeypatch, n, k):
    """Nothing tells the caller of push_only when its values have been read: the kernel gets a copy of its own, made in
    the order of the caller's stream, and the container's stream starts behind that stream."""
    kv = _container(n, k)
    waited = []
    kv._begin = waited.append
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    for name, values in _forms(n, k):
        want = torch.as_tensor(values).detach().to(torch.float32).reshape(-1).clone()
        kv.push_only(torch.arange(n), values)
        if not isinstance(values, torch.Tensor):
            values = torch.from_numpy(values)
        with torch.no_grad():
            base = values._base if values._base is not None else values
            base.fill_(77.0)
        assert torch.equal(kv.plane.values.detach(), want), name
        assert waited.pop() is None and not waited
    kv = _container(0, k)
    kv._begin = waited.append
    assert kv.push_only(torch.arange(0), None) == 0        # a round without keys needs no values


@pytest.mark.parametrize("current,container", [(0, 0), (0, 1), (1, 0)])
def test_push_enters_a_stream_of_another_device(monkeypatch, current, container):
    """Values and keys that are read where they are spare a push the entry into its stream, but not where another device than
    the container's is the current one: entering makes its device the current one."""
    from parameter_server_b200.ops import _lib
    kv = _container(5, 1)
    kv.stream = types.SimpleNamespace(device=torch.device("cuda", container))
    kv._time, kv._push_round_of = -1, {}
    kv._begin = kv._finish = lambda *a: None
    kv._apply_half = lambda rnd, channel: None
    kv._in_place = lambda values: True
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current)
    entered = []
    monkeypatch.setattr(_lib, "on_stream", lambda s: entered.append(s) or contextlib.nullcontext())
    kv.push(torch.arange(5), torch.ones(5))
    assert entered == [None if current == container else kv.stream]
    kv.push(torch.arange(5, dtype=torch.int32), torch.ones(5))
    assert entered[1] is kv.stream
