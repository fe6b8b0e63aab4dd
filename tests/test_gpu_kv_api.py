"""Device KVMap / KVVector Push/Pull API: timestamps, wait dependencies, callbacks."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_kv_vector_push_pull_timestamps_and_callbacks(cuda_lib, tmp_path):
    from parameter_server_b200.parameter.kv import DeviceKVVector
    kv = DeviceKVVector.create(table_capacity=1 << 12, max_keys=1 << 10)
    keys = np.array([3, 17, 1 << 40, (1 << 63) + 5], dtype=np.uint64)
    called = []
    t0 = kv.push(keys, [1.0, 2.0, 3.0, 4.0])
    t1 = kv.push(keys[1:3], [10.0, 20.0], callback=lambda: called.append("p1"))
    t2 = kv.pull(keys, wait=[t1], callback=lambda: called.append("pull"))
    assert (t0, t1, t2) == (0, 1, 2)
    kv.wait(t1); kv.wait(t2)
    assert called == ["p1", "pull"]
    assert kv.result(t2).cpu().tolist() == [1.0, 12.0, 23.0, 4.0]
    t3 = kv.pull(np.array([5, 17], dtype=np.uint64), ts=10)        # explicit timestamp, an absent key reads 0
    assert t3 == 10 and kv.pull(keys[:1]) == 11
    kv.wait(10)
    assert kv.result(10).cpu().tolist() == [0.0, 12.0]
    kv.write_to_file(str(tmp_path / "dump_S0"))
    lines = open(tmp_path / "dump_S0").read().splitlines()
    assert lines[0] == "3\t1" and lines[1] == "17\t12" and len(lines) == 4


def test_kv_map_ftrl_entries(cuda_lib):
    from parameter_server_b200.parallel.dataplane import OptimizerConfig
    from parameter_server_b200.parameter.kv import DeviceKVMap
    from parameter_server_b200.utils import oracle
    opt = OptimizerConfig(algo="ftrl", alpha=0.1, beta=1.0, l1=0.01, l2=0.1)
    kv = DeviceKVMap.create(table_capacity=1 << 12, max_keys=1 << 10, opt=opt)
    ot = oracle.OracleTable(opt)
    rng = np.random.default_rng(0)
    universe = np.unique(rng.integers(0, 1 << 62, 200, dtype=np.uint64))
    for _ in range(5):
        k = np.sort(rng.choice(universe, 50, replace=False))
        g = rng.normal(size=50).astype(np.float32)
        kv.push(k, g)
        ot.push(k, g)
    ts = kv.pull(universe)
    kv.wait(ts)
    assert np.allclose(kv.result(ts).cpu().numpy(), ot.pull(universe), rtol=1e-4, atol=1e-6)


def test_key_caching_inside_the_exchange_pull(cuda_lib):
    """A pull with the key list of the previous pull sends no keys: the request areas are poisoned
    after the first pull and the second still answers correctly (the owner used the slots it
    remembered); a different list afterwards is a miss and sends its keys again."""
    from parameter_server_b200.parameter.kv import DeviceKVVector
    kv = DeviceKVVector.create(table_capacity=1 << 14, max_keys=1 << 12, key_cache=True)
    plane = kv.plane
    rng = np.random.default_rng(5)
    keys = np.unique(rng.integers(0, 1 << 62, 3000, dtype=np.uint64))
    vals = rng.normal(size=len(keys)).astype(np.float32)
    kv.push(keys, vals)
    t1 = kv.pull(keys)
    kv.wait(t1)
    assert np.allclose(kv.result(t1).cpu().numpy(), vals)
    req = plane.fabric.view(plane.layout["req_keys"], (2 * plane.S * plane.cfg.inbox_cap,), torch.int64)
    req.fill_(0x1234)
    t2 = kv.pull(keys)                       # same list: a hit, nothing is read from the request areas
    kv.wait(t2)
    assert np.allclose(kv.result(t2).cpu().numpy(), vals)
    assert int((req == 0x1234).all().item()) == 1, "keys were sent although the list did not change"
    other = keys[::3]
    t3 = kv.pull(other)                      # another list: a miss
    kv.wait(t3)
    assert np.allclose(kv.result(t3).cpu().numpy(), vals[::3])
    assert int((req != 0x1234).any().item()) == 1
    t4 = kv.pull(other)                      # and a hit again, right after new values arrived
    kv.push(other, np.ones(len(other), np.float32))
    t5 = kv.pull(other)
    kv.wait(t4); kv.wait(t5)
    assert np.allclose(kv.result(t4).cpu().numpy(), vals[::3])
    assert np.allclose(kv.result(t5).cpu().numpy(), vals[::3] + 1)


@pytest.mark.parametrize("S,k,quant", [(1, 8, "none"), (3, 8, "none"), (2, 64, "none"), (3, 5, "int8")])
def test_kv_vector_of_width_k_with_channels(cuda_lib, S, k, quant):
    """KVVector with k values per key and two channels, on S emulated shards: pushes are summed per
    key over workers and rounds, pulls return (n, k) arrays, channels do not mix."""
    from parameter_server_b200.parallel.dataplane import DataPlane, OptimizerConfig, PlaneConfig, heap_layout
    from parameter_server_b200.parallel.fabric import Fabric
    from parameter_server_b200.parameter.kv import DeviceKVVector
    pc = PlaneConfig(table_capacity=1 << 12, inbox_cap=1 << 10, ring=4, pull_cap=1 << 10, width=k, channels=2, quant=quant)
    fabs = Fabric.emulated(S, heap_layout(pc, S).total())
    kvs = [DeviceKVVector(DataPlane(f, pc, OptimizerConfig(algo="sum")), 1 << 10) for f in fabs]
    rng = np.random.default_rng(S * 100 + k)
    universe = np.unique(rng.integers(0, np.iinfo(np.uint64).max, 600, dtype=np.uint64))
    state = [dict(), dict()]
    for rnd in range(3):
        chl = rnd % 2
        per = []
        for r in range(S):
            keys = np.sort(rng.choice(universe, 150, replace=False))
            vals = rng.normal(size=(len(keys), k)).astype(np.float32)
            per.append((keys, vals))
            for kk, vv in zip(keys.tolist(), vals):
                state[chl][kk] = state[chl].get(kk, np.zeros(k, np.float32)) + vv
        for r in range(S):               # emulated ranks: every worker's push first, then every owner's apply
            kv = kvs[r]
            b = kv._buffer(kv._as_keys(per[r][0], kv.dev))
            b.grad[:per[r][1].size].copy_(torch.from_numpy(per[r][1]).flatten())
            kv.plane.push(b, rnd, with_gradient=False)
        for r in range(S):
            kvs[r].plane.apply(rnd, channel=chl)
    tol = dict(rtol=1e-4, atol=1e-5) if quant == "none" else dict(rtol=0.05, atol=0.05)
    for chl in range(2):
        ask = np.sort(rng.choice(universe, 200, replace=False))
        stamps = []
        for phase in (1, 2, 4):          # the three roles of the exchange pull as separate launches
            for r in range(S):
                kv = kvs[r]
                b = kv._buffer(kv._as_keys(ask if r == 0 else np.zeros(0, np.uint64), kv.dev))
                kv.plane.pull_exchange(b, chl, need_applied=3, with_margins=False, channel=chl, phases=phase,
                                       wait_iters=1 << 12)
        torch.cuda.synchronize()
        got = kvs[0].plane.response_weights(chl, len(ask)).cpu().numpy()
        exp = np.stack([state[chl].get(kk, np.zeros(k, np.float32)) for kk in ask.tolist()])
        assert got.shape == (len(ask), k)
        assert np.allclose(got, exp, **tol), float(np.abs(got - exp).max())
    for kv in kvs:
        kv.plane.check_status()


def test_buffered_kv_vector_aggregation_idiom(cuda_lib):
    """buffer_value=True: a push round is kept per source for the owner to look at; the owner merges it
    explicitly; a later pull sees the merged sum (test/kv_vector_buffer_ps.cc:10-59)."""
    from parameter_server_b200.parameter.kv import DeviceKVVector
    kv = DeviceKVVector.create(table_capacity=1 << 12, max_keys=1 << 10, k=2, buffer_value=True)
    keys = np.array([5, 9, 1 << 50], dtype=np.uint64)
    vals = np.array([[1, 2], [3, 4], [5, 6]], dtype=np.float32)
    t0 = kv.push(keys, vals)
    t1 = kv.pull(keys)
    kv.wait(t1)
    assert float(kv.result(t1).abs().sum()) == 0.0            # nothing merged yet
    (bk, bv), = kv.buffer(t0)
    assert np.array_equal(bk, keys) and np.array_equal(bv.cpu().numpy(), vals)
    kv.apply_buffer(t0)
    kv.apply_buffer(t0)                                      # merging is the owner's decision: here twice
    t2 = kv.pull(keys)
    kv.wait(t2)
    assert np.array_equal(kv.result(t2).cpu().numpy(), 2 * vals)


@pytest.mark.parametrize("n", [1, 3, 1025, 4095, 4096])
def test_crowded_table_probes_past_collisions(cuda_lib, n):
    """Keys far from their first slot (up to a completely full table, with wrap-around): look-ups and updates
    of four keys side by side find and insert every one of them, whatever the keys of a thread collide with."""
    from parameter_server_b200.parameter.kv import DeviceKVVector
    rng = np.random.default_rng(n)
    kv = DeviceKVVector.create(None, table_capacity=4096, max_keys=4096)
    keys = np.sort(rng.choice(1 << 40, size=n, replace=False).astype(np.uint64))
    vals = rng.integers(-8, 9, size=n).astype(np.float32)
    ts = kv.push(keys, vals)                               # inserted by the push
    ts = kv.push(keys, 2 * vals, wait=[ts])                # found by the push
    got = kv.pull(keys, wait=[ts])                         # found by the pull
    kv.wait(got)
    np.testing.assert_array_equal(kv.result(got).cpu().numpy(), 3 * vals)
    kv = DeviceKVVector.create(None, table_capacity=4096, max_keys=4096)
    got = kv.pull(keys)                                    # inserted by the pull
    kv.wait(got)
    assert not kv.result(got).any()
    kv.wait(kv.push(keys, vals))
    have = dict(zip(*(t.tolist() for t in kv.plane.dump_nonzero())))
    assert have == {int(k): float(v) for k, v in zip(keys, vals) if v}


@pytest.mark.parametrize("n", [1, 31, 129, 5000])
@pytest.mark.parametrize("k,quant", [(1, "none"), (1, "int8"), (3, "none"), (3, "fp16"), (8, "none"), (8, "int8"), (64, "int8"),
                                     (64, "fp16")])
def test_request_sizes_widths_and_filters(cuda_lib, n, k, quant):
    """Requests of a few to thousands of keys on one plane, values that start off a 16-byte boundary, groups of
    32 values that end inside a row. Each of the two pushes is off by at most half a code step of its group."""
    from parameter_server_b200.parameter.kv import DeviceKVVector
    rng = np.random.default_rng(n * k)
    kv = DeviceKVVector.create(table_capacity=1 << 14, max_keys=5001, k=k, quant=quant)
    keys = np.unique(rng.integers(1, 1 << 60, 2 * n + 8).astype(np.uint64))[:n]
    vals = torch.randn(n * k + 1, device="cuda")[1:].view(n, k)
    t0 = kv.push(keys, vals)
    t1 = kv.push(keys, vals, wait=[t0])
    got = kv.pull(keys, wait=[t1])
    kv.wait(got)
    got = kv.result(got).view(n, k)
    flat = torch.nn.functional.pad(vals.flatten(), (0, -n * k % 32)).view(-1, 32)
    step = {"none": 0.0, "int8": 1 / 254, "fp16": 2.0 ** -11}[quant]
    bound = (flat.abs().amax(1, keepdim=True) * 2 * step * 1.001 + flat.abs() * 2.0 ** -22).expand_as(flat).flatten()[:n * k].view(n, k)
    assert ((got - 2 * vals).abs() <= bound).all()


@pytest.mark.parametrize("exchange", [True, False])
def test_pushed_values_of_any_stride(cuda_lib, exchange):
    """A column, a step slice and an expanded tensor are pushed as the numbers they show."""
    from parameter_server_b200.parameter.kv import DeviceKVVector
    n = 700
    keys = np.arange(1, n + 1, dtype=np.uint64) << np.uint64(40)
    m = torch.randn(2 * n, 5, device="cuda")
    for vals in (m[:n, 3], m[:n, 3:4], m[::2, 1], m.flatten()[:2 * n:2], torch.full((1,), 2.5, device="cuda").expand(n)):
        kv = DeviceKVVector.create(table_capacity=1 << 12, max_keys=n, exchange=exchange)
        kv.wait(kv.push(keys, vals))
        got = kv.pull(keys)
        kv.wait(got)
        assert torch.equal(kv.result(got), vals.flatten())
    b = kv._bufs[0]
    for bad in (m[:n, 3], m[:n].double(), m.flatten()[:n - 1]):
        with pytest.raises(AssertionError):
            kv.plane.push(b, 100, with_gradient=False, values=bad)


@pytest.mark.parametrize("k", [1, 8])
def test_push_only_values_may_be_overwritten_after_the_call(cuda_lib, k):
    """The worker half of a push records no event: values that the caller's stream writes before and after the call,
    while the container's stream is still busy with something else, are pushed as they were at the call."""
    from parameter_server_b200.parameter.kv import DeviceKVVector
    n = 3000
    kv = DeviceKVVector.create(table_capacity=1 << 13, max_keys=n, k=k)
    keys = torch.arange(1, n + 1, device="cuda") << 40
    vals = torch.zeros(n * k, device="cuda")
    for rnd in range(3):
        with torch.cuda.stream(kv.stream):
            torch.cuda._sleep(20_000_000)                  # about ten milliseconds
        torch.cuda._sleep(2_000_000)
        vals.fill_(rnd + 1.0)                              # not there yet when push_only is called
        r = kv.push_only(keys, vals.view(n, k))
        vals.fill_(100.0)
        kv.apply_round(r)
    got = kv.pull(keys)
    kv.wait(got)
    assert (kv.result(got) == 6.0).all()


def test_memory_of_a_key_list_is_not_reused_before_it_is_read(cuda_lib):
    """Requests run ahead of the container's stream: the device copy of the first one's keys is let go when the
    second one comes, and the caller's stream allocates and writes tensors of the same size meanwhile."""
    from parameter_server_b200.parameter.kv import DeviceKVVector
    n = 5000
    kv = DeviceKVVector.create(table_capacity=1 << 15, max_keys=n)
    lists = [np.arange(1 + i * n, 1 + (i + 1) * n, dtype=np.uint64) << np.uint64(32) for i in range(3)]
    with torch.cuda.stream(kv.stream):
        torch.cuda._sleep(40_000_000)                      # about twenty milliseconds
    junk, ts = [], []
    for i, keys in enumerate(lists):
        ts.append(kv.push(keys, np.full(n, i + 1, np.float32)))
        junk += [torch.full((n,), 7, dtype=torch.int64, device="cuda") for _ in range(4)]
    torch.cuda.current_stream().synchronize()
    for t in ts:
        kv.wait(t)
    for i, keys in enumerate(lists):
        got = kv.pull(keys)
        kv.wait(got)
        assert (kv.result(got) == i + 1.0).all(), i


def test_wait_reports_the_status_that_a_pull_left(cuda_lib):
    """The status word travels with the pull; an error in it is raised once and cleared, as when wait() reads the word itself."""
    from parameter_server_b200.ops._lib import PsbCudaError
    from parameter_server_b200.parameter.kv import DeviceKVVector
    kv = DeviceKVVector.create(table_capacity=1 << 12, max_keys=1 << 10)
    keys = torch.arange(1, 6, dtype=torch.int64, device="cuda")
    pushed = kv.push(keys, torch.ones(5, device="cuda"))
    kv.plane.status.fill_(1)
    first, second = kv.pull(keys), kv.pull(keys, wait=[pushed])
    with pytest.raises(PsbCudaError):
        kv.wait(first)
    kv.wait(second)
    kv.wait(pushed)
    assert kv.result(second).tolist() == [1.0] * 5
    kv.plane.status.fill_(1)
    again = kv.push(keys, torch.ones(5, device="cuda"))
    with pytest.raises(PsbCudaError):
        kv.wait(again)                                 # (behind a push the word is read by wait())


def test_no_wait_takes_back_what_another_pull_left(cuda_lib, monkeypatch):
    """A pull that fails while wait() of another request looks at the status word is still reported by its own wait()."""
    from parameter_server_b200.ops._lib import PsbCudaError
    from parameter_server_b200.parameter.kv import DeviceKVVector
    kv = DeviceKVVector.create(table_capacity=1 << 12, max_keys=1 << 10)
    keys = torch.arange(1, 6, dtype=torch.int64, device="cuda")
    pushed, pulled = kv.push(keys, torch.ones(5, device="cuda")), []
    look = kv.plane.check_status

    def and_then_a_pull_fails(what):
        look(what)
        kv.plane.status.fill_(1)
        pulled.append(kv.pull(keys))
        torch.cuda.synchronize()
    with monkeypatch.context() as m:
        m.setattr(kv.plane, "check_status", and_then_a_pull_fails)
        kv.wait(pushed)
    with pytest.raises(PsbCudaError):
        kv.wait(pulled[0])


def test_status_words_of_pulls_that_nobody_waits_for(cuda_lib):
    """More pulls in flight than there are words, discarded ones, and a push with the timestamp of a pull."""
    from parameter_server_b200.ops._lib import PsbCudaError
    from parameter_server_b200.parameter.kv import DeviceKVVector
    kv = DeviceKVVector.create(table_capacity=1 << 12, max_keys=1 << 10)
    keys = torch.arange(1, 6, dtype=torch.int64, device="cuda")
    kv.push(keys, torch.ones(5, device="cuda"))
    pulls = [kv.pull(keys) for _ in range(150)]
    for ts in pulls[:50]:
        kv.discard(ts)
    kv.plane.status.fill_(1)
    bad = [kv.pull(keys) for _ in range(100)]
    with pytest.raises(PsbCudaError):
        kv.wait(bad[0])
    for ts in bad[1:] + pulls[50:]:
        kv.wait(ts)
        assert kv.result(ts).tolist() == [1.0] * 5
    assert kv.pull(keys, ts=7000) == kv.push(keys, torch.ones(5, device="cuda"), ts=7000)
    torch.cuda.synchronize()
    kv.plane.status.fill_(1)
    with pytest.raises(PsbCudaError):
        kv.wait(7000)


def test_a_dropped_container_gives_its_pinned_words_back_when_idle(cuda_lib):
    """A container dropped with a pull in flight, which still has its status word to write, ends behind it."""
    import weakref
    from parameter_server_b200.parameter.kv import DeviceKVVector
    kv = DeviceKVVector.create(table_capacity=1 << 12, max_keys=1 << 10)
    keys = torch.arange(1, 6, dtype=torch.int64, device="cuda")
    busy = torch.zeros(1 << 26, device="cuda")
    kv.wait(kv.pull(keys))
    for _ in range(200):                               # about 16 ms in front of the pull
        busy += 1
    kv.pull(keys)
    stream, words, plane = kv.stream, kv._status_host, kv.plane      # (a plane that goes too waits for the device)
    gone = weakref.ref(kv)
    del kv
    assert gone() is None and stream.query() and not words.any()


def test_on_stream_is_left_as_it_was_entered(cuda_lib):
    from parameter_server_b200.ops._lib import on_stream, run_behind
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    before = torch.cuda.current_stream()
    with on_stream(a):
        assert torch.cuda.current_stream() == a
        with pytest.raises(ZeroDivisionError), on_stream(b):
            assert torch.cuda.current_stream() == b
            1 / 0
        assert torch.cuda.current_stream() == a
        with on_stream(None):
            assert torch.cuda.current_stream() == a
    assert torch.cuda.current_stream() == before
    x = torch.zeros(1 << 24, device="cuda")
    run_behind(a, before)
    with on_stream(a):
        for _ in range(50):
            x += 1
    run_behind(before, a)
    assert float(x.sum()) == 50.0 * x.numel()
