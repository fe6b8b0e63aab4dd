"""Radix sort and minibatch localisation against NumPy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand_keys(n, rng, skew=False, bits=64):
    if skew:
        ids = (rng.pareto(1.05, n) * 3).astype(np.uint64) % np.uint64(1 << 20)
        from parameter_server_b200.utils.oracle import hash_id_to_key
        k = hash_id_to_key(ids, 7)
    else:
        k = rng.integers(0, 1 << 63, n, dtype=np.uint64) * np.uint64(2) + rng.integers(0, 2, n, dtype=np.uint64)
    if bits < 64:
        k = k >> np.uint64(64 - bits)
    return k


@pytest.mark.parametrize("n", [1, 31, 4096, 4097, 100_003, 1_500_000])
@pytest.mark.parametrize("skew", [False, True])
def test_sort_pairs_matches_numpy(cuda_lib, n, skew):
    from parameter_server_b200.ops.localize import sort_pairs
    rng = np.random.default_rng(n + skew)
    k = _rand_keys(n, rng, skew)
    kt = torch.from_numpy(k.view(np.int64)).cuda()
    sk, sv = sort_pairs(kt)
    torch.cuda.synchronize()
    order = np.argsort(k, kind="stable")
    assert np.array_equal(sk.cpu().numpy().view(np.uint64), k[order])
    assert np.array_equal(sv.cpu().numpy().astype(np.int64), order)  # stable => identical permutation


def test_sort_partial_bits_and_payload(cuda_lib):
    from parameter_server_b200.ops.localize import sort_pairs
    rng = np.random.default_rng(3)
    n = 50_000
    k = _rand_keys(n, rng, bits=26)
    pay = rng.integers(0, 1 << 31, n, dtype=np.int64).astype(np.int32)
    sk, sv = sort_pairs(torch.from_numpy(k.view(np.int64)).cuda(), torch.from_numpy(pay).cuda(), 0, 26)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(sk.cpu().numpy().view(np.uint64), k[order])
    assert np.array_equal(sv.cpu().numpy(), pay[order])


@pytest.mark.parametrize("S", [1, 2, 8])
@pytest.mark.parametrize("fixed", [True, False])
def test_localize_matches_numpy(cuda_lib, S, fixed):
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.utils.range import Range, shard_bounds
    rng = np.random.default_rng(11 + S)
    rows, z = 700, 37
    if fixed:
        row_ptr = np.arange(rows + 1) * z
    else:
        lens = rng.integers(0, 2 * z, rows)
        row_ptr = np.concatenate([[0], np.cumsum(lens)])
    nnz = int(row_ptr[-1])
    keys = _rand_keys(nnz, rng, skew=True)
    vals = rng.random(nnz, dtype=np.float32)
    b = LocalBatch(rows, nnz, S, "cuda", real_values=True)
    bounds_h = shard_bounds(Range.all(), S)
    bounds = torch.tensor([x if x < (1 << 63) else x - (1 << 64) for x in bounds_h], dtype=torch.int64).cuda()
    ids = torch.from_numpy(keys.view(np.int64)).cuda()
    kw = dict(fixed_z=z) if fixed else dict(row_ptr=torch.from_numpy(row_ptr.astype(np.int32)).cuda())
    b.localize(ids, None, bounds, vals=torch.from_numpy(vals).cuda(), hash_seed=None, method="sort", **kw)
    torch.cuda.synchronize()
    u, inv, cnt = np.unique(keys, return_inverse=True, return_counts=True)
    U = int(b.n_unique.item())
    assert U == len(u)
    assert np.array_equal(b.ukeys[:U].cpu().numpy().view(np.uint64), u)
    assert np.array_equal(b.csr_col[:nnz].cpu().numpy(), inv)
    seg = b.seg_off[:U + 1].cpu().numpy()
    assert np.array_equal(np.diff(seg), cnt)
    # CSC rows/values: each segment lists the rows containing that key, in position order
    rows_of = np.repeat(np.arange(rows), np.diff(row_ptr))
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(b.csc_row[:nnz].cpu().numpy(), rows_of[order])
    assert np.allclose(b.csc_val[:nnz].cpu().numpy(), vals[order])
    own = b.own_off.cpu().numpy()
    exp = [int(np.searchsorted(u, np.uint64(x))) for x in bounds_h[:-1]] + [U]
    assert list(own) == exp
    # head bitmap consistent with segment offsets
    fb = b.flagbits[:(nnz + 31) // 32].cpu().numpy().view(np.uint32)
    heads = np.zeros(nnz, dtype=bool); heads[seg[:-1]] = True
    bits = np.unpackbits(fb.view(np.uint8), bitorder="little")[:nnz].astype(bool)
    assert np.array_equal(bits, heads)
    wb = b.wordbase[:(nnz + 31) // 32].cpu().numpy()
    assert np.array_equal(wb, np.concatenate([[0], np.cumsum(heads)])[0:nnz:32])


def test_hash_on_device_matches_oracle(cuda_lib):
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.utils.oracle import hash_id_to_key
    rng = np.random.default_rng(5)
    ids = rng.integers(0, 1 << 26, 64 * 50, dtype=np.int64).astype(np.int32)
    b = LocalBatch(64, ids.size, 1, "cuda")
    bounds = torch.tensor([0, -1], dtype=torch.int64).cuda()
    b.localize(torch.from_numpy(ids).cuda(), None, bounds, fixed_z=50, hash_seed=9)
    U = int(b.n_unique.item())
    assert np.array_equal(b.ukeys[:U].cpu().numpy().view(np.uint64), np.unique(hash_id_to_key(ids, 9)))


def test_sort_skips_constant_digits_and_narrow_hash(cuda_lib):
    """Keys with 40 significant bits (top bits): the three low digit passes are
    skipped on the device, the result is still the stable sorted order; and the
    device hash with 40 bits matches the NumPy restatement."""
    from parameter_server_b200.ops.localize import LocalBatch, sort_pairs
    from parameter_server_b200.utils.oracle import hash_id_to_key
    rng = np.random.default_rng(8)
    ids = rng.integers(0, 1 << 26, 64 * 300, dtype=np.int64).astype(np.int32)
    k = hash_id_to_key(ids, 0, 40)
    sk, sv = sort_pairs(torch.from_numpy(k.view(np.int64)).cuda())
    order = np.argsort(k, kind="stable")
    assert np.array_equal(sk.cpu().numpy().view(np.uint64), k[order])
    assert np.array_equal(sv.cpu().numpy().astype(np.int64), order)
    # already sorted input with identical keys: every pass is skipped, payload = index
    same = torch.full((5000,), 77, dtype=torch.int64, device="cuda")
    sk2, sv2 = sort_pairs(same)
    assert torch.equal(sv2.cpu(), torch.arange(5000, dtype=torch.int32)) and torch.equal(sk2, same)
    b = LocalBatch(64, ids.size, 2, "cuda")
    bounds = torch.tensor([0, -(1 << 63), -1], dtype=torch.int64).cuda()
    b.localize(torch.from_numpy(ids).cuda(), None, bounds, fixed_z=300, hash_seed=0, hash_bits=40, method="sort")
    U = int(b.n_unique.item())
    u = np.unique(k)
    assert np.array_equal(b.ukeys[:U].cpu().numpy().view(np.uint64), u)
    assert b.own_off.cpu().tolist() == [0, int(np.searchsorted(u, np.uint64(1 << 63))), U]
    rows_of = np.repeat(np.arange(64), 300)
    assert np.array_equal(b.csc_row[:ids.size].cpu().numpy(), rows_of[order])


@pytest.mark.parametrize("hash_bits,rows,z", [(40, 512, 100), (48, 300, 37), (20, 200, 64)])
def test_packed_positions_match_pair_sort(cuda_lib, hash_bits, rows, z):
    """Narrow hashed keys: sorting (key | position) single words gives exactly the
    same localised batch as sorting (key, position) pairs."""
    from parameter_server_b200.ops.localize import LocalBatch
    rng = np.random.default_rng(31)
    ids = (rng.zipf(1.3, rows * z) % (1 << 22)).astype(np.int32)
    vals = rng.random(rows * z, dtype=np.float32)
    bounds = torch.tensor([0, 1 << 62, -(1 << 63), -1], dtype=torch.int64).cuda()
    out = []
    for packed in (True, False):
        b = LocalBatch(rows, ids.size, 3, "cuda", real_values=True)
        b.localize(torch.from_numpy(ids).cuda(), None, bounds, fixed_z=z, vals=torch.from_numpy(vals).cuda(),
                   hash_seed=3, hash_bits=hash_bits, key_bits=(64 - hash_bits, 64), packed=packed, method="sort")
        torch.cuda.synchronize()
        assert (b.pack_bits > 0) == packed
        U = int(b.n_unique.item())
        out.append((U, b.ukeys[:U].cpu(), b.seg_off[:U + 1].cpu(), b.csr_col[:ids.size].cpu(),
                    b.csc_row[:ids.size].cpu(), b.csc_val[:ids.size].cpu(), b.own_off.cpu(),
                    b.flagbits[:(ids.size + 31) // 32].cpu(), b.wordbase[:(ids.size + 31) // 32].cpu()))
    assert out[0][0] == out[1][0] and out[0][0] > 1
    for x, y in zip(out[0][1:], out[1][1:]):
        assert torch.equal(x, y)


def _check_grouped(b, keys, row_ptr, vals, bounds_h, rows):
    """Every output of a localised batch against NumPy, with the rows of a key's
    CSC segment compared as a set (the bucket path does not order them)."""
    nnz = keys.size
    u, inv, cnt = np.unique(keys, return_inverse=True, return_counts=True)
    U = int(b.n_unique.item())
    assert U == len(u)
    assert np.array_equal(b.ukeys[:U].cpu().numpy().view(np.uint64), u)
    assert np.array_equal(b.csr_col[:nnz].cpu().numpy(), inv)
    seg = b.seg_off[:U + 1].cpu().numpy().astype(np.int64)
    assert seg[0] == 0 and seg[-1] == nnz
    assert np.array_equal(np.diff(seg), cnt)
    rows_of = np.repeat(np.arange(rows), np.diff(row_ptr))
    order = np.argsort(keys, kind="stable")
    seg_id = np.repeat(np.arange(U), cnt)
    got_rows = b.csc_row[:nnz].cpu().numpy().astype(np.int64)
    exp_rows = rows_of[order]
    if vals is None:
        assert np.array_equal(np.sort(seg_id * (rows + 1) + got_rows), np.sort(seg_id * (rows + 1) + exp_rows))
    else:
        # (row, value) pairs per segment, as sets
        got_v = b.csc_val[:nnz].cpu().numpy()
        g = np.lexsort((got_v, got_rows, seg_id))
        e = np.lexsort((vals[order], exp_rows, seg_id))
        assert np.array_equal(got_rows[g], exp_rows[e])
        assert np.array_equal(got_v[g], vals[order][e])
    own = b.own_off.cpu().numpy()
    assert list(own) == [int(np.searchsorted(u, np.uint64(x))) for x in bounds_h[:-1]] + [U]
    fb = b.flagbits[:(nnz + 31) // 32].cpu().numpy().view(np.uint32)
    heads = np.zeros(nnz, dtype=bool); heads[seg[:-1]] = True
    bits = np.unpackbits(fb.view(np.uint8), bitorder="little")[:nnz].astype(bool)
    assert np.array_equal(bits, heads)
    wb = b.wordbase[:(nnz + 31) // 32].cpu().numpy()
    assert np.array_equal(wb, np.concatenate([[0], np.cumsum(heads)])[0:nnz:32])


def _bounds(S):
    from parameter_server_b200.utils.range import Range, shard_bounds
    bounds_h = shard_bounds(Range.all(), S)
    return bounds_h, torch.tensor([x if x < (1 << 63) else x - (1 << 64) for x in bounds_h], dtype=torch.int64).cuda()


@pytest.mark.parametrize("hash_bits,rows,z,S", [(40, 2048, 100, 1), (40, 4096, 200, 8), (0, 1500, 64, 3), (52, 700, 37, 2)])
def test_bucket_localize_hashed_ids(cuda_lib, hash_bits, rows, z, S):
    """Bucket path on device-hashed ids with a heavy head (frequent keys go through
    the counting path, the rest through the per-bucket tables)."""
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.utils.oracle import hash_id_to_key
    rng = np.random.default_rng(hash_bits + rows)
    ids = (rng.zipf(1.2, rows * z) % (1 << 24)).astype(np.int32)
    keys = hash_id_to_key(ids, 5, hash_bits or 64)
    bounds_h, bounds = _bounds(S)
    b = LocalBatch(rows, ids.size, S, "cuda")
    b.localize(torch.from_numpy(ids).cuda(), None, bounds, fixed_z=z, hash_seed=5, hash_bits=hash_bits, method="bucket")
    torch.cuda.synchronize()
    assert int(b.gate.item()) == 0, "the bucket path gave up on evenly spread keys"
    assert int(b.status.item()) == 0
    _check_grouped(b, keys, np.arange(rows + 1) * z, None, bounds_h, rows)


def test_bucket_localize_raw_keys_rows_and_values(cuda_lib):
    """Raw 64-bit keys (no device hash, positions in their own array), CSR row
    offsets and real values."""
    from parameter_server_b200.ops.localize import LocalBatch
    rng = np.random.default_rng(77)
    rows = 3000
    lens = rng.integers(0, 60, rows)
    row_ptr = np.concatenate([[0], np.cumsum(lens)])
    nnz = int(row_ptr[-1])
    keys = _rand_keys(nnz, rng, skew=True)
    vals = rng.random(nnz, dtype=np.float32)
    bounds_h, bounds = _bounds(4)
    b = LocalBatch(rows, nnz, 4, "cuda", real_values=True)
    b.localize(torch.from_numpy(keys.view(np.int64)).cuda(), None, bounds,
               row_ptr=torch.from_numpy(row_ptr.astype(np.int32)).cuda(), vals=torch.from_numpy(vals).cuda(),
               hash_seed=None, method="bucket")
    torch.cuda.synchronize()
    assert int(b.gate.item()) == 0 and int(b.status.item()) == 0
    _check_grouped(b, keys, row_ptr, vals, bounds_h, rows)


def test_bucket_localize_all_distinct_and_all_equal(cuda_lib):
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.utils.oracle import hash_id_to_key
    bounds_h, bounds = _bounds(2)
    rows, z = 1024, 64
    for ids in (np.arange(rows * z, dtype=np.int32), np.full(rows * z, 12345, dtype=np.int32)):
        keys = hash_id_to_key(ids, 1, 40)
        b = LocalBatch(rows, ids.size, 2, "cuda")
        b.localize(torch.from_numpy(ids).cuda(), None, bounds, fixed_z=z, hash_seed=1, hash_bits=40, method="bucket")
        torch.cuda.synchronize()
        assert int(b.gate.item()) == 0 and int(b.status.item()) == 0
        _check_grouped(b, keys, np.arange(rows + 1) * z, None, bounds_h, rows)


def test_auto_falls_back_to_sort_on_clustered_keys(cuda_lib):
    """Small integer keys all fall into the first bucket: the bucket path raises its
    flag on the device and the gated sort path produces the result."""
    from parameter_server_b200.ops.localize import LocalBatch
    rng = np.random.default_rng(9)
    rows, z = 2000, 50
    keys = rng.integers(1, 200_000, rows * z, dtype=np.int64).astype(np.uint64)
    bounds_h, bounds = _bounds(2)
    b = LocalBatch(rows, keys.size, 2, "cuda")
    b.localize(torch.from_numpy(keys.view(np.int64)).cuda(), None, bounds, fixed_z=z, hash_seed=None, method="auto")
    torch.cuda.synchronize()
    assert int(b.gate.item()) == 1 and int(b.status.item()) == 0
    _check_grouped(b, keys, np.arange(rows + 1) * z, None, bounds_h, rows)
    # the same buffers, next minibatch with spread keys: the bucket path runs again
    keys2 = _rand_keys(rows * z, rng, skew=True)
    b.localize(torch.from_numpy(keys2.view(np.int64)).cuda(), None, bounds, fixed_z=z, hash_seed=None, method="auto")
    torch.cuda.synchronize()
    assert int(b.gate.item()) == 0 and int(b.status.item()) == 0
    _check_grouped(b, keys2, np.arange(rows + 1) * z, None, bounds_h, rows)


@pytest.mark.parametrize("hash_bits", [None, 40, 0])
@pytest.mark.parametrize("lens", ["one_row", "empty_rows", "one_each", "last_rows_empty", "long_then_short"])
def test_bucket_localize_rows_of_all_lengths(cuda_lib, lens, hash_bits):
    """The row of a nonzero, found between the hints of its block of 32 positions and of the next one, and carried
    with its position: raw keys, hashed ids with room for positions in the keys, and without."""
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.utils.oracle import hash_id_to_key
    rng = np.random.default_rng(5)
    n = {"one_row": [5003], "empty_rows": (rng.random(40000) < 0.13) * rng.integers(1, 3, 40000), "one_each": np.ones(4097, int),
         "last_rows_empty": np.concatenate([rng.integers(0, 9, 1500), np.zeros(700, int)]),
         "long_then_short": np.concatenate([[6000], rng.integers(0, 4, 900)])}[lens]
    row_ptr = np.concatenate([[0], np.cumsum(n)])
    rows, nnz = len(n), int(row_ptr[-1])
    if hash_bits is None:
        keys = _rand_keys(nnz, rng, skew=True)
        ids = keys.view(np.int64)
    else:
        ids = (rng.zipf(1.3, nnz) % (1 << 22)).astype(np.int32)
        keys = hash_id_to_key(ids, 3, hash_bits or 64)
    bounds_h, bounds = _bounds(2)
    b = LocalBatch(rows, nnz, 2, "cuda")
    b.localize(torch.from_numpy(ids).cuda(), None, bounds, row_ptr=torch.from_numpy(row_ptr.astype(np.int32)).cuda(),
               hash_seed=None if hash_bits is None else 3, hash_bits=hash_bits or 0, method="bucket")
    torch.cuda.synchronize()
    assert nnz >= b.BUCKET_MIN_NNZ and int(b.gate.item()) == 0 and int(b.status.item()) == 0
    _check_grouped(b, keys, row_ptr, None, bounds_h, rows)


@pytest.mark.parametrize("n", [4096, 4097, 16385, 65537, 131071, 262144, 262145, 900001])
@pytest.mark.parametrize("hash_bits", [40, 0])
def test_bucket_localize_sizes(cuda_lib, n, hash_bits):
    """Around the sizes at which the number of buckets, the sample and the walk grid change."""
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.utils.oracle import hash_id_to_key
    rng = np.random.default_rng(n)
    ids = (rng.zipf(1.3, n) % (1 << 22)).astype(np.int32)
    keys = hash_id_to_key(ids, 3, hash_bits or 64)
    bounds_h, bounds = _bounds(3)
    b = LocalBatch(n, n, 3, "cuda")
    for _ in range(2):
        b.localize(torch.from_numpy(ids).cuda(), None, bounds, fixed_z=1, hash_seed=3, hash_bits=hash_bits, method="auto")
        torch.cuda.synchronize()
        assert int(b.gate.item()) == 0 and int(b.status.item()) == 0
        _check_grouped(b, keys, np.arange(n + 1), None, bounds_h, n)


@pytest.mark.parametrize("n", [4096, 5001, 70000, 1500001])
def test_gated_sort_path_sizes(cuda_lib, n):
    """The sort-based path behind the gate, one launch for the sort and one for the rest, from less than a tile
    to more tiles than CTAs; the barrier words it shares with the next call are left as they were."""
    from parameter_server_b200.ops.localize import LocalBatch
    rng = np.random.default_rng(n)
    bounds_h, bounds = _bounds(2)
    b = LocalBatch(n, n, 2, "cuda", real_values=True)
    for _ in range(3):
        keys = rng.integers(1, 1 + n // 3, n, dtype=np.int64).astype(np.uint64)
        vals = rng.random(n, dtype=np.float32)
        b.localize(torch.from_numpy(keys.view(np.int64)).cuda(), None, bounds, fixed_z=1, hash_seed=None,
                   vals=torch.from_numpy(vals).cuda(), method="auto")
        torch.cuda.synchronize()
        assert int(b.gate.item()) == 1 and int(b.status.item()) == 0
        _check_grouped(b, keys, np.arange(n + 1), vals, bounds_h, n)


@pytest.mark.parametrize("n,method,hash_bits,ragged", [(5000, "auto", 40, False), (5000, "auto", 0, True), (5000, "bucket", 40, True),
                                                       (5000, "sort", 40, False), (5000, "sort", 0, False), (100, "auto", 40, False)])
def test_localize_counts_its_launches(cuda_lib, n, method, hash_bits, ragged):
    """The launch counter grows by the number of kernels that a captured call consists of."""
    from parameter_server_b200.ops import _lib
    from parameter_server_b200.ops.localize import LocalBatch
    rt = pytest.importorskip("cuda.bindings.runtime")
    ids = torch.randint(0, 1 << 20, (n,), dtype=torch.int32, device="cuda")
    rows = {"row_ptr": torch.arange(0, n + 1, 10, dtype=torch.int32, device="cuda")} if ragged else {"fixed_z": 10}
    _, bounds = _bounds(2)
    b = LocalBatch(n, n, 2, "cuda")
    b.localize(ids, None, bounds, hash_seed=3, hash_bits=hash_bits, method=method, **rows)
    torch.cuda.synchronize()
    before = _lib.LAUNCHES
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        b.localize(ids, None, bounds, hash_seed=3, hash_bits=hash_bits, method=method, **rows)
    graph = rt.cudaGraph_t(init_value=g.raw_cuda_graph())
    _, _, count = rt.cudaGraphGetNodes(graph)
    _, nodes, _ = rt.cudaGraphGetNodes(graph, count)
    kernels = sum(rt.cudaGraphNodeGetType(x)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for x in nodes)
    assert kernels == _lib.LAUNCHES - before


@pytest.mark.parametrize("split", [0, 1, 2, 3])
def test_bucket_localize_long_run_of_empty_rows(cuda_lib, split):
    """300,000 empty rows between two nonzeros, wherever the gap lies among the four nonzeros of a thread: the rows
    are right, and no thread walks the gap row by row (70 ns a row: 21 ms; all of it takes 0.1 ms)."""
    from parameter_server_b200.ops.localize import LocalBatch
    rng = np.random.default_rng(split)
    n = np.concatenate([np.full(900, 4), [1 + split], np.zeros(300000, int), np.full(900, 4)])
    row_ptr = np.concatenate([[0], np.cumsum(n)])
    rows, nnz = len(n), int(row_ptr[-1])
    keys = _rand_keys(nnz, rng, skew=True)
    bounds_h, bounds = _bounds(2)
    b = LocalBatch(rows, nnz, 2, "cuda")
    ids, rp = torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(row_ptr.astype(np.int32)).cuda()
    ms = []
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        b.localize(ids, None, bounds, row_ptr=rp, hash_seed=None, method="bucket")
        e1.record()
        e1.synchronize()
        ms.append(e0.elapsed_time(e1))
    assert int(b.gate.item()) == 0 and int(b.status.item()) == 0
    _check_grouped(b, keys, row_ptr, None, bounds_h, rows)
    assert min(ms) < 5.0


@pytest.mark.parametrize("lens", [[150_001], [8192], [8193], [16384, 8192, 24_576], [3, 8192, 5, 8193, 1, 16384, 0, 0, 22_501, 7, 70_000, 31],
                                  [0, 1, 10_000, 0, 0, 8191, 8250, 100, 200_000, 0]])
def test_bucket_localize_very_long_rows(cuda_lib, lens):
    """Row hints beyond a warp's share: rows around 8192 positions and far beyond, wherever they begin and end."""
    from parameter_server_b200.ops.localize import LocalBatch
    rng = np.random.default_rng(len(lens))
    lens = np.concatenate([lens, rng.integers(0, 40, 3000)]) if len(lens) > 3 else np.array(lens)
    row_ptr = np.concatenate([[0], np.cumsum(lens)])
    rows, nnz = len(lens), int(row_ptr[-1])
    keys = _rand_keys(nnz, rng, skew=True)
    bounds_h, bounds = _bounds(2)
    b = LocalBatch(rows, nnz, 2, "cuda")
    b.bucket_scratch.fill_(255)
    b.localize(torch.from_numpy(keys.view(np.int64)).cuda(), None, bounds, row_ptr=torch.from_numpy(row_ptr.astype(np.int32)).cuda(),
               method="bucket")
    torch.cuda.synchronize()
    assert int(b.gate.item()) == 0 and int(b.status.item()) == 0
    _check_grouped(b, keys, row_ptr, None, bounds_h, rows)


@pytest.mark.parametrize("method", ["bucket", "sort"])
@pytest.mark.parametrize("n", [4096, 200_001])
def test_nonzeros_without_rows_are_row_0s(cuda_lib, n, method):
    """Row offsets of one element: no row to look for, and nothing of the offsets or the row hints is read."""
    from parameter_server_b200.ops.localize import LocalBatch
    rng = np.random.default_rng(n)
    keys = _rand_keys(n, rng, skew=True)
    bounds_h, bounds = _bounds(2)
    b = LocalBatch(1, n, 2, "cuda")
    b.bucket_scratch.fill_(255)                        # (hints of another minibatch)
    b.localize(torch.from_numpy(keys.view(np.int64)).cuda(), None, bounds, row_ptr=torch.zeros(1, dtype=torch.int32, device="cuda"),
               method=method)
    torch.cuda.synchronize()
    assert int(b.gate.item()) == 0 and int(b.status.item()) == 0
    u, inv = np.unique(keys, return_inverse=True)
    assert np.array_equal(b.ukeys[:len(u)].cpu().numpy().view(np.uint64), u)
    assert np.array_equal(b.csr_col[:n].cpu().numpy(), inv) and not b.csc_row[:n].any()


@pytest.mark.parametrize("values", [False, True])
@pytest.mark.parametrize("hash_bits,rows", [(40, 3000), (52, 4096), (52, 4097), (24, 3001), (0, 3000)])
@pytest.mark.parametrize("ragged", [False, True])
def test_bucket_localize_what_travels_beside_a_key(cuda_lib, ragged, hash_bits, rows, values):
    """A row rides in the zero bits of its key as long as every row fits (4096 rows in 12 bits, 4097 do not), else
    beside it; a value always beside it."""
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.utils.oracle import hash_id_to_key
    rng = np.random.default_rng(rows + values)
    n = rng.integers(0, 17, rows) if ragged else np.full(rows, 7)
    row_ptr = np.concatenate([[0], np.cumsum(n)])
    nnz = int(row_ptr[-1])
    ids = (rng.zipf(1.3, nnz) % (1 << 22)).astype(np.int32)
    keys = hash_id_to_key(ids, 3, hash_bits or 64)
    vals = rng.random(nnz, dtype=np.float32) if values else None
    bounds_h, bounds = _bounds(5)
    b = LocalBatch(rows, nnz, 5, "cuda", real_values=values)
    kw = dict(row_ptr=torch.from_numpy(row_ptr.astype(np.int32)).cuda()) if ragged else dict(fixed_z=7)
    b.localize(torch.from_numpy(ids).cuda(), None, bounds, vals=torch.from_numpy(vals).cuda() if values else None, hash_seed=3,
               hash_bits=hash_bits, method="bucket", **kw)
    torch.cuda.synchronize()
    assert int(b.gate.item()) == 0 and int(b.status.item()) == 0
    _check_grouped(b, keys, row_ptr, vals, bounds_h, rows)


@pytest.mark.parametrize("hash_bits", [0, 40])
@pytest.mark.parametrize("given", ["neither", "vals", "csc_val", "both"])
def test_bucket_localize_values_move_only_where_both_sides_are_given(cuda_lib, given, hash_bits):
    """The C entry with values and no room for them by key, and the other way round: nothing is read or written there."""
    from parameter_server_b200.ops import _lib
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.utils.oracle import hash_id_to_key
    rng = np.random.default_rng(1)
    rows, z = 1500, 6
    ids = (rng.zipf(1.3, rows * z) % (1 << 22)).astype(np.int32)
    vals = rng.random(rows * z, dtype=np.float32)
    bounds_h, bounds = _bounds(2)
    b = LocalBatch(rows, rows * z, 2, "cuda", real_values=True)
    b.csc_val_buf.fill_(-1)
    i, v, ptr = torch.from_numpy(ids).cuda(), torch.from_numpy(vals).cuda(), _lib.ptr
    _lib.check(_lib.lib().psb_bucket_localize(
        ptr(i), 1, 3 | hash_bits << 56, rows * z, 64 - hash_bits if hash_bits else 0, 0, rows, z, ptr(v) if given in ("vals", "both") else 0,
        ptr(bounds), 2, ptr(b.keys_a), ptr(b.pos_a), ptr(b.keys_b), ptr(b.ukeys), ptr(b.seg_off), ptr(b.csr_col), ptr(b.csc_row_buf),
        ptr(b.csc_val_buf) if given in ("csc_val", "both") else 0, ptr(b.flagbits), ptr(b.wordbase), ptr(b.n_unique), ptr(b.own_off),
        ptr(b.bucket_scratch), ptr(b.status), ptr(b.gate), _lib.stream_ptr()), "bucket localize", kernels=10)
    torch.cuda.synchronize()
    b.nnz, b.csc_row, b.csc_val = rows * z, b.csc_row_buf, b.csc_val_buf
    _check_grouped(b, hash_id_to_key(ids, 3, hash_bits or 64), np.arange(rows + 1) * z, vals if given == "both" else None, bounds_h, rows)
    assert given == "both" or (b.csc_val_buf == -1).all()


@pytest.mark.parametrize("z", [1, 3, 5000])
def test_bucket_localize_more_slices_than_sms(cuda_lib, z):
    """A slice of the input is at most as long as a nonzero's place in it has bits: from 148 x 2^18 nonzeros on there are
    more slices than SMs."""
    from parameter_server_b200.ops import _lib
    from parameter_server_b200.ops.localize import LocalBatch
    n = ((_lib.lib().psb_device_sm_count() << 18) // 15000 + 1) * 15000
    g = torch.Generator(device="cuda").manual_seed(z)
    # half of the nonzeros on a thousand ids, the rest on half a million
    ids = torch.where(torch.rand(n, device="cuda", generator=g) < 0.5, torch.randint(0, 1000, (n,), device="cuda", generator=g),
                      torch.randint(0, 1 << 19, (n,), device="cuda", generator=g)).to(torch.int32)
    b = LocalBatch(n // z, n, 1, "cuda")
    b.localize(ids, None, _bounds(1)[1], fixed_z=z, hash_seed=0, hash_bits=40, method="bucket")
    torch.cuda.synchronize()
    assert int(b.gate.item()) == 0 and int(b.status.item()) == 0
    U = int(b.n_unique.item())
    wide, keys = ids.long(), torch.empty(n, dtype=torch.int64, device="cuda")
    _lib.check(_lib.lib().psb_hash_ids(0, _lib.ptr(wide), _lib.ptr(keys), n, 40 << 56, _lib.stream_ptr()), "hash")
    sign = -(1 << 63)
    u, inv, count = torch.unique(keys ^ sign, return_inverse=True, return_counts=True)
    assert U == u.numel() and torch.equal(b.ukeys[:U], u ^ sign) and torch.equal(b.csr_col[:n].long(), inv)
    assert torch.equal((b.seg_off[1:U + 1] - b.seg_off[:U]).long(), count)
    segment = torch.repeat_interleave(torch.arange(U, device="cuda"), count)
    rows = torch.arange(n, device="cuda") // z
    got = torch.sort(segment * (n // z + 1) + b.csc_row[:n].long())[0]
    assert torch.equal(got, torch.sort(inv * (n // z + 1) + rows)[0])
