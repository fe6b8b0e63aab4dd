"""Wide-value path: tcgen05 pull+GEMM, row sums, push and AdaGrad apply against PyTorch fp32."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(S, N, rows=300, z=12, n_feat=2500, seed=0, pull_cap=0):
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.parallel.fabric import Fabric
    from parameter_server_b200.parallel.wide import WideConfig, WidePlane, wide_layout
    from parameter_server_b200.utils.oracle import hash_id_to_key
    rng = np.random.default_rng(seed)
    cfg = WideConfig(table_capacity=1 << 13, inbox_cap=rows * z, ring=2, alpha=0.1, beta=1.0, pull_cap=pull_cap)
    fabs = Fabric.emulated(S, wide_layout(cfg, S).total())
    planes = [WidePlane(f, cfg) for f in fabs]
    all_ids = np.arange(n_feat)
    all_keys = hash_id_to_key(all_ids, 11)
    table = (torch.randn(n_feat, 64) * 0.5).to(torch.bfloat16)
    known = rng.random(n_feat) < 0.8                  # 20 % of the keys are not in the table yet
    for p in planes:
        lo, hi = p.bounds_host[p.rank], p.bounds_host[p.rank + 1]
        sel = known & (all_keys >= np.uint64(lo)) & (all_keys < np.uint64(min(hi, (1 << 64) - 1)))
        p.load(all_keys[sel], table[torch.from_numpy(sel)])
    ids = np.minimum((rng.pareto(1.2, rows * z) * 3).astype(np.int64), n_feat - 1).astype(np.int32)
    y = np.where(rng.random(rows) < 0.5, 1.0, -1.0).astype(np.float32)
    b = LocalBatch(rows, rows * z, S, "cuda")
    b.localize(torch.from_numpy(ids).cuda(), torch.from_numpy(y).cuda(), planes[0].bounds, fixed_z=z, hash_seed=11)
    ctx = (torch.randn(N, 64) * 0.3).to(torch.bfloat16).cuda()
    torch.cuda.synchronize()
    return planes, b, ctx, table, known, all_keys, ids, y, rows, z


@pytest.mark.parametrize("S,N", [(1, 64), (2, 128), (1, 128)])
def test_wide_pull_gemm_matches_fp32_matmul(cuda_lib, S, N):
    planes, b, ctx, table, known, all_keys, ids, y, rows, z = _setup(S, N)
    U = int(b.n_unique.item())
    P = torch.zeros(b.max_nnz, N, device="cuda")
    V = torch.zeros(b.max_nnz, 64, dtype=torch.bfloat16, device="cuda")
    planes[0].pull_gemm(b, ctx, P, V)
    torch.cuda.synchronize()
    planes[0].check_status()
    uk = b.ukeys[:U].cpu().numpy().view(np.uint64)
    idx = {int(k): i for i, k in enumerate(all_keys.tolist())}
    rows_ref = torch.stack([table[idx[int(k)]] if known[idx[int(k)]] else torch.zeros(64, dtype=torch.bfloat16) for k in uk.tolist()])
    assert torch.equal(V[:U].cpu(), rows_ref)                                  # the gather is exact
    ref = rows_ref.float() @ ctx.cpu().float().T
    assert torch.allclose(P[:U].cpu(), ref, rtol=1e-3, atol=1e-3), float((P[:U].cpu() - ref).abs().max())


@pytest.mark.parametrize("n_rows,fused", [(300, False), (900, False), (900, True)])
def test_wide_training_step_matches_reference(cuda_lib, n_rows, fused):
    """With 900 rows the most frequent key owns about 3,000 nonzeros: its gradient is
    reduced by several warps (segments above 256 nonzeros are split into chunks).
    ``fused``: the pull kernel adds the products into the rows' margins itself and no
    product matrix is stored."""
    S, N = 2, 64
    planes, b, ctx, table, known, all_keys, ids, y, rows, z = _setup(S, N, rows=n_rows, seed=4)
    assert int((b.seg_off[1:int(b.n_unique.item()) + 1] - b.seg_off[:int(b.n_unique.item())]).max().item()) > (256 if n_rows == 900 else 0)
    U = int(b.n_unique.item())
    w = planes[0]
    P = torch.zeros(b.max_nnz, N, device="cuda")
    if fused:
        w.pull_gemm(b, ctx, None, fuse_margins=True)
        w.rowloss(b)
    else:
        w.pull_gemm(b, ctx, P)
        w.rowsum(b, P, N)
    w.push(b, ctx, 0)
    # the other (virtual) worker pushes nothing: publish an empty round for it
    from parameter_server_b200.ops.localize import LocalBatch
    empty = LocalBatch(4, 16, S, "cuda")
    empty.n_unique.zero_(); empty.own_off.zero_(); empty.seg_off.zero_()
    planes[1].push(empty, ctx, 0)
    for p in planes:
        p.apply(0)
    torch.cuda.synchronize()
    for p in planes:
        p.check_status()
    # reference in fp32
    idx = {int(k): i for i, k in enumerate(all_keys.tolist())}
    uk = b.ukeys[:U].cpu().numpy().view(np.uint64)
    col = b.csr_col[:rows * z].cpu().numpy().reshape(rows, z)
    Vref = torch.stack([table[idx[int(k)]].float() if known[idx[int(k)]] else torch.zeros(64) for k in uk.tolist()])
    Pref = Vref @ ctx.cpu().float().T
    n_of_row = np.arange(rows) % N
    margin = Pref[torch.from_numpy(col), torch.from_numpy(n_of_row)[:, None]].sum(1)
    assert torch.allclose(b.margin[:rows].cpu(), margin, rtol=2e-3, atol=2e-3)
    ym = torch.from_numpy(y) * margin
    gcoef = -torch.from_numpy(y) * torch.sigmoid(-ym)
    assert torch.allclose(b.gcoef[:rows].cpu(), gcoef, rtol=2e-3, atol=2e-3)
    G = torch.zeros(U, 64)
    C = ctx.cpu().float()
    for r in range(rows):
        for j in range(z):
            G[col[r, j]] += gcoef[r] * C[n_of_row[r]]
    Gb = G.to(torch.bfloat16).float()                        # gradients travel as bf16
    acc = Gb * Gb
    Wref = (Vref - 0.1 / (acc.sqrt() + 1.0) * Gb).to(torch.bfloat16)
    got = torch.zeros(U, 64, dtype=torch.bfloat16)
    for p in planes:
        lo, hi = p.bounds_host[p.rank], p.bounds_host[p.rank + 1]
        sel = (uk >= np.uint64(lo)) & (uk < np.uint64(min(hi, (1 << 64) - 1)))
        got[torch.from_numpy(sel)] = p.lookup(uk[sel])
    diff = (got.float() - Wref.float()).abs()
    assert float(diff.max()) < 0.02 and float((diff > 0.004).float().mean()) < 0.02


@pytest.mark.parametrize("S,N", [(1, 64), (2, 128), (3, 64)])
def test_wide_exchange_pull_matches_fp32_matmul(cuda_lib, S, N):
    """Exchange form of the pull (keys to the owners, rows back in bulk, tcgen05 product on
    the local copy), ranks emulated on one GPU: the three roles run as separate launches."""
    from parameter_server_b200.ops.localize import LocalBatch
    rows, z = 300, 12
    planes, b, ctx, table, known, all_keys, ids, y, rows, z = _setup(S, N, rows=rows, z=z, seed=5, pull_cap=rows * z)
    U = int(b.n_unique.item())
    batches = [b]
    for _ in range(1, S):
        e = LocalBatch(4, rows * z, S, "cuda")
        e.n_unique.zero_(); e.own_off.zero_(); e.seg_off.zero_()
        batches.append(e)
    Ps = [torch.zeros(rows * z, N, device="cuda") for _ in range(S)]
    for rnd in range(2):                                   # two rounds: both parities of the buffers
        for phase in (1, 2, 4):
            for p, bb, P in zip(planes, batches, Ps):
                # the second round also adds the products into the rows' margins (fused form)
                p.pull_xgemm(bb, ctx, P, rnd, phases=phase, wait_iters=1 << 12, fuse_margins=rnd == 1)
        if rnd == 1:
            planes[0].rowloss(b)               # the fused margins are complete after the long segments are added
        torch.cuda.synchronize()
        for p in planes:
            p.check_status()
        idx = {int(k): i for i, k in enumerate(all_keys.tolist())}
        uk = b.ukeys[:U].cpu().numpy().view(np.uint64)
        Vref = torch.stack([table[idx[int(k)]].float() if known[idx[int(k)]] else torch.zeros(64) for k in uk.tolist()])
        assert torch.equal(planes[0].pulled_rows(rnd, U).cpu().float(), Vref)
        Pref = Vref @ ctx.cpu().float().T
        assert torch.allclose(Ps[0][:U].cpu(), Pref, rtol=2e-3, atol=2e-3)
        if rnd == 1:
            col = b.csr_col[:rows * z].cpu().numpy().reshape(rows, z)
            n_of_row = np.arange(rows) % N
            margin = Pref[torch.from_numpy(col), torch.from_numpy(n_of_row)[:, None]].sum(1)
            assert torch.allclose(b.margin[:rows].cpu(), margin, rtol=2e-3, atol=2e-3)
        Ps[0].zero_()


@pytest.mark.parametrize("rows,z,N", [(1, 1, 64), (3, 70, 128), (37, 5, 64), (2050, 9, 128)])
def test_wide_rows_push_and_apply_sizes(cuda_lib, rows, z, N):
    """Row sums, gradient rows and AdaGrad steps at sizes around the tiles that a warp takes (4 to 32 keys or
    records, eight lanes per row), with keys of one to thousands of nonzeros, against fp64."""
    planes, b, ctx, table, known, all_keys, ids, y, rows, z = _setup(1, N, rows=rows, z=z, seed=rows)
    w = planes[0]
    U = int(b.n_unique.item())
    P = torch.zeros(b.max_nnz, N, device="cuda")
    w.pull_gemm(b, ctx, P)
    w.rowsum(b, P, N)
    w.push(b, ctx, 0)
    w.apply(0)
    torch.cuda.synchronize()
    w.check_status()
    col = b.csr_col[:rows * z].long()
    cx = torch.arange(rows, device="cuda") % N
    margin = P.double()[col, cx.repeat_interleave(z)].view(rows, z).sum(1)
    assert (b.margin[:rows] - margin).norm() <= 1e-6 * margin.norm() + 1e-6      # 32-bit sums of z terms
    yy = torch.from_numpy(y).cuda().double()
    gcoef = -yy * torch.sigmoid(-yy * margin)
    assert torch.allclose(b.gcoef[:rows].double(), gcoef, rtol=1e-5, atol=1e-6)
    C = ctx.double()
    G = torch.zeros(U, 64, dtype=torch.float64, device="cuda").index_add_(0, col, (gcoef[:, None] * C[cx]).repeat_interleave(z, 0))
    uk = b.ukeys[:U].cpu().numpy().view(np.uint64)
    at = np.searchsorted(all_keys, uk, sorter=np.argsort(all_keys))
    at = np.argsort(all_keys)[at]
    V = torch.where(torch.from_numpy(known[at])[:, None], table[torch.from_numpy(at)].double(), 0.0).cuda()
    want = V - 0.1 / (G.abs() + 1.0) * G
    # the gradient travels as bf16 (2^-9 of |G|, whose step is at most 0.1 |G|) and the weight is stored as bf16
    err = (w.lookup(uk).cuda().double() - want).abs()
    assert (err <= 0.1 * G.abs() * 2.0 ** -8 + want.abs() * 2.0 ** -8 + 1e-5).all()


@pytest.mark.parametrize("N", [64, 128])
def test_wide_exchange_pull_reports_rows_that_never_come(cuda_lib, N):
    """The worker's role alone, for rounds that no owner has answered: every tile group's wait runs out, the kernel
    returns with a status, and the plane serves the next round."""
    from parameter_server_b200.ops._lib import PsbCudaError
    rows, z = 300, 12
    planes, b, ctx, *_ = _setup(1, N, rows=rows, z=z, seed=5, pull_cap=rows * z)
    w = planes[0]
    P = torch.zeros(rows * z, N, device="cuda")
    for rnd in range(2):
        w.pull_xgemm(b, ctx, P, rnd, phases=4, wait_iters=1 << 8)
        torch.cuda.synchronize()
        with pytest.raises(PsbCudaError):
            w.check_status()
    assert not P.any()
    w.pull_xgemm(b, ctx, P, 2)
    torch.cuda.synchronize()
    w.check_status()
    U = int(b.n_unique.item())
    want = w.pulled_rows(2, U).float() @ ctx.float().T
    assert torch.allclose(P[:U], want, rtol=2e-3, atol=2e-3) and P[:U].any()


@pytest.mark.parametrize("keys,each", [(100, 200), (100, 129), (70, 1500)])
def test_wide_push_with_more_long_segments_than_the_list_holds(cuda_lib, keys, each):
    """An inbox for the keys of a minibatch that repeats them often: the list of long segments is sized by the inbox
    and fills up, and the rest are summed where they are. Same weights as with an inbox for every nonzero."""
    from parameter_server_b200.ops.localize import LocalBatch
    from parameter_server_b200.parallel.fabric import Fabric
    from parameter_server_b200.parallel.wide import WideConfig, WidePlane, wide_layout
    g = torch.Generator().manual_seed(keys + each)
    ids = torch.arange(keys, dtype=torch.int32).repeat(each, 1).cuda()
    y = torch.where(torch.rand(each, generator=g) < 0.5, 1.0, -1.0).cuda()
    ctx = (torch.randn(64, 64, generator=g) * 0.3).to(torch.bfloat16).cuda()
    rows = torch.randn(keys, 64, generator=g) * 0.5
    got = []
    for inbox in (keys, keys * each):
        cfg = WideConfig(table_capacity=1 << 10, inbox_cap=inbox, ring=2)
        w = WidePlane(Fabric.single(wide_layout(cfg, 1).total()), cfg)
        assert (w.long_cap < keys) == (inbox == keys)
        b = LocalBatch(each, keys * each, 1, "cuda")
        b.localize(ids.flatten(), y, w.bounds, fixed_z=keys, hash_seed=3)
        uk = b.ukeys[:keys].cpu().numpy().view(np.uint64)
        w.load(uk, rows)
        P = torch.zeros(b.max_nnz, 64, device="cuda")
        for rnd in range(3):                               # the list and its sums are left clean for the next round
            w.pull_gemm(b, ctx, P)
            w.rowsum(b, P, 64)
            w.push(b, ctx, rnd)
            w.apply(rnd)
        torch.cuda.synchronize()
        w.check_status()
        got.append(w.lookup(uk).float())
    # 32-bit sums in another order: in each of three rounds a gradient (whose step is at most 0.1) and a weight may be
    # rounded to the next bf16 value
    assert (got[0] - got[1]).abs().le(3 * 2.0 ** -8 * (got[1].abs() + 0.1)).all()
    assert not torch.equal(got[0], rows.to(torch.bfloat16).float())


@pytest.mark.parametrize("z", [10, 40, 96])
def test_wide_row_sums_of_eight_lanes_are_as_close_as_those_of_a_warp(cuda_lib, z):
    """The error of the margins against 64 bits (root mean square over 4000 rows) is no larger than that of a warp per
    row in 32 bits (32 lanes in sequence, then a tree; emulated here)."""
    planes, b, ctx, *_ = _setup(1, 64, rows=4000, z=z, seed=z)
    rows = 4000
    P = torch.randn(b.max_nnz, 64, device="cuda")
    planes[0].rowsum(b, P, 64)
    torch.cuda.synchronize()
    terms = P[b.csr_col[:rows * z].long(), (torch.arange(rows, device="cuda") % 64).repeat_interleave(z)].view(rows, z).cpu().numpy()
    want = terms.astype(np.float64).sum(1)
    lane = np.zeros((rows, 32), np.float32)
    for j in range(0, z, 32):
        lane[:, :min(32, z - j)] += terms[:, j:j + 32]
    while lane.shape[1] > 1:
        lane = lane[:, :lane.shape[1] // 2] + lane[:, lane.shape[1] // 2:]
    rms = lambda e: float(np.sqrt(np.mean(np.square(e))))
    assert rms(b.margin[:rows].cpu().numpy() - want) <= rms(lane[:, 0] - want)
