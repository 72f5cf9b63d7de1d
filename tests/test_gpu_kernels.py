"""GPU numerics tests: every CUDA kernel against the PyTorch fp32 oracle.

The multi-rank exchange kernels are exercised with all P ranks emulated on one
GPU in a single cooperative launch (peer pointers are local pointers), which
runs the full protocol: pushes, flags, epochs, merges, re-selects, broadcast
and residual put-back.
"""
import math

import pytest
import torch

from gtopkssgd_b200.ops import oracle

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


def _selector(d, k, **kw):
    from gtopkssgd_b200.ops.select import TopkSelector
    return TopkSelector(d, k, DEV, **kw)


def _check_select(sel, g, r_before, k, scale=1.0):
    """Compare the selector's output with the oracle on the same inputs."""
    r_ref = r_before.clone().cpu()
    idx_ref, val_ref = oracle.compress(g.cpu(), r_ref, k, scale)
    idx, val = sel.pairs()
    assert idx.numel() == min(k, g.numel())
    got = dict(zip(idx.cpu().tolist(), val.cpu().tolist()))
    ref = dict(zip(idx_ref.tolist(), val_ref.tolist()))
    assert len(got) == idx.numel(), "duplicate indices in the selection"
    assert set(got) == set(ref)
    for j in ref:
        assert got[j] == pytest.approx(ref[j], rel=1e-6, abs=1e-7)
    return r_ref


@pytest.mark.parametrize("d,k", [(1, 1), (7, 3), (1000, 1), (4099, 17), (100003, 100), (1 << 20, 1048), (3_000_001, 3000)])
def test_k1_select_matches_oracle(d, k):
    torch.manual_seed(d)
    sel = _selector(d, k)
    r = torch.zeros(d, device=DEV)
    for it in range(4):  # call 0: exact path; later calls: predicted threshold
        g = torch.randn(d, device=DEV) * (1.0 + 0.05 * it)
        r_before = r.clone()
        sel.select(g, r, k)
        r_ref = _check_select(sel, g, r_before, k)
        assert torch.allclose(r.cpu(), r_ref, rtol=1e-6, atol=1e-7)
        assert sel.status() == (0, 0)
    assert sel.stats()["n_calls"] == 4


def test_k1_large_vector_dynamic_stream_pass():
    """From 20 M elements on the stream pass hands its work out through ticket
    counters; compared here against the oracle computed on the device."""
    d, k = 50_000_003, 50_000
    torch.manual_seed(7)
    sel = _selector(d, k)
    r = torch.zeros(d, device=DEV)
    for it in range(3):  # exact path, then predicted thresholds
        g = torch.randn(d, device=DEV)
        r_ref = r.clone()
        idx_ref, val_ref = oracle.compress(g, r_ref, k)
        sel.select(g, r, k)
        idx, val = sel.pairs()
        assert sel.status() == (0, 0) and idx.numel() == k
        order, order_ref = idx.argsort(), idx_ref.argsort()
        assert torch.equal(idx[order], idx_ref[order_ref])
        assert torch.allclose(val[order], val_ref[order_ref], rtol=1e-6, atol=1e-7)
        assert torch.allclose(r, r_ref, rtol=1e-6, atol=1e-7)
        del g, r_ref
    st = sel.stats()  # the residual grows over these calls, so a second exact pass is legitimate
    assert st["n_calls"] == 3 and st["n_fallbacks"] < 3


def test_k1_threshold_prediction_carries_steady_state():
    """With a stationary input distribution only the first call (no threshold
    yet) may take the exact dense path."""
    torch.manual_seed(11)
    d, k = 1 << 20, 1048
    sel = _selector(d, k)
    r = torch.zeros(d, device=DEV)
    for it in range(10):
        g = torch.randn(d, device=DEV) * (1.0 + 0.03 * math.sin(it))
        r.zero_()
        sel.select(g, r, k)
    st = sel.stats()
    assert st["n_calls"] == 10 and st["n_fallbacks"] == 1, st
    assert k <= st["n_cand"] <= sel.cap


def test_k1_unaligned_views_and_scale():
    torch.manual_seed(5)
    d, k = 50001, 50
    big_g = torch.randn(d + 8, device=DEV)
    big_r = torch.zeros(d + 8, device=DEV)
    scale = torch.tensor([0.5], device=DEV)
    for off in (1, 2, 3):
        g, r = big_g[off:off + d], big_r[off:off + d]
        big_r.zero_()
        sel = _selector(d, k)
        for _ in range(2):
            r_before = r.clone()
            sel.select(g, r, k, g_scale=scale)
            r_ref = _check_select(sel, g, r_before, k, 0.5)
            assert torch.allclose(r.cpu(), r_ref, rtol=1e-6, atol=1e-7)
        # nothing outside the view was touched
        assert float(big_r[:off].abs().sum()) == 0.0 and float(big_r[off + d:].abs().sum()) == 0.0


def test_k1_non_finite_entries_are_selected_on_both_paths():
    """NaN and +-Inf count as the largest magnitudes (NaN above Inf), as
    torch.topk(|acc|) of the reference ranks them (compression.py:43): they are
    selected and leave the residual on the exact path (first call) and on the
    predicted-threshold path (later calls) alike."""
    torch.manual_seed(9)
    d, k = 300_000, 300
    sel = _selector(d, k)
    r = torch.zeros(d, device=DEV)
    planted = {0: [(17, float("nan")), (d - 1, float("inf"))],              # call 0: exact path
               2: [(4096, float("-inf")), (123_457, float("nan")), (3, float("nan"))]}  # call 2: predicted threshold
    for it in range(4):
        g = torch.randn(d, device=DEV)
        for j, v in planted.get(it, []):
            g[j] = v
        r_before = r.clone()
        sel.select(g, r, k)
        idx, val = sel.pairs()
        assert sel.status() == (0, 0) and idx.numel() == k
        got = dict(zip(idx.cpu().tolist(), val.cpu().tolist()))
        assert len(got) == k
        bad = planted.get(it, [])
        for j, v in bad:
            assert j in got, "call %d: non-finite entry %d not selected" % (it, j)
            assert (math.isnan(v) and math.isnan(got[j])) or got[j] == v
            assert float(r[j]) == 0.0
        # the finite rest: the k - len(bad) largest finite magnitudes, residual = acc off the selection
        acc = (g + r_before).cpu()
        finite = acc.clone()
        for j, _ in bad:
            finite[j] = 0.0
        top = set(torch.topk(finite.abs(), k - len(bad)).indices.tolist())
        assert set(got) - {j for j, _ in bad} == top
        keep = torch.ones(d, dtype=torch.bool)
        keep[list(got)] = False
        assert torch.equal(r.cpu()[keep], acc[keep])
        assert torch.isfinite(r).all()
        if it == 2:
            assert sel.stats()["fallback"] == 0, "call 2 was meant to run on the predicted threshold"


def test_k1_scale_jump_and_ties():
    """A 5x scale jump overflows or starves the candidate list: the exact path
    must take over; repeated values must still give exactly k entries."""
    torch.manual_seed(6)
    d, k = 200000, 200
    sel = _selector(d, k)
    r = torch.zeros(d, device=DEV)
    for scale in (1.0, 1.0, 5.0, 0.2, 1.0):
        g = torch.randn(d, device=DEV) * scale
        r.zero_()
        sel.select(g, r, k)
        _check_select(sel, g, torch.zeros(d, device=DEV), k)
    g = torch.ones(d, device=DEV)  # all tied
    r.zero_()
    sel.select(g, r, k)
    idx, val = sel.pairs()
    assert idx.numel() == k and idx.unique().numel() == k and torch.all(val == 1.0)
    assert float(r.sum()) == d - k
    g = torch.zeros(d, device=DEV)  # all zero
    r.zero_()
    sel.select(g, r, k)
    idx, val = sel.pairs()
    assert idx.numel() == k and torch.all(val == 0)


def test_k1_density_one():
    d = 1000
    sel = _selector(d, d)
    g = torch.randn(d, device=DEV)
    r = torch.zeros(d, device=DEV)
    sel.select(g, r, d)
    idx, val = sel.pairs()
    assert idx.numel() == d and float(r.abs().sum()) == 0.0
    assert torch.equal(val[torch.argsort(idx)], g)


def _pairs_tensor(idx, val, cap):
    from gtopkssgd_b200.ops.select import tensors_to_pairs
    out = torch.zeros((cap, 2), dtype=torch.int32, device=DEV)
    tensors_to_pairs(idx.to(DEV), val.to(DEV), out)
    return out


@pytest.mark.parametrize("momentum,nesterov,wd,damp", [(0.9, False, 1e-4, 0.0), (0.9, True, 5e-4, 0.0),
                                                      (0.0, False, 0.0, 0.0), (0.5, False, 0.0, 0.1)])
def test_k3_sparse_plus_dense_equals_reference_sgd(momentum, nesterov, wd, damp):
    from gtopkssgd_b200.ops.sgd import SgdHyper, sgd_dense, sgd_sparse
    torch.manual_seed(7)
    d, k, P = 100003, 101, 4
    p = torch.randn(d, device=DEV)
    buf = torch.zeros(d, device=DEV)
    p_ref, buf_ref = p.cpu().clone(), buf.cpu().clone()
    h = SgdHyper(lr=0.1, momentum=momentum, dampening=damp, weight_decay=wd, nesterov=nesterov)
    for step in range(3):
        idx = torch.randperm(d)[:k]
        val = torch.randn(k)
        pairs = _pairs_tensor(idx, val, k)
        counts = torch.tensor([k], dtype=torch.int32, device=DEV)
        sgd_dense(p, buf, h, first_step=(step == 0))
        sgd_sparse(p, buf, pairs, counts, 1, k, h, first_step=(step == 0), scale=1.0 / P)
        dense = oracle.scatter_average((idx, val), d, P)
        oracle.sgd_step(p_ref, buf_ref, dense, 0.1, momentum, damp, wd, nesterov, first_step=(step == 0))
    assert torch.allclose(p.cpu(), p_ref, rtol=1e-5, atol=1e-6)
    if momentum:
        assert torch.allclose(buf.cpu(), buf_ref, rtol=1e-5, atol=1e-6)


def test_k3_dense_mode_and_scatter():
    from gtopkssgd_b200.ops.sgd import SgdHyper, scatter_dense, sgd_dense, sgd_sparse
    torch.manual_seed(8)
    d, P = 70001, 8
    p = torch.randn(d + 1, device=DEV)[1:]  # unaligned view
    buf = torch.zeros(d + 1, device=DEV)[1:]
    g = torch.randn(d + 1, device=DEV)[1:]
    coef = torch.tensor([0.25], device=DEV)
    p_ref, buf_ref = p.cpu().clone(), buf.cpu().clone()
    h = SgdHyper(lr=0.05, momentum=0.9, weight_decay=1e-4)
    sgd_dense(p, buf, h, True, g=g, scale=1.0 / P, coef=coef)
    oracle.sgd_step(p_ref, buf_ref, g.cpu() * (0.25 / P), 0.05, 0.9, 0.0, 1e-4, False, True)
    assert torch.allclose(p.cpu(), p_ref, rtol=1e-5, atol=1e-6)
    assert torch.allclose(buf.cpu(), buf_ref, rtol=1e-5, atol=1e-6)
    # atomic mode with repeated indices over two segments
    k = 64
    idx = torch.randint(0, 100, (2 * k,))
    val = torch.randn(2 * k)
    pairs = _pairs_tensor(idx, val, 2 * k)
    counts = torch.tensor([k, k - 3], dtype=torch.int32, device=DEV)
    dense = torch.empty(d, device=DEV)
    scatter_dense(dense, pairs, counts, 2, k, 0.5, use_atomics=True)
    ref = torch.zeros(d)
    ref.index_add_(0, idx[:k], val[:k] * 0.5)
    ref.index_add_(0, idx[k:2 * k - 3], val[k:2 * k - 3] * 0.5)
    assert torch.allclose(dense.cpu(), ref, atol=1e-6)
    q = torch.zeros(d, device=DEV)
    sgd_sparse(q, None, pairs, counts, 2, k, SgdHyper(lr=1.0), False, 0.5, use_atomics=True)
    assert torch.allclose(q.cpu(), -ref, atol=1e-6)


def test_k4_clip_norm():
    from gtopkssgd_b200.ops.clip import ClipNorm
    torch.manual_seed(9)
    d = 1_000_003
    x = torch.randn(d + 1, device=DEV)[1:]
    c = ClipNorm(DEV)
    c.add_dense(x)
    coef = c.finalize(0.25)
    norm = float(x.double().norm())
    assert c.last_norm() == pytest.approx(norm, rel=1e-5)
    assert float(coef) == pytest.approx(0.25 / (norm + 1e-6), rel=1e-5)
    # sparse pairs, scaled by 1/P, no clipping needed -> coef 1; accumulator was cleared
    k = 1000
    val = torch.randn(k) * 1e-3
    pairs = _pairs_tensor(torch.arange(k), val, k)
    counts = torch.tensor([k], dtype=torch.int32, device=DEV)
    c.add_pairs(pairs, counts, 1, k)
    coef = c.finalize(400.0, scale=0.125)
    assert float(coef) == 1.0
    assert c.last_norm() == pytest.approx(float(val.double().norm()) / 8, rel=1e-5)


def _emulated_world(P, d, k, mode="gtopk"):
    from gtopkssgd_b200.ops import exchange as ex
    with_ag = mode != "gtopk"
    regions = ex.SymmetricRegion.create_emulated(P, ex.region_bytes(k, with_ag), DEV)
    ranks = []
    for r in range(P):
        sel = _selector(d, k)
        resid = torch.zeros(d, device=DEV)
        ranks.append(ex.ExchangeRank(r, P, d, k, sel, resid, regions[r], with_allgather=with_ag,
                                     reselect=(mode == "topk2")))
    desc = torch.cat([r.desc for r in ranks])
    return ranks, desc


def _read_gout(rank, parity):
    from gtopkssgd_b200.ops.select import pairs_to_tensors
    n = int(rank.n_global.item())
    off = rank.layout[2] + parity * rank.kcap * 8
    raw = rank.region.tensor()[off:off + n * 8].view(torch.int32).view(n, 2)
    return pairs_to_tensors(raw, n)


@pytest.mark.parametrize("P", [2, 4, 8])
@pytest.mark.parametrize("d,k,nctas", [(4096, 8, 1), (50000, 50, 1), (300000, 3000, 4), (2_000_000, 20000, 8),
                                       (2_000_000, 20000, 12)])  # 1 CTA; clusters of 4 and 8; software barrier
def test_k2_gtopk_exchange_emulated(P, d, k, nctas):
    from gtopkssgd_b200.ops import exchange as ex
    torch.manual_seed(100 * P + k)
    ranks, desc = _emulated_world(P, d, k)
    res_ref = [torch.zeros(d) for _ in range(P)]
    for epoch in (1, 2, 3):  # both parities, flag reuse
        grads = [torch.randn(d, device=DEV) for _ in range(P)]
        for r, g in zip(ranks, grads):
            r.selector.select(g, r.resid, k)
        ex.launch_gtopk(ranks, desc, 0, P, k, nctas=nctas, limit_ms=2000)
        torch.cuda.synchronize()
        for r in ranks:
            assert r.status() == (0, 0)
        glob, _ = oracle.simulate_gtopk_step([g.cpu() for g in grads], res_ref, k)
        ref = dict(zip(glob[0].tolist(), glob[1].tolist()))
        for r in ranks:
            gi, gv = _read_gout(r, r.last_parity())
            got = dict(zip(gi.cpu().tolist(), gv.cpu().tolist()))
            assert len(got) == gi.numel()
            assert set(got) == set(ref), "rank %d" % r.rank
            for j in ref:
                assert got[j] == pytest.approx(ref[j], rel=1e-5, abs=1e-6)
            assert torch.allclose(r.resid.cpu(), res_ref[r.rank], rtol=1e-5, atol=1e-6)
            assert r.region.guards_intact(), "a store landed outside the slots of rank %d" % r.rank


@pytest.mark.parametrize("nctas", [1, 4, 12])
def test_k2_reselect_when_the_threshold_prediction_misses(nctas):
    """The re-select of a tree round reads its first two radix digits from histograms built on the
    fly around a predicted threshold digit (this rank's own k-th magnitude, then the previous round's
    threshold).  Ranks whose gradients differ in scale by orders of magnitude put the union's
    threshold far outside that window, so the counting sweep has to take over; tiny and huge ranks
    alternate so that both receivers and senders of every round are affected."""
    from gtopkssgd_b200.ops import exchange as ex
    P, d, k = 4, 300_000, 3000
    torch.manual_seed(4242 + nctas)
    ranks, desc = _emulated_world(P, d, k)
    res_ref = [torch.zeros(d) for _ in range(P)]
    scales = [1.0, 3.0e3, 1.0e-3, 5.0e1]
    for epoch in range(3):
        grads = [torch.randn(d, device=DEV) * scales[(r + epoch) % P] for r in range(P)]
        for r, g in zip(ranks, grads):
            r.selector.select(g, r.resid, k)
        ex.launch_gtopk(ranks, desc, 0, P, k, nctas=nctas, limit_ms=2000)
        torch.cuda.synchronize()
        assert all(r.status() == (0, 0) for r in ranks)
        glob, _ = oracle.simulate_gtopk_step([g.cpu() for g in grads], res_ref, k)
        ref = dict(zip(glob[0].tolist(), glob[1].tolist()))
        for r in ranks:
            gi, gv = _read_gout(r, r.last_parity())
            got = dict(zip(gi.cpu().tolist(), gv.cpu().tolist()))
            assert set(got) == set(ref), "rank %d epoch %d" % (r.rank, epoch)
            for j in ref:
                assert got[j] == pytest.approx(ref[j], rel=1e-5, abs=1e-9)
            assert torch.allclose(r.resid.cpu(), res_ref[r.rank], rtol=1e-5, atol=1e-9)


def test_region_guard_bands_detect_a_stray_write():
    """The canary bands around a peer-visible region are checked by reading
    them back; an ordinary torch write into the band (inside the same
    allocation) must be noticed."""
    from gtopkssgd_b200.ops import exchange as ex
    regions = ex.SymmetricRegion.create_emulated(2, ex.region_bytes(64, True), DEV)
    assert all(r.guards_intact() for r in regions)
    assert regions[0].tensor().numel() == regions[0].nbytes
    regions[0].tensor().fill_(7)              # the whole usable region may be written
    assert regions[0].guards_intact()
    regions[1]._owner[ex.GUARD_BYTES + regions[1].nbytes + 3] = 0   # first band byte range after the region
    assert not regions[1].guards_intact() and regions[0].guards_intact()


@pytest.mark.parametrize("mode", ["topk", "topk2"])
@pytest.mark.parametrize("P", [2, 3, 4])  # the all-gather modes need no power-of-two world
def test_k2t_allgather_emulated(P, mode):
    from gtopkssgd_b200.ops import exchange as ex
    from gtopkssgd_b200.ops.select import pairs_to_tensors
    torch.manual_seed(P)
    d, k = 200000, 500
    ranks, desc = _emulated_world(P, d, k, mode)
    seg_counts = torch.zeros(P * ex.MAX_PEERS, dtype=torch.int32, device=DEV)
    res_ref = [torch.zeros(d) for _ in range(P)]
    for epoch in (1, 2):
        grads = [torch.randn(d, device=DEV) for _ in range(P)]
        for r, g in zip(ranks, grads):
            r.selector.select(g, r.resid, k)
        ex.launch_allgather(ranks, desc, seg_counts, 0, P, k, reselect=(mode == "topk2"), nctas=2,
                            limit_ms=2000)
        torch.cuda.synchronize()
        local = [oracle.compress(g.cpu(), rr, k) for g, rr in zip(grads, res_ref)]
        for r in ranks:
            assert r.status() == (0, 0)
            counts = seg_counts[r.rank * ex.MAX_PEERS:r.rank * ex.MAX_PEERS + P].cpu().tolist()
            assert counts == [k] * P
            assert r.last_parity() == epoch & 1
            base = r.layout[1] + r.last_parity() * ex.MAX_PEERS * k * 8
            for q in range(P):
                raw = r.region.tensor()[base + q * k * 8: base + (q + 1) * k * 8].view(torch.int32).view(k, 2)
                qi, qv = pairs_to_tensors(raw, k)
                assert set(qi.cpu().tolist()) == set(local[q][0].tolist())
        if mode == "topk2":
            gi_ref, gv_ref = oracle.topk2_reselect(local, k)
            ref = dict(zip(gi_ref.tolist(), gv_ref.tolist()))
            for rr, loc in zip(res_ref, local):
                oracle.put_back(rr, loc, gi_ref)
            for r in ranks:
                gi, gv = _read_gout(r, r.last_parity())
                got = dict(zip(gi.cpu().tolist(), gv.cpu().tolist()))
                assert set(got) == set(ref)
                for j in ref:
                    assert got[j] == pytest.approx(ref[j], rel=1e-5, abs=1e-6)
                assert torch.allclose(r.resid.cpu(), res_ref[r.rank], rtol=1e-5, atol=1e-6)


def test_k2_bounded_wait_reports_timeout():
    """A receiver whose partner never sends must give up after the limit and
    report a status; the context stays usable.  Rank 0 of a 2-rank world is
    launched alone (its partner's kernel is simply not launched)."""
    from gtopkssgd_b200.ops import exchange as ex
    d, k = 10000, 10
    ranks, desc = _emulated_world(2, d, k)
    g = torch.randn(d, device=DEV)
    ranks[0].selector.select(g, ranks[0].resid, k)
    ex.launch_gtopk(ranks[:1], ranks[0].desc, 0, 2, k, nctas=2, limit_ms=50)
    torch.cuda.synchronize()
    status, where = ranks[0].status()
    assert status == 1 and 210 <= where < 220
    assert int(ranks[0].n_global.item()) == 0  # an empty global set: the consumer applies nothing
    assert int(ranks[0].epoch.item()) == 1     # the aborted call did not advance the counter
    # a failed exchange stays failed: the next call returns at once (no second wait), still empty
    import time
    ranks[0].n_global.fill_(123)
    t0 = time.time()
    ex.launch_gtopk(ranks[:1], ranks[0].desc, 0, 2, k, nctas=2, limit_ms=5000)
    ranks[0].mirror_status()
    torch.cuda.synchronize()
    assert time.time() - t0 < 2.0
    assert int(ranks[0].n_global.item()) == 0 and ranks[0].status()[0] == 1
    assert ranks[0].failed_on_host_mirror()[0] == 1  # what the host sees without synchronising
    # the host clears the failure (all ranks together); the device is healthy and a complete exchange works
    ranks[0].clear_failure()
    assert ranks[0].status() == (0, 0)
    for r in ranks:
        r.selector.select(torch.randn(d, device=DEV), r.resid, k)
    ex.launch_gtopk(ranks, desc, 0, 2, k, nctas=1, limit_ms=2000)
    torch.cuda.synchronize()
    assert all(r.status() == (0, 0) for r in ranks)
    assert [int(r.epoch.item()) for r in ranks] == [2, 2]
    assert int(ranks[1].n_global.item()) == k


def _check_selection(idx, val, r, acc, k):
    """k distinct entries of acc, none left out larger than any taken (which of
    two equal ones is taken is free), residual = acc off them, 0 on them."""
    assert idx.numel() == k and idx.unique().numel() == k and torch.equal(val, acc[idx])
    assert torch.equal(val.abs().sort().values, torch.topk(acc.abs(), k).values.sort().values)
    want = acc.clone()
    want[idx] = 0.0
    assert torch.equal(r, want)


@pytest.mark.parametrize("d,k", [(1, 1), (5, 2), (4097, 4097), (300_001, 300), (2_000_003, 6000), (20_000_010, 20_000)])
def test_k1_compress_leaves_g_sparsified(d, k):
    """The compressor's form of K1: the vector keeps acc on the selection and 0
    off it, indices and values come as separate lists (exact path on the first
    call, predicted thresholds after it; static and dynamic stream pass)."""
    torch.manual_seed(d + k)
    sel = _selector(d, k)
    r = torch.zeros(d, device=DEV)
    for it in range(3):
        g = torch.randn(d, device=DEV)
        acc = g + r
        idx, val = sel.compress(g, r, k)
        assert sel.status() == (0, 0) and idx.dtype == torch.int64
        _check_selection(idx, val, r, acc, k)
        want = torch.zeros(d, device=DEV)
        want[idx] = val
        assert torch.equal(g, want)


@pytest.mark.parametrize("d,k", [(60_000, 4000), (200_000, 4096), (400_000, 30_000), (3_000_000, 65_536), (4_000_000, 400_000)])
@pytest.mark.parametrize("off", [0, 3])
def test_k1_pick_in_one_cta_a_cluster_and_by_shares(d, k, off):
    """Candidate counts on both sides of the borders between one CTA, a cluster and
    shares over all CTAs, on aligned and unaligned views."""
    torch.manual_seed(k + off)
    sel = _selector(d, k)
    g, r = torch.empty(d + 4, device=DEV)[off:off + d], torch.zeros(d + 4, device=DEV)[off:off + d]
    for it in range(4):
        g.normal_()
        acc = g + r
        sel.select(g, r, k)
        assert sel.status() == (0, 0)
        _check_selection(*sel.pairs(), r, acc, k)
    assert sel.stats()["n_fallbacks"] < 4


@pytest.mark.parametrize("P", [2, 8])
@pytest.mark.parametrize("d,k", [(64, 1), (1500, 1024), (30_000, 1025), (3000, 2000), (400_000, 2048)])
def test_k2_small_exchange_matches_oracle(P, d, k):
    """One CTA per rank, set in shared memory, flags inside the data: k at the
    edges of the CTA's 1024 threads, sets that overlap almost completely, scales
    that put the threshold outside the predicted band, and the largest k."""
    from gtopkssgd_b200.ops import exchange as ex
    torch.manual_seed(7 * P + k)
    ranks, desc = _emulated_world(P, d, k)
    res_ref = [torch.zeros(d) for _ in range(P)]
    for epoch, scales in enumerate(([1.0], [1.0, 1.0, 300.0, 1e-3], [1.0])):
        grads = [torch.randn(d, device=DEV) * scales[r % len(scales)] for r in range(P)]
        for r, g in zip(ranks, grads):
            r.selector.select(g, r.resid, k)
        ex.launch_gtopk(ranks, desc, 0, P, k, nctas=1, limit_ms=2000)
        torch.cuda.synchronize()
        assert all(r.status() == (0, 0) for r in ranks)
        glob, _ = oracle.simulate_gtopk_step([g.cpu() for g in grads], res_ref, k)
        ref = dict(zip(glob[0].tolist(), glob[1].tolist()))
        for r in ranks:
            gi, gv = _read_gout(r, r.last_parity())
            got = dict(zip(gi.cpu().tolist(), gv.cpu().tolist()))
            assert len(got) == gi.numel() and set(got) == set(ref), "rank %d epoch %d" % (r.rank, epoch)
            for j in ref:
                assert got[j] == pytest.approx(ref[j], rel=1e-5, abs=1e-9)
            assert torch.allclose(r.resid.cpu(), res_ref[r.rank], rtol=1e-5, atol=1e-9)
            assert r.region.guards_intact()


def test_k2_small_bounded_wait_reports_timeout():
    """The one-CTA form gives up like the other one when its partner never sends,
    and works again after ``clear_failure``."""
    from gtopkssgd_b200.ops import exchange as ex
    d, k = 10000, 10
    ranks, desc = _emulated_world(2, d, k)
    ranks[0].selector.select(torch.randn(d, device=DEV), ranks[0].resid, k)
    ex.launch_gtopk(ranks[:1], ranks[0].desc, 0, 2, k, nctas=1, limit_ms=50)
    torch.cuda.synchronize()
    status, where = ranks[0].status()
    assert status == 1 and 210 <= where < 220
    assert int(ranks[0].n_global.item()) == 0 and int(ranks[0].epoch.item()) == 1
    ranks[0].clear_failure()
    for r in ranks:
        r.selector.select(torch.randn(d, device=DEV), r.resid, k)
    ex.launch_gtopk(ranks, desc, 0, 2, k, nctas=1, limit_ms=2000)
    torch.cuda.synchronize()
    assert all(r.status() == (0, 0) for r in ranks) and int(ranks[1].n_global.item()) == k


@pytest.mark.parametrize("P,d,k,nctas", [(2, 200_000, 3, 1), (5, 100_000, 4000, 3), (4, 3_000_000, 30_000, 16)])
def test_k2t_reselect_in_and_outside_the_predicted_band(P, d, k, nctas):
    """'topk2' with ranks of one scale (the threshold lies in the band above the
    own k-th magnitude) and of very different scales (the counting sweeps), over
    both control blocks."""
    from gtopkssgd_b200.ops import exchange as ex
    torch.manual_seed(P + k)
    ranks, desc = _emulated_world(P, d, k, "topk2")
    seg_counts = torch.zeros(P * ex.MAX_PEERS, dtype=torch.int32, device=DEV)
    res_ref = [torch.zeros(d) for _ in range(P)]
    for scales in ([1.0], [1.0], [1.0, 200.0, 1e-3], [1.0]):
        grads = [torch.randn(d, device=DEV) * scales[r % len(scales)] for r in range(P)]
        for r, g in zip(ranks, grads):
            r.selector.select(g, r.resid, k)
        ex.launch_allgather(ranks, desc, seg_counts, 0, P, k, reselect=True, nctas=nctas, limit_ms=2000)
        torch.cuda.synchronize()
        local = [oracle.compress(g.cpu(), rr, k) for g, rr in zip(grads, res_ref)]
        gi_ref, gv_ref = oracle.topk2_reselect(local, k)
        ref = dict(zip(gi_ref.tolist(), gv_ref.tolist()))
        for rr, loc in zip(res_ref, local):
            oracle.put_back(rr, loc, gi_ref)
        for r in ranks:
            assert r.status() == (0, 0)
            gi, gv = _read_gout(r, r.last_parity())
            got = dict(zip(gi.cpu().tolist(), gv.cpu().tolist()))
            assert set(got) == set(ref)
            for j in ref:
                assert got[j] == pytest.approx(ref[j], rel=1e-5, abs=1e-6)
            assert torch.allclose(r.resid.cpu(), res_ref[r.rank], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("sizes,k", [([5], 2), ([1, 2, 3, 4, 5, 130], 9), ([64] * 300, 100), ([100_003, 7, 1_000_001, 10, 999], 1000),
                                     ([20_000_001, 3, 4_000_000], 20_000)])
def test_k1_select_reads_one_tensor_per_parameter(sizes, k):
    """The gradient in one tensor per parameter, some of them at odd addresses
    and one missing, equals the same select over one vector; static and dynamic
    stream pass, tails of 1 to 3 elements, segments shorter than a warp's row."""
    from gtopkssgd_b200.ops.select import segment_table
    torch.manual_seed(sum(sizes))
    offsets, at = [], 0
    for n in sizes:
        offsets.append(at)
        at = (at + n + 3) // 4 * 4
    d = offsets[-1] + sizes[-1]
    sel = _selector(d, k)
    table = segment_table(offsets, sizes, d, DEV)
    r = torch.zeros(d, device=DEV)
    for it in range(3):
        grads = [torch.randn(n + 1, device=DEV)[i % 2:][:n] for i, n in enumerate(sizes)]
        missing = 1 if len(sizes) > 1 and it == 2 else -1
        g = torch.zeros(d, device=DEV)
        for i, (o, t) in enumerate(zip(offsets, grads)):
            if i != missing:
                g[o:o + t.numel()] = t
        acc = g + r
        sel.select_segments([0 if i == missing else t.data_ptr() for i, t in enumerate(grads)], table, r, k)
        assert sel.status() == (0, 0)
        _check_selection(*sel.pairs(), r, acc, k)


@pytest.mark.parametrize("mode,P,k,nctas", [("topk2", 2, 9000, 2), ("topk2", 3, 4097, 1), ("topk2", 5, 2500, 4),
                                            ("gtopk", 2, 4097, 2), ("gtopk", 2, 9000, 4), ("gtopk", 4, 9000, 3)])
def test_exchange_of_the_same_indices_over_again(mode, P, k, nctas):
    """More entries per thread than its registers hold, and call after call with
    the same selections: received words, look-up tables and merge buffers still
    carry the same indices from the calls before, at other positions."""
    from gtopkssgd_b200.ops import exchange as ex
    d = 40000
    torch.manual_seed(P * k)
    ranks, desc = _emulated_world(P, d, k, mode)
    seg_counts = torch.zeros(P * ex.MAX_PEERS, dtype=torch.int32, device=DEV)
    common = torch.randn(d, device=DEV)
    grads = [common + torch.randn(d, device=DEV) for _ in range(P)]
    res_ref = [torch.zeros(d) for _ in range(P)]
    if mode == "topk2":
        local = [oracle.compress(g.cpu(), rr, k) for g, rr in zip(grads, res_ref)]
        gi, gv = oracle.topk2_reselect(local, k)
        for rr, loc in zip(res_ref, local):
            oracle.put_back(rr, loc, gi)
    else:
        (gi, gv), _ = oracle.simulate_gtopk_step([g.cpu() for g in grads], res_ref, k)
    order = torch.argsort(gi)
    for call in range(6):
        for r, g in zip(ranks, grads):
            r.resid.zero_()
            r.selector.select(g, r.resid, k)
        if mode == "topk2":
            ex.launch_allgather(ranks, desc, seg_counts, 0, P, k, reselect=True, nctas=nctas, limit_ms=2000)
        else:
            ex.launch_gtopk(ranks, desc, 0, P, k, nctas=nctas, limit_ms=2000)
        torch.cuda.synchronize()
        for r in ranks:
            assert r.status() == (0, 0)
            qi, qv = _read_gout(r, r.last_parity())
            o = torch.argsort(qi)
            assert torch.equal(qi[o].cpu().long(), gi[order].long())
            assert torch.allclose(qv[o].cpu(), gv[order], rtol=1e-5, atol=1e-6)
            assert torch.allclose(r.resid.cpu(), res_ref[r.rank], rtol=1e-5, atol=1e-6)
            assert r.region.guards_intact()


@pytest.mark.parametrize("step", [0.0, 2.0 ** -12, 2.0 ** -6, 0.5])  # continuous; 4, 260 and 10 000s of equal entries
@pytest.mark.parametrize("k,form", [(40_000, "select"), (200_000, "select"), (200_000, "compress")])
def test_k1_pick_settles_the_thresholds_bin_apart(k, form, step):
    """Many candidates: those in the threshold's bin are put aside and settled by
    one CTA, unless they are too many, which equal magnitudes make them."""
    d = 3_000_000
    torch.manual_seed(k)
    sel = _selector(d, k)
    r = torch.zeros(d, device=DEV)
    for it in range(4):
        g = torch.randn(d, device=DEV)
        if step:
            g = (g / step).round() * step
            r.copy_((r / step).round() * step)
        acc = g + r
        if form == "compress":
            idx, val = sel.compress(g, r, k)
        else:
            sel.select(g, r, k)
            idx, val = sel.pairs()
            idx, val = idx.long(), val.clone()
        assert sel.status() == (0, 0)
        _check_selection(idx, val, r, acc, k)


def test_selector_refuses_what_the_kernels_cannot_read():
    """Strided vectors, which the kernels would take for contiguous ones, and a
    segment table of another number of tensors."""
    from gtopkssgd_b200.ops.select import segment_table
    from gtopkssgd_b200.parallel.compression import TopKCompressor, compressors
    d, k = 1000, 10
    sel = _selector(d, k)
    wide = torch.randn(2 * d, device=DEV)
    kept, r = wide.clone(), torch.zeros(d, device=DEV)
    for g, res in ((wide[::2], r), (torch.randn(d, device=DEV), wide[::2])):
        with pytest.raises(AssertionError):
            sel.compress(g, res, k)
    TopKCompressor.clear()
    with pytest.raises(AssertionError):
        compressors["gtopk"].compress(wide[::2], "strided", ratio=0.01)
    TopKCompressor.clear()
    g = torch.randn(d, device=DEV)
    table = segment_table([0, 500], [500, 500], d, DEV)
    for addresses, t, res in (([g.data_ptr()] * 2, table, wide[::2]), ([g.data_ptr()] * 3, table, r),
                              ([g.data_ptr()], table, r), ([g.data_ptr()] * 2, table.long(), r)):
        with pytest.raises(AssertionError):
            sel.select_segments(addresses, t, res, k)
    torch.cuda.synchronize()
    assert torch.equal(wide, kept)


def test_tables_may_be_written_by_the_kernel_just_before():
    """The rank descriptors of an exchange and the segment table of a select are
    read behind the wait for the predecessor: it may be the kernel that wrote
    them.  (Before, they hold another valid set.)"""
    from gtopkssgd_b200.ops import exchange as ex
    from gtopkssgd_b200.ops.select import segment_table
    torch.manual_seed(2)
    P, d, k = 4, 20_000, 500
    worlds = [_emulated_world(P, d, k) for _ in range(2)]
    desc = worlds[0][1].clone()
    for it in range(6):
        ranks, _ = worlds[it & 1]
        grads = [torch.randn(d, device=DEV) for _ in range(P)]
        for r, g in zip(ranks, grads):
            r.resid.zero_()
            r.selector.select(g, r.resid, k)
        epochs = [int(r.epoch.item()) for w, _ in worlds for r in w]
        torch.cat([r.desc for r in ranks], out=desc)
        ex.launch_gtopk(ranks, desc, 0, P, k, nctas=1, limit_ms=2000)
        torch.cuda.synchronize()
        res = [torch.zeros(d) for _ in range(P)]
        (gi, gv), _ = oracle.simulate_gtopk_step([g.cpu() for g in grads], res, k)
        for r, want in zip(ranks, res):
            assert r.status() == (0, 0) and set(_read_gout(r, r.last_parity())[0].tolist()) == set(gi.tolist())
            assert torch.allclose(r.resid.cpu(), want, rtol=1e-5, atol=1e-9)
        now = [int(r.epoch.item()) for w, _ in worlds for r in w]
        assert [b - a for a, b in zip(epochs, now)] == [int(w == (it & 1)) for w in range(2) for _ in range(P)]
    sizes = [[400, 1600], [1600, 400]]
    tables = [segment_table([0, s[0]], s, 2000, DEV) for s in sizes]
    table, sel, r = tables[0].clone(), _selector(2000, 20), torch.zeros(2000, device=DEV)
    for it in range(6):
        s = sizes[it & 1]
        grads = [torch.randn(1600, device=DEV) for _ in s]
        acc = torch.cat([g[:n] for g, n in zip(grads, s)]) + r
        torch.add(tables[it & 1], 0, out=table)
        sel.select_segments([g.data_ptr() for g in grads], table, r, 20)
        _check_selection(*sel.pairs(), r, acc, 20)


@pytest.mark.parametrize("mode,P,k,nctas", [("gtopk", 2, 1000, 1), ("gtopk", 4, 2000, 1), ("gtopk", 2, 6000, 4), ("gtopk", 4, 9000, 3),
                                            ("gtopk", 2, 30_000, 40), ("topk2", 2, 1000, 1), ("topk2", 4, 6000, 4)])
def test_exchange_of_gradients_that_cancel(mode, P, k, nctas):
    """Ranks in pairs with almost opposite gradients: most of the largest entries
    cancel, so that the sums' k-th magnitude lies far below every rank's own, the
    bottom of the band that the re-select predicts.  (Sums of numbers of about 2
    are multiples of 2^-23 or so: at 30 000 of them over a range of 0.2, two at
    the k-th place may be equal, and either may be kept.)"""
    from gtopkssgd_b200.ops import exchange as ex
    d = 30 * k
    torch.manual_seed(P + k)
    ranks, desc = _emulated_world(P, d, k, mode)
    seg_counts = torch.zeros(P * ex.MAX_PEERS, dtype=torch.int32, device=DEV)
    for call in range(3):
        res_ref = [torch.zeros(d) for _ in range(P)]
        grads = []
        for r in range(0, P, 2):
            g = torch.randn(d, device=DEV)
            grads += [g, -g + 0.2 * torch.randn(d, device=DEV)]
        own = []
        for r, g in zip(ranks, grads):
            r.resid.zero_()
            r.selector.select(g, r.resid, k)
            own.append(float(r.selector.state[6:7].view(torch.float32)))
        if mode == "topk2":
            ex.launch_allgather(ranks, desc, seg_counts, 0, P, k, reselect=True, nctas=nctas, limit_ms=2000)
            local = [oracle.compress(g.cpu(), rr, k) for g, rr in zip(grads, res_ref)]
            gi, gv = oracle.topk2_reselect(local, k)
            for rr, loc in zip(res_ref, local):
                oracle.put_back(rr, loc, gi)
        else:
            ex.launch_gtopk(ranks, desc, 0, P, k, nctas=nctas, limit_ms=2000)
            (gi, gv), _ = oracle.simulate_gtopk_step([g.cpu() for g in grads], res_ref, k)
        torch.cuda.synchronize()
        cut = float(gv.abs().min())
        assert cut < 0.5 * min(own)
        ref = dict(zip(gi.tolist(), gv.tolist()))
        for r, want in zip(ranks, res_ref):
            assert r.status() == (0, 0)
            qi, qv = _read_gout(r, r.last_parity())
            got = dict(zip(qi.cpu().tolist(), qv.cpu().tolist()))
            assert len(got) == qi.numel() == len(ref)
            swapped = set(got) ^ set(ref)
            assert len(swapped) <= 2 and all(abs({**ref, **got}[j]) == pytest.approx(cut, rel=1e-6) for j in swapped)
            for j in set(got) & set(ref):
                assert got[j] == pytest.approx(ref[j], rel=1e-5, abs=1e-6)
            same = torch.ones(d, dtype=torch.bool)
            same[list(swapped)] = False
            assert torch.allclose(r.resid.cpu()[same], want[same], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("mode,P,k,nctas", [("topk2", 8, 60_000, None), ("gtopk", 2, 200_000, None),
                                            ("topk2", 8, 60_000, 4), ("gtopk", 2, 200_000, 3)])
def test_exchange_stages_many_entries_per_cta(mode, P, k, nctas):
    """1 300 to 1 650 winners per CTA with the CTA counts that the exchange takes
    by itself, so that the stage in shared memory (emptied above 1 536) fills at the
    end of a call if at all; 15 000 and 66 000 with few CTAs, where it fills and
    empties 9 and 43 times in every call.  All threads of a CTA have to agree on when
    it is full: where they did not, 8 ranks of 170 000 entries (4 600 winners per CTA)
    lost their place in the output list in about one call of 50."""
    from gtopkssgd_b200.ops import exchange as ex
    d = 1_000_000
    torch.manual_seed(P)
    ranks, desc = _emulated_world(P, d, k, mode)
    seg_counts = torch.zeros(P * ex.MAX_PEERS, dtype=torch.int32, device=DEV)
    grads = [torch.randn(d, device=DEV) for _ in range(P)]
    total = torch.zeros(d, device=DEV)
    for r, g in zip(ranks, grads):
        r.selector.select(g, r.resid, k)
        idx, val = r.selector.pairs()
        total[idx] += val
    want = total.abs().topk(k).values[-1]
    for call in range(60):
        if mode == "topk2":
            ex.launch_allgather(ranks, desc, seg_counts, 0, P, k, reselect=True, nctas=nctas, limit_ms=1000)
        else:
            ex.launch_gtopk(ranks, desc, 0, P, k, nctas=nctas, limit_ms=1000)
    torch.cuda.synchronize()
    for r in ranks:
        assert r.status() == (0, 0)
        gi, gv = _read_gout(r, r.last_parity())
        assert gi.unique().numel() == k
        assert torch.allclose(gv, total[gi], rtol=1e-5, atol=1e-6)
        assert float(gv.abs().min()) == pytest.approx(float(want), rel=1e-5)


@pytest.mark.parametrize("n,capacity,nseg", [(0, 5, 1), (1, 1, 1), (257, 300, 3), (256, 100_000, 2), (4_849_665, 4_900_000, 1)])
@pytest.mark.parametrize("momentum", [0.0, 0.9])
def test_k3_sparse_covers_lists_below_at_and_beyond_its_grid(n, capacity, nseg, momentum):
    """List lengths at the edge of a CTA, capacities far above the length, and
    more entries than the largest grid has threads; with the order of a list's
    entries at random, distinct within a segment."""
    from gtopkssgd_b200.ops.sgd import SgdHyper, sgd_sparse
    d = max(4 * capacity, 64)
    torch.manual_seed(n + nseg)
    gen = torch.Generator(device=DEV).manual_seed(n)
    p0 = torch.randn(d, device=DEV, generator=gen)
    p, buf = p0.clone(), torch.zeros(d, device=DEV)
    pairs = torch.zeros((nseg * capacity, 2), dtype=torch.int32, device=DEV)
    want = torch.zeros(d, dtype=torch.float64, device=DEV)
    for s in range(nseg):
        idx = torch.randperm(d, device=DEV, generator=gen)[:n]
        val = torch.randn(n, device=DEV, generator=gen)
        pairs[s * capacity:s * capacity + n, 0] = idx.int()
        pairs[s * capacity:s * capacity + n, 1] = val.view(torch.int32)
        want.index_add_(0, idx, val.double())
    counts = torch.full((nseg,), n, dtype=torch.int32, device=DEV)
    h = SgdHyper(lr=0.1, momentum=momentum)
    sgd_sparse(p, buf if momentum else None, pairs, counts, nseg, capacity, h, True, 0.5, use_atomics=nseg > 1)
    # each addition rounds once to 24 bits: values below 8, at most 2 * nseg roundings
    assert torch.allclose(p.double(), p0.double() - 0.05 * want, rtol=0, atol=2 * nseg * 8 * 2.0 ** -24)
    if momentum:
        assert torch.allclose(buf.double(), 0.5 * want, rtol=0, atol=2 * nseg * 8 * 2.0 ** -24)


@pytest.mark.parametrize("n,capacity,nseg,max_count", [(300, 300, 1, 0), (300, 300, 3, 0), (300, 1000, 3, 300), (2000, 2000, 3, 100),
                                                       (100_000, 100_000, 3, 0), (1_300_000, 1_400_000, 1, 1_300_000)])
@pytest.mark.parametrize("momentum", [0.0, 0.9])
def test_k3_sparse_takes_the_live_half_of_two(n, capacity, nseg, max_count, momentum):
    """Lists that alternate between two halves, as the exchanges leave them:
    the half of the call counter is applied, whether entries are read ahead of it
    (few, in a tensor that holds both halves), behind it (many, or a tensor that
    ends before the second half's lists do), or in a loop (lists longer than
    expected, or than the largest grid)."""
    from gtopkssgd_b200.ops.sgd import SgdHyper, sgd_sparse
    d, stride = 4 * capacity, 4 * capacity  # (room for four lists per half)
    gen = torch.Generator(device=DEV).manual_seed(n + nseg)
    p0 = torch.randn(d, device=DEV, generator=gen)
    pairs = torch.zeros((2 * stride, 2), dtype=torch.int32, device=DEV)
    want = torch.zeros((2, d), dtype=torch.float64, device=DEV)
    for half in range(2):
        for s in range(nseg):
            at = half * stride + s * capacity
            idx = torch.randperm(d, device=DEV, generator=gen)[:n]
            val = torch.randn(n, device=DEV, generator=gen)
            pairs[at:at + n, 0] = idx.int()
            pairs[at:at + n, 1] = val.view(torch.int32)
            want[half].index_add_(0, idx, val.double())
    counts = torch.full((nseg,), n, dtype=torch.int32, device=DEV)
    h = SgdHyper(lr=0.1, momentum=momentum)
    for word in (1, 2, 3):
        for given in (pairs, pairs[:nseg * capacity]):  # the second one's later half lies behind its end
            p, buf = p0.clone(), torch.zeros(d, device=DEV)
            sgd_sparse(p, buf if momentum else None, given, counts, nseg, capacity, h, True, 0.5, use_atomics=nseg > 1,
                       parity_word=torch.tensor([word], dtype=torch.int32, device=DEV), parity_stride=stride,
                       max_count=max_count)
            step = 0.5 * want[(word - 1) & 1]
            # each addition rounds once to 24 bits: values below 16, at most 2 * nseg roundings
            assert torch.allclose(p.double(), p0.double() - 0.1 * step, rtol=0, atol=2 * nseg * 16 * 2.0 ** -24)
            if momentum:
                assert torch.allclose(buf.double(), step, rtol=0, atol=2 * nseg * 16 * 2.0 ** -24)


@pytest.mark.parametrize("d,k", [(19_000, 18_001), (100_000, 18_000), (100_000, 18_001), (3_000_000, 12_289), (6_000_000, 130_000),
                                 (5_000_000, 1_300_000), (33_000, 32_769), (49_152, 16_001), (100_000, 22_001),
                                 (200_000, 12_289), (800_000, 18_001)])
@pytest.mark.parametrize("form", ["select", "compress", "ties"])
def test_k1_pick_shares_many_candidates_out(d, k, form):
    """The pick without clusters, from its smallest k on (compress's lies below
    select's): nearly everything selected, shares of less and of more than one round, few CTAs and all of
    them, and candidates so often equal that the threshold's bin is counted by
    finer levels or is a single magnitude."""
    torch.manual_seed(k)
    sel = _selector(d, k)
    r = torch.zeros(d, device=DEV)
    for it in range(4):
        g = torch.randn(d, device=DEV)
        if form == "ties":
            g = (g * 8).round() / 8
            r.zero_()
        acc = g + r
        if form == "compress":
            idx, val = sel.compress(g, r, k)
            want = torch.zeros(d, device=DEV)
            want[idx] = val
            assert torch.equal(g, want)
        else:
            sel.select(g, r, k)
            idx, val = sel.pairs()
        assert sel.status() == (0, 0)
        _check_selection(idx, val, r, acc, k)


@pytest.mark.parametrize("d,k,form", [(100_000, 22_001, "select"), (3_000_000, 12_289, "select"), (6_000_000, 130_000, "select"),
                                      (200_000, 12_289, "compress"), (4_000_000, 20_000, "compress")])
def test_k1_pick_without_clusters_predicts_and_recovers(d, k, form):
    """Steady inputs take one exact pass, the first.  Too few candidates, or more
    than their list holds, take another, which first puts back into the residual
    what the stream pass took out of it."""
    torch.manual_seed(d)
    sel = _selector(d, k)
    r = torch.zeros(d, device=DEV)

    def call(g):
        r.normal_().mul_(1e-3)
        acc = g + r
        if form == "compress":
            idx, val = sel.compress(g, r, k)
            want = torch.zeros(d, device=DEV)
            want[idx] = val
            assert torch.equal(g, want)
        else:
            sel.select(g, r, k)
            idx, val = sel.pairs()
        assert sel.status() == (0, 0)
        _check_selection(idx, val, r, acc, k)
        return sel.stats()

    for it in range(6):
        st = call(torch.randn(d, device=DEV))
        assert st["n_fallbacks"] == 1 and (it == 0 or k <= st["n_cand"] <= sel.cap)
    g = torch.randn(d, device=DEV) * 1e-3
    g[torch.randperm(d, device=DEV)[:k // 2]] = 50.0
    st = call(g)
    assert st["n_cand"] == k // 2 and st["n_fallbacks"] == 2
    call(torch.randn(d, device=DEV))
    call(torch.randn(d, device=DEV))
    before = sel.stats()["n_fallbacks"]
    st = call(torch.randn(d, device=DEV) * 1000.0)
    assert st["n_cand"] > 0.9 * d and st["n_fallbacks"] == before + (1 if st["n_cand"] > sel.cap else 0)
    assert (st["n_cand"] > sel.cap) == (32 * k < 0.9 * d)


@pytest.mark.parametrize("d,max_k,kcap", [(20_000, 300, 1000), (400_000, 3000, 9000)])  # one CTA per rank, several
def test_exchange_with_selections_shorter_than_its_k(d, max_k, kcap):
    """The exchange may be set up for more entries than its selectors ever
    deliver: all of them stay, and nothing from behind them gets in.  (That the kernels
    are told where a selection's buffer ends is checked on the host.)"""
    from gtopkssgd_b200.ops import exchange as ex
    torch.manual_seed(d)
    P = 2
    regions = ex.SymmetricRegion.create_emulated(P, ex.region_bytes(kcap, False), DEV)
    ranks, sels, grads = [], [], [torch.randn(d, device=DEV) for _ in range(P)]
    for r in range(P):
        sel, resid = _selector(d, max_k), torch.zeros(d, device=DEV)
        ranks.append(ex.ExchangeRank(r, P, d, kcap, sel, resid, regions[r]))
        sel.select(grads[r], resid, max_k)
        sels.append(sel.pairs())
    ex.launch_gtopk(ranks, torch.cat([r.desc for r in ranks]), 0, P, kcap, limit_ms=2000)
    torch.cuda.synchronize()
    total = torch.zeros(d, device=DEV)
    for idx, val in sels:
        total[idx] += val
    for r in ranks:
        assert r.status() == (0, 0)
        gi, gv = _read_gout(r, r.last_parity())
        assert sorted(gi.tolist()) == total.nonzero().view(-1).tolist()
        assert torch.equal(gv, total[gi])
