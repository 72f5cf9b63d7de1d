"""GPU end-to-end tests: the DistributedOptimizer on CUDA (fused select,
fused sparse SGD step, side stream) replayed against the oracle, on one GPU
and -- when the box has them -- on 2 and 4 GPUs through the peer-store
exchange kernel over CUDA IPC."""
import gc

import pytest
import torch

import _workers
from test_distributed_cpu import replay_and_check
from gtopkssgd_b200.ops import oracle
from gtopkssgd_b200.utils.launch import spawn_ranks

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release_trainers():
    """A trainer and its captured graphs form cycles; collected here, their memory
    is not given back in the middle of a later test that watches the allocator."""
    yield
    gc.collect()


@pytest.mark.parametrize("compressor", ["gtopk", "none"])
def test_single_gpu_training_matches_oracle(compressor):
    traces = spawn_ranks(_workers.resnet20_gtopk_worker, 1, args=(4, 0.001, compressor, "cuda"), timeout_s=300)
    replay_and_check(traces, 0.001, compressor, rtol=1e-4, atol=1e-5)


def test_single_gpu_three_merge_groups_overlap_backward():
    """Three merged groups: the select of a finished group runs on the side
    stream while backward continues."""
    traces = spawn_ranks(_workers.resnet20_gtopk_worker, 1, args=(4, 0.001, "gtopk", "cuda", 100000), timeout_s=300)
    assert len(traces[0]["groups"]) == 3
    replay_and_check(traces, 0.001, "gtopk", rtol=1e-4, atol=1e-5)


@pytest.mark.multigpu
def test_two_gpu_three_merge_groups():
    traces = spawn_ranks(_workers.resnet20_gtopk_worker, 2, args=(4, 0.001, "gtopk", "cuda", 100000), timeout_s=300,
                         env={"NCCL_NVLS_ENABLE": "0"})
    replay_and_check(traces, 0.001, "gtopk", rtol=1e-4, atol=1e-5)


@pytest.mark.multigpu
@pytest.mark.parametrize("compressor", ["gtopk", "topk", "topk2", "none"])
def test_two_gpu_training_matches_oracle(compressor):
    env = {"NCCL_NVLS_ENABLE": "0"}
    traces = spawn_ranks(_workers.resnet20_gtopk_worker, 2, args=(4, 0.001, compressor, "cuda"), timeout_s=300,
                         env=env)
    replay_and_check(traces, 0.001, compressor, rtol=1e-4, atol=1e-5)


@pytest.mark.multigpu
@pytest.mark.parametrize("compressor", ["gtopk", "topk2"])
def test_two_gpu_staged_transport_matches_oracle(compressor):
    """Ranks without GPU peer access (several hosts) exchange through the host
    and gloo; forced here on one host."""
    env = {"NCCL_NVLS_ENABLE": "0", "GTOPK_TRANSPORT": "staged"}
    traces = spawn_ranks(_workers.resnet20_gtopk_worker, 2, args=(4, 0.001, compressor, "cuda"), timeout_s=300,
                         env=env)
    replay_and_check(traces, 0.001, compressor, rtol=1e-4, atol=1e-5)


@pytest.mark.multigpu
def test_four_gpu_gtopk_matches_oracle():
    if torch.cuda.device_count() < 4:
        pytest.skip("needs 4 GPUs")
    traces = spawn_ranks(_workers.resnet20_gtopk_worker, 4, args=(3, 0.001, "gtopk", "cuda"), timeout_s=300,
                         env={"NCCL_NVLS_ENABLE": "0"})
    replay_and_check(traces, 0.001, "gtopk", rtol=1e-4, atol=1e-5)


@pytest.mark.multigpu
def test_eight_gpu_gtopk_matches_oracle():
    if torch.cuda.device_count() < 8:
        pytest.skip("needs 8 GPUs")
    traces = spawn_ranks(_workers.resnet20_gtopk_worker, 8, args=(3, 0.001, "gtopk", "cuda"), timeout_s=300,
                         env={"NCCL_NVLS_ENABLE": "0"})
    replay_and_check(traces, 0.001, "gtopk", rtol=1e-4, atol=1e-5)


def _check_real_peer_exchange(out, world, d, k, epochs):
    res_ref = [torch.zeros(d) for _ in range(world)]
    for e in range(epochs):
        # the same Philox stream as in the workers (seed-determined, whatever the device index)
        grads = [torch.randn(d, device="cuda:0", generator=torch.Generator(device="cuda:0").manual_seed(1000 * e + r)).cpu()
                 for r in range(world)]
        glob, local = oracle.simulate_gtopk_step(grads, res_ref, k)
        ref = dict(zip(glob[0].tolist(), glob[1].tolist()))
        for r in range(world):
            ep = out[r]["epochs"][e]
            assert tuple(ep["status"]) == (0, 0) and ep["guards"], (e, r, ep["status"])
            assert set(ep["local"][0].tolist()) == set(local[r][0].tolist()), "epoch %d rank %d: local selection" % (e, r)
            got = dict(zip(ep["global"][0].tolist(), ep["global"][1].tolist()))
            assert len(got) == k and set(got) == set(ref), \
                "epoch %d rank %d: %d extra, %d missing in the global set" % (e, r, len(set(got) - set(ref)), len(set(ref) - set(got)))
            for j, v in ref.items():
                assert got[j] == pytest.approx(v, rel=1e-5, abs=1e-6)
            assert torch.allclose(ep["resid"], res_ref[r], rtol=1e-5, atol=1e-6)


@pytest.mark.multigpu
@pytest.mark.parametrize("d,k,nctas", [(1_000_000, 1000, 1), (1_000_000, 5000, 4), (2_000_000, 14000, 16),
                                       (2_000_000, 20000, 24)])  # one CTA; clusters of 4 and 16; software barrier
def test_exchange_kernel_between_real_gpus_matches_oracle(d, k, nctas):
    """The multi-CTA forms of the exchange over NVLink peers: what the emulated single-GPU tests cannot
    see is whether a partner's flag can overtake data still in flight from other SMs."""
    world = 4 if torch.cuda.device_count() >= 4 else 2
    epochs = 6
    out = spawn_ranks(_workers.real_peer_exchange_worker, world, args=(d, k, nctas, epochs), timeout_s=300,
                      env={"NCCL_NVLS_ENABLE": "0"})
    _check_real_peer_exchange(out, world, d, k, epochs)


@pytest.mark.multigpu
@pytest.mark.parametrize("nctas", [1, 8])
def test_allgather_reselect_kernel_between_real_gpus_matches_oracle(nctas):
    """'topk2' over NVLink peers with one and with several CTAs per rank: every rank pushes its pairs into
    every peer's all-gather slots, merges the P lists in rank order and re-selects."""
    world = 4 if torch.cuda.device_count() >= 4 else 2
    d, k, epochs = 1_000_000, 4000, 4
    out = spawn_ranks(_workers.real_peer_exchange_worker, world, args=(d, k, nctas, epochs, "topk2"), timeout_s=300,
                      env={"NCCL_NVLS_ENABLE": "0"})
    res_ref = [torch.zeros(d) for _ in range(world)]
    for e in range(epochs):
        grads = [torch.randn(d, device="cuda:0", generator=torch.Generator(device="cuda:0").manual_seed(1000 * e + r)).cpu()
                 for r in range(world)]
        local = [oracle.compress(g, r, k) for g, r in zip(grads, res_ref)]
        gi_ref, gv_ref = oracle.topk2_reselect(local, k)
        for r, loc in zip(res_ref, local):
            oracle.put_back(r, loc, gi_ref)
        ref = dict(zip(gi_ref.tolist(), gv_ref.tolist()))
        for r in range(world):
            ep = out[r]["epochs"][e]
            assert tuple(ep["status"]) == (0, 0) and ep["guards"]
            got = dict(zip(ep["global"][0].tolist(), ep["global"][1].tolist()))
            assert len(got) == k and set(got) == set(ref), "epoch %d rank %d" % (e, r)
            for j, v in ref.items():
                assert got[j] == pytest.approx(v, rel=1e-5, abs=1e-6)
            assert torch.allclose(ep["resid"], res_ref[r], rtol=1e-5, atol=1e-6)


@pytest.mark.multigpu
def test_exchange_kernel_between_eight_gpus_matches_oracle():
    if torch.cuda.device_count() < 8:
        pytest.skip("needs 8 GPUs")
    d, k, epochs = 2_000_000, 14000, 4
    out = spawn_ranks(_workers.real_peer_exchange_worker, 8, args=(d, k, 16, epochs), timeout_s=300,
                      env={"NCCL_NVLS_ENABLE": "0"})
    _check_real_peer_exchange(out, 8, d, k, epochs)


def test_single_gpu_cuda_graph_step_matches_oracle():
    traces = spawn_ranks(_workers.graphed_step_worker, 1, args=(7, "gtopk"), timeout_s=300)
    assert traces[0]["graphs"] == 1
    replay_and_check(traces, 0.001, "gtopk", rtol=1e-4, atol=1e-5)


@pytest.mark.multigpu
@pytest.mark.parametrize("compressor,graphs", [("gtopk", 1), ("none", 0)])
def test_two_gpu_cuda_graph_step_matches_oracle(compressor, graphs):
    """gTop-k iterations are captured (peer-store exchange inside the graph);
    dense multi-GPU iterations stay eager by design."""
    traces = spawn_ranks(_workers.graphed_step_worker, 2, args=(7, compressor), timeout_s=240,
                         env={"NCCL_NVLS_ENABLE": "0"})
    assert traces[0]["graphs"] == graphs
    replay_and_check(traces, 0.001, compressor, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("graph", [False, True])
def test_train_step_leaves_backwards_own_gradients(graph):
    """An iteration that the trainer runs takes the gradients where backward left
    them; ``zero_grad`` and the flat gradient buffer work as before around it."""
    from gtopkssgd_b200 import settings
    from gtopkssgd_b200.parallel.compression import compressors
    from gtopkssgd_b200.parallel.distributed_optimizer import DistributedOptimizer
    from gtopkssgd_b200.trainer.dl_trainer import DLTrainer
    settings.PIN_DENSITY = True
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    t = DLTrainer(0, 1, dist=False, ngpus=1, batch_size=8, data_dir="synthetic", dataset="cifar10", dnn="resnet20", lr=0.1,
                  nworkers=1, device=dev, synthetic_train_size=640, cuda_graph=graph)
    opt = DistributedOptimizer(t.optimizer, t.net.named_parameters(), compression=compressors["gtopk"], is_sparse=True,
                               density=0.01)
    t.update_optimizer(opt)
    fb = opt._flat
    batch = (torch.randn(8, 3, 32, 32, device=dev), torch.randint(0, 10, (8,), device=dev))
    for it in range(6):
        before = fb.residual.clone()
        t.train_step(data=batch)
        assert not fb.grads_attached()
        want = torch.cat([p.grad.flatten() for p in (s.param for s in fb.slots.values())])
        got = torch.cat([fb.grad[s.offset:s.offset + s.numel] for s in fb.slots.values()])
        assert torch.equal(want, got)
        idx, val = opt._allreducer.engines[0].selector.pairs()
        acc = (fb.grad + before)[:fb.numel]
        assert torch.equal(val, acc[idx])
        acc[idx] = 0.0
        assert torch.equal(fb.residual[:fb.numel], acc)
    opt.zero_grad()
    assert fb.grads_attached() and float(fb.grad.abs().sum()) == 0.0
    t.criterion(t.net(batch[0]), batch[1]).backward()   # an iteration of the user's own
    assert fb.grads_attached() and float(fb.grad.abs().sum()) > 0.0
    opt.step()
    opt.check_status()
    opt.stop()


def test_graft_smoke():
    import __graft_entry__ as g
    g.smoke()


def test_prefetched_batches_train_like_host_batches():
    """DLTrainer.prefetch copies a pinned batch on a side stream.  The consumer
    sees exactly the host data (also while the compute stream is busy), and
    ``train_step`` takes the handle in the eager and the CUDA-graph path: the
    first step, which depends only on the initial weights and the batch, gives
    the same loss as with the host batch."""
    import torch
    from gtopkssgd_b200.trainer.dl_trainer import DLTrainer, PrefetchedBatch

    def trainer(graph):
        torch.manual_seed(0)
        return DLTrainer(0, 1, dist=False, ngpus=1, batch_size=8, data_dir="synthetic", dataset="cifar10",
                         dnn="resnet20", lr=0.1, nworkers=1, device=torch.device("cuda", 0), synthetic_train_size=64,
                         cuda_graph=graph)

    g = torch.Generator().manual_seed(1)
    batches = [(torch.randn(8, 3, 32, 32, generator=g).pin_memory(),
                torch.randint(0, 10, (8,), generator=g).pin_memory()) for _ in range(6)]
    t = trainer(False)
    busy = torch.randn(4096, 4096, device="cuda")
    for b in batches * 3:
        h = t.prefetch(b)
        assert isinstance(h, PrefetchedBatch) and t.prefetch(h) is h
        busy = busy @ busy * 1e-4          # keeps the compute stream occupied while the copy runs
        x, y, _, _ = t._to_device(h)
        assert torch.equal(x.cpu(), b[0]) and torch.equal(y.cpu(), b[1])

    for graph in (False, True):
        first = {}
        for prefetch in (False, True):
            t = trainer(graph)
            nxt, losses = None, []
            for i, b in enumerate(batches):
                if prefetch:
                    cur = nxt if nxt is not None else t.prefetch(b)
                    nxt = t.prefetch(batches[i + 1]) if i + 1 < len(batches) else None
                else:
                    cur = b
                t.train_step(data=cur)
                losses.append(t.loss)
            assert all(l == l and l < 1e3 for l in losses)
            first[prefetch] = losses[0]
        assert abs(first[False] - first[True]) < 1e-4, first


@pytest.mark.multigpu
@pytest.mark.parametrize("leaver", [0, 1])
def test_two_gpu_planned_departure(leaver):
    """One of two GPU ranks announces its departure (between iterations,
    nothing in flight); the other closes its peer mappings, leaves the NCCL
    group and trains on alone from the agreed iteration."""
    total = 12
    out = spawn_ranks(_workers.elastic_worker, 2, args=("gtopk", leaver, 3, total, "cuda"), timeout_s=300,
                      env={"NCCL_NVLS_ENABLE": "0"})
    other = 1 - leaver
    at = out[leaver]["left_at"]
    assert at == 6 and out[leaver]["iters"] == at
    o = out[other]
    assert o["iters"] == total and o["calls"] == [(1, 0)]
    assert [h[1] for h in o["hist"]] == [2] * at + [1] * (total - at)
    import torch
    assert torch.isfinite(o["params"]).all() and not torch.equal(o["params"], out[leaver]["params"])


@pytest.mark.parametrize("rows,classes", [(1, 1), (33, 10), (128, 31), (64, 1000), (2000, 100)])
def test_top1_accuracy_matches_library(rows, classes):
    from gtopkssgd_b200.ops import accuracy
    torch.manual_seed(rows)
    x = torch.randn(rows, classes, device="cuda")
    y = torch.randint(0, classes, (rows,), device="cuda")
    x[0, classes - 1] = float("nan")
    assert accuracy.takes(x, y)
    want = 100.0 * x.topk(1, 1).indices[:, 0].eq(y).float().mean()
    assert float(accuracy.top1_percent(x, y)) == pytest.approx(float(want), abs=1e-4)


def test_batch_counters_advance_like_the_layers_do():
    from gtopkssgd_b200.models import create_net
    from gtopkssgd_b200.trainer.dl_trainer import BatchCounters
    nets = []
    for _ in range(2):
        torch.manual_seed(0)
        nets.append(create_net(10, "resnet20")[0].cuda())
    frozen = [n.stage_2[0].bn_a.eval() for n in nets]
    x = torch.randn(4, 3, 32, 32, device="cuda")
    counters = BatchCounters(nets[0])
    for _ in range(3):
        a, b = counters.forward(nets[0], x), nets[1](x)
    assert torch.allclose(a, b, atol=1e-5) and int(frozen[0].num_batches_tracked) == 0
    for (k, u), v in zip(nets[0].state_dict().items(), nets[1].state_dict().values()):
        assert torch.allclose(u, v, atol=1e-5) if u.is_floating_point() else torch.equal(u, v), k


def test_direct_layer_calls_keep_hooks_and_results():
    """The residual block's direct library calls give the layers' results bit for
    bit, and a layer with a hook is called as a layer."""
    from gtopkssgd_b200.models import create_net, direct
    torch.manual_seed(0)
    net = create_net(10, "resnet20")[0].cuda()
    x = torch.randn(4, 16, 32, 32, device="cuda")
    block = net.stage_1[0]
    for conv, bn in ((block.conv_a, block.bn_a), (block.conv_b, block.bn_b)):
        y = direct.conv(conv, x)
        assert torch.equal(y, conv(x))
        before = bn.running_mean.clone()
        a = direct.batch_norm(bn, y)
        moved, bn.running_mean[:] = bn.running_mean.clone(), before
        assert torch.equal(a, bn(y)) and torch.equal(moved, bn.running_mean) and int(bn.num_batches_tracked) == 2
    seen = []
    handle = block.conv_a.register_forward_hook(lambda *a: seen.append(1))
    block(x)
    handle.remove()
    block.eval()(x)
    assert len(seen) == 1


def _on_a_side_stream(opt):
    """A single worker's optimizer reduces on the side stream, as those of several workers do."""
    opt._overlap = opt._allreducer.concurrent = True
    opt._ready = [torch.cuda.Event() for _ in opt._flat.groups]


@pytest.mark.parametrize("graph", [False, True])
def test_reduction_is_launched_before_the_dense_part(graph, monkeypatch):
    """With one merged group nothing has launched the reduction when ``step``
    begins: it goes out first, the dense part behind this iteration's select, in
    eager iterations, in a captured one and in an eager one after it, with the
    results of a reduction on the compute stream."""
    from gtopkssgd_b200 import settings
    from gtopkssgd_b200.parallel import distributed_optimizer as do
    from gtopkssgd_b200.parallel.compression import compressors
    from gtopkssgd_b200.trainer.dl_trainer import DLTrainer
    monkeypatch.setattr(settings, "PIN_DENSITY", True)
    monkeypatch.setattr(torch.backends.cudnn, "deterministic", True)
    order = []
    plain_dense = do.sgd_dense
    monkeypatch.setattr(do, "sgd_dense", lambda *a, **kw: (order.append("dense"), plain_dense(*a, **kw)))
    dev = torch.device("cuda", 0)
    batches = [(torch.randn(8, 3, 32, 32, device=dev), torch.randint(0, 10, (8,), device=dev)) for _ in range(7)]
    results = []
    for side in (False, True):
        torch.manual_seed(0)
        t = DLTrainer(0, 1, dist=False, ngpus=1, batch_size=8, data_dir="synthetic", dataset="cifar10", dnn="resnet20",
                      lr=0.1, nworkers=1, device=dev, synthetic_train_size=640, cuda_graph=graph)
        opt = do.DistributedOptimizer(t.optimizer, t.net.named_parameters(), compression=compressors["gtopk"],
                                      is_sparse=True, density=0.01)
        t.update_optimizer(opt)
        if side:
            _on_a_side_stream(opt)
        reduce_group = opt._allreducer.reduce_group
        monkeypatch.setattr(opt._allreducer, "reduce_group",
                            lambda *a, f=reduce_group: (order.append("reduce"), f(*a)))
        del order[:]
        for i, b in enumerate(batches):
            t.train_step(data=b, cuda_graph=graph and i < 6)
        if side:   # eager iterations, and the captured one once
            assert order == ["reduce", "dense"] * (5 if graph else 7)
        opt.check_status()
        results.append([opt._flat.param.clone(), opt._flat.momentum.clone(), opt._flat.residual.clone()])
        opt.stop()
    for a, b in zip(*results):
        assert torch.equal(a, b)


def test_parameters_carry_the_gradient_of_the_last_replay():
    """Two captured batch shapes in turn, with an iteration of the user's own in
    between: ``p.grad`` is the gradient of the last iteration each time."""
    from gtopkssgd_b200 import settings
    from gtopkssgd_b200.parallel.compression import compressors
    from gtopkssgd_b200.parallel.distributed_optimizer import DistributedOptimizer
    from gtopkssgd_b200.trainer.dl_trainer import DLTrainer
    settings.PIN_DENSITY = True
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    t = DLTrainer(0, 1, dist=False, ngpus=1, batch_size=8, data_dir="synthetic", dataset="cifar10", dnn="resnet20", lr=0.1,
                  nworkers=1, device=dev, synthetic_train_size=640, cuda_graph=True)
    opt = DistributedOptimizer(t.optimizer, t.net.named_parameters(), compression=compressors["gtopk"], is_sparse=True,
                               density=0.01)
    t.update_optimizer(opt)
    fb = opt._flat
    params = [s.param for s in fb.slots.values()]

    def selected_from_gradients(before):
        """What the step selected, against the sum of residual and ``p.grad``."""
        idx, val = opt._allreducer.engines[0].selector.pairs()
        g = torch.zeros_like(before)
        for s in fb.slots.values():
            assert s.param.grad is not None
            g[s.offset:s.offset + s.numel] = s.param.grad.flatten()
        assert torch.equal(val, (g + before)[idx]) and torch.equal(fb.grad, g)

    for own, rows in ((0, 8), (0, 8), (0, 8), (0, 8), (0, 5), (0, 8), (0, 5), (1, 6), (0, 5), (0, 8), (2, 6), (0, 8)):
        batch = (torch.randn(rows, 3, 32, 32, device=dev), torch.randint(0, 10, (rows,), device=dev))
        before = fb.residual.clone()
        if own:   # the user's own loop, with the optimizer's zero_grad or the network's
            (opt if own == 1 else t.net).zero_grad()
            t.criterion(t.net(batch[0]), batch[1]).backward()
            opt.step()
        else:
            t.train_step(data=batch)
        selected_from_gradients(before)
    assert len(t._graphed.graphs) == 2
    opt.stop()


def test_gradients_replaced_by_the_user_are_taken_as_they_are():
    """A loop with the network's own ``zero_grad`` (``p.grad`` None) gives what the
    optimizer's gives, also for a parameter without a gradient in one iteration."""
    import test_framework_cpu as cpu
    cpu.check_replaced_gradients("cuda")


def test_top1_accuracy_of_another_device_takes_the_librarys_way(monkeypatch):
    from gtopkssgd_b200.ops import accuracy
    from gtopkssgd_b200.trainer.dl_trainer import DLTrainer
    x, y = torch.randn(6, 4, device="cuda:0"), torch.randint(0, 4, (6,), device="cuda:0")
    want = float(DLTrainer.cal_accuracy(x, y)[0])
    assert accuracy.takes(x, y)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    assert not accuracy.takes(x, y)
    assert float(DLTrainer.cal_accuracy(x, y)[0]) == pytest.approx(want, abs=1e-4)
