"""The work that users of this framework have it do on one GPU, as timed cases.

Five kinds of pass, each through the public entry points:

``train``     a whole iteration of a named model: ``DLTrainer.train_step`` with
              the wrapped optimizer (eager or as a captured CUDA graph).
``update``    a user's own training loop around ``DistributedOptimizer``:
              ``zero_grad``, gradients from backward, ``step``, for a parameter
              list of a given total size and layer count.
``select``    ``TopkSelector.select`` (residual add, exact top-k, residual
              write-back) and ``sgd_sparse`` with the selected pairs: the sparse
              path of one worker over a flat gradient.
``compress``  the stand-alone compressor, ``compressors[...].compress``.
``exchange``  one sparse exchange between P ranks held by one GPU
              (``launch_gtopk`` / ``launch_allgather``) with the residual
              put-back, and rank 0's sparse update with the global set.

Gradients are N(0, 1e-2), another one in every pass (windows of one buffer of
noise), and the residual starts in the state that error feedback keeps it in
after many iterations: an entry walks at random until it is sent, so its value
is spread like a triangle between plus and minus the sending threshold.  Which of
two entries of exactly equal magnitude is kept at the k-th place is not part of
the operation's meaning, so ``prepare`` moves such ties apart in its inputs.
"""
from __future__ import annotations

import math
import random

import torch

from gtopkssgd_b200 import settings
from gtopkssgd_b200.ops import exchange as ex
from gtopkssgd_b200.ops.oracle import num_selected
from gtopkssgd_b200.ops.select import TopkSelector
from gtopkssgd_b200.ops.sgd import SgdHyper, sgd_sparse
from gtopkssgd_b200.parallel.compression import TopKCompressor, compressors
from gtopkssgd_b200.parallel.distributed_optimizer import DistributedOptimizer
from gtopkssgd_b200.trainer.dl_trainer import DLTrainer

DEV = "cuda"
SIGMA = 1e-2     # scale of a gradient entry
WINDOWS = 32     # gradients that a state goes through
SHIFT = 64       # elements between the starts of two windows

# model -> data set, learning rate, clip norm, parameters, forward multiply-adds per sample
MODELS = {
    "resnet20": ("cifar10", 0.1, None, 269_722, 41e6),
    "resnet56": ("cifar10", 0.1, None, 853_018, 126e6),
    "vgg16": ("cifar10", 0.1, None, 14_728_266, 313e6),
    "resnet50": ("imagenet", 0.1, None, 25_557_032, 4.1e9),
    "lstm": ("ptb", 22.0, 0.25, 66_034_000, 35 * 51e6),
}


def listed():
    return [
        # CIFAR ResNet-20, 32 samples per worker, eager: the smallest network, launches and host work count
        {"name": "train-resnet20-eager", "kind": "train", "model": "resnet20", "batch": 32, "graph": False},
        # CIFAR VGG-16, 128 samples per worker, whole-iteration graph
        {"name": "train-vgg16-graph", "kind": "train", "model": "vgg16", "batch": 128, "graph": True},
        # PTB LSTM, 20 sequences of 35 tokens, gradient-norm clip, no momentum
        {"name": "train-lstm-graph", "kind": "train", "model": "lstm", "batch": 20, "graph": True},
        # ResNet-50, 64 images per worker: the headline configuration
        {"name": "train-resnet50-graph", "kind": "train", "model": "resnet50", "batch": 64, "graph": True},
        # own loop, ResNet-50's parameter count and number of tensors, momentum and weight decay
        {"name": "update-gtopk-25m", "kind": "update", "d": 25_557_032, "tensors": 161, "density": 0.001,
         "compressor": "gtopk", "momentum": 0.9, "weight_decay": 5e-4, "nesterov": False},
        # the dense path ('none') at VGG-16's size
        {"name": "update-dense-14m", "kind": "update", "d": 14_728_266, "tensors": 54, "density": 0.001,
         "compressor": "none", "momentum": 0.9, "weight_decay": 1e-4, "nesterov": False},
        # the smallest and the largest vector of the sparse all-reduce benchmark, at its two densities
        {"name": "select-1m", "kind": "select", "d": 1_000_000, "density": 0.001},
        {"name": "select-138m", "kind": "select", "d": 138_000_000, "density": 0.01},
        # stand-alone compressor on an odd length
        {"name": "compress-4m", "kind": "compress", "d": 4_000_037, "density": 0.001},
        # tree exchange of 8 ranks with small sets: a chain of short rounds
        {"name": "exchange-gtopk-8x1m", "kind": "exchange", "mode": "gtopk", "ranks": 8, "d": 1_000_000, "density": 0.001},
        # tree exchange of 2 ranks at the LSTM's size
        {"name": "exchange-gtopk-2x66m", "kind": "exchange", "mode": "gtopk", "ranks": 2, "d": 66_034_000, "density": 0.001},
        # all-gather with re-selection, 4 ranks at VGG-16's size
        {"name": "exchange-topk2-4x14m", "kind": "exchange", "mode": "topk2", "ranks": 4, "d": 14_728_266, "density": 0.001},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["train", "update", "update", "select", "select", "compress", "exchange", "exchange"])
    density = math.exp(rng.uniform(math.log(0.001), math.log(0.01)))
    if kind == "train":
        model = rng.choice(["resnet20", "resnet56", "vgg16", "lstm", "resnet50"])
        lo, hi = {"resnet20": (16, 256), "resnet56": (16, 128), "vgg16": (16, 192), "lstm": (10, 40),
                  "resnet50": (8, 48)}[model]
        return {"kind": kind, "model": model, "batch": _log_int(rng, lo, hi), "graph": rng.random() < 0.6}
    if kind == "update":
        d = _log_int(rng, 250_000, 138_000_000)
        return {"kind": kind, "d": d, "tensors": rng.randint(8, 200), "density": density,
                "compressor": rng.choice(["gtopk", "gtopk", "none"]), "momentum": rng.choice([0.9, 0.9, 0.0]),
                "weight_decay": rng.choice([1e-4, 5e-4, 0.0]), "nesterov": rng.random() < 0.25}
    if kind == "select":
        return {"kind": kind, "d": _log_int(rng, 250_000, 138_000_000), "density": density}
    if kind == "compress":
        return {"kind": kind, "d": _log_int(rng, 250_000, 64_000_000), "density": density}
    ranks = rng.choice([2, 4, 8])
    return {"kind": kind, "mode": rng.choice(["gtopk", "gtopk", "topk", "topk2"]), "ranks": ranks,
            "d": _log_int(rng, 250_000, 138_000_000 // ranks), "density": density}


# -- inputs -------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _untie(g, acc, k):
    """Raises tied entries at the k-th magnitude of ``acc`` (through ``g``, in
    place, ``acc`` alike) until the k largest are separate from the rest.
    Returns the indices of the k largest."""
    n = acc.numel()
    for _ in range(4):
        mag, idx = torch.topk(acc.abs(), min(k + 1, n), sorted=True)
        if k >= n or bool(mag[k - 1] > mag[k]):
            break
        t = mag[k]
        tied = (acc.abs() == t).nonzero().view(-1)
        tied = tied[:k - int((mag[:k] > t).sum())]
        step = acc[tied].sign() * (t * 1e-3)
        g[tied] += step
        acc[tied] += step
    return idx[:k]


def _residual(d, density, gen):
    """Steady state of the residual: entries leave at about sigma / sqrt(density)."""
    r = torch.rand(d, device=DEV, generator=gen)
    r += torch.rand(d, device=DEV, generator=gen)
    return r.sub_(1.0).mul_(SIGMA / math.sqrt(density))


def _gradients(d, k, density, gen):
    """(residual, list of gradients), with the selection boundary of the first
    four passes free of ties."""
    noise = torch.randn(d + WINDOWS * SHIFT, device=DEV, generator=gen).mul_(SIGMA)
    starts = [(7 * i % WINDOWS) * SHIFT for i in range(WINDOWS)]
    grads = [noise[at:at + d] for at in starts]
    r0 = _residual(d, density, gen)
    r = r0.clone()
    for g in grads[:4]:
        idx = _untie(g, g + r, k)
        r += g
        r[idx] = 0.0
    return r0, grads


def _layer_sizes(d, tensors):
    """Sizes of a parameter list of ``d`` elements: weights that grow along the
    network, each followed by a small bias or scale."""
    rng = random.Random(d * 1009 + tensors)
    small = [min(rng.choice([10, 16, 64, 100, 256, 512, 1000, 1500]), max(1, d // (8 * tensors)))
             for _ in range(tensors // 2)]
    n_big = tensors - len(small)
    weights = [math.exp(4.0 * i / n_big + rng.uniform(-0.7, 0.7)) for i in range(n_big)]
    rest = d - sum(small)
    big = [max(1, int(rest * w / sum(weights))) for w in weights]
    big[-1] += rest - sum(big)
    out = []
    for i in range(n_big):
        out.append(big[i])
        if i < len(small):
            out.append(small[i])
    return out


# -- states -------------------------------------------------------------------
def _setup():
    settings.PIN_DENSITY = True          # the named density from the first step on
    settings.logger.setLevel("WARNING")
    torch.backends.cudnn.benchmark = False
    torch.backends.cudnn.deterministic = True
    torch.backends.cudnn.allow_tf32 = False      # strict fp32
    torch.backends.cuda.matmul.allow_tf32 = False


def _flat_view(t):
    """All of the storage that a parameter of the wrapped optimizer lives in."""
    return torch.empty(0, dtype=t.dtype, device=t.device).set_(t.untyped_storage())


def _prepare_train(case, seed):
    dataset, lr, clip, _, _ = MODELS[case["model"]]
    dev = torch.device(DEV, torch.cuda.current_device())
    torch.manual_seed(seed)
    size = None if dataset == "ptb" else 100_000_000     # no epoch boundary inside a measurement
    t = DLTrainer(0, 1, dist=False, ngpus=1, batch_size=case["batch"], data_dir="synthetic", dataset=dataset,
                  dnn=case["model"], lr=lr, nworkers=1, device=dev, synthetic_train_size=size,
                  cuda_graph=case["graph"])
    opt = DistributedOptimizer(t.optimizer, t.net.named_parameters(), compression=compressors["gtopk"], is_sparse=True,
                               density=0.001)
    t.update_optimizer(opt)
    gen = _generator(seed)
    b = case["batch"]
    if dataset == "ptb":
        tokens = torch.randint(0, 10000, (b, 36), device=DEV, generator=gen)
        batch = (tokens[:, :-1].contiguous(), tokens[:, 1:].contiguous())
    else:
        side, classes = (224, 1000) if dataset == "imagenet" else (32, 10)
        batch = (torch.randn(b, 3, side, side, device=DEV, generator=gen),
                 torch.randint(0, classes, (b,), device=DEV, generator=gen))
    hidden = t.net.init_hidden() if case["model"] == "lstm" else None
    return {"kind": "train", "trainer": t, "batch": batch, "hidden": hidden, "clip": clip,
            "params": _flat_view(next(t.net.parameters()))}


def _run_train(s):
    s["hidden"] = s["trainer"].train_step(data=s["batch"], hidden=s["hidden"], clip_norm=s["clip"])
    return {"params": s["params"], "hidden": s["hidden"]}


def _prepare_update(case, seed):
    gen = _generator(seed)
    sizes = _layer_sizes(case["d"], case["tensors"])
    params = [torch.nn.Parameter(torch.randn(n, device=DEV, generator=gen).mul_(0.05)) for n in sizes]
    named = [("p%03d" % i, p) for i, p in enumerate(params)]
    sgd = torch.optim.SGD(params, lr=0.1, momentum=case["momentum"], weight_decay=case["weight_decay"],
                          nesterov=case["nesterov"] and case["momentum"] != 0)
    sparse = case["compressor"] != "none"
    opt = DistributedOptimizer(sgd, named, compression=compressors[case["compressor"]], is_sparse=sparse,
                               density=case["density"])
    r0, grads = _gradients(case["d"], num_selected(case["d"], case["density"]), case["density"], gen)
    if sparse:
        opt.load_residual_state({n: t for (n, _), t in zip(named, r0.split(sizes))})
    outputs = {"params": _flat_view(params[0])}
    if sparse:
        outputs["residual"] = opt._flat.residual
    if case["momentum"]:
        outputs["momentum"] = opt._flat.momentum
    return {"kind": "update", "opt": opt, "params": params, "grads": [list(g.split(sizes)) for g in grads], "i": 0,
            "outputs": outputs}


def _run_update(s):
    opt, g = s["opt"], s["grads"][s["i"] % WINDOWS]
    s["i"] += 1
    opt.zero_grad()
    torch.autograd.backward(s["params"], g)
    opt.step()
    return s["outputs"]


def _prepare_select(case, seed):
    d, gen = case["d"], _generator(seed)
    k = num_selected(d, case["density"])
    r0, grads = _gradients(d, k, case["density"], gen)
    return {"kind": "select", "sel": TopkSelector(d, k, torch.device(DEV)), "k": k, "r": r0, "grads": grads, "i": 0,
            "p": torch.randn(d, device=DEV, generator=gen).mul_(0.05), "h": SgdHyper(lr=0.1)}


def _run_select(s):
    g, sel = s["grads"][s["i"] % WINDOWS], s["sel"]
    s["i"] += 1
    sel.select(g, s["r"], s["k"])
    sgd_sparse(s["p"], None, sel.sel, sel.n_sel_tensor, 1, sel.max_k, s["h"], False, 1.0)
    return {"residual": s["r"], "params": s["p"]}


def _prepare_compress(case, seed):
    d, gen = case["d"], _generator(seed)
    k = num_selected(d, case["density"])
    name = "case-%d-%r-%d" % (d, case["density"], seed)
    for store in (TopKCompressor.residuals, TopKCompressor.values, TopKCompressor.indexes, TopKCompressor.selectors):
        store.pop(name, None)
    g = torch.randn(d, device=DEV, generator=gen).mul_(SIGMA)
    r = TopKCompressor.get_residuals(name, g)
    r.copy_(_residual(d, case["density"], gen))
    for _ in range(2):   # the sum is rounded, so look once more at what came of a moved tie
        _untie(g, g + r, k)
    return {"kind": "compress", "tensor": g, "name": name, "ratio": case["density"], "residual": r}


def _run_compress(s):
    # the vector comes back sparsified; together with the residual it adds up to the same sum again
    tensor, _ = compressors["gtopk"].compress(s["tensor"], s["name"], ratio=s["ratio"])
    return {"tensor": tensor, "residual": s["residual"]}


def _prepare_exchange(case, seed):
    d, P, mode, gen = case["d"], case["ranks"], case["mode"], _generator(seed)
    dev = torch.device(DEV, torch.cuda.current_device())
    k = num_selected(d, case["density"])
    gather = mode != "gtopk"
    regions = ex.SymmetricRegion.create_emulated(P, ex.region_bytes(k, gather), dev)
    grads = [torch.randn(d, device=DEV, generator=gen).mul_(SIGMA) for _ in range(P)]
    top = [_untie(g, g.clone(), k) for g in grads]
    # magnitudes of all ranks' selections apart from one another, so that no union has a tie at its k-th place
    for attempt in range(3):
        vals = torch.cat([g[i] for g, i in zip(grads, top)])
        mag, order = vals.abs().sort()
        same = torch.zeros_like(mag, dtype=torch.bool)
        same[1:] = mag[1:] == mag[:-1]
        if not bool(same.any()):
            break
        at = order[same]
        vals[at] *= 1.0 + 1e-3 * (1.0 + torch.rand(at.numel(), device=DEV, generator=gen))
        for g, i, v in zip(grads, top, vals.split(k)):
            g[i] = v
    ranks = []
    for r in range(P):
        sel, resid = TopkSelector(d, k, dev), torch.zeros(d, device=DEV)
        ranks.append(ex.ExchangeRank(r, P, d, k, sel, resid, regions[r], with_allgather=gather, reselect=mode == "topk2"))
        sel.select(grads[r], resid, k)
    rc = ranks[0]
    s = {"kind": "exchange", "mode": mode, "ranks": ranks, "desc": torch.cat([r.desc for r in ranks]), "P": P, "k": k,
         "p": torch.randn(d, device=DEV, generator=gen).mul_(0.05), "h": SgdHyper(lr=0.1)}
    if mode == "topk":
        s["pairs"] = ex.pairs_view(rc.ag_ptr(0), 2 * ex.MAX_PEERS * k, dev)
    else:
        s["pairs"] = ex.pairs_view(rc.gout_ptr(0), 2 * k, dev)
    if gather:
        s["counts"] = torch.zeros(P * ex.MAX_PEERS, dtype=torch.int32, device=dev)
    return s


def _run_exchange(s):
    ranks, P, k, rc = s["ranks"], s["P"], s["k"], s["ranks"][0]
    if s["mode"] == "gtopk":
        ex.launch_gtopk(ranks, s["desc"], 0, P, k)
    else:
        ex.launch_allgather(ranks, s["desc"], s["counts"], 0, P, k, reselect=s["mode"] == "topk2")
    if s["mode"] == "topk":
        sgd_sparse(s["p"], None, s["pairs"], s["counts"], P, k, s["h"], False, 1.0 / P, use_atomics=True,
                   parity_word=rc.epoch, parity_stride=rc.ag_parity_stride)
    else:
        sgd_sparse(s["p"], None, s["pairs"], rc.n_global, 1, k, s["h"], False, 1.0 / P, parity_word=rc.epoch,
                   parity_stride=rc.parity_stride)
    return {"params": s["p"], "residuals": [r.resid for r in ranks]}


_PREPARE = {"train": _prepare_train, "update": _prepare_update, "select": _prepare_select, "compress": _prepare_compress,
            "exchange": _prepare_exchange}
_RUN = {"train": _run_train, "update": _run_update, "select": _run_select, "compress": _run_compress,
        "exchange": _run_exchange}


def prepare(case, seed):
    _setup()
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def work(case):
    """Bytes and operations of one pass.  Per element of a flat vector: gradient
    read (4), residual read and written (8), parameter and velocity read and
    written (8 each, where the step touches all of them)."""
    kind = case["kind"]
    if kind == "train":
        dataset, _, _, d, macs = MODELS[case["model"]]
        step = 0 if case["model"] == "lstm" else 16
        sample = {"cifar10": 3 * 32 * 32 * 4, "imagenet": 3 * 224 * 224 * 4, "ptb": 2 * 35 * 8}[dataset]
        return {"bytes": (12 + step) * d + sample * case["batch"], "flops": 6.0 * macs * case["batch"]}
    d = case["d"]
    k = num_selected(d, case["density"])
    if kind == "update":
        dense = (16 if case["momentum"] else 8) * d
        if case["compressor"] == "none":
            return {"bytes": 4 * d + dense, "flops": 5.0 * d}
        if not case["momentum"] and not case["weight_decay"]:
            dense = 8 * k
        return {"bytes": 12 * d + dense + 8 * k, "flops": 5.0 * d}
    if kind == "select":
        return {"bytes": 12 * d + 16 * k, "flops": 1.0 * d}
    if kind == "compress":
        return {"bytes": 16 * d + 12 * k, "flops": 1.0 * d}
    # exchange, per rank: the selection read, the global set written, the residual of what came back updated
    P = case["ranks"]
    sent = P * k if case["mode"] == "topk" else k
    back = 0 if case["mode"] == "topk" else 8 * k
    return {"bytes": P * (8 * k + 8 * sent + back) + 8 * sent, "flops": 2.0 * P * k}


def tolerance(case):
    # fp32 throughout.  A training step adds thousands of products in an order that another library version may change,
    # and where that moves an entry across the selection boundary its parameter differs by one update.
    if case["kind"] == "train":
        return {"rel": 1e-4, "max": 0.05}
    return {"rel": 1e-5, "max": 1e-3}
