"""Performance cases: the work that users of this package have it do on one GPU, over the range of sizes they bring.

Four kinds, each through the calls a training program makes:

``train``     a whole iteration of a model (forward, loss, backward, sparse exchange, sparse optimiser) through the
              wrapper's ``train_step`` in its captured form, as the training driver and the benchmark run it.
``step``      the engine's own part of an iteration for the parameter tensors of a model: a backward pass hands over one
              gradient per parameter, and the engine's hooks select, exchange and apply.  ``launch`` is "graph" (a
              captured iteration, the product path) or "eager".  The gradients themselves cost nothing here, so that the
              time is the engine's and not a model's.
``rank``      one rank's share of a job of several GPUs: select with a store into every rank's receive area, then the
              merge of all ranks' streams and the optimiser.  The peers' memory is local memory and the peers' streams
              have arrived before the pass begins.
``compress``  ``compress(name, tensor, ratio)`` of one tensor, and the dense tensor that its receiver rebuilds from the
              pairs.

Gradients differ in scale from tensor to tensor and are heavy-tailed inside a tensor, as those of real models are.
"""
from __future__ import annotations

import gc
import itertools
import math

import torch
import torch.nn as nn

import stellatrain_b200 as st
from stellatrain_b200.models.registry import build_model, is_language_model, synthetic_batch
from stellatrain_b200.models.wrapper import FasterDpModelWrapper
from stellatrain_b200.parallel import buckets as B
from stellatrain_b200.parallel.engine import EngineConfig, SparseDPEngine
from stellatrain_b200.parallel.gpu_bucket import CandidateScratch, GpuBucket, Wiring
from stellatrain_b200.parallel.graphs import GraphedStep

#: A convolutional net of eight small tensors, 6,000 parameters in all: the size at which only latency counts.
SMALL_NET = [216, 8, 576, 8, 4736, 37, 370, 10]

_LR = {"adam": 1e-3, "sgd": 0.1}


def listed() -> list[dict]:
    return [
        # the benchmark's workload: ResNet-152 at 32 images, 1 % of the gradient entries, sparse Adam
        dict(name="train resnet152", kind="train", model="resnet152", batch=32, size=224, compressor="thresholdv16",
             optimizer="adam", ratio=0.99),
        # a model so small that a step is nothing but launches
        dict(name="train gpt2-tiny", kind="train", model="gpt2-tiny", batch=8, size=64, compressor="topk", optimizer="adam",
             ratio=0.99),
        # the smallest models people try the package with, without graph capture
        dict(name="step small net eager", kind="step", model="small", launch="eager", compressor="topk", optimizer="sgd",
             ratio=0.9, grad_mode="steal", wire="wide", bucket_mb=64.0),
        # ordinary eager training of a mid-size model
        dict(name="step resnet18 eager", kind="step", model="resnet18", launch="eager", compressor="thresholdv",
             optimizer="sgd", ratio=0.99, grad_mode="steal", wire="wide", bucket_mb=64.0),
        # ResNet-50, top-k 1 %, SGD with momentum
        dict(name="step resnet50", kind="step", model="resnet50", launch="graph", compressor="topk", optimizer="sgd",
             ratio=0.99, grad_mode="steal", wire="wide", bucket_mb=64.0),
        # the engine's share of the benchmark's iteration
        dict(name="step resnet152", kind="step", model="resnet152", launch="graph", compressor="thresholdv16",
             optimizer="adam", ratio=0.99, grad_mode="steal", wire="wide", bucket_mb=64.0),
        # ViT-B/16, top-k 0.1 %, Adam
        dict(name="step vit_b_16", kind="step", model="vit_b_16", launch="graph", compressor="topk", optimizer="adam",
             ratio=0.999, grad_mode="steal", wire="wide", bucket_mb=64.0),
        # GPT-2 small, top-k 1 %, Adam: one tensor of 38.6 million elements next to 147 others
        dict(name="step gpt2", kind="step", model="gpt2", launch="graph", compressor="topk", optimizer="adam", ratio=0.99,
             grad_mode="steal", wire="wide", bucket_mb=64.0),
        # the largest: GPT-2 medium in large buckets
        dict(name="step gpt2-medium", kind="step", model="gpt2-medium", launch="graph", compressor="thresholdv16",
             optimizer="adam", ratio=0.99, grad_mode="steal", wire="wide", bucket_mb=256.0),
        # one of eight GPUs: every stream goes to eight places and eight streams are merged
        dict(name="rank of 8 resnet152", kind="rank", model="resnet152", world=8, compressor="thresholdv16", optimizer="adam",
             ratio=0.99, wire="wide", bucket_mb=64.0),
        # compression of a single tensor by itself, small and large (the embedding of GPT-2)
        dict(name="compress 10000", kind="compress", n=10_000, compressor="thresholdv16", ratio=0.99),
        dict(name="compress 38.6M", kind="compress", n=50257 * 768, compressor="topk", ratio=0.99),
    ]


def _log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    kind = rng.choice(["train", "step", "step", "step", "step", "step", "rank", "rank", "compress", "compress"])
    ratio = round(1.0 - _log_uniform(rng, 0.001, 0.1), 6)
    compressor = rng.choice(["thresholdv16", "thresholdv16", "thresholdv16", "topk", "topk", "topk", "thresholdv", "thresholdv",
                             "randomk"])
    optimizer = rng.choice(["adam", "sgd"])
    if kind == "compress":
        return dict(kind=kind, n=int(_log_uniform(rng, 1_000, 38_000_000)), compressor=compressor, ratio=ratio)
    if kind == "train":
        model = rng.choice(["gpt2-tiny", "resnet18", "resnet34", "resnet50"])
        lm = is_language_model(model)
        return dict(kind=kind, model=model, batch=rng.randint(1, 24), size=rng.randint(17, 64) if lm else 32 * rng.randint(2, 7),
                    compressor=compressor, optimizer=optimizer, ratio=ratio)
    # a made-up model: a number of tensors, their sizes spread over three orders of magnitude around the mean of the model
    total = _log_uniform(rng, 5_000, 100_000_000)
    tensors = int(min(_log_uniform(rng, 1, 400), total / 16))
    common = dict(tensors=max(1, tensors), total=int(total), layout_seed=rng.randrange(1 << 30), compressor=compressor,
                  optimizer=optimizer, ratio=ratio, wire=rng.choice(["wide", "wide", "wide", "narrow"]),
                  bucket_mb=rng.choice([16.0, 64.0, 64.0, 256.0]))
    if kind == "rank":
        common["total"] = min(common["total"], 60_000_000)
        return dict(kind=kind, world=rng.choice([2, 4, 8]), **common)
    return dict(kind=kind, launch=rng.choice(["graph", "graph", "eager"]), grad_mode=rng.choice(["steal", "steal", "steal", "flat"]),
                **common)


# ------------------------------------------------------------------------------------------------ shapes
_shapes: dict = {}


def _model_numels(name: str) -> list[int]:
    if name == "small":
        return list(SMALL_NET)
    if name not in _shapes:
        with torch.device("meta"):
            _shapes[name] = [p.numel() for p in build_model(name, 100).parameters()]
    return _shapes[name]


def _numels(case: dict) -> list[int]:
    if "model" in case:
        return _model_numels(case["model"])
    import random

    rng = random.Random(case["layout_seed"])
    share = [_log_uniform(rng, 1.0, 1000.0) for _ in range(case["tensors"])]
    scale = case["total"] / sum(share)
    return [max(1, int(s * scale)) for s in share]


def _entries(case: dict, world: int = 1) -> int:
    return sum(B.entries_for(n, case["ratio"], world) for n in _numels(case))


# ------------------------------------------------------------------------------------------------ inputs
def _gradient(n: int, gen: torch.Generator) -> torch.Tensor:
    """Normal values times a log-normal factor for every 64 neighbours."""
    g = torch.randn(n, device="cuda", generator=gen)
    rows = torch.randn((n + 63) // 64, device="cuda", generator=gen).mul_(0.8).exp_()
    return g.mul_(rows.repeat_interleave(64)[:n])


def _gradients(numels: list[int], gen: torch.Generator, scales: list[float]) -> list[torch.Tensor]:
    offs, pos = [], 0
    for n in numels:
        offs.append(pos)
        pos += (n + 63) // 64 * 64          # every gradient starts on a 256-byte boundary, as the allocator's do
    flat = _gradient(pos, gen)
    return [flat[o : o + n].mul_(s) for o, n, s in zip(offs, numels, scales)]


def _scales(count: int, seed: int) -> list[float]:
    import random

    rng = random.Random(seed)
    return [_log_uniform(rng, 1e-4, 1e-2) for _ in range(count)]


class _HandOver(torch.autograd.Function):
    """A backward pass that hands one ready gradient to every parameter."""

    @staticmethod
    def forward(ctx, owner, *params):
        ctx.owner = owner
        return owner.loss.detach()

    @staticmethod
    def backward(ctx, _):
        return (None, *[g.detach() for g in ctx.owner.gradients])


class Parameters(nn.Module):
    """The parameter tensors of a model and, in place of its layers, the gradients of two batches."""

    def __init__(self, numels: list[int], seed: int) -> None:
        super().__init__()
        gen = torch.Generator(device="cuda").manual_seed(seed)
        self.items = nn.ParameterList(nn.Parameter(torch.randn(n, device="cuda", generator=gen).mul_(0.02)) for n in numels)
        scales = _scales(len(numels), seed)
        self.batches = [_gradients(numels, gen, scales) for _ in range(2)]
        self.gradients = self.batches[0]
        self.loss = torch.zeros((), device="cuda")

    def forward(self):
        return _HandOver.apply(self, *self.items)


def _engine_config(case: dict) -> EngineConfig:
    options = {"lr": _LR[case["optimizer"]]}
    if case["optimizer"] == "sgd":
        options["momentum"] = 0.9
    return EngineConfig(compressor=case["compressor"], ratio=case["ratio"], optimizer=case["optimizer"], optimizer_options=options,
                        bucket_mb=case.get("bucket_mb", 64.0), grad_mode=case.get("grad_mode", "steal"),
                        wire_format=case.get("wire", "wide"))


# ------------------------------------------------------------------------------------------------ states
class _Train:
    def __init__(self, case: dict, seed: int) -> None:
        torch.manual_seed(seed)
        lm = is_language_model(case["model"])
        with torch.device("cuda"):
            model = build_model(case["model"], 100)
        if not lm:
            model = model.to(memory_format=torch.channels_last)
        self.net = FasterDpModelWrapper(model, sequential=False, graph=True, graph_warmup=3)
        self.net.engine = SparseDPEngine(self.net.module, _engine_config(case))
        gen = torch.Generator(device="cuda").manual_seed(seed)
        self.data = []
        for _ in range(2):
            if lm:
                x, y = synthetic_batch(case["model"], case["batch"], seq_len=case["size"], device="cuda", generator=gen)
            else:
                x = torch.randn(case["batch"], 3, case["size"], case["size"], device="cuda", generator=gen)
                x = x.contiguous(memory_format=torch.channels_last)
                y = torch.randint(0, 100, (case["batch"],), device="cuda", generator=gen)
            self.data.append((x, y))
        self.passes = 0
        for _ in range(5):                  # three eager iterations, the capture, one replay
            self.run()

    def run(self):
        x, y = self.data[self.passes & 1]
        self.passes += 1
        loss = self.net.train_step(x, y)
        return {"loss": loss, "param": [rt.bucket.param for rt in self.net.engine.buckets]}


class _Step:
    def __init__(self, case: dict, seed: int) -> None:
        self.module = Parameters(_numels(case), seed)
        self.engine = SparseDPEngine(self.module, _engine_config(case))
        self.passes = 0
        self.graphs = []
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for i in range(3):
                self.module.gradients = self.module.batches[i & 1]
                self._iteration()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        if case["launch"] == "graph":
            for batch in self.module.batches:
                self.module.gradients = batch
                self.graphs.append(GraphedStep(self.engine, self._iteration, [], warmup=0, stream=side))

    def _iteration(self):
        loss = self.module()
        loss.backward()
        return loss

    def run(self):
        which = self.passes & 1
        self.passes += 1
        if self.graphs:
            self.graphs[which].replay()
        else:
            self.module.gradients = self.module.batches[which]
            self._iteration()
        return _updated([rt.bucket for rt in self.engine.buckets])


def _updated(buckets: list) -> dict:
    out = {"param": [b.param for b in buckets], "resid": [b.resid for b in buckets], "m": [b.m for b in buckets]}
    if buckets[0].v is not None:
        out["v"] = [b.v for b in buckets]
    return out


class _Rank:
    """Rank 0 of ``world``.  Arrival flags and acknowledgements of the peers say "everything up to a far epoch", and their
    streams, one per slot, come from selects over gradients of their own."""

    FAR = 1 << 40

    def __init__(self, case: dict, seed: int) -> None:
        numels = list(reversed(_numels(case)))
        world = case["world"]
        dev = torch.device("cuda", torch.cuda.current_device())
        gen = torch.Generator(device="cuda").manual_seed(seed)
        scales = _scales(len(numels), seed)
        scratch = CandidateScratch(dev)
        self.buckets, self.passes, self.keep = [], 0, []
        for bi, grp in enumerate(B.plan_buckets(numels, int(case["bucket_mb"] * (1 << 20) / 4))):
            sizes, sc = [numels[i] for i in grp], [scales[i] for i in grp]
            make = lambda r: GpuBucket(bi, B.BucketLayout([f"t{i}" for i in grp], sizes, narrow_wire=case["wire"] == "narrow"), dev,  # noqa: E731
                                       compressor=case["compressor"], ratio=case["ratio"], world=world, rank=r,
                                       optimizer=case["optimizer"], scratch=scratch)
            b = make(0)
            recv = [torch.zeros(b.recv_bytes(), dtype=torch.uint8, device=dev) for _ in range(world)]
            words = lambda: torch.full((2 * world,), self.FAR, dtype=torch.int64, device=dev)  # noqa: E731
            flags, acks = [words() for _ in range(world)], [words() for _ in range(world)]
            ptrs = lambda ts: [t.data_ptr() for t in ts]  # noqa: E731
            for r in range(1, world):
                peer = make(r)
                peer.wire(Wiring(world, r, recv[0], [recv[0].data_ptr()] * world, None, [0] * world, None, [0] * world))
                for _ in range(2):
                    self._fill(peer, sizes, sc, gen)
                    peer.select()
            b.wire(Wiring(world, 0, recv[0], ptrs(recv), flags[0], ptrs(flags), acks[0], ptrs(acks), use_flags=True, use_acks=True))
            b.set_optimizer_options(lr=_LR[case["optimizer"]], momentum=0.9)
            b.param.normal_(0.0, 0.02, generator=gen)
            b.use_grad_table()
            batches = []
            for _ in range(2):
                self._fill(b, sizes, sc, gen)
                flat = b.grad.clone()
                table = torch.tensor([flat.data_ptr() + 4 * s.off for s in b.layout.segments], dtype=torch.int64, device=dev)
                batches.append((flat, table))
            self.buckets.append((b, batches))
            self.keep += [recv, flags, acks]
        for _ in range(3):
            self.run()

    @staticmethod
    def _fill(b, sizes, scales, gen) -> None:
        for i, g in enumerate(_gradients(sizes, gen, scales)):
            b.view(b.grad, i).copy_(g)

    def run(self):
        which = self.passes & 1
        self.passes += 1
        for b, batches in self.buckets:
            b.grad_tab_dev.copy_(batches[which][1])
            b.select()
            b.apply()
        return _updated([b for b, _ in self.buckets])


_names = itertools.count()


class _Compress:
    def __init__(self, case: dict, seed: int) -> None:
        gen = torch.Generator(device="cuda").manual_seed(seed)
        st.configure_compression(case["compressor"])
        self.name = f"tensor {next(_names)}"          # threshold compressors keep a threshold per name
        self.ratio = case["ratio"]
        self.tensors = [_gradient(case["n"], gen).mul_(1e-2) for _ in range(2)]
        self.passes = 0

    def run(self):
        t = self.tensors[self.passes & 1]
        self.passes += 1
        idx, val = st.compress(self.name, t, self.ratio)
        return torch.zeros_like(t).scatter_(0, idx.long(), val)


_KINDS = {"train": _Train, "step": _Step, "rank": _Rank, "compress": _Compress}


def prepare(case: dict, seed: int):
    gc.collect()        # an engine and its module refer to each other: give an earlier one's memory back
    return _KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
#: multiply-adds of one forward pass at 224 x 224
_MACS = {"resnet18": 1.82e9, "resnet34": 3.67e9, "resnet50": 4.11e9, "resnet152": 11.53e9}


def work(case: dict) -> dict:
    if case["kind"] == "compress":
        k = int((1.0 - case["ratio"]) * case["n"])
        return {"bytes": 4.0 * case["n"] + 8.0 * k + 4.0 * case["n"], "flops": 0.0}
    n, world = sum(_numels(case)), case.get("world", 1)
    k = _entries(case, world)
    state = 16.0 if case["optimizer"] == "adam" else 8.0
    # gradient and residual read, residual written; a sent entry is written to every rank; a received one is read, and its
    # parameter and optimiser state are read and written
    sparse = 12.0 * n + 8.0 * k * world + (8.0 + 8.0 + state) * k * world
    if case["kind"] != "train":
        return {"bytes": sparse, "flops": 0.0}
    if is_language_model(case["model"]):
        flops = 6.0 * n * case["batch"] * case["size"]
    else:
        flops = 6.0 * _MACS[case["model"]] * case["batch"] * (case["size"] / 224.0) ** 2
    # the parameters are read once forward and once backward, the gradients written
    return {"bytes": sparse + 12.0 * n, "flops": flops}


def tolerance(case: dict):
    if case["kind"] == "compress":
        return "exact"          # the pairs are copies of the input's values
    if case["kind"] == "train":
        # an entry on the edge of a tensor's budget may go in either of two neighbouring iterations
        return {"rel": 1e-3, "max": 0.5}
    # against the same steps in 64 bits: 5e-8 for parameters, residuals and first moments, 1.3e-5 for Adam's second
    # moment, whose factor 1 - 0.999 has that error in 32 bits
    return {"rel": 5e-5 if case["optimizer"] == "adam" else 1e-5, "max": 1e-3}
