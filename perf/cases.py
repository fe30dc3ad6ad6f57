"""The work this library is used for, as cases that can be timed and compared.

Every case is one call of a public entry point on one batch: host arrays in, pooler output or class
probabilities out (``encode`` / ``classify``: what the engine's replicas and a request handler call),
device-resident inputs (``device``: a program that keeps its batches in HBM), or the final hidden states
of every token (``hidden``: feature extraction through ``Cuda_Inference``).

Models: the four model / mode pairs of the benchmark workloads (``synth.CONFIGS``): BERT-base and
BERT-large with bf16 weights, BERT-base in fp32, BERT-large with FP8 weights.  Weights are seeded and
random with random biases, gammas and betas; a process keeps one handle per pair, as a server does, and
all its batches go through that handle.
"""
import math
import tempfile

import numpy as np
import torch

from cudabert_b200 import synth
from cudabert_b200.config import Engin_Config
from cudabert_b200.cuda_model import Cuda_BERT

# model name -> (BERT-large, precision mode)
MODELS = {
    "base-fp32": (False, "fp32"),
    "base-bf16": (False, "bf16"),
    "large-bf16": (True, "bf16"),
    "large-fp8": (True, "fp8"),
}
WEIGHT_BYTES = {"fp32": 4, "bf16": 2, "fp8": 1}


def listed():
    return [
        # one short query, answered on its own: the smallest call, all latency
        dict(name="one_query_base", model="base-bf16", entry="encode", batch=1, seq=24, dist="full", mask=True),
        # one passage through the large model with the classifier head: a request handler without batching
        dict(name="one_passage_large", model="large-bf16", entry="classify", batch=1, seq=128, dist="full", mask=True),
        # a handful of requests gathered for a few milliseconds; FP8 weights, odd ragged lengths
        dict(name="few_requests_fp8", model="large-fp8", entry="classify", batch=5, seq=37, dist="uniform:4:37", mask=True),
        # the specification's small batch (8 x 128, lengths U[32,128]) with bf16 weights ...
        dict(name="small_batch_base", model="base-bf16", entry="encode", batch=8, seq=128, dist="uniform:32:128", mask=True),
        # ... and in fp32, where it is the accuracy baseline
        dict(name="small_batch_fp32", model="base-fp32", entry="encode", batch=8, seq=128, dist="uniform:32:128", mask=True),
        # an fp32 batch of ordinary size without a mask, odd length
        dict(name="batch_fp32", model="base-fp32", entry="encode", batch=24, seq=101, dist="full", mask=False),
        # feature extraction on documents: hidden states of every token, long ragged rows
        dict(name="hidden_documents", model="large-bf16", entry="hidden", batch=16, seq=384, dist="uniform:64:384", mask=True),
        # what the engine makes of a stream of lines: one full batch of one length bucket, right-trimmed
        dict(name="engine_bucket", model="large-bf16", entry="classify", batch=128, seq=93, dist="uniform:92:93", mask=True),
        # the headline workload: untrimmed ragged batch with the classifier head
        dict(name="headline_large", model="large-bf16", entry="classify", batch=128, seq=200, dist="uniform:16:200", mask=True),
        # the bulk workload on the base model, batches resident in HBM
        dict(name="bulk_base", model="base-bf16", entry="device", batch=256, seq=128, dist="tnormal:60:25:8:128", mask=True),
        # full-length documents: the attention-heavy regime
        dict(name="full_length_large", model="large-bf16", entry="encode", batch=32, seq=512, dist="full", mask=True),
        # many short lines with FP8 weights: the largest batch
        dict(name="many_short_fp8", model="large-fp8", entry="encode", batch=1024, seq=64, dist="uniform:8:64", mask=True),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: any model, entry point and length distribution, batches of 1 to 1024 rows
    of 8 to 512 positions, at most as much work as the largest listed case (fp32, which multiplies six
    times as much: at most what 32 full rows of 128 tokens take)."""
    most = max(work(c)["flops"] for c in listed())
    while True:
        model = rng.choice(sorted(MODELS))
        large, precision = MODELS[model]
        seq = _log_uniform(rng, 8, 512)
        batch = _log_uniform(rng, 1, 1024)
        lo = rng.randint(1, seq)
        dist = rng.choice(["full", "uniform:%d:%d" % (lo, seq), "uniform:%d:%d" % (max(1, seq // 12), seq),
                           "tnormal:%d:%d:%d:%d" % (max(1, seq * 47 // 100), max(1, seq // 5), max(1, seq // 16), seq)])
        case = dict(model=model, entry=rng.choice(["encode", "classify", "device", "hidden"]), batch=batch, seq=seq,
                    dist=dist, mask=True if dist != "full" else rng.random() < 0.5)
        if batch * seq > (4096 if precision == "fp32" else 65536):
            continue
        if work(case)["flops"] <= most:
            return case


_handles = {}


def _handle(model):
    """The process's handle of a model.  Both modes of a size are loaded from one weight directory."""
    if model not in _handles:
        large = MODELS[model][0]
        with tempfile.TemporaryDirectory() as folder:
            synth.write_weight_dir(folder, synth.make_weights(large, 7 + large, affine=True))
            for name, (is_large, precision) in MODELS.items():
                if is_large == large:
                    config = Engin_Config()
                    config.is_large, config.model_npy_pth, config.precision = large, folder, precision
                    _handles[name] = Cuda_BERT(0, config)
    return _handles[model]


class _DeviceArray:
    """A library-owned device buffer for torch.as_tensor (no copy)."""

    def __init__(self, pointer, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (int(pointer), False), "version": 3}


def prepare(case, seed):
    handle = _handle(case["model"])
    ids, seg, mask = synth.make_inputs(seed, case["batch"], case["seq"], case["dist"])
    batch = [ids, seg, mask if case["mask"] else None]
    if case["entry"] == "device":
        batch = [None if t is None else torch.from_numpy(t).cuda() for t in batch]
        torch.cuda.synchronize()
    return dict(case=case, handle=handle, batch=batch)


def run(state):
    case, handle, batch = state["case"], state["handle"], state["batch"]
    entry, rows, seq = case["entry"], case["batch"], case["seq"]
    if entry == "encode":
        return handle.encode(batch)
    if entry == "classify":
        return handle.classify(batch)
    pybert, model = handle._pybert, handle.model
    if entry == "device":
        ids, seg, mask = (None if t is None else t.data_ptr() for t in batch)
        pybert.forward_dev(model, ids, seg, mask, rows, seq)
        pybert.sync(model)
        pybert.check(model)
        return torch.as_tensor(_DeviceArray(pybert.pooled_dev(model), (rows, handle.hidden_size)), device="cuda")
    result = pybert.inference(model, batch[0], batch[1], rows, seq, batch[2])
    pybert.check(model)
    return [torch.as_tensor(_DeviceArray(result.tensor, (rows, seq, handle.hidden_size)), device="cuda"),
            torch.as_tensor(_DeviceArray(result.Pooled_Output, (rows, handle.hidden_size)), device="cuda")]


def _mean_lengths(case):
    """Expected length and squared length of a row."""
    parts = case["dist"].split(":")
    if parts[0] == "full":
        return float(case["seq"]), float(case["seq"]) ** 2
    lens = synth.make_lengths(np.random.default_rng(1), 4096, case["seq"], case["dist"]).astype(np.float64)
    return float(lens.mean()), float((lens * lens).mean())


def work(case):
    """What one call cannot do without, on the valid tokens alone: 24 H^2 multiply-adds per token and layer,
    4 H per query-key pair; without hidden states asked for, the last layer needs K and V of every token and
    the rest for the first token of each row.  Bytes: the encoder's weights once in the mode's format, the
    looked-up embedding rows, the ids, the results."""
    large, precision = MODELS[case["model"]]
    d = synth.model_dims(large)
    H, L, rows = d["hidden"], d["layers"], case["batch"]
    mean, mean_sq = _mean_lengths(case)
    tokens, pairs = rows * mean, rows * mean_sq
    full = L if case["entry"] == "hidden" else L - 1
    flops = full * (24 * H * H * tokens + 4 * H * pairs) + 2 * H * H * rows
    if full < L:
        flops += 4 * H * H * tokens + 20 * H * H * rows + 4 * H * tokens
    out = rows * H if case["entry"] != "hidden" else rows * case["seq"] * H + rows * H
    nbytes = 12 * L * H * H * WEIGHT_BYTES[precision] + 4 * H * H + 4 * H * min(tokens, 30522) + 12 * rows * case["seq"] + 4 * out
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """Measured by running the cases with other kernels, i.e. their sums in another order (the CUDA-core
    fp32 GEMM, `mma.sync` attention, LayerNorms folded into the GEMMs): at most 6.2e-5 (2-norm) and 2.4e-4
    (largest) in fp32, 8.6e-4 and 5.6e-3 in the 16-bit modes, whose activations are rounded to fp16 at other
    places and pass through 12 or 24 layers of random weights.  Four times that is stated."""
    if MODELS[case["model"]][1] == "fp32":
        return {"rel": 2.5e-4, "max": 1e-3}
    return {"rel": 3.5e-3, "max": 2.5e-2}
