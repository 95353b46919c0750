"""The work this framework is used for, as cases that can be prepared, run and compared: recorded training steps of the
three architectures (`CudaStep`), the reference's own micro-batch loop (`trainLMGpuResident`), scoring of held-out
windows and token-by-token decoding, at the shapes of `arch.py` and over the sizes, precisions, optimizers and options a
user picks for them.

A case is a dict of plain values:
  kind       "step" | "loop" | "score" | "decode"
  shape      "tiny" | "smollm2" | "gemma3" | "qwen3": a configuration of arch.py; layers: how many of its layers are kept
  batch, seq sequences per step and tokens per sequence ("loop": micro-batches per step; "score": windows;
             "decode": new tokens after a prompt of seq tokens)
  precision  "fp32" (the backend's default) or "tf32"
  optimizer  "adamw" | "muon"; recompute; lossChunk (vocabulary span of the fused readout loss, 0 = dense);
  lora       adapter rank on a frozen base, 0 = train every parameter; masked: share of the targets that is ignored
  steps      optimizer steps of one "loop" call
"""
from __future__ import annotations

import dataclasses
import json
import math
import weakref

import numpy as np
import torch

from gguf_trainer_b200 import autograd as ag
from gguf_trainer_b200.arch import LanguageModel, gemma3_95M, isGlobalLayer, paramCount, qwen3_0_6B, smolLM2_135M, tinyLlama
from gguf_trainer_b200.backend import requireGPU
from gguf_trainer_b200.lora import applyLora, clearLora
from gguf_trainer_b200.optim import AdamWGpu, MuonGpu
from gguf_trainer_b200.rng import Mulberry32
from gguf_trainer_b200.train import CudaStep, freezeForScoring, sequenceLoss, trainLMGpuResident

SHAPES = {"tiny": tinyLlama, "smollm2": smolLM2_135M, "gemma3": gemma3_95M, "qwen3": qwen3_0_6B}
DEFAULTS = dict(kind="step", precision="tf32", optimizer="adamw", recompute=False, lossChunk=0, lora=0, masked=0.0, steps=1)
MAX_WEIGHTS = 60     # updated weights returned beside the losses and the gradient arena


def _case(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # The smallest job: the CPU-sized llama of the parity configurations, strict f32, one recorded step. Launches count.
        _case("tiny_step_f32", shape="tiny", layers=2, batch=4, seq=128, precision="fp32"),
        # The same model in the loop a user of the reference calls, with its per-op host work and two syncs per step: an odd
        # sequence length, three micro-batches, a supervision mask, weights back on the host at the end.
        _case("tiny_loop_f32", kind="loop", shape="tiny", layers=2, batch=3, seq=333, precision="fp32", steps=4, masked=0.3),
        # Pretraining at the shape and sequence length of the benchmark's 135M llama: the ordinary big step. (Half of its
        # layers in most cases here: a layer is a layer, and the model is prepared many times.)
        _case("smollm2_step", shape="smollm2", layers=15, batch=4, seq=2048),
        # The same model at the full batch with recompute and Muon on the hidden matrices: memory-bound users and the
        # optimizer of the multi-GPU configuration.
        _case("smollm2_recompute_muon", shape="smollm2", layers=8, batch=8, seq=2048, recompute=True, optimizer="muon"),
        # A short, odd sequence length whose rows fill no whole tile: fine-tuning on documents.
        _case("smollm2_ragged", shape="smollm2", layers=15, batch=3, seq=777),
        # The default precision mode at model size: parity runs and users who want 1e-5.
        _case("smollm2_f32", shape="smollm2", layers=8, batch=1, seq=512, precision="fp32"),
        # The reference's loop at model size: micro-batches launched op by op.
        _case("smollm2_loop", kind="loop", shape="smollm2", layers=30, batch=2, seq=256, steps=2),
        # Heads of 256, sliding windows on five of six layers, sandwich norms: the gemma3 pretraining configuration.
        _case("gemma3_step", shape="gemma3", layers=12, batch=8, seq=2048),
        # LoRA fine-tuning of the 0.6B shape as configured for it: frozen base, rank 16, half of the targets masked, recompute,
        # chunked readout loss over 151936 tokens.
        _case("qwen3_lora", shape="qwen3", layers=14, batch=4, seq=2048, lora=16, masked=0.5, recompute=True, lossChunk=32768),
        # One sequence at the context limit (maxSeq 8192), a few layers of it: attention is the largest part.
        _case("qwen3_long", shape="qwen3", layers=4, batch=1, seq=8192, lossChunk=32768),
        # Held-out loss of a frozen model, window by window: forward only, four bytes back per window.
        _case("smollm2_score", kind="score", shape="smollm2", layers=15, batch=2, seq=512),
        # Decoding without a cache, one forward over the growing context per token: the smallest forward calls.
        _case("smollm2_decode", kind="decode", shape="smollm2", layers=30, batch=4, seq=37),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "loop", "score", "decode"])
    shape = rng.choice(["tiny", "smollm2", "smollm2", "gemma3", "qwen3"])
    precision = "fp32" if shape == "tiny" or rng.random() < 0.15 else "tf32"
    if shape == "tiny" and rng.random() < 0.3:
        precision = "tf32"
    full = SHAPES[shape]().nLayers
    layers = _log(rng, 1, min(full, 8 if shape == "qwen3" else full))
    kw = dict(kind=kind, shape=shape, layers=layers, precision=precision)
    if kind == "decode":
        return _case(batch=rng.randint(1, 4), seq=_log(rng, 5, 400), **kw)
    rows = 768 if precision == "fp32" and shape != "tiny" else (4096 if shape == "qwen3" else 8192)
    rows = min(rows, 64_000 // layers)
    seq = _log(rng, 32, min(rows, 4096))
    batch = _log(rng, 1, max(1, min(16, rows // seq)))
    if kind == "score":
        return _case(batch=min(batch, 4), seq=min(seq, 1024), lossChunk=rng.choice([0, 0, 4096]), **kw)
    kw.update(optimizer=rng.choice(["adamw", "adamw", "muon"]), recompute=rng.random() < 0.3,
              lossChunk=rng.choice([0, 0, 4096]), masked=rng.choice([0.0, 0.0, 0.5]))
    if kind == "loop":
        return _case(batch=min(batch, 3), seq=min(seq, 512), steps=rng.randint(1, 3), **dict(kw, layers=min(layers, 12)))
    if shape == "qwen3" and rng.random() < 0.5:
        kw.update(lora=rng.choice([8, 16]), optimizer="adamw")
    return _case(batch=batch, seq=seq, **kw)


# --------------------------------------------------------------------------------------------- what a program keeps
class _Device:
    """The process's one backend (one context per process and GPU), shared by the states of a case and closed with the
    last of them."""

    def __init__(self, precision):
        self.gpu = requireGPU("the cases", precision=precision)

    def __del__(self):
        if getattr(self, "gpu", None) is not None:
            self.gpu.destroy()


_current = [None, None]     # key, weak reference


def _device(case) -> _Device:
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    dev = _current[1]() if _current[1] is not None else None
    if dev is None or _current[0] != key:
        dev = _Device(case["precision"])
        _current[:] = [key, weakref.ref(dev)]
    return dev


class _Held:
    """Keeps a state's device memory alive for as long as one of its outputs is; gives the recorded step's buffers back to
    the pool after that."""

    def __init__(self, dev):
        self.dev, self.step = dev, None

    def __del__(self):
        if self.step is not None and self.step.graph is not None and self.dev.gpu.ctx is not None:
            self.step.graph.destroy()


class _Raw:
    def __init__(self, held, addr, count):
        self.held = held
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (addr, False), "version": 2, "strides": None}


def _view(held, addr, count) -> torch.Tensor:
    """The library's device memory as a tensor, in place."""
    return torch.as_tensor(_Raw(held, addr, count), device="cuda")


class _Normals:
    """Stands in for the model's generator: the same distributions, drawn on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def randn(self, shape, std):
        return torch.randn(int(np.prod(shape)), generator=self.g, device="cuda").mul_(std).cpu().numpy()


def _config(case):
    return dataclasses.replace(SHAPES[case["shape"]](), nLayers=case["layers"])


def _zipf(rng, n, vocab):
    """Zipf(1.1) token ids: what a tokenised text looks like."""
    cdf = np.cumsum(1.0 / np.arange(1, vocab + 1, dtype=np.float64) ** 1.1)
    return np.minimum(np.searchsorted(cdf / cdf[-1], rng.random(n)), vocab - 1).astype(np.int64)


def _optimizer(case, gpu, model, trainable):
    adamw = dict(lr=1e-3, beta1=0.9, beta2=0.95, weightDecay=0.1, clip=1.0)
    if case["optimizer"] == "muon":
        g = model.paramGroups()
        return MuonGpu(gpu, g["muon"], g["aux"], lr=0.02, momentum=0.95, nesterov=True, nsSteps=5, aux=dict(adamw, weightDecay=0.0))
    return AdamWGpu(gpu, trainable, **adamw)


def prepare(case, seed):
    case = dict(DEFAULTS, **case)
    cfg = _config(case)
    rng = np.random.default_rng(seed)
    dev = _device(case)
    gpu, held = dev.gpu, _Held(dev)
    B, T = case["batch"], case["seq"]
    model = LanguageModel(cfg, _Normals(seed))
    state = dict(case=case, held=held, gpu=gpu, model=model)

    if case["kind"] in ("score", "decode"):
        freezeForScoring(model)
        n = T + B if case["kind"] == "decode" else B * T + 1
        state["tokens"] = _zipf(rng, n, cfg.vocabSize)
        gpu.uploadParams(model.params())
        return state

    if case["kind"] == "loop":
        n = max(20_000, 4 * T)
        state["tokens"] = _zipf(rng, n, cfg.vocabSize)
        state["supervised"] = (rng.random(n) >= case["masked"]).astype(np.uint8) if case["masked"] else None
        state["opt"] = _optimizer(case, gpu, model, model.params())
        state["seed"] = int(seed)
        return state

    # a recorded step: model and optimizer on the device, gradients in one arena, forward and backward captured
    ids = _zipf(rng, B * (T + 1), cfg.vocabSize).reshape(B, T + 1)
    targets = ids[:, 1:].reshape(-1).copy()
    if case["masked"]:
        targets[rng.random(targets.size) < case["masked"]] = -1
    state["ids"], state["targets"] = ids[:, :-1].reshape(-1).copy(), targets
    ag.setCheckpointing(case["recompute"])
    try:
        trainable = model.params()
        if case["lora"]:
            trainable = applyLora(model, case["lora"], 2.0 * case["lora"], _Normals(seed + 1)).groups["aux"]
            b = _Normals(seed + 2)
            for t in trainable[1::2]:           # a run under way: B has left its zero start
                t.data[:] = b.randn(t.shape, 0.02)
        base, total, _ = gpu.reserveGradArena(list(reversed(trainable)))
        for p in trainable:
            gpu.keepGradOnDevice(p)
        state["opt"] = _optimizer(case, gpu, model, trainable)
        step = state["step"] = held.step = CudaStep(model, gpu, B, T, lossChunk=case["lossChunk"])
        step.run(state["ids"], state["targets"])    # records
        gpu.sync([])
    finally:
        ag.setCheckpointing(False)
        if case["lora"]:
            clearLora()
    state["ticket"] = None
    # The gradients are whole, in one array. A deep model has more weight tensors than can be returned one by one: then those
    # of the first layers and of the embedding come; every weight goes into the next pass's losses and gradients.
    state["out"] = {"losses": _view(held, step.graph.outputs["loss"][0], 1 + B), "grads": _view(held, base, total),
                    "weights": [_view(held, gpu.buffersFor(p)["data"], p.size) for p in trainable[:MAX_WEIGHTS]]}
    return state


def run(state):
    case, gpu, model = state["case"], state["gpu"], state["model"]
    T = case["seq"]
    if case["kind"] == "step":
        step = state["step"]
        step.run(state["ids"], state["targets"])
        state["opt"].recordStep()
        # the loss of a step is collected one step late, as a training program does to keep the device busy
        ticket = step.lossesBegin()
        if state["ticket"] is not None:
            step.lossesEnd(state["ticket"])
        state["ticket"] = ticket
        return state["out"]
    if case["kind"] == "loop":
        ag.setCheckpointing(case["recompute"])
        try:
            history = trainLMGpuResident(model, gpu, state["tokens"], T, case["steps"], case["batch"], state["opt"], logEvery=1,
                                         rng=Mulberry32(state["seed"]), supervised=state["supervised"],
                                         reclaimTransients=True, lossChunk=case["lossChunk"])
        finally:
            ag.setCheckpointing(False)
        return {"losses": np.array([h["loss"] for h in history], np.float32),
                "weights": [p.data for p in model.params()[:MAX_WEIGHTS]]}
    tokens, rows = state["tokens"], []
    gpu.install()
    try:
        for i in range(case["batch"]):
            if case["kind"] == "score":
                loss = sequenceLoss(model, tokens[i * T:(i + 1) * T], tokens[i * T + 1:(i + 1) * T + 1], case["lossChunk"])
                gpu.sync([loss])
                rows.append(float(loss.data[0]))
            else:
                n = T + i
                logits = model.forward(tokens[:n])
                gpu.sync([logits])
                rows.append(logits.data.reshape(n, -1)[-1].copy())
    finally:
        gpu.uninstall()
    return np.array(rows, np.float32)


def work(case):
    """Products and attention of the forward pass once, of the backward pass twice (the input gradients alone where the base
    is frozen), without recompute; parameters, optimizer state and gradients moved once each."""
    case = dict(DEFAULTS, **case)
    cfg, T, B = _config(case), case["seq"], case["batch"]
    h, q, kv = cfg.hiddenSize, cfg.nHeads * cfg.headDim, cfg.nKVHeads * cfg.headDim
    layer = h * (q + 2 * kv) + q * h + 3 * h * cfg.ffnDim
    readout = cfg.vocabSize * h
    params = paramCount(cfg)

    def forward(n):      # one sequence of n tokens: (products, attention) in flop
        attn = 0
        for il in range(cfg.nLayers):
            w = 0 if cfg.arch != "gemma3" or isGlobalLayer(cfg, il) else cfg.slidingWindow
            m = min(w, n) if w else n
            pairs = m * (m + 1) // 2 + (n - m) * m
            attn += 4 * q * pairs
        return 2 * n * (cfg.nLayers * layer + readout), attn

    if case["kind"] in ("score", "decode"):
        lens = [T] * B if case["kind"] == "score" else [T + i for i in range(B)]
        out = 1 if case["kind"] == "score" else cfg.vocabSize
        return {"bytes": sum(4.0 * params + 4 * out + 8 * n for n in lens), "flops": float(sum(sum(forward(n)) for n in lens))}
    gemm, attn = forward(T)
    steps = case["steps"] if case["kind"] == "loop" else 1
    if case["lora"]:
        thin = cfg.nLayers * case["lora"] * sum(o + i for o, i in ((q, h), (kv, h), (kv, h), (h, q), (cfg.ffnDim, h), (cfg.ffnDim, h), (h, cfg.ffnDim)))
        flops, bytes_ = 2.0 * gemm + 3.5 * attn + 6 * T * thin, 4.0 * params + 28 * thin
        return {"bytes": bytes_, "flops": B * flops}
    moved = 28.0 * params if case["optimizer"] == "adamw" else 20.0 * params
    return {"bytes": steps * moved + (4.0 * params if case["kind"] == "loop" else 0), "flops": steps * B * (3.0 * gemm + 3.5 * attn)}


def tolerance(case):
    """Strict f32: order of summation through the depth of the model, and AdamW's first update, which is nearly the sign of a
    gradient element and flips where that sits at the rounding floor. TF32: 11 significant bits per operand put 2e-3 to 6e-3
    on a deep model's gradients; an element of a weight can again differ by a whole update."""
    if dict(DEFAULTS, **case)["precision"] == "fp32":
        return {"rel": 2e-4, "max": 0.2}
    return {"rel": 6e-3, "max": 0.4}
