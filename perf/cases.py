"""Performance cases of the `cuda` device: what a training or generating program has it do.

Each case goes through the public entry points: the kernel callables that a graph runtime binds
(`backend.get_forward_kernel(op)(inputs, outputs)`, `fill_storage2`, `adamw_step`, the stage
methods) or `FusedLayerStep`.  Inputs are torch tensors on the GPU whose memory is handed over by
address, as a torch program would do it; the gradient buffers are zero-filled in every pass, as the
graph runtime does before its backward pass.

A case is a dict of plain values with a `kind`:
  step       one training step of a GPT-shaped model: every fused layer kernel, forward and backward
  generate   one token for each of a few sequences through every layer: the fused layer kernels of decoding
  sublayer   residual add + LayerNorm and GELU of one layer, as graph nodes, forward and backward
  qwen       RMSNorm, RoPE and SwiGLU of one layer, fp32 or bf16 activations, forward and backward
  embed      token embedding: gather and the deterministic scatter-add of its gradient
  head       linear + cross-entropy head, with or without RMSNorm and per-row weights
  project    linear + bias + residual projection
  optimizer  AdamW over a model's parameters
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

import autograd_b200 as ag
from autograd_b200 import dp, hostgraph as hg
from autograd_b200.step import FusedLayerStep, StepConfig
from autograd_b200.storage import CudaMemPointer, Storage

PRECISION = {"3xtf32": ag.AG_CE_3XTF32, "bf16": ag.AG_CE_BF16, "bf16x3": ag.AG_CE_BF16X3}


def listed():
    return [
        # the smallest training step that the tests run: a smoke run or a unit-sized model, all launches and host work
        {"name": "step-tiny", "kind": "step", "layers": 2, "heads": 1, "head_dim": 128, "seq": 64, "batch": 3,
         "vocab": 640, "precision": "3xtf32"},
        # the depth-6 GPT of the published training log: 32 sequences of 512, hidden 384
        {"name": "step-depth6", "kind": "step", "layers": 6, "heads": 6, "head_dim": 64, "seq": 512, "batch": 32,
         "vocab": 32768, "precision": "3xtf32"},
        # the benchmark's own step: depth 20, hidden 1280, 32768 token rows
        {"name": "step-depth20", "kind": "step", "layers": 20, "heads": 10, "head_dim": 128, "seq": 2048, "batch": 16,
         "vocab": 32768, "precision": "3xtf32"},
        # sampling from the depth-20 model, 8 sequences at a time: many launches over a few rows
        {"name": "generate-depth20", "kind": "generate", "layers": 20, "heads": 10, "head_dim": 128, "batch": 8,
         "pos": 700, "vocab": 32768},
        # a hidden size and a row count that no vector width divides: an odd-width experiment
        {"name": "sublayer-ragged", "kind": "sublayer", "rows": 3001, "cols": 1026, "train": True},
        # one layer at Qwen-1.5B widths with bf16 activations, 4 sequences of 2048
        {"name": "qwen-bf16", "kind": "qwen", "batch": 4, "seq": 2048, "heads": 12, "kv_heads": 2, "head_dim": 128,
         "inner": 8960, "dtype": "bf16", "train": True},
        # the same layer on a short batch of prompts in fp32: 3 sequences of 333
        {"name": "qwen-short-f32", "kind": "qwen", "batch": 3, "seq": 333, "heads": 12, "kv_heads": 2, "head_dim": 128,
         "inner": 8960, "dtype": "f32", "train": True},
        # 65536 Zipf-distributed token ids into a Qwen-sized table: fine-tuning on text
        {"name": "embed-zipf", "kind": "embed", "ids": 65536, "cols": 1536, "vocab": 151936, "zipf": True,
         "grad": "f32", "train": True},
        # policy-gradient head of a Qwen-sized model: RMSNorm, per-row weights, ignored prompt rows, bf16 operands
        {"name": "head-rl-bf16", "kind": "head", "rows": 4096, "cols": 1536, "vocab": 151936, "norm": True,
         "weighted": True, "valid_mean": False, "ignored": 0.05, "precision": "bf16", "train": True},
        # a last, partly filled batch through a small head with an odd vocabulary
        {"name": "head-ragged", "kind": "head", "rows": 333, "cols": 392, "vocab": 5003, "norm": False,
         "weighted": False, "valid_mean": True, "ignored": 0.05, "precision": "3xtf32", "train": True},
        # the MLP down-projection of the depth-20 model over 8 sequences
        {"name": "project-down", "kind": "project", "rows": 16384, "inner": 5120, "cols": 1280, "precision": "3xtf32",
         "train": True},
        # one optimizer step of the depth-6 GPT: a few large matrices and many small vectors
        {"name": "adamw-depth6", "kind": "optimizer", "layers": 6, "cols": 384, "vocab": 32768, "grad": "f32"},
    ]


# ------------------------------------------------------------------ drawn cases
def _log(rng, low, high):
    """An integer spread evenly over the logarithm of [low, high]."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["step", "generate", "sublayer", "qwen", "embed", "head", "project", "optimizer"])
    precision = rng.choice(["3xtf32", "3xtf32", "bf16x3", "bf16"])  # fp32-grade is the default
    train = rng.random() < 0.75                                     # the others: evaluation, no gradients
    if kind == "step":
        head_dim = rng.choice([32, 64, 128])
        heads = _log(rng, 1, 1280 // head_dim)
        seq = _log(rng, 16, 2048)
        return {"kind": kind, "layers": _log(rng, 1, 12), "heads": heads, "head_dim": head_dim, "seq": seq,
                "batch": _log(rng, 1, max(1, 16384 // seq)), "vocab": _log(rng, 65, 50257), "precision": precision}
    if kind == "generate":
        head_dim = rng.choice([32, 64, 128])
        return {"kind": kind, "layers": _log(rng, 2, 24), "heads": _log(rng, 1, 2048 // head_dim), "head_dim": head_dim,
                "batch": _log(rng, 1, 64), "pos": rng.randint(0, 2047), "vocab": _log(rng, 65, 50257)}
    if kind == "sublayer":
        return {"kind": kind, "rows": _log(rng, 1, 32768), "cols": _log(rng, 48, 4100), "train": train}
    if kind == "qwen":
        seq = _log(rng, 1, 4096)
        return {"kind": kind, "batch": _log(rng, 1, max(1, 8192 // seq)), "seq": seq, "heads": 2 * _log(rng, 1, 14),
                "kv_heads": 2, "head_dim": rng.choice([64, 128]), "inner": 8 * _log(rng, 32, 1120),
                "dtype": rng.choice(["f32", "bf16"]), "train": train}
    if kind == "embed":
        return {"kind": kind, "ids": _log(rng, 1, 131072), "cols": _log(rng, 32, 2048), "vocab": _log(rng, 65, 151936),
                "zipf": rng.random() < 0.5, "grad": rng.choice(["f32", "f32", "bf16"]), "train": train}
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 16, 8192), "cols": 8 * _log(rng, 8, 192), "vocab": _log(rng, 256, 65536),
                "norm": rng.random() < 0.5, "weighted": rng.random() < 0.3, "valid_mean": rng.random() < 0.5,
                "ignored": rng.choice([0.0, 0.05]), "precision": precision, "train": train}
    if kind == "project":
        return {"kind": kind, "rows": _log(rng, 8, 16384), "inner": 8 * _log(rng, 8, 640), "cols": 8 * _log(rng, 8, 256),
                "precision": "bf16" if precision == "bf16" else "3xtf32", "train": train}
    return {"kind": kind, "layers": _log(rng, 1, 12), "cols": _log(rng, 64, 1280), "vocab": _log(rng, 65, 32768),
            "grad": rng.choice(["f32", "bf16"])}


# ------------------------------------------------------------------ what a pass cannot do without
def _optimizer_shapes(case):
    """Parameters of a GPT without biases: embedding, head, and per layer two norms and four matrices."""
    c, shapes = case["cols"], [(case["vocab"], case["cols"])] * 2
    for _ in range(case["layers"]):
        shapes += [(c,), (c,), (c, 3 * c), (c, c), (c,), (c,), (c, 4 * c), (4 * c, c)]
    return shapes + [(c,), (c,)]


def _distinct(case):
    """How many different rows of the table the ids of an embedding case are expected to name."""
    v = case["vocab"]
    p = np.arange(1, v + 1, dtype=np.float64) ** (-1.1 if case["zipf"] else 0.0)
    return int(np.sum(1.0 - (1.0 - p / p.sum()) ** case["ids"])) or 1


def work(case):
    """Bytes and operations of one pass: every call's operands read once and its results written once."""
    kind, flops = case["kind"], 0
    if kind == "step":
        n, c = case["seq"] * case["batch"], case["heads"] * case["head_dim"]
        v, layers = case["vocab"], case["layers"]
        norms = 2 * layers + 1
        rows = min(n, v)
        nbytes = 4 * (n + rows) * c + norms * 32 * n * c - 4 * n * c     # gather; norms forward and backward
        nbytes += layers * 32 * n * c + layers * 20 * n * 4 * c          # RoPE on q and k, GELU, both ways
        nbytes += 4 * n * c + 8 * rows * c                               # scatter-add
        nbytes += 8 * (n + v) * c + 4 * (n + v) * c                      # the head's operands and gradients; zero-fills
        flops = 6 * n * c * v
    elif kind == "generate":
        n, c = case["batch"], case["heads"] * case["head_dim"]
        nbytes = 8 * n * c + case["layers"] * (2 * 16 * n * c + 16 * n * c + 32 * n * c + 16 * c) + 16 * n * c + 8 * c
    elif kind == "sublayer":
        n = case["rows"] * case["cols"]
        nbytes = 16 * n + 32 * n                                         # h, y from x, r; GELU on the wide rows
        if case["train"]:
            nbytes += 12 * n + 12 * n + 48 * n + (12 + 16) * n           # norm and add backward, GELU backward, zero-fills
    elif kind == "qwen":
        n, es = case["batch"] * case["seq"], 4 if case["dtype"] == "f32" else 2
        d = case["head_dim"]
        c, qk = case["heads"] * d, (case["heads"] + case["kv_heads"]) * d
        nbytes = n * es * (2 * c + 2 * qk) + n * case["inner"] * (12 + 3 * es)      # the projection's result arrives converted
        if case["train"]:
            nbytes += n * es * (4 * c + 2 * qk + 5 * case["inner"])
    elif kind == "embed":
        n, c, rows = case["ids"], case["cols"], _distinct(case)
        nbytes = 4 * (n + rows) * c
        if case["train"]:
            es = 4 if case["grad"] == "f32" else 2
            nbytes += 4 * n * c + (case["vocab"] + 2 * rows) * c * es
    elif kind == "head":
        n, c, v = case["rows"], case["cols"], case["vocab"]
        nbytes, flops = 4 * (n + v) * c, 2 * n * c * v
        if case["train"]:
            nbytes, flops = nbytes + 4 * 4 * (n + v) * c, flops + 4 * n * c * v
    elif kind == "project":
        n, k, c = case["rows"], case["inner"], case["cols"]
        nbytes, flops = 4 * (n * k + k * c + 2 * n * c), 2 * n * k * c
        if case["train"]:
            nbytes, flops = nbytes + 4 * (5 * n * c + 4 * n * k + 4 * k * c), flops + 4 * n * k * c
    else:
        count = sum(math.prod(s) for s in _optimizer_shapes(case))
        nbytes = count * (24 + (4 if case["grad"] == "f32" else 2))
    return {"bytes": int(nbytes), "flops": int(flops)}


def tolerance(case):
    """fp32 sums in another order: 1e-5.  The heads and projections add thousands of products per element on tensor
    cores: 1e-4 in fp32-grade modes, 1e-2 with bf16 operands.  bf16 storage: its rounding."""
    bf16_grad = case["kind"] == "embed" and case["grad"] == "bf16" and case["train"]
    if case.get("precision") == "bf16" or case.get("dtype") == "bf16" or bf16_grad:
        return {"rel": 1e-2, "max": 0.1}
    if "precision" in case:
        return {"rel": 1e-4, "max": 1e-2}
    return {"rel": 1e-5, "max": 1e-3}


# ------------------------------------------------------------------ the device, and torch memory handed to it
_DEVICE = None


def _device():
    """(context, allocator, backend): one per process, as a program has it."""
    global _DEVICE
    if _DEVICE is None:
        _DEVICE = ag.create(0)
    return _DEVICE


_NUMPY = {torch.float32: np.float32, torch.bfloat16: np.uint16, torch.int32: np.int32}


def _wrap(t, grad=None):
    """A torch tensor's memory as a tensor of the backend; bf16 travels as 16-bit words."""
    dtype = _NUMPY[t.dtype]
    h = hg.HostTensor(tuple(t.shape), dtype, requires_grad=grad is not None)
    h.storage = Storage(CudaMemPointer(t.data_ptr()), tuple(t.shape), dtype, "cuda", t.numel() * t.element_size())
    if grad is not None:
        h.grad = _wrap(grad)
    return h


class _Inputs:
    """Seeded inputs on the GPU; keeps every tensor it makes, since the backend holds addresses only."""

    def __init__(self, seed):
        self.generator = torch.Generator(device="cuda")
        self.generator.manual_seed(seed)
        self.kept = []

    def keep(self, t):
        self.kept.append(t)
        return t

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        t = torch.empty(shape, device="cuda", dtype=torch.float32)
        t.normal_(mean, std, generator=self.generator)
        return self.keep(t if dtype == torch.float32 else t.to(dtype))

    def empty(self, *shape, dtype=torch.float32):
        return self.keep(torch.zeros(shape, device="cuda", dtype=dtype))

    def uniform_ids(self, count, below):
        t = torch.randint(0, below, (count,), device="cuda", generator=self.generator)
        return self.keep(t.to(torch.int32))

    def zipf_ids(self, count, below):
        """Ids whose frequency falls as rank^-1.1, as words do in text."""
        p = torch.arange(1, below + 1, device="cuda", dtype=torch.float64).pow(-1.1)
        at = torch.cumsum(p, 0)
        u = torch.rand(count, device="cuda", dtype=torch.float64, generator=self.generator) * at[-1]
        return self.keep(torch.searchsorted(at, u).clamp_(max=below - 1).to(torch.int32))

    def rope_tables(self, seq, head_dim, theta):
        angle = torch.arange(seq, device="cuda", dtype=torch.float32)[:, None] * theta ** (
            -torch.arange(0, head_dim, 2, device="cuda", dtype=torch.float32)[None, :] / head_dim)
        return self.keep(angle.cos().contiguous()), self.keep(angle.sin().contiguous())


def _zero(backend, *tensors):
    for t in tensors:
        backend.fill_storage2(t.grad.storage, 0)


# ------------------------------------------------------------------ one training step
class _Owner:
    """Closes a step when nothing refers to it any more: neither the state nor a tensor over its memory."""

    def __init__(self, step):
        self.step = step

    def __del__(self):
        self.step.close()

    def tensor(self, address, count):
        view = dp.DeviceArrayView(address, count)
        view.owner = self  # torch keeps the view alive as long as the tensor
        return torch.as_tensor(view, device="cuda")


class _Step:
    """A FusedLayerStep with its batch in pinned memory."""

    def __init__(self, case, seed):
        ctx, alloc, backend = _device()
        cfg = StepConfig(n_layer=case["layers"], n_embd=case["heads"] * case["head_dim"], n_head=case["heads"],
                         head_dim=case["head_dim"], seq_len=case["seq"], vocab=case["vocab"], batch=case["batch"],
                         ce_precision=PRECISION[case["precision"]])
        generator = torch.Generator(device="cuda")

        def fill_normal(address, count, seed_, std):
            generator.manual_seed(seed_)
            dp.as_torch(address, count).normal_(0.0, std, generator=generator)
            torch.cuda.synchronize()

        self.step = FusedLayerStep(ctx, alloc, backend, cfg, seed=1000 * seed, fill_normal=fill_normal)
        draw_ids = torch.Generator()
        draw_ids.manual_seed(seed)
        self.batch = torch.randint(0, cfg.vocab, (2, cfg.tokens), dtype=torch.int32, generator=draw_ids).pin_memory()
        s, own = self.step, _Owner(self.step)
        self.outputs = {"loss": own.tensor(s.loss, 1), "norm_grads": own.tensor(s.small_bucket, s.n_small),
                        "table_grad": own.tensor(s.dtable, s.V * s.C), "stream_grad": own.tensor(s.dh, s.N * s.C),
                        "gelu": own.tensor(s.g, s.N * s.I), "gelu_grad": own.tensor(s.du, s.N * s.I),
                        "stream": own.tensor(s.h_final, s.N * s.C), "normed": own.tensor(s.y[0], s.N * s.C)}

    def run(self):
        self.step.load_batch(self.batch[0].data_ptr(), self.batch[1].data_ptr())
        self.step.step()
        return self.outputs


# ------------------------------------------------------------------ one generated token
class _Generate:
    """Gather, then per layer add + LayerNorm, RoPE at the current position, add + LayerNorm, GELU; a last LayerNorm.
    The projections and attention between them belong to the program: their results are inputs here."""

    def __init__(self, case, seed):
        self.ctx, _, self.backend = _device()
        make, n = _Inputs(seed), case["batch"]
        heads, d, layers = case["heads"], case["head_dim"], case["layers"]
        c = heads * d
        self.make = make
        cos, sin = make.rope_tables(2048, d, 1e5)
        at = case["pos"]
        self.cos, self.sin = _wrap(cos[at:at + 1]), _wrap(sin[at:at + 1])
        gather = hg.make_node(hg.make_op("GatherOp"), [_wrap(make.uniform_ids(n, case["vocab"])),
                                                       _wrap(make.normal(case["vocab"], c, std=0.02))],
                              [_wrap(make.empty(n, c))])
        self.gather = gather, self.backend.get_forward_kernel(gather.op)
        self.layers, stream = [], gather.outputs[0]
        for _ in range(layers):
            one = SimpleNamespace(x=stream)
            one.r, one.a = _wrap(make.normal(n, c)), _wrap(make.normal(n, c))
            one.g1, one.b1, one.g2, one.b2 = (_wrap(make.normal(c, std=0.02, mean=m)) for m in (1.0, 0.0, 1.0, 0.0))
            one.h1, one.y1, one.h2, one.y2 = (_wrap(make.empty(n, c)) for _ in range(4))
            q = make.normal(n, 1, heads, d)
            one.q, one.k = _wrap(q), _wrap(make.normal(n, 1, heads, d))
            hidden = make.empty(n, 4 * c)
            node = hg.make_node(hg.make_op("GELUOp"), [_wrap(make.normal(n, 4 * c))], [_wrap(hidden)])
            one.gelu = node, self.backend.get_forward_kernel(node.op)
            stream = one.h2
            self.layers.append(one)
        last = make.empty(n, c)
        node = hg.make_node(hg.make_op("LayerNormOp", eps=1e-5, normalized_dim=-1),
                            [stream, _wrap(make.normal(c, std=0.02, mean=1.0)), _wrap(make.normal(c, std=0.02))],
                            [_wrap(last)])
        self.norm = node, self.backend.get_forward_kernel(node.op)
        self.outputs = {"normed": last, "gelu": hidden, "q": q}

    def run(self):
        backend = self.backend
        node, fn = self.gather
        fn(node.inputs, node.outputs)
        for one in self.layers:
            backend.fused_add_layernorm_forward(one.x, one.r, one.g1, one.b1, one.h1, one.y1, 1e-5)
            backend.rope_qk(one.q, one.k, self.cos, self.sin)
            backend.fused_add_layernorm_forward(one.h1, one.a, one.g2, one.b2, one.h2, one.y2, 1e-5)
            node, fn = one.gelu
            fn(node.inputs, node.outputs)
        node, fn = self.norm
        fn(node.inputs, node.outputs)
        return self.outputs


# ------------------------------------------------------------------ residual add + LayerNorm, GELU
class _Sublayer:
    def __init__(self, case, seed):
        self.ctx, _, self.backend = _device()
        be, make, n, c = self.backend, _Inputs(seed), case["rows"], case["cols"]
        self.make, self.train = make, case["train"]
        grad = (lambda *shape: make.empty(*shape)) if self.train else (lambda *shape: None)
        self.grads = [grad(n, c), grad(n, c), grad(n, c), grad(c), grad(c), grad(n, 4 * c)]
        x_g, r_g, h_g, gamma_g, beta_g, u_g = self.grads
        h, y, hidden = make.empty(n, c), make.empty(n, c), make.empty(n, 4 * c)
        dy, dhidden = (make.normal(n, c), make.normal(n, 4 * c)) if self.train else (None, None)
        add = hg.make_node(hg.make_op("AddOp"), [_wrap(make.normal(n, c), x_g), _wrap(make.normal(n, c), r_g)],
                           [_wrap(h, h_g)])
        norm = hg.make_node(hg.make_op("LayerNormOp", eps=1e-5, normalized_dim=-1),
                            [add.outputs[0], _wrap(make.normal(c, std=0.02, mean=1.0), gamma_g),
                             _wrap(make.normal(c, std=0.02), beta_g)], [_wrap(y, dy)])
        gelu = hg.make_node(hg.make_op("GELUOp"), [_wrap(make.normal(n, 4 * c), u_g)], [_wrap(hidden, dhidden)])
        self.add, self.norm, self.gelu = add, norm, gelu
        self.gelu_forward, self.gelu_backward = be.get_forward_kernel(gelu.op), be.get_backward_kernel(gelu.op)
        self.norm_backward, self.add_backward = be.get_backward_kernel(norm.op), be.bind_add_backward(add)
        self.outputs = [h, y, hidden] + self.grads

    def run(self):
        be, add, norm, gelu = self.backend, self.add, self.norm, self.gelu
        be.fused_add_layernorm_forward(add.inputs[0], add.inputs[1], norm.inputs[1], norm.inputs[2], add.outputs[0],
                                       norm.outputs[0], 1e-5)
        self.gelu_forward(gelu.inputs, gelu.outputs)
        if self.train:
            _zero(be, *add.inputs, *norm.inputs, gelu.inputs[0])
            self.gelu_backward(gelu.inputs, gelu.outputs)
            self.norm_backward(norm.inputs, norm.outputs)
            self.add_backward(add.inputs, add.outputs)
        return self.outputs


# ------------------------------------------------------------------ RMSNorm, RoPE, SwiGLU
class _Qwen:
    """The gate and up projections belong to the program; their result arrives in the other precision and is
    converted, so that the in-place SwiGLU backward has fresh operands in every pass."""

    def __init__(self, case, seed):
        self.ctx, _, self.backend = _device()
        make, b, t = _Inputs(seed), case["batch"], case["seq"]
        heads, kv, d, inner = case["heads"], case["kv_heads"], case["head_dim"], case["inner"]
        n, c = b * t, heads * d
        self.make, self.train, self.bf16, self.count = make, case["train"], case["dtype"] == "bf16", n * 2 * inner
        dt, other = (torch.bfloat16, torch.float32) if self.bf16 else (torch.float32, torch.bfloat16)
        self.cos, self.sin = (_wrap(x) for x in make.rope_tables(t, d, 1e6))
        self.x, self.gamma = _wrap(make.normal(n, c, dtype=dt)), _wrap(make.normal(c, std=0.02, mean=1.0))
        z, q, k = make.empty(n, c, dtype=dt), make.normal(b, t, heads, d, dtype=dt), make.normal(b, t, kv, d, dtype=dt)
        self.z, self.q, self.k = _wrap(z), _wrap(q), _wrap(k)
        self.projected = make.normal(n, 2 * inner, dtype=other)
        gu, hidden = make.empty(n, 2 * inner, dtype=dt), make.empty(n, inner, dtype=dt)
        self.gu, self.hidden = _wrap(gu), _wrap(hidden)
        self.outputs = [z, q, k, hidden, gu]
        if self.train:
            self.dhidden, self.dz = _wrap(make.normal(n, inner, dtype=dt)), _wrap(make.normal(n, c, dtype=dt))
            self.dres = _wrap(make.normal(n, c, dtype=dt))
            dx, dgamma = make.empty(n, c, dtype=dt), make.empty(c)
            self.dx, self.dgamma = _wrap(dx), _wrap(dgamma)
            self.outputs += [dx, dgamma]

    def run(self):
        be, ctx = self.backend, self.ctx
        be.rmsnorm_forward(self.x, self.gamma, self.z, 1e-6)
        be.rope_qk(self.q, self.k, self.cos, self.sin)
        projected, gu = self.projected.data_ptr(), self.gu.storage.ptr.address
        if self.bf16:
            ctx.f32_to_bf16(projected, gu, self.count)
        else:
            ctx.bf16_to_f32(projected, gu, self.count)
        be.swiglu_forward(self.gu, self.hidden)
        if self.train:
            be.swiglu_backward(self.gu, self.dhidden)
            be.rope_qk(self.q, self.k, self.cos, self.sin, sin_sign=-1)
            be.fill_storage2(self.dgamma.storage, 0)
            be.rmsnorm_backward(self.dz, self.x, self.gamma, 1e-6, self.dx, self.dgamma, dres=self.dres)
        return self.outputs


# ------------------------------------------------------------------ one graph node with a forward and a backward kernel
class _Node:
    """A node of the graph, run as the runtime runs it: forward; gradients zero-filled; backward."""

    def __init__(self, make, op, inputs, outputs, train, results):
        _, _, self.backend = _device()
        self.make, self.node, self.train, self.outputs = make, hg.make_node(op, inputs, outputs), train, results
        self.forward, self.backward = self.backend.get_forward_kernel(op), self.backend.get_backward_kernel(op)
        self.with_grad = [t for t in self.node.inputs if t is not None and t.grad is not None]

    def run(self):
        node = self.node
        self.forward(node.inputs, node.outputs)
        if self.train:
            _zero(self.backend, *self.with_grad)
            self.backward(node.inputs, node.outputs)
        return self.outputs


def _embed(case, seed):
    make, n, c, v = _Inputs(seed), case["ids"], case["cols"], case["vocab"]
    ids = make.zipf_ids(n, v) if case["zipf"] else make.uniform_ids(n, v)
    out, results = make.empty(n, c), []
    grad = dout = None
    if case["train"]:
        grad = make.empty(v, c, dtype=torch.float32 if case["grad"] == "f32" else torch.bfloat16)
        dout = make.normal(n, c)
        results = [grad]
    return _Node(make, hg.make_op("GatherOp"), [_wrap(ids), _wrap(make.normal(v, c, std=0.02), grad)],
                 [_wrap(out, dout)], case["train"], [out] + results)


class _Head(_Node):
    """The precision of the head is a setting of the backend, made before the calls as a program does."""

    def __init__(self, case, seed):
        make, n, c, v = _Inputs(seed), case["rows"], case["cols"], case["vocab"]
        train = case["train"]
        x_g, w_g, gamma_g = (make.empty(n, c), make.empty(v, c), make.empty(c)) if train else (None, None, None)
        x, w = _wrap(make.normal(n, c), x_g), _wrap(make.normal(v, c, std=0.02), w_g)
        targets = make.uniform_ids(n, v)
        if case["ignored"]:
            targets[torch.rand(n, device="cuda", generator=make.generator) < case["ignored"]] = -1
        weights = [_wrap(make.keep(torch.rand(n, device="cuda", generator=make.generator) / n))] if case["weighted"] else []
        loss = make.empty(1)
        out = _wrap(loss, make.keep(torch.ones(1, device="cuda")) if train else None)
        if case["norm"]:
            op = hg.make_op("FusedRMSNormLinearCrossEntropyOp", eps=1e-6)
            inputs = [x, w, _wrap(make.normal(c, std=0.02, mean=1.0), gamma_g), _wrap(targets)] + weights
        else:
            op = hg.make_op("FusedLinearCrossEntropyOp")
            inputs = [x, w, _wrap(targets)] + weights
        results = [loss] + ([x_g, w_g] + ([gamma_g] if case["norm"] else []) if train else [])
        super().__init__(make, op, inputs, [out], train, results)
        self.precision = PRECISION[case["precision"]]
        self.reduction = ag.AG_CE_MEAN_VALID if case["valid_mean"] else ag.AG_CE_MEAN_ALL_ROWS

    def run(self):
        self.backend.ce_precision, self.backend.ce_reduction = self.precision, self.reduction
        return super().run()


class _Project(_Node):
    def __init__(self, case, seed):
        make, n, k, c = _Inputs(seed), case["rows"], case["inner"], case["cols"]
        train = case["train"]
        grads = [make.empty(*s) for s in ((n, c), (n, k), (k, c), (c,))] if train else [None] * 4
        inputs = [_wrap(make.normal(n, c), grads[0]), _wrap(make.normal(n, k), grads[1]),
                  _wrap(make.normal(k, c, std=0.02), grads[2]), _wrap(make.normal(c, std=0.02), grads[3])]
        out = make.empty(n, c)
        super().__init__(make, hg.make_op("FusedLinearAddOp"), inputs, [_wrap(out, make.normal(n, c) if train else None)],
                         train, [out] + (grads if train else []))
        self.precision = PRECISION[case["precision"]]

    def run(self):
        self.backend.ce_precision = self.precision
        return super().run()


# ------------------------------------------------------------------ AdamW
class _Optimizer:
    """Parameters, gradients and moments lie in one buffer each, every parameter on a 256-byte boundary; the
    optimizer steps them one after the other."""

    def __init__(self, case, seed):
        _, _, self.backend = _device()
        self.make = make = _Inputs(seed)
        shapes, at, offsets = _optimizer_shapes(case), 0, []
        for s in shapes:
            offsets.append(at)
            at += (math.prod(s) + 127) // 128 * 128
        dt = torch.float32 if case["grad"] == "f32" else torch.bfloat16
        p, g = make.normal(at, std=0.02), make.normal(at, std=0.01, dtype=dt)
        m, v = make.normal(at, std=0.01), make.keep(make.normal(at, std=0.01).square())
        self.params = [tuple(_wrap(t[o:o + math.prod(s)].view(s)).storage for t in (p, g, m, v))
                       for s, o in zip(shapes, offsets)]
        self.outputs = [p, m, v]

    def run(self):
        step = self.backend.adamw_step
        for p, g, m, v in self.params:
            step(p, g, m, v, None, 3e-4, 2.9e-4, 0.9, 0.95, 1e-8, 0.1)
        return self.outputs


# ------------------------------------------------------------------ the interface
_KINDS = {"step": _Step, "generate": _Generate, "sublayer": _Sublayer, "qwen": _Qwen, "embed": _embed, "head": _Head,
          "project": _Project, "optimizer": _Optimizer}


def prepare(case, seed):
    state = _KINDS[case["kind"]](case, seed)
    torch.cuda.synchronize()  # the inputs were made on torch's stream, the backend works on its own
    return state


def run(state):
    return state.run()
