"""The work that a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public C interface (include/ckb200*.h), reached over ctypes as the reference's own tools reach a model:

  gemv     one activation row through one quantised matrix, host pointers as generated code passes them (weights registered) or
           device pointers as a runtime of the user's own does
  gemm     the rows of a prompt through one quantised matrix, device pointers
  decode   a few tokens generated by a whole model, token ids in and logits out at every step, for one sequence or a batch
  prompt   a prompt, or a later turn of a conversation, through a whole model: ids in, the last token's logits out, the cache filled
  request  a prompt and the tokens generated after it through a layer-stack model

Weights are random blocks whose values have mean zero and variance 1 / columns, less for what is added to the residual, so that activations
and attention scores have the spread they have in trained models and the arithmetic is as well conditioned."""
from __future__ import annotations

import ctypes as C
import json
import math
import os
import tempfile

import numpy as np
import torch

import __graft_entry__ as graft

pkg = graft.load_package()
api = pkg.model_api
vptr, fptr = api.vptr, api.fptr

# block formats: name -> (value of the fmt_* fields, bytes of a block, elements of a block, spread of its values at d = 1)
FORMATS = {"q4_k": (0, 144, 256, 258.0), "q6_k": (1, 210, 256, 342.0), "q8_0": (2, 34, 32, 73.0), "q5_0": (3, 22, 32, 9.2)}
FMT_NAME = {v[0]: k for k, v in FORMATS.items()}

# what fmt_q, fmt_k, fmt_v, fmt_o, fmt_gate_up, fmt_down, fmt_lm_head are in the files people run
MIXES = {
    "q4_k_m": dict(fmt_q=0, fmt_k=0, fmt_v=1, fmt_o=0, fmt_gate_up=0, fmt_down=1, fmt_lm_head=1),
    # models whose width is no multiple of 256 keep their projections in 32-element blocks
    "q5_0": dict(fmt_q=3, fmt_k=3, fmt_v=3, fmt_o=3, fmt_gate_up=3, fmt_down=1, fmt_lm_head=1),
}
SHAPES = {
    "qwen2-0.5b": dict(embed_dim=896, num_heads=14, num_kv_heads=2, head_dim=64, intermediate_size=4864, num_layers=24, vocab_size=151936, rms_eps=1e-6, rope_theta=1.0e6),
    "llama3-8b": dict(embed_dim=4096, num_heads=32, num_kv_heads=8, head_dim=128, intermediate_size=14336, num_layers=32, vocab_size=128256, rms_eps=1e-5, rope_theta=5.0e5),
    "llama3-70b": dict(embed_dim=8192, num_heads=64, num_kv_heads=8, head_dim=128, intermediate_size=28672, num_layers=80, vocab_size=128256, rms_eps=1e-5, rope_theta=5.0e5),
}
STACK_VOCAB = 32768
LN1, WQ, WK, WV, WO, LN2, W1, W2 = range(8)
FINAL_GAMMA, LM_HEAD = 100, 101


def listed():
    return [
        # one call of generated code that was linked against the library: quantise the row, multiply, all pointers on the host
        dict(name="gemv host q4_k 4096x4096", kind="gemv", fmt="q4_k", rows=4096, cols=4096, host=True),
        # the LM head of a small model that a runtime of its own keeps resident
        dict(name="gemv device q8_0 151936x896", kind="gemv", fmt="q8_0", rows=151936, cols=896, host=False),
        # the gate/up projection of an 8B layer for a prompt of odd length
        dict(name="gemm q4_k 333 tokens", kind="gemm", fmt="q4_k", tokens=333, rows=28672, cols=4096),
        # chat with a small model: latency of a token
        dict(name="decode qwen2-0.5b ctx 1024", kind="decode", shape="qwen2-0.5b", layers=24, mix="q4_k_m", batch=1, ctx=1024, steps=8, kv_f16=False),
        # the same model's short question, and the file format in which it is mostly shipped on a longer one
        dict(name="prompt qwen2-0.5b 77", kind="prompt", shape="qwen2-0.5b", layers=24, mix="q4_k_m", ctx=0, tokens=77),
        dict(name="prompt qwen2-0.5b q5_0 256", kind="prompt", shape="qwen2-0.5b", layers=24, mix="q5_0", ctx=0, tokens=256),
        # an assistant on one GPU: a token, the first prompt, a later turn of the conversation
        dict(name="decode llama3-8b ctx 4096", kind="decode", shape="llama3-8b", layers=32, mix="q4_k_m", batch=1, ctx=4096, steps=8, kv_f16=False),
        dict(name="prompt llama3-8b 512", kind="prompt", shape="llama3-8b", layers=32, mix="q4_k_m", ctx=0, tokens=512),
        dict(name="turn llama3-8b 129 after 1024", kind="prompt", shape="llama3-8b", layers=32, mix="q4_k_m", ctx=1024, tokens=129),
        # a server with 32 sequences in flight: one of ten pipeline stages of the largest shape
        dict(name="decode llama3-70b/10 batch 32", kind="decode", shape="llama3-70b", layers=8, mix="q4_k_m", batch=32, ctx=4096, steps=4, kv_f16=False),
        # layer-stack models: a long prompt, and a short one with the answer generated after it
        dict(name="request puzevik 2048+0", kind="request", design="puzevik", width=4096, periods=1, tokens=2048, steps=0),
        dict(name="request sipadra 100+32", kind="request", design="sipadra", width=2048, periods=2, tokens=100, steps=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """gemv and gemm: each format, 256 to 32768 rows (GEMV: up to a vocabulary), 256 to 14336 columns; models: each shape and mix the
    executor takes, one sequence or 2 to 32, contexts of 16 to 4096 tokens in either cache type, prompts of 16 to 512 tokens that start a
    conversation or go on with one of up to 2048; layer stacks of either design."""
    kind = rng.choice(["gemv", "gemm", "decode", "decode", "prompt", "prompt", "prompt", "request"])
    if kind == "gemv":
        fmt = rng.choice(sorted(FORMATS))
        unit = FORMATS[fmt][2]
        return dict(kind=kind, fmt=fmt, rows=_log(rng, 256, 151936), cols=max(256, _log(rng, 256, 14336) // unit * unit), host=rng.random() < 0.5)
    if kind == "gemm":
        fmt = rng.choice(["q4_k", "q4_k", "q6_k", "q8_0"])
        unit = FORMATS[fmt][2]
        return dict(kind=kind, fmt=fmt, tokens=_log(rng, 2, 512), rows=_log(rng, 256, 32768), cols=max(256, _log(rng, 896, 14336) // unit * unit))
    if kind == "decode":
        shape = rng.choice(sorted(SHAPES))
        small = shape == "qwen2-0.5b"
        batch = 1 if small or rng.random() < 0.4 else _log(rng, 2, 32)
        layers = {"qwen2-0.5b": 24, "llama3-8b": 32, "llama3-70b": 8}[shape] if batch == 1 else 8
        return dict(kind=kind, shape=shape, layers=layers, mix=rng.choice(["q4_k_m", "q5_0"]) if small else "q4_k_m", batch=batch, ctx=_log(rng, 16, 4000 if not small else 2000),
                    steps=rng.randint(2, 8) if batch == 1 else rng.randint(2, 4), kv_f16=rng.random() < 0.4)
    if kind == "prompt":
        small = rng.random() < 0.5
        return dict(kind=kind, shape="qwen2-0.5b" if small else "llama3-8b", layers=24 if small else 32, mix=rng.choice(["q4_k_m", "q5_0"]) if small else "q4_k_m",
                    ctx=0 if rng.random() < 0.6 else _log(rng, 16, 2048), tokens=_log(rng, 16, 500))
    design = rng.choice(["puzevik", "sipadra"])
    return dict(kind=kind, design=design, width=rng.choice([2048, 4096]), periods=1, tokens=_log(rng, 16, 1500), steps=rng.choice([0, rng.randint(1, 24)]))


# ------------------------------------------------------------------ inputs

_lib = None


def lib():
    global _lib
    if _lib is None:
        torch.cuda.init()
        torch.cuda.current_stream()
        _lib = pkg.load_lib()
        api.bind_model_api(_lib)
        for name in ("ckb200_q6_k_planar_bytes", "ckb200_q8_0_planar_bytes", "ckb200_q5_0_planar_bytes"):
            getattr(_lib, name).restype = C.c_size_t
        if _lib.ckb200_init(0) != 0:
            raise RuntimeError(_lib.ckb200_last_error_message().decode())
    return _lib


def ok(rc):
    if rc:
        raise RuntimeError((lib().ckb200_last_error_message() or b"call failed").decode())


def p(t):
    return C.c_void_p(t.data_ptr())


def generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def make_blocks(fmt, rows, cols, gen, scale=1.0):
    """uint8 [rows, blocks, block bytes] on the GPU, values of mean 0 and variance scale^2 / cols."""
    _, size, unit, spread = FORMATS[fmt]
    nb = rows * (cols // unit)
    raw = torch.randint(-2 ** 63, 2 ** 63 - 1, (nb * size // 8 + 1,), dtype=torch.int64, device="cuda", generator=gen).view(torch.uint8)[:nb * size].view(nb, size)
    d = (torch.rand(nb, device="cuda", generator=gen) + 0.5) * (scale / (spread * math.sqrt(cols)))

    def put(at, v):
        raw[:, at:at + 2] = v.to(torch.float16).view(torch.uint8).view(nb, 2)

    if fmt == "q4_k":
        put(0, d)
        put(2, 7.5 * d)
    elif fmt == "q6_k":
        raw[:, 192:208] = ((raw[:, 192:208].to(torch.int16) & 63) - 32).to(torch.int8).view(torch.uint8)
        put(208, d)
    else:
        put(0, d)
        if fmt == "q8_0":
            q = raw[:, 2:].view(torch.int8)
            q[q == -128] = -127
    return raw.view(rows, cols // unit, size)


def act_bytes(fmt, cols):
    return cols // 32 * 34 if fmt in ("q8_0", "q5_0") else cols // 256 * 292


def model_cfg(case):
    need = case["ctx"] + case.get("steps", 0) + case.get("tokens", 0)
    return dict(SHAPES[case["shape"]], num_layers=case["layers"], max_seq_len=max(256, (need + 255) // 256 * 256), **MIXES[case["mix"]])


def matrices(cfg):
    """(layer, tensor, format, rows, columns) of every matrix, columns as the executor pads them."""
    D, A, kv, F = cfg["embed_dim"], cfg["num_heads"] * cfg["head_dim"], cfg["num_kv_heads"] * cfg["head_dim"], cfg["intermediate_size"]

    def pad(fmt, k):
        unit = FORMATS[FMT_NAME[fmt]][2]
        return (k + unit - 1) // unit * unit

    for layer in range(cfg["num_layers"]):
        for which, f, rows, k in ((WQ, cfg["fmt_q"], A, D), (WK, cfg["fmt_k"], kv, D), (WV, cfg["fmt_v"], kv, D), (WO, cfg["fmt_o"], D, A), (W1, cfg["fmt_gate_up"], 2 * F, D), (W2, cfg["fmt_down"], D, F)):
            yield layer, which, FMT_NAME[f], rows, pad(f, k)
    yield -1, LM_HEAD, FMT_NAME[cfg["fmt_lm_head"]], cfg["vocab_size"], pad(cfg["fmt_lm_head"], D)


def matrix_bytes(fmt, rows, cols):
    return rows * (cols // FORMATS[fmt][2]) * FORMATS[fmt][1]


class Handle:
    """A model of the library, freed when nothing uses it or its memory any more."""

    def __init__(self, ptr):
        self.ptr = ptr

    def __del__(self):
        lib().ckb200_model_free(self.ptr)


class DeviceArray:
    """Memory of a model as something torch can view; the view keeps the model."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "typestr": kind, "version": 3, "strides": None}


class Model:
    """A decoder of random weights, its cache filled to `ctx`."""

    def __init__(self, case, seed):
        L = lib()
        self.cfg = model_cfg(case)
        self.batch = case.get("batch", 1)
        L.ckb200_tune_set(b"model_kv_f16", int(case.get("kv_f16", False)))
        try:
            self.handle = L.ckb200_model_create(C.byref(api.make_cfg(self.cfg, batch=self.batch)))
        finally:
            L.ckb200_tune_set(b"model_kv_f16", 0)
        if not self.handle:
            ok(1)
        self.owner = Handle(self.handle)
        gen = generator(seed)
        staging = None

        def upload(layer, which, t):
            nonlocal staging
            flat = t.reshape(-1).view(torch.uint8)
            if staging is None or staging.numel() < flat.numel():
                staging = torch.empty(flat.numel(), dtype=torch.uint8, pin_memory=True)
            staging[:flat.numel()].copy_(flat)
            ok(L.ckb200_model_upload_tensor(self.handle, layer, which, C.c_void_p(staging.data_ptr()), flat.numel()))

        biggest = max(matrix_bytes(f, r, c) for _, _, f, r, c in matrices(self.cfg))
        staging = torch.empty(biggest, dtype=torch.uint8, pin_memory=True)
        for layer, which, fmt, rows, cols in matrices(self.cfg):
            # what a layer adds to the residual is small beside it; the table that is both embedding and LM head has entries of variance 1
            scale = {WO: (2 * self.cfg["num_layers"]) ** -0.5, W2: (2 * self.cfg["num_layers"]) ** -0.5, LM_HEAD: math.sqrt(cols)}.get(which, 1.0)
            upload(layer, which, make_blocks(fmt, rows, cols, gen, scale))
        D, Da = self.cfg["embed_dim"], (self.cfg["embed_dim"] + 255) // 256 * 256
        for layer in range(self.cfg["num_layers"]):
            for which in (LN1, LN2):
                upload(layer, which, self._gamma(D, Da, gen))
        upload(-1, FINAL_GAMMA, self._gamma(D, Da, gen))
        ok(L.ckb200_model_fill_kv_synthetic(self.handle, case["ctx"], int(seed) & 0x7FFFFFFF))
        c = self.cfg
        kind = "<f2" if case.get("kv_f16") else "<f4"
        self.kv = torch.as_tensor(DeviceArray(self.owner, L.ckb200_model_kv_device(self.handle, 0, 0),
                                              (c["num_layers"], 2, self.batch, c["num_kv_heads"], c["max_seq_len"], c["head_dim"]), kind), device="cuda")
        self.L = L

    @staticmethod
    def _gamma(D, Da, gen):
        g = torch.zeros(Da, device="cuda")
        g[:D] = 1 + 0.1 * torch.randn(D, device="cuda", generator=gen)
        return g

    def weights(self, layer, which, fmt, rows, cols):
        """The blocks as they lie on the device."""
        self.L.ckb200_model_tensor_ptr.restype = C.c_void_p
        self.L.ckb200_model_tensor_ptr.argtypes = [C.c_void_p, C.c_int, C.c_int]
        ptr = self.L.ckb200_model_tensor_ptr(self.handle, layer, which)
        if fmt is None:
            return torch.as_tensor(DeviceArray(self.owner, ptr, (cols,), "<f4"), device="cuda")
        return torch.as_tensor(DeviceArray(self.owner, ptr, (rows, cols // FORMATS[fmt][2], FORMATS[fmt][1]), "|u1"), device="cuda")


class Gemv:
    def __init__(self, case, seed):
        L = self.L = lib()
        fmt, rows, cols = case["fmt"], case["rows"], case["cols"]
        self.rows, self.cols, self.w_host = rows, cols, None
        gen = generator(seed)
        blocks = make_blocks(fmt, rows, cols, gen)
        x = torch.randn(cols, device="cuda", generator=gen)
        if case["host"]:
            self.w_host = blocks.reshape(-1).cpu().numpy()
            self.x, self.xq, self.y = x.cpu().numpy(), np.zeros(act_bytes(fmt, cols), np.uint8), np.zeros(rows, np.float32)
            ok(L.ckb200_register_weights(vptr(self.w_host), C.c_size_t(self.w_host.nbytes)))
            self.quantise = getattr(L, "quantize_row_q8_0" if fmt in ("q8_0", "q5_0") else "quantize_row_q8_k")
            self.multiply = getattr(L, f"gemv_{fmt}_" + ("q8_0" if fmt in ("q8_0", "q5_0") else "q8_k"))
            self.quantise.restype = self.multiply.restype = None
        else:
            self.x, self.xq, self.y = x, torch.zeros(act_bytes(fmt, cols) + 64, dtype=torch.uint8, device="cuda"), torch.zeros(rows, device="cuda")
            self.w = resident(L, fmt, blocks, rows, cols)
            self.quantise = getattr(L, "ckb200_dev_quantize_" + ("q8_0" if fmt in ("q8_0", "q5_0") else "q8_k"))
            self.multiply = getattr(L, {"q4_k": "ckb200_dev_gemv_q4_k_q8_k", "q6_k": "ckb200_dev_gemv_q6_k_planar_q8_k",
                                        "q8_0": "ckb200_dev_gemv_q8_0_planar_q8_0", "q5_0": "ckb200_dev_gemv_q5_0_planar_q8_0"}[fmt])

    def run(self):
        if self.w_host is not None:
            self.quantise(fptr(self.x), vptr(self.xq), C.c_int(self.cols))
            self.multiply(fptr(self.y), vptr(self.w_host), vptr(self.xq), C.c_int(self.rows), C.c_int(self.cols))
            pkg.check(self.L)
        else:
            ok(self.quantise(p(self.x), p(self.xq), 1, self.cols, None))
            ok(self.multiply(p(self.y), p(self.w), p(self.xq), self.rows, self.cols, None))
        return {"y": self.y}

    def __del__(self):
        if getattr(self, "w_host", None) is not None:
            self.L.ckb200_unregister_weights(vptr(self.w_host))


def resident(L, fmt, blocks, rows, cols):
    """The form in which a runtime keeps a matrix on the device: Q4_K rows as they are, the others row-planar."""
    if fmt == "q4_k":
        return torch.cat([blocks.reshape(-1), torch.zeros(256, dtype=torch.uint8, device="cuda")])
    w = torch.zeros(getattr(L, f"ckb200_{fmt}_planar_bytes")(rows, cols) + 256, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ok(getattr(L, f"ckb200_dev_{fmt}_to_planar")(p(w), p(blocks), rows, cols, None))
    ok(L.ckb200_synchronize())
    return w


class Gemm:
    def __init__(self, case, seed):
        L = self.L = lib()
        fmt, T, rows, cols = case["fmt"], case["tokens"], case["rows"], case["cols"]
        self.args = T, rows, cols
        gen = generator(seed)
        blocks = make_blocks(fmt, rows, cols, gen)
        self.x = torch.randn(T, cols, device="cuda", generator=gen)
        self.xq = torch.zeros(T * act_bytes(fmt, cols) + 64, dtype=torch.uint8, device="cuda")
        self.y = torch.zeros(T, rows, device="cuda")
        self.w = resident(L, fmt, blocks, rows, cols) if fmt == "q6_k" else torch.cat([blocks.reshape(-1), torch.zeros(256, dtype=torch.uint8, device="cuda")])
        self.quantise = getattr(L, "ckb200_dev_quantize_" + ("q8_0" if fmt == "q8_0" else "q8_k"))
        self.multiply = getattr(L, {"q4_k": "ckb200_dev_gemm_nt_q4_k_q8_k", "q6_k": "ckb200_dev_gemm_nt_q6_k_planar_q8_k", "q8_0": "ckb200_dev_gemm_nt_q8_0_q8_0"}[fmt])

    def run(self):
        T, rows, cols = self.args
        ok(self.quantise(p(self.x), p(self.xq), T, cols, None))
        ok(self.multiply(p(self.xq), p(self.w), None, p(self.y), T, rows, cols, None))
        return {"y": self.y}


class Decode:
    def __init__(self, case, seed):
        self.model = Model(case, seed)
        self.ctx, self.steps, self.batch = case["ctx"], case["steps"], case["batch"]
        V = self.model.cfg["vocab_size"]
        self.ids = np.random.default_rng(seed).integers(0, V, (self.steps, self.batch)).astype(np.int32)
        self.logits = np.zeros((self.steps, self.batch, V), np.float32)

    def run(self):
        L, h = self.model.L, self.model.handle
        ok(L.ckb200_model_set_pos(h, self.ctx))
        for i in range(self.steps):
            ok(L.ckb200_model_decode(h, vptr(self.ids[i]), vptr(self.logits[i])))
        return {"logits": self.logits, "kv": self.model.kv[:, :, :, :, self.ctx:self.ctx + self.steps]}


class Prompt:
    def __init__(self, case, seed):
        self.model = Model(dict(case, batch=1), seed)
        self.ctx, self.tokens = case["ctx"], case["tokens"]
        V = self.model.cfg["vocab_size"]
        self.ids = np.random.default_rng(seed).integers(0, V, (self.tokens, 1)).astype(np.int32)
        self.logits = np.zeros((1, 1, V), np.float32)

    def run(self):
        L, h = self.model.L, self.model.handle
        # a conversation starts from an empty cache, a later turn behind what the earlier ones left
        ok(L.ckb200_model_reset(h) if self.ctx == 0 else L.ckb200_model_set_pos(h, self.ctx))
        ok(L.ckb200_model_prefill(h, vptr(self.ids), self.tokens, vptr(self.logits)))
        return {"logits": self.logits, "kv": self.model.kv[:, :, :, :, self.ctx:self.ctx + self.tokens]}


def stack_config(design, width, periods):
    heads, ff, q_rank = width // 128, {2048: 5632, 4096: 14336}[width], {2048: 768, 4096: 1536}[width]
    mlp = {"kind": "dense", "ff": ff}
    if design == "puzevik":
        delta = {"type": "channel_delta", "mlp": mlp, "mixer": {"heads": heads, "kv_heads": heads, "dim": 128, "vdim": 128, "conv": 4, "a_rank": 128, "g_rank": 128}}
        ret = {"type": "retention", "mlp": mlp, "mixer": {"heads": heads, "dim": 128, "vdim": 128, "decay": [1 - 2.0 ** (-5 - h % 8) for h in range(heads)], "rot": {"base": 1.0e6, "dims": 128}}}
        lat = {"type": "latent_attention", "mlp": mlp, "mixer": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": q_rank, "kv_rank": 512, "scale": 192 ** -0.5,
                                                                 "rot": {"base": 1.0e4, "dims": 64}}}
        return {"architecture": "Puzevik", "width": width, "vocab": STACK_VOCAB, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "layers": [delta, ret, lat, delta] * periods}
    mix = {"type": "wkv", "mlp": mlp, "mixer": {"heads": width // 64, "dim": 64, "a_rank": 64}}
    rot = {"base": 1.0e6, "dims": 64, "scaling": {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}}
    both = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": heads, "kv_heads": max(heads // 4, 1), "dim": 128, "vdim": 128, "mask": {"size": 1024}, "rot": rot, "scale": 128 ** -0.5}, "left_scale": 0.7,
        "right": {"heads": heads // 2, "dim": 128, "vdim": 128, "decay": [1 - 2.0 ** (-5 - h % 8) for h in range(heads // 2)]}, "right_scale": 0.7}}
    return {"architecture": "Sipadra", "width": width, "vocab": STACK_VOCAB, "norm": {"eps": 1e-6}, "logit_softcap": 30.0, "layers": [mix, mix, both, mix] * periods}


class Request:
    def __init__(self, case, seed):
        fd, path = tempfile.mkstemp(suffix=".json")
        try:
            with os.fdopen(fd, "w") as f:
                json.dump(stack_config(case["design"], case["width"], case["periods"]), f)
            self.session = api.Session(lib(), f"synthetic:{path}:{int(seed) & 0x7FFFFFFF}", 2304)
        finally:
            os.unlink(path)
        self.weight_bytes = lib().ckb200_model_weight_bytes(self.session.handle)
        rng = np.random.default_rng(seed)
        self.ids = rng.integers(0, STACK_VOCAB, case["tokens"]).astype(np.int32)
        self.more = rng.integers(0, STACK_VOCAB, case["steps"]).astype(np.int32)

    def run(self):
        self.session.reset()
        logits = [self.session.extend(self.ids, [len(self.ids) - 1])]
        for t in self.more:
            logits.append(self.session.extend([t], [0]))
        return {"logits": np.concatenate(logits)}

    def __del__(self):
        if hasattr(self, "session"):
            self.session.close()


KINDS = {"gemv": Gemv, "gemm": Gemm, "decode": Decode, "prompt": Prompt, "request": Request}


def prepare(case, seed):
    return KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind == "gemv":
        return {"bytes": matrix_bytes(case["fmt"], case["rows"], case["cols"]) + 4 * (case["rows"] + case["cols"]), "flops": 2 * case["rows"] * case["cols"]}
    if kind == "gemm":
        T, rows, cols = case["tokens"], case["rows"], case["cols"]
        return {"bytes": matrix_bytes(case["fmt"], rows, cols) + 4 * T * (rows + cols), "flops": 2 * T * rows * cols}
    if kind == "request":
        # weights of the layers and the output projection in 16 bits; a multiply-add per weight and token, the output projection for the tokens whose logits are read
        width, n = case["width"], 4 * case["periods"]
        ff = {2048: 5632, 4096: 14336}[width]
        per_layer = 3 * width * ff + (5 if case["design"] == "sipadra" else 4) * width * width
        head = STACK_VOCAB * width
        passes, tokens = 1 + case["steps"], case["tokens"] + case["steps"]
        return {"bytes": 2 * passes * (n * per_layer + head) + 4 * passes * STACK_VOCAB, "flops": 2 * (tokens * n * per_layer + passes * head)}
    cfg = model_cfg(case)
    every = list(matrices(cfg))
    head = every[-1]
    layer_params = sum(r * c for _, _, _, r, c in every[:-1])
    weight_bytes = sum(matrix_bytes(f, r, c) for _, _, f, r, c in every)
    row = cfg["num_layers"] * 2 * cfg["num_kv_heads"] * cfg["head_dim"] * (2 if case.get("kv_f16") else 4)      # cache bytes of a position
    attn = cfg["num_layers"] * 4 * cfg["num_heads"] * cfg["head_dim"]                                         # multiply-adds of a query and a key, twice
    if kind == "decode":
        n, B = case["steps"], case["batch"]
        keys = sum(case["ctx"] + i + 1 for i in range(n))
        return {"bytes": n * weight_bytes + B * keys * row + 4 * n * B * cfg["vocab_size"], "flops": 2 * n * B * (layer_params + head[3] * head[4]) + B * keys * attn}
    T = case["tokens"]
    return {"bytes": weight_bytes + (case["ctx"] + T) * row + 4 * cfg["vocab_size"],
            "flops": 2 * T * layer_params + 2 * head[3] * head[4] + attn * sum(case["ctx"] + i + 1 for i in range(T))}


def tolerance(case):
    """One product: sums of exact integers in 32-bit, 1e-7 from the 64-bit result.  Whole models round activations to 8 bits between the
    products; where the 32-bit sums before it differ in the last place some values go to the other side of a step, the next product spreads
    that over all its rows, and a few layers on two correct implementations round independently: they differ by what the rounding itself costs,
    about a hundredth.  Layer stacks round activations to bfloat16."""
    if case["kind"] in ("gemv", "gemm"):
        return {"rel": 5e-6}
    if case["kind"] == "request":
        return {"rel": 0.02}
    return {"rel": 0.03, "max": 0.5}


# ------------------------------------------------------------------ the same in 64 bits

def dequantise(fmt, blocks):
    """float64 [rows, columns] of uint8 [rows, blocks, bytes]."""
    rows, nb, _ = blocks.shape

    def half(at):
        return blocks[:, :, at:at + 2].contiguous().view(torch.float16).double()

    if fmt == "q8_0":
        return (half(0) * blocks[:, :, 2:].contiguous().view(torch.int8).double()).reshape(rows, -1)
    if fmt == "q5_0":
        bits = blocks[:, :, 2:6].contiguous().view(torch.int32)
        fifth = (bits >> torch.arange(32, device=blocks.device, dtype=torch.int32)) & 1
        nib = blocks[:, :, 6:22].to(torch.int32)
        return (half(0) * (torch.cat([nib & 15, nib >> 4], 2) + 16 * fifth - 16).double()).reshape(rows, -1)
    if fmt == "q6_k":
        ql = blocks[:, :, :128].to(torch.int16).view(rows, nb, 2, 64)
        qh = blocks[:, :, 128:192].to(torch.int16).view(rows, nb, 2, 32)
        lo, hi = ql[..., :32], ql[..., 32:]
        q = torch.stack([(lo & 15) | ((qh & 3) << 4), (hi & 15) | ((qh >> 2 & 3) << 4), (lo >> 4) | ((qh >> 4 & 3) << 4), (hi >> 4) | ((qh >> 6 & 3) << 4)], 3) - 32
        sc = blocks[:, :, 192:208].contiguous().view(torch.int8).double()
        return (half(208).unsqueeze(-1) * sc.unsqueeze(-1) * q.reshape(rows, nb, 16, 16).double()).reshape(rows, -1)
    s = blocks[:, :, 4:16].to(torch.int16)
    sc = torch.cat([s[:, :, 0:4] & 63, (s[:, :, 8:12] & 15) | (s[:, :, 0:4] >> 6 << 4)], 2).double()
    mn = torch.cat([s[:, :, 4:8] & 63, (s[:, :, 8:12] >> 4) | (s[:, :, 4:8] >> 6 << 4)], 2).double()
    qs = blocks[:, :, 16:].view(rows, nb, 4, 32)
    q = torch.stack([qs & 15, qs >> 4], 3).reshape(rows, nb, 8, 32).double()
    return ((half(0) * sc).unsqueeze(-1) * q - (half(2) * mn).unsqueeze(-1)).reshape(rows, -1)


def quantised(fmt, x):
    """The values that activations [n, cols] have after the path's own 8-bit rounding, which is defined in 32-bit arithmetic."""
    n, cols = x.shape
    x = x.float()
    if fmt in ("q8_0", "q5_0"):
        b = x.view(n, -1, 32)
        top = b.abs().amax(2, keepdim=True)
        q = torch.round(b * torch.where(top > 0, torch.full_like(top, 127.0) / top, 0.0))
        return (q.double() * (top / torch.full_like(top, 127.0)).to(torch.float16).double()).view(n, cols)
    b = x.view(n, -1, 256)
    pick = torch.gather(b, 2, b.abs().argmax(2, keepdim=True))
    scale = torch.where(pick != 0, torch.full_like(pick, -127.0) / pick, 0.0)
    q = torch.round(scale * b).clamp(-128, 127)
    return torch.where(pick != 0, q.double() * (1.0 / scale).double(), 0.0).view(n, cols)


def product(fmt, blocks, x):
    """float64 [n, rows]: rows of `x` (padded with zeros to the matrix) after their rounding, through the matrix."""
    cols = blocks.shape[1] * FORMATS[fmt][2]
    xq = quantised(fmt, torch.nn.functional.pad(x, (0, cols - x.shape[1])) if x.shape[1] < cols else x)
    step = max(256, (1 << 28) // cols)
    return torch.cat([xq @ dequantise(fmt, blocks[i:i + step]).t() for i in range(0, blocks.shape[0], step)], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "request":
        return None         # the weights exist only inside the library, which draws them on the device and has no way to read them back
    if kind in ("gemv", "gemm"):
        gen = generator(seed)
        blocks = make_blocks(case["fmt"], case["rows"], case["cols"], gen)
        x = torch.randn(case["tokens"], case["cols"], device="cuda", generator=gen) if kind == "gemm" else torch.randn(case["cols"], device="cuda", generator=gen).view(1, -1)
        y = product(case["fmt"], blocks, x)
        return {"y": y if kind == "gemm" else y[0]}
    state = prepare(case, seed)
    out = exact_model(state.model, case, torch.from_numpy(state.ids).cuda().long())
    return out


def exact_model(model, case, ids):
    cfg = model.cfg
    T, B = ids.shape
    D, H, G, d, F, eps = cfg["embed_dim"], cfg["num_heads"], cfg["num_kv_heads"], cfg["head_dim"], cfg["intermediate_size"], cfg["rms_eps"]
    ctx, f16 = case["ctx"], case.get("kv_f16", False)
    every = {(layer, which): (fmt, model.weights(layer, which, fmt, rows, cols)) for layer, which, fmt, rows, cols in matrices(cfg)}

    def norm(x, layer, which):
        g = model.weights(layer, which, None, 1, D).double()
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * g

    freq = cfg["rope_theta"] ** (-torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d)
    angle = torch.arange(ctx, ctx + T, device="cuda", dtype=torch.float64)[:, None] * freq
    cos, sin = angle.cos()[:, None, None], angle.sin()[:, None, None]

    def rotate(x):          # [T, B, heads, d]
        a, b = x[..., :d // 2], x[..., d // 2:]
        return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)

    fmt, table = every[-1, LM_HEAD]
    x = dequantise(fmt, table[ids.reshape(-1)])[:, :D]
    seen = torch.arange(ctx + T, device="cuda")[None, :] <= torch.arange(ctx, ctx + T, device="cuda")[:, None]
    new = []
    for layer in range(cfg["num_layers"]):
        h = norm(x, layer, LN1)
        q = rotate(product(*every[layer, WQ], h).view(T, B, H, d))
        k = rotate(product(*every[layer, WK], h).view(T, B, G, d))
        v = product(*every[layer, WV], h).view(T, B, G, d)
        kv = torch.stack([k, v]).permute(0, 2, 3, 1, 4)                         # [2, B, G, T, d]
        if f16:
            kv = kv.to(torch.float16).double()
        new.append(kv)
        a = torch.empty(T, B, H, d, device="cuda", dtype=torch.float64)
        for b in range(B):
            keys, values = torch.cat([model.kv[layer, :, b, :, :ctx].double(), kv[:, b]], 2)
            s = torch.einsum("tghd,gsd->ghts", q[:, b].view(T, G, H // G, d), keys) / math.sqrt(d)
            w = torch.softmax(s.masked_fill(~seen, -math.inf), -1)
            a[:, b] = torch.einsum("ghts,gsd->tghd", w, values).reshape(T, H, d)
        x = x + product(*every[layer, WO], a.reshape(T * B, H * d))
        gu = product(*every[layer, W1], norm(x, layer, LN2))
        x = x + product(*every[layer, W2], torch.nn.functional.silu(gu[:, :F]) * gu[:, F:])
    last = x.view(T, B, D) if case["kind"] == "decode" else x.view(T, B, D)[-1:]
    logits = product(*every[-1, LM_HEAD], norm(last.reshape(-1, D), -1, FINAL_GAMMA))
    return {"logits": logits.view(*last.shape[:2], -1), "kv": torch.stack(new)}
