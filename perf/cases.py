"""What this framework is asked to do, as calls that can be timed and checked.

Four kinds of work, all through public entry points:

  linear        one quantized Linear on device buffers at decode sizes (`cmlb200_gemv`, 1 to 32 rows of activations), through
                `layers` weights of the same shape in turn, as a decode step goes from layer to layer: with enough of them the
                weights come from memory and not from the L2 cache
  prompt        the same Linear at prompt sizes (`cmlb200_gemm_bf16`, 33 rows and more)
  llama_decode  a LLaMA from a GGUF file, `batch` sequences behind `context` cached tokens: `steps` batched decode steps whose logits
                come back (`cml_llama_forward_batch`), then back to the context (`cml_llama_truncate`)
  llama_prompt  a prompt of a new sequence (`cml_llama_prefill_sequence`) and the logits behind its last token
  layered       a model folder (config.json, safetensors) through the step function: `batch` new sequences, their prompts as one
                step, `steps` decode steps with logits, and the sequences closed

Weights are random with the quantized formats' own value ranges; models have the layer sizes of the 7B model (or the layered
models' 2048) and fewer layers."""
import ctypes
import math
import random
import shutil
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import __graft_entry__ as entry  # noqa: E402

pkg = entry.load_package()
synth = entry.load_synth()
lib = pkg.lib

TYPES = {"q4_0": 2, "q4_1": 3, "q8_0": 7, "q4_k": 12, "q5_k": 13, "q6_k": 14, "nf4": 100}
BLOCK_BYTES = {"q4_0": (32, 18), "q4_1": (32, 20), "q8_0": (32, 34), "q4_k": (256, 144), "q5_k": (256, 176), "q6_k": (256, 210)}
NF4_BLOCK = 64
NORM_EPS = 1e-5
ROPE_BASE = 10000.0
WINDOW = 1024

LLAMA_7B = {"hidden": 4096, "inter": 11008, "heads": 32, "kv_heads": 32, "layers": 4, "vocab": 32000}
LAYERED = {"width": 2048, "ff": 5632, "heads": 16, "kv_heads": 4, "layers": 4, "vocab": 32000}


def listed():
    return [
        # The smallest calls: small projections for one token, a matter of latency and launches.
        {"name": "linear q8_0 4096x4096 m1", "kind": "linear", "type": "q8_0", "rows": 4096, "cols": 4096, "m": 1, "layers": 2},
        # The headline: the 7B feed-forward's up projection for one token, weights from memory.
        {"name": "linear q4_0 11008x4096 m1", "kind": "linear", "type": "q4_0", "rows": 11008, "cols": 4096, "m": 1, "layers": 4},
        # The same with a full batch of decoded tokens.
        {"name": "linear q4_0 11008x4096 m32", "kind": "linear", "type": "q4_0", "rows": 11008, "cols": 4096, "m": 32, "layers": 4},
        # The down projection in the format most GGUF files come in, one token.
        {"name": "linear q4_k 4096x11008 m1", "kind": "linear", "type": "q4_k", "rows": 4096, "cols": 11008, "m": 1, "layers": 4},
        # The vocabulary projection of such files, a ragged batch.
        {"name": "linear q6_k 32000x4096 m7", "kind": "linear", "type": "q6_k", "rows": 32000, "cols": 4096, "m": 7, "layers": 1},
        # A QLoRA base weight, a small batch.
        {"name": "linear nf4 4096x4096 m4", "kind": "linear", "type": "nf4", "rows": 4096, "cols": 4096, "m": 4, "layers": 8},
        # A short ragged prompt over a QLoRA base weight.
        {"name": "prompt nf4 4096x4096 m77", "kind": "prompt", "type": "nf4", "rows": 4096, "cols": 4096, "m": 77, "layers": 8},
        # A long prompt through the feed-forward's up projection.
        {"name": "prompt q4_0 11008x4096 m2048", "kind": "prompt", "type": "q4_0", "rows": 11008, "cols": 4096, "m": 2048, "layers": 2},
        # One user's decode steps behind a conversation.
        {"name": "llama decode b1", "kind": "llama_decode", "type": "q4_0", **LLAMA_7B, "batch": 1, "context": 600, "steps": 8},
        # A prompt of 512 tokens.
        {"name": "llama prompt 512", "kind": "llama_prompt", "type": "q4_0", **LLAMA_7B, "prompt": 512},
        # Eight short requests decoded together by a dense bf16 model.
        {"name": "layered decode b8", "kind": "layered", **LAYERED, "batch": 8, "prompt": 48, "steps": 16},
        # A long prompt of such a model, longer than its attention window.
        {"name": "layered prompt 2000", "kind": "layered", **LAYERED, "batch": 1, "prompt": 2000, "steps": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear"] * 6 + ["prompt"] * 3 + ["llama_decode"] * 2 + ["llama_prompt"] * 2 + ["layered"] * 2)
    if kind in ("linear", "prompt"):
        type_ = rng.choice(["q4_0", "q4_0", "q8_0", "q4_k", "q6_k", "q5_k", "q4_1", "nf4"] if kind == "linear" else ["q4_0", "nf4", "q8_0"])
        rows = _log(rng, 512, 32000)
        if rng.random() < 0.7:
            rows = rows // 64 * 64                           # most models' sizes; the others are a shard's or a vocabulary's
        step = 256 if type_ in ("q4_k", "q5_k", "q6_k") or rng.random() < 0.7 else 32 if type_ != "nf4" else 64
        cols = max(step, _log(rng, 1024, 14336) // step * step)
        while rows * cols > 32000 * 4096:
            rows = max(512, rows // 2 // 64 * 64)
        m = _log(rng, 1, 32) if kind == "linear" else _log(rng, 33, 2048)
        layers = max(1, min(8, 100_000_000 // (rows * cols)))
        return {"kind": kind, "type": type_, "rows": rows, "cols": cols, "m": m, "layers": layers}
    if kind == "layered":
        if rng.random() < 0.5:
            return {"kind": kind, **LAYERED, "batch": _log(rng, 1, 32), "prompt": _log(rng, 4, 64), "steps": rng.randint(8, 16)}
        return {"kind": kind, **LAYERED, "batch": rng.randint(1, 3), "prompt": _log(rng, 65, 660), "steps": 1}
    size = dict(LLAMA_7B, layers=rng.randint(2, 4))
    if rng.random() < 0.4:                                   # heads that share keys and values
        size.update(kv_heads=8)
    type_ = rng.choice(["q4_0", "q4_0", "q8_0", "q4_k"])
    if kind == "llama_decode":
        return {"kind": kind, "type": type_, **size, "batch": _log(rng, 1, 16), "context": _log(rng, 16, 1500), "steps": 8}
    return {"kind": kind, "type": type_, **size, "prompt": _log(rng, 33, 512 if type_ != "q4_k" else 128)}


# ---- what a user has in hand -----------------------------------------------------------------------------------------
class Weight:
    """A quantized weight on the device, laid out once as a loader does it."""

    def __init__(self, type_, rows, cols, m, rng):
        t = TYPES[type_]
        tiles, block = None, 32
        if type_ == "nf4":
            qs, scales = synth.nf4_weight(rng, rows, cols, NF4_BLOCK)
            block = NF4_BLOCK
        else:
            blocks = weight_blocks(rng, type_, rows, cols)
            if type_ in ("q4_0", "q8_0"):
                qs, scales = pkg.repack_gguf(t, blocks, rows, cols)
                if type_ == "q8_0" and 4 < m <= 32 and cols % 128 == 0:      # as the LLaMA loader does for batches
                    tiles = torch.from_numpy(pkg.repack_tiles(t, blocks, rows, cols)).cuda()
            else:
                qs, scales, block = blocks, None, BLOCK_BYTES[type_][0]
        self.tiles = tiles
        self.qs = torch.from_numpy(np.ascontiguousarray(qs)).cuda()
        self.scales = None if scales is None else torch.from_numpy(np.ascontiguousarray(scales)).cuda()
        self.q = pkg.QMat(t, rows, cols, block, self.qs.data_ptr(), None if scales is None else self.scales.data_ptr(), 0,
                          None if tiles is None else tiles.data_ptr())


def weight_blocks(rng, type_, rows, cols):
    if type_ == "q4_0":
        return synth.q4_0_blocks(rng, rows, cols)
    if type_ == "q8_0":
        return synth.q8_0_blocks(rng, rows, cols)
    return synth.gguf_blocks(rng, TYPES[type_], rows, cols, 0.05 if type_ == "q6_k" else 0.02)     # scales that are normal halves


def activations(case, seed):
    rng = np.random.default_rng([seed, 1])
    return rng.standard_normal((case["m"], case["cols"]), dtype=np.float32)


class Linear:
    def __init__(self, case, seed):
        rng = np.random.default_rng([seed, 2])
        prompt = case["kind"] == "prompt"
        self.weights = [Weight(case["type"], case["rows"], case["cols"], case["m"], rng) for _ in range(case["layers"])]
        self.m = case["m"]
        self.x = torch.from_numpy(activations(case, seed)).cuda()
        if prompt:
            self.x = self.x.to(torch.bfloat16)
        self.y = [torch.empty(case["m"], case["rows"], dtype=torch.bfloat16 if prompt else torch.float32, device="cuda") for _ in self.weights]
        self.call = lib.cmlb200_gemm_bf16 if prompt else lib.cmlb200_gemv
        self.stream = torch.cuda.current_stream().cuda_stream

    def run(self):
        x = self.x.data_ptr()
        for w, y in zip(self.weights, self.y):
            pkg.check(self.call(w.q, x, y.data_ptr(), self.m, self.stream), "linear")
        return self.y


def llama_tensors(case):
    """(name, dims, type id, bytes) of every tensor of the model's file; all layers hold the same values."""
    rng = np.random.default_rng(7)
    H, inter, V = case["hidden"], case["inter"], case["vocab"]
    kv = H // case["heads"] * case["kv_heads"]
    t = TYPES[case["type"]]

    def norm():
        return (1 + 0.05 * rng.standard_normal(H)).astype(np.float16).tobytes()

    def weight(rows, cols):
        b = synth.gguf_blocks(rng, t, rows, cols)
        if case["type"] == "q4_0":                           # a model's weights have no mean: nibbles of 0 become 8
            q = b.reshape(-1, 18)[:, 2:]
            q += (q & 15 == 0).astype(np.uint8) * 8 + (q >> 4 == 0).astype(np.uint8) * 128
        return b.tobytes()

    embed = ((rng.random((V, H), dtype=np.float32) - 0.5) * 1.7).astype(np.float16).tobytes()
    layer = [("attn_norm", (H,), 1, norm()), ("attn_q", (H, H), t, weight(H, H)), ("attn_k", (H, kv), t, weight(kv, H)),
             ("attn_v", (H, kv), t, weight(kv, H)), ("attn_output", (H, H), t, weight(H, H)), ("ffn_norm", (H,), 1, norm()),
             ("ffn_gate", (H, inter), t, weight(inter, H)), ("ffn_up", (H, inter), t, weight(inter, H)), ("ffn_down", (inter, H), t, weight(H, inter))]
    out = [("token_embd.weight", (H, V), 1, embed)]
    for i in range(case["layers"]):
        out += [(f"blk.{i}.{name}.weight", dims, ty, raw) for name, dims, ty, raw in layer]
    return out + [("output_norm.weight", (H,), 1, norm()), ("output.weight", (H, V), t, weight(V, H))]


def layered_config(case):
    layer = synth.layered_layer(case["heads"], case["kv_heads"], 128, 128, WINDOW, case["ff"])
    return synth.layered_config(case["vocab"], case["width"], [layer] * case["layers"], NORM_EPS)


def layered_weights(case):
    """Name -> values of one layer's tensors (all layers alike), the embedding and the head."""
    rng = np.random.default_rng(8)
    made = {}

    def weight(name, shape):
        key = name.split(".", 1)[1] if name[0] == "l" else name
        if key not in made:
            if len(shape) == 1:
                a = 1 + 0.2 * rng.standard_normal(shape, dtype=np.float32)
            else:
                a = (rng.random(shape, dtype=np.float32) - 0.5) * (3.4 if name == "embed" else 3.4 / math.sqrt(shape[1]))
            made[key] = torch.from_numpy(a).to(torch.bfloat16).float().numpy()
        return made[key]
    return weight


_model_file = {}          # what the model is -> its file or folder; one at a time


def model_file(case):
    keys = ("kind", "type", "hidden", "inter", "heads", "kv_heads", "layers", "vocab", "width", "ff")
    key = tuple((k, str(case.get(k)).replace("llama_prompt", "llama_decode")) for k in keys)
    if key not in _model_file:
        for old in _model_file.values():
            shutil.rmtree(old, ignore_errors=True)
        _model_file.clear()
        folder = Path(tempfile.mkdtemp(prefix="model_"))
        if case["kind"] == "layered":
            synth.write_layered(folder, layered_config(case), layered_weights(case), alias_layers=True)
        else:
            synth.write_gguf(folder / "model.gguf", llama_tensors(case))
        _model_file[key] = folder
    return _model_file[key]


def tokens_of(case, seed):
    """Prompt (or context) and decoded tokens of every sequence: [batch][n], [steps][batch]."""
    rng = np.random.default_rng([seed, 3])
    batch, steps = case.get("batch", 1), case.get("steps", 1)
    if case["kind"] == "layered" and batch > 1:              # requests are never of one length
        sizes = [max(1, int(case["prompt"] * f)) for f in rng.uniform(0.6, 1.0, batch)]
    else:
        sizes = [case.get("prompt", case.get("context"))] * batch
    prompts = [rng.integers(0, case["vocab"], n).astype(np.int32) for n in sizes]
    return prompts, rng.integers(0, case["vocab"], (steps, batch)).astype(np.int32)


class Llama:
    def __init__(self, case, seed):
        self.case = case
        self.prompts, self.decoded = tokens_of(case, seed)
        c = pkg.LlamaConfig(case["vocab"], case["hidden"], case["inter"], case["layers"], case["heads"], case["kv_heads"], 2048, ROPE_BASE, NORM_EPS, 1, 0)
        self.model = lib.cml_llama_create(ctypes.byref(c))
        pkg.check(lib.cml_llama_set_options(self.model, 0, case.get("batch", 1)), "options")
        pkg.check(lib.cml_llama_load_gguf(self.model, str(model_file(case) / "model.gguf").encode()), "load")
        if case["kind"] == "llama_decode":
            for i, p in enumerate(self.prompts):
                pkg.check(lib.cml_llama_prefill_sequence(self.model, i, pkg.np_ptr(p), len(p)), "prefill")

    def __del__(self):
        lib.cml_llama_free(self.model)

    def logits(self, tokens):
        t = lib.cml_llama_forward_batch(self.model, pkg.np_ptr(tokens), len(tokens))
        if not t:
            raise pkg.CmlB200Error("cml_llama_forward_batch failed")
        return pkg.tensor_to_numpy(t)

    def run(self):
        if self.case["kind"] == "llama_prompt":
            p = self.prompts[0]
            lib.cml_llama_reset(self.model)
            pkg.check(lib.cml_llama_prefill_sequence(self.model, 0, pkg.np_ptr(p), len(p) - 1), "prefill")
            return self.logits(p[-1:])
        for i, p in enumerate(self.prompts):
            pkg.check(lib.cml_llama_truncate(self.model, i, len(p)), "truncate")
        return [self.logits(t) for t in self.decoded]


class Layered:
    def __init__(self, case, seed):
        self.prompts, self.decoded = tokens_of(case, seed)
        rows = sum(len(p) for p in self.prompts)
        room = sum((len(p) + len(self.decoded) + 31) // 16 * 16 for p in self.prompts)
        self.model = pkg.LanguageModel(model_file(case), max_tokens=room, max_sequences=len(self.prompts), max_step_rows=rows)

    def __del__(self):
        if hasattr(self, "model"):
            self.model.close()

    def run(self):
        m = self.model
        seqs = [m.open() for _ in self.prompts]
        m.step([(s, p, []) for s, p in zip(seqs, self.prompts)])
        out = [np.concatenate(m.step([(s, t[i:i + 1], None) for i, s in enumerate(seqs)])) for t in self.decoded]
        for s in seqs:
            m.end(s)
        return out


def prepare(case, seed):
    if case["kind"] in ("linear", "prompt"):
        return Linear(case, seed)
    return Layered(case, seed) if case["kind"] == "layered" else Llama(case, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def weight_bytes(type_, n):
    if type_ == "nf4":
        return n / 2 + n / NF4_BLOCK * 4
    if type_ == "bf16":
        return 2 * n
    elements, size = BLOCK_BYTES[type_]
    return n / elements * size


def work(case):
    if case["kind"] in ("linear", "prompt"):
        n, m, each = case["rows"] * case["cols"], case["m"], 2 if case["kind"] == "prompt" else 4
        return {"bytes": case["layers"] * (weight_bytes(case["type"], n) + each * m * (case["rows"] + case["cols"])), "flops": 2.0 * case["layers"] * m * n}
    if case["kind"] == "layered":
        width, ff, type_ = case["width"], case["ff"], "bf16"
        q, kv = case["heads"] * 128, case["kv_heads"] * 128
        prompts, decoded = tokens_of(case, 0)
        sizes, steps = [len(p) for p in prompts], len(decoded)
        window = WINDOW
    else:
        width, ff, type_ = case["hidden"], case["inter"], case["type"]
        q, kv = width, width // case["heads"] * case["kv_heads"]
        batch = case.get("batch", 1)
        decode = case["kind"] == "llama_decode"
        sizes, steps = ([case["context"]] * batch, case["steps"]) if decode else ([case["prompt"] - 1], 1)
        window = 1 << 30
    per = 2 * width * q + 2 * width * kv + 3 * width * ff
    head = width * case["vocab"]
    B = len(sizes)
    with_prompt = case["kind"] != "llama_decode"
    rows = (sum(sizes) if with_prompt else 0) + B * steps
    passes = steps + (1 if with_prompt else 0)                # the weights are read once a step
    seen = [min(n + t + 1, window) for n in sizes for t in range(steps)]          # keys of decoded tokens
    pairs = sum(seen) + (sum(min(i + 1, window) for n in sizes for i in range(n)) if with_prompt else 0)
    cache = case["layers"] * 2 * kv * 2
    return {"bytes": passes * case["layers"] * weight_bytes(type_, per) + steps * weight_bytes(type_, head) + cache * (sum(seen) + rows) + 4 * B * steps * case["vocab"],
            "flops": 2.0 * rows * case["layers"] * per + 2.0 * B * steps * head + 4.0 * case["layers"] * q * pairs}


# ---- how far another correct implementation may be -------------------------------------------------------------------------
def tolerance(case):
    # Linear: 32-bit sums. Prompts: bf16 operands and results. Models: caches in 16 bits, prompts in bf16.
    if case["kind"] == "linear":
        return {"rel": 2e-6, "max": 2e-5}
    if case["kind"] == "prompt":
        return {"rel": 1e-2, "max": 6e-2}
    return {"rel": 2e-2, "max": 2e-1}


# ---- the same in 64 bits, in plain torch -------------------------------------------------------------------------------------
# C-ML's table: the published NF4 values to four digits.
NF4_TABLE = [-1.0, -0.6962, -0.5251, -0.3949, -0.2844, -0.1848, -0.0911, 0.0, 0.0796, 0.1609, 0.2461, 0.3379, 0.4407, 0.5626, 0.7230, 1.0]


def _halves(b):
    return b.contiguous().view(torch.float16).double()


def _interleaved(parts):
    return torch.stack(parts, -1).flatten(-2)


def dequantized(type_, blocks, rows, cols):
    """The weight that GGUF blocks (file order) stand for, fp64 [rows, cols] on the GPU."""
    elements, size = BLOCK_BYTES[type_]
    b = torch.from_numpy(np.frombuffer(blocks, np.uint8).reshape(-1, size).copy()).cuda()
    n = len(b)
    if type_ == "q8_0":
        w = b[:, 2:].view(torch.int8).double() * _halves(b[:, :2])
    elif type_ in ("q4_0", "q4_1"):
        q = b[:, size - 16:]
        q = torch.cat([q & 15, q >> 4], 1).double()
        w = (q - 8) * _halves(b[:, :2]) if type_ == "q4_0" else q * _halves(b[:, :2]) + _halves(b[:, 2:4])
    elif type_ == "q6_k":
        low = _interleaved([b[:, :128] & 15, b[:, :128] >> 4])
        high = _interleaved([(b[:, 128:192] >> s) & 3 for s in (0, 2, 4, 6)])
        scale = b[:, 192:208].contiguous().view(torch.int8).double().repeat_interleave(16, 1)
        w = _halves(b[:, 208:210]) * scale * ((low | (high << 4)).double() - 32)
    else:
        s = b[:, 4:16]
        scale = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | ((s[:, :4] >> 6) << 4)], 1).double()
        least = torch.cat([s[:, 4:8] & 63, (s[:, 8:] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1).double()
        q = b[:, size - 128:].reshape(n, 8, 16)
        q = torch.cat([q & 15, q >> 4], 2)
        if type_ == "q5_k":
            q = q | (_interleaved([(b[:, 16:48] >> i) & 1 for i in range(8)]).reshape(n, 8, 32) << 4)
        w = q.double() * (_halves(b[:, :2]) * scale)[:, :, None] - (_halves(b[:, 2:4]) * least)[:, :, None]
    return w.reshape(rows, cols)


def exact_linear(case, seed):
    rng = np.random.default_rng([seed, 2])
    x = torch.from_numpy(activations(case, seed)).cuda()
    x = (x.to(torch.bfloat16) if case["kind"] == "prompt" else x).double()
    out = []
    for _ in range(case["layers"]):
        if case["type"] == "nf4":
            packed, scales = (torch.from_numpy(a).cuda() for a in synth.nf4_weight(rng, case["rows"], case["cols"], NF4_BLOCK))
            w = torch.tensor(NF4_TABLE, dtype=torch.float64, device="cuda")[_interleaved([packed >> 4, packed & 15]).long()]
            w = (w.reshape(-1, NF4_BLOCK) * scales.double()[:, None]).reshape(case["rows"], case["cols"])
        else:
            w = dequantized(case["type"], weight_blocks(rng, case["type"], case["rows"], case["cols"]), case["rows"], case["cols"])
        out.append(x @ w.T)
    return out


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + NORM_EPS) * w


def _heads(x, n):
    return x.reshape(len(x), n, -1).transpose(0, 1)


def exact_llama(case, seed):
    w = {}
    for name, dims, t, raw in llama_tensors(case):
        if name in w or (name.startswith("blk.") and not name.startswith("blk.0.")):
            continue
        if t == 1:
            w[name] = torch.from_numpy(np.frombuffer(raw, np.float16).copy()).cuda().double().reshape(dims[::-1])
        else:
            w[name] = dequantized(case["type"], raw, dims[1], dims[0])
    prompts, decoded = tokens_of(case, seed)
    if case["kind"] == "llama_prompt":
        prompts, decoded = [prompts[0][:-1]], prompts[0][-1:].reshape(1, 1)
    H, heads, kv, steps = case["hidden"], case["heads"], case["kv_heads"], len(decoded)
    dim = H // heads
    out = torch.empty(steps, len(prompts), case["vocab"], dtype=torch.float64, device="cuda")
    for i, p in enumerate(prompts):
        tokens = torch.from_numpy(np.concatenate([p, decoded[:, i]])).cuda().long()
        n = len(tokens)
        angle = torch.arange(n, device="cuda").double()[:, None] * (ROPE_BASE ** (-torch.arange(0, dim, 2, device="cuda").double() / dim))
        cos, sin = angle.cos(), angle.sin()

        def rotated(x):
            a, b = x[..., 0::2], x[..., 1::2]
            return _interleaved([a * cos - b * sin, a * sin + b * cos])
        mask = torch.ones(n, n, device="cuda", dtype=torch.bool).tril()
        x = w["token_embd.weight"][tokens]
        for _ in range(case["layers"]):
            def at(name):
                return w[f"blk.0.{name}.weight"]
            h = _rms(x, at("attn_norm"))
            q, k = rotated(_heads(h @ at("attn_q").T, heads)), rotated(_heads(h @ at("attn_k").T, kv))
            v = _heads(h @ at("attn_v").T, kv)
            k, v = k.repeat_interleave(heads // kv, 0), v.repeat_interleave(heads // kv, 0)
            s = (q @ k.transpose(1, 2) / math.sqrt(dim)).masked_fill(~mask, -math.inf).softmax(-1)
            x = x + (s @ v).transpose(0, 1).reshape(n, H) @ at("attn_output").T
            h = _rms(x, at("ffn_norm"))
            x = x + (torch.nn.functional.silu(h @ at("ffn_gate").T) * (h @ at("ffn_up").T)) @ at("ffn_down").T
        out[:, i] = _rms(x[-steps:], w["output_norm.weight"]) @ w["output.weight"].T
    return out[0] if case["kind"] == "llama_prompt" else list(out)


def exact_layered(case, seed):
    cfg, weight = layered_config(case), layered_weights(case)
    w = {}
    for name, shape in synth.layered_shapes(cfg).items():
        key = name.split(".", 1)[1] if name.startswith("l0.") else name
        if not name.startswith("l") or name.startswith("l0."):
            w[key] = torch.from_numpy(weight(name, shape)).cuda().double()
    mixer = cfg["layers"][0]["mixer"]
    heads, kv, width = case["heads"], case["kv_heads"], case["width"]
    slopes = 2.0 ** (-8.0 * torch.arange(1, heads + 1, device="cuda").double() / heads)
    prompts, decoded = tokens_of(case, seed)
    steps = len(decoded)
    out = torch.empty(steps, len(prompts), case["vocab"], dtype=torch.float64, device="cuda")
    for i, p in enumerate(prompts):
        tokens = torch.from_numpy(np.concatenate([p, decoded[:, i]])).cuda().long()
        n = len(tokens)
        pos = torch.arange(n, device="cuda").double()
        at = torch.arange(width, device="cuda")
        angle = pos[:, None] * 10000.0 ** (-(2.0 * (at // 2).double()) / width)
        x = w["embed"][tokens] + torch.where(at % 2 == 0, angle.sin(), angle.cos())
        far = pos[:, None] - pos[None, :]
        hidden = (far < 0) | (far >= WINDOW)
        warmth = 1 + mixer["q_temp"]["coef"] * torch.log(torch.floor((pos + 1) / mixer["q_temp"]["every"]) + 1)
        for _ in range(case["layers"]):
            h = _rms(x, w["norm1"])
            q = _heads(_rms(h @ w["mix.q"].T, w["mix.q.norm"]) * warmth[:, None], heads)
            k, v = _heads(_rms(h @ w["mix.k"].T, w["mix.k.norm"]), kv), _heads(h @ w["mix.v"].T, kv)
            k, v = k.repeat_interleave(heads // kv, 0), v.repeat_interleave(heads // kv, 0)
            s = (q @ k.transpose(1, 2) * mixer["scale"] - slopes[:, None, None] * far).masked_fill(hidden, -math.inf)
            most = s.amax(-1, keepdim=True).clamp(min=0)
            e = torch.exp(s - most)
            o = (e / (torch.exp(-most) + e.sum(-1, keepdim=True))) @ v
            o = o.transpose(0, 1) * torch.sigmoid(h @ w["mix.g"].T)[:, :, None]
            x = x + _rms(o.reshape(n, -1) @ w["mix.o"].T, w["norm1b"])
            h = _rms(x, w["norm2"])
            x = x + _rms((torch.nn.functional.gelu(h @ w["mlp.gate"].T, approximate="tanh") * (h @ w["mlp.up"].T)) @ w["mlp.down"].T, w["norm2b"])
        out[:, i] = _rms(x[-steps:], w["final.norm"]) @ w["head"].T
    return list(out)


def exact(case, seed):
    if case["kind"] in ("linear", "prompt"):
        return exact_linear(case, seed)
    return exact_layered(case, seed) if case["kind"] == "layered" else exact_llama(case, seed)


if __name__ == "__main__":
    for c in listed() + [draw(random.Random(i)) for i in range(6)]:
        print(c, work(c), tolerance(c))
