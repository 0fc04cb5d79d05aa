"""The work a user of this framework has it do, as cases that can be timed and compared.

Two families, both through the public entry points:

* "model": a model is loaded once and kept (weights, KV cache, a conversation already in the
  cache), and a pass is what a host program does with it: one decode step whose logits come back
  to the host, a greedy run on the device, or the evaluation of a prompt in chunks of 64 tokens;
* "product": one weight matrix on the device and fresh f32 activations: a pass quantizes the
  activations as the weight type asks for and multiplies (a single row in decoding, up to 64 rows
  in a prompt chunk).

The shapes are those of the benchmark configurations: the TinyLlama shape, the Qwen3-8B shape,
and the matrix shapes of the quant-type sweep.
"""
from __future__ import annotations

import functools

import numpy as np
import torch

import __graft_entry__ as graft

CHUNK = 64        # tokens per prompt batch, the reference's batch size
N_CTX = 2048
KINDS = {"f32": 0, "f16": 1, "bf16": 2, "q4_0": 3, "q5_0": 4, "q8_0": 5, "q4_k": 6, "q5_k": 7, "q6_k": 8}

# dim, hidden, layers, query heads, KV heads, head_dim, vocab, RoPE base, per-head q/k norm + NEOX RoPE
SHAPES = {
    "tinyllama": (2048, 5632, 22, 32, 4, 64, 32000, 1e4, False),
    "qwen3-8b": (4096, 12288, 36, 32, 8, 128, 151936, 1e6, True),
}


def listed():
    return [
        # ffn_up of the TinyLlama shape for one token: the smallest call of all, a few microseconds of launches
        dict(name="matvec q4_k 5632x2048", family="product", kind="q4_k", rows=5632, cols=2048, m=1),
        # an unquantized output head for one token: the largest matrix, bound by memory
        dict(name="matvec f16 128256x4096", family="product", kind="f16", rows=128256, cols=4096, m=1),
        # FFN matrices of an 8B model against a full prompt chunk
        dict(name="matmul q8_0 14336x4096 m64", family="product", kind="q8_0", rows=14336, cols=4096, m=64),
        dict(name="matmul q6_k 4096x14336 m64", family="product", kind="q6_k", rows=4096, cols=14336, m=64),
        # the last, ragged chunk of a prompt on an unquantized attention matrix
        dict(name="matmul bf16 4096x4096 m37", family="product", kind="bf16", rows=4096, cols=4096, m=37),
        # a sampling program: one token in, the logits out to the host
        dict(name="decode tinyllama q4_k_m", family="model", shape="tinyllama", mix="q4_k_m", what="forward", pos=160, n=1),
        # greedy decoding near the end of the context, where attention grows
        dict(name="greedy tinyllama long", family="model", shape="tinyllama", mix="q4_k_m", what="generate", pos=1700, n=16),
        # greedy decoding of the other common quantization
        dict(name="greedy tinyllama q4_0", family="model", shape="tinyllama", mix="q4_0", what="generate", pos=160, n=16),
        # greedy decoding of a large model after a 545-token conversation
        dict(name="greedy qwen3-8b", family="model", shape="qwen3-8b", mix="q4_k_m", what="generate", pos=545, n=16),
        # a long prompt from scratch, in whole chunks
        dict(name="prompt tinyllama 512", family="model", shape="tinyllama", mix="q4_k_m", what="prompt", pos=0, n=512),
        # a short chat turn appended to a conversation
        dict(name="turn tinyllama 7", family="model", shape="tinyllama", mix="q4_k_m", what="prompt", pos=300, n=7),
        # a prompt of a large model that does not fill its last chunk
        dict(name="prompt qwen3-8b 201", family="model", shape="qwen3-8b", mix="q4_k_m", what="prompt", pos=0, n=201),
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    if rng.random() < 0.5:
        kind = rng.choice(["q4_0", "q5_0", "q8_0", "q4_k", "q5_k", "q6_k", "f16", "bf16"])
        m = 1 if rng.random() < 0.4 else _log_int(rng, 2, 64)
        rows = _log_int(rng, 256, 32768)
        if rng.random() < 0.75:  # most matrices have rows in whole tiles; vocabularies and fused slices may not
            rows = max(256, rows // 64 * 64)
        return dict(family="product", kind=kind, rows=rows, cols=256 * _log_int(rng, 1, 56), m=m)
    shape = rng.choice(["tinyllama", "tinyllama", "qwen3-8b"])
    mix = "q4_k_m" if shape == "qwen3-8b" else rng.choice(["q4_k_m", "q4_k_m", "q4_0", "q8_0"])
    what = rng.choice(["forward", "generate", "prompt", "prompt"])
    if what == "prompt":
        n = _log_int(rng, 2, 201 if shape == "qwen3-8b" else 512)
        pos = 0 if rng.random() < 0.5 else _log_int(rng, 16, 1500)
    else:
        n = 1 if what == "forward" else _log_int(rng, 2, 10)
        pos = _log_int(rng, 16, 2000)
    return dict(family="model", shape=shape, mix=mix, what=what, pos=pos, n=n)


# ---- weights ---------------------------------------------------------------------------------------
def _f16_bytes(x):
    return x.to(torch.float16).view(torch.uint8).view(-1, 2)


def _random_rows(kind, rows, cols, std, gen):
    """`rows` x `cols` weights of about standard deviation `std` as the raw bytes of a GGUF tensor:
    quants uniform, block scales within a factor of two of each other."""
    dev = gen.device
    if kind in ("f32", "f16", "bf16"):
        dt = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[kind]
        out = torch.empty(rows * cols, dtype=dt, device=dev)
        step = 1 << 26
        for i in range(0, out.numel(), step):
            n = min(step, out.numel() - i)
            out[i:i + n] = (torch.randn(n, generator=gen, device=dev) * std).to(dt)
        return out.view(torch.uint8)
    size, per = {"q4_0": (18, 32), "q5_0": (22, 32), "q8_0": (34, 32), "q4_k": (144, 256), "q5_k": (176, 256), "q6_k": (210, 256)}[kind]
    n = rows * cols // per
    b = torch.randint(0, 256, (n, size), dtype=torch.uint8, generator=gen, device=dev)
    # what one unit of the block scale is worth, by the spread of uniform quants (and sub-block scales)
    unit = {"q4_0": 4.6, "q5_0": 9.2, "q8_0": 73.9, "q4_k": 258.0, "q5_k": 520.0, "q6_k": 684.0}[kind]
    d = (std / unit) * (0.7 + 0.6 * torch.rand(n, generator=gen, device=dev))
    if kind == "q6_k":
        b[:, 192:208] = (b[:, 192:208].to(torch.int16) // 2 - 64).to(torch.int8).view(torch.uint8)
        b[:, 208:210] = _f16_bytes(d)
    else:
        b[:, 0:2] = _f16_bytes(d)
        if kind in ("q4_k", "q5_k"):
            b[:, 2:4] = _f16_bytes(d * (7.5 if kind == "q4_k" else 15.5))
    return b.view(-1)


def _kind_of(mix, layer, tensor):
    """Which type each matrix of a file has: the usual K mix, or one type with a Q6_K output head."""
    if tensor == "output":
        return "q6_k"
    if mix == "q4_k_m":
        return "q6_k" if tensor in ("wv", "down") and layer % 2 == 0 else "q4_k"
    return mix


# ---- what a program keeps ----------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _context():
    return graft.import_package().Context(torch.cuda.current_device())


class _View:
    """A device buffer of the library for torch.as_tensor, without a copy."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}


class _Model:
    """A loaded model: its weights are uploaded once; its cache holds the rows of a conversation."""

    def __init__(self, shape, mix):
        pkg = graft.import_package()
        L = pkg.lib
        dim, hidden, n_layer, n_head, n_kv, hd, vocab, base, qwen = SHAPES[shape]
        qd, kvd = n_head * hd, n_kv * hd
        gen = torch.Generator(device="cuda").manual_seed(0x5EED)
        parts, off = [], 0

        def add(kind, rows, cols, std, mean=0.0):
            nonlocal off
            if kind == "f32":
                raw = (mean + std * torch.randn(rows * cols, generator=gen, device="cuda")).view(torch.uint8)
            else:
                raw = _random_rows(kind, rows, cols, std, gen)
            t = L.Tensor(kind=KINDS[kind], present=1, off=off, len=raw.numel(), rows=rows, cols=cols)
            parts.append((off, raw.cpu().numpy()))
            off = -(-(off + raw.numel()) // 32) * 32
            return t

        def matrix(layer, tensor, rows, cols):
            return add(_kind_of(mix, layer, tensor), rows, cols, cols ** -0.5)

        embd = add("q4_k" if mix == "q4_k_m" else mix, vocab, dim, 1.0)
        layers = []
        for i in range(n_layer):
            y = L.Layer()
            y.attn_norm, y.ffn_norm = add("f32", 1, dim, 0.2, 1.0), add("f32", 1, dim, 0.2, 1.0)
            y.wq, y.wk, y.wv = matrix(i, "wq", qd, dim), matrix(i, "wk", kvd, dim), matrix(i, "wv", kvd, dim)
            y.wo = matrix(i, "wo", dim, qd)
            y.gate, y.up, y.down = matrix(i, "gate", hidden, dim), matrix(i, "up", hidden, dim), matrix(i, "down", dim, hidden)
            if qwen:
                y.q_norm, y.k_norm = add("f32", 1, hd, 0.2, 1.0), add("f32", 1, hd, 0.2, 1.0)
            layers.append(y)
        norm, out = add("f32", 1, dim, 0.2, 1.0), matrix(-1, "output", vocab, dim)
        dims = L.Dims(dim=dim, hidden=hidden, n_layer=n_layer, n_head=n_head, n_kv_head=n_kv, head_dim=hd, rot_dim=hd, vocab=vocab,
                      n_ctx_train=N_CTX, eps=1e-6 if qwen else 1e-5, rope_base=base, rope_scale=1.0, rope_base_local=1e4,
                      rope_scale_local=1.0, qk_norm=int(qwen), rope_neox=int(qwen))
        weights = np.empty(off, dtype=np.uint8)
        for at, raw in parts:
            weights[at:at + raw.size] = raw
        head = L.ModelHead(dims=dims, token_embd=embd, output_norm=norm, output=out)
        self.gpu = pkg.Gpu(_context(), head, layers, weights, N_CTX, CHUNK)
        self.vocab = vocab
        self.cache = [torch.as_tensor(_View(self.gpu.buf_ptr(b), (n_layer, N_CTX, kvd)), device="cuda") for b in ("KCache", "VCache")]
        self.at = None

    def converse(self, pos):
        """Positions [0, pos) of one long conversation in the cache."""
        if self.at != pos:
            toks = np.random.default_rng(7).integers(0, self.vocab, N_CTX).astype(np.uint32)
            _evaluate(self.gpu, toks[:pos], 0, False)
            self.at = pos


@functools.lru_cache(maxsize=1)
def _model(shape, mix):
    return _Model(shape, mix)


def _evaluate(gpu, tokens, pos, want_logits):
    """A prompt in chunks, with logits for its last token only."""
    n = len(tokens)
    for a in range(0, n, CHUNK):
        b = min(a + CHUNK, n)
        if b - a == 1:
            gpu.forward(int(tokens[a]), pos + a, want_logits and b == n)
        else:
            gpu.forward_batch(tokens[a:b], pos + a, want_logits and b == n)


# ---- the interface -----------------------------------------------------------------------------------
def prepare(case, seed):
    if case["family"] == "model":
        m = _model(case["shape"], case["mix"])
        m.converse(case["pos"])
        toks = np.random.default_rng(seed).integers(0, m.vocab, case["n"]).astype(np.uint32)
        rows = [c[:, case["pos"]:case["pos"] + case["n"]] for c in m.cache]
        return dict(what=case["what"], gpu=m.gpu, model=m, pos=case["pos"], n=case["n"], tokens=toks, rows=rows)
    kind, rows, cols, m = KINDS[case["kind"]], case["rows"], case["cols"], case["m"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    raw = _random_rows(case["kind"], rows, cols, cols ** -0.5, gen)
    w = torch.zeros(raw.numel() + 256, dtype=torch.uint8, device="cuda")  # the entry points may read past the last row
    w[:raw.numel()] = raw
    del raw
    x = torch.randn(m, cols, generator=gen, device="cuda")
    act = graft.import_package().lib.activation(kind)
    blocks = {"q8_k": cols // 256 * 292, "q8_0": cols // 32 * 36, "f32": 0}[act]
    xq = torch.empty(m * blocks, dtype=torch.uint8, device="cuda")
    out = torch.empty(m, rows, device="cuda")
    torch.cuda.synchronize()  # the library works on a stream of its own
    return dict(what="product", ctx=_context(), kind=kind, act=act, rows=rows, cols=cols, m=m, w=w, x=x, xq=xq, out=out, pw=w.data_ptr(),
                px=x.data_ptr(), pq=xq.data_ptr(), po=out.data_ptr(), bx=_Ptr(x.data_ptr()), bq=_Ptr(xq.data_ptr()))


class _Ptr:
    """A device pointer where the quantizers take a buffer."""

    def __init__(self, ptr):
        self.ptr = ptr


def run(s):
    what = s["what"]
    if what == "product":
        ctx, xs = s["ctx"], s["px"]
        if s["act"] == "q8_k":
            ctx.quantize_q8_k(s["bx"], s["m"] * s["cols"], s["bq"])
            xs = s["pq"]
        elif s["act"] == "q8_0":
            ctx.quantize_q8_0(s["bx"], s["m"] * s["cols"], s["bq"])
            xs = s["pq"]
        if s["m"] == 1:
            ctx.matvec(s["kind"], s["po"], s["pw"], xs, s["rows"], s["cols"])
        else:
            ctx.matmul(s["kind"], s["po"], s["pw"], xs, s["m"], s["rows"], s["cols"])
        return {"out": s["out"], "activations": s["xq"]}
    g = s["gpu"]
    if what == "generate":
        ids, _ = g.generate(int(s["tokens"][0]), s["pos"], s["n"])
        return {"ids": ids, "rows": s["rows"]}
    if what == "forward":
        g.forward(int(s["tokens"][0]), s["pos"], True)
    else:
        _evaluate(g, s["tokens"], s["pos"], True)
    return {"logits": g.logits(), "rows": s["rows"]}


_ROW = {"f32": 4.0, "f16": 2.0, "bf16": 2.0, "q4_0": 18 / 32, "q5_0": 22 / 32, "q8_0": 34 / 32, "q4_k": 144 / 256, "q5_k": 176 / 256, "q6_k": 210 / 256}


def work(case):
    if case["family"] == "product":
        rows, cols, m = case["rows"], case["cols"], case["m"]
        return {"bytes": rows * cols * _ROW[case["kind"]] + 4 * m * (rows + cols), "flops": 2.0 * m * rows * cols}
    dim, hidden, n_layer, n_head, n_kv, hd, vocab, _, _ = SHAPES[case["shape"]]
    qd, kvd, pos, n, mix = n_head * hd, n_kv * hd, case["pos"], case["n"], case["mix"]
    per, weights = 0.0, 0.0
    for i in range(n_layer):
        for t, r, c in (("wq", qd, dim), ("wk", kvd, dim), ("wv", kvd, dim), ("wo", dim, qd), ("gate", hidden, dim), ("up", hidden, dim), ("down", dim, hidden)):
            weights += r * c
            per += r * c * _ROW[_kind_of(mix, i, t)]
    head = vocab * dim
    attn = sum(4.0 * qd * (pos + i + 1) for i in range(n)) * n_layer  # q.k and p.v
    if case["what"] == "prompt":  # weights once a chunk, cached rows once a chunk
        starts = range(0, n, CHUNK)
        kv = sum(2.0 * 4 * kvd * n_layer * (pos + min(a + CHUNK, n)) for a in starts)
        return {"bytes": per * len(starts) + head * _ROW["q6_k"] + kv, "flops": 2.0 * weights * n + 2.0 * head + attn}
    kv = sum(2.0 * 4 * kvd * n_layer * (pos + i + 1) for i in range(n))
    return {"bytes": n * (per + head * _ROW["q6_k"]) + kv, "flops": n * 2.0 * (weights + head) + attn}


def tolerance(case):
    """The framework's results are bit-identical to its CPU oracle for every path: integer block
    sums are exact and every f32 operation has its place in a fixed order."""
    return "exact"
