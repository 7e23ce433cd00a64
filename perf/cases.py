"""The calls whose time this backend is judged by, over the ranges its users meet.

Four kinds of call, all through the public entry points of ``spy_b200.backend``:

``matmul``   one ``B200Backend.submit(MatMul)`` against an uploaded constant: the operator a Spy graph issues seven times per
             layer and once for the head.
``layer``    the operators of one decoder layer, submitted one after the other as the reference's scheduler walks its graph
             (RMSNorm, projections, RoPE, KV append into the strided caches, masked attention, SwiGLU FFN, residuals).
model calls  on a GGUF model that is loaded once and kept, as a server keeps it:
  ``reply``     a prompt through ``LlamaModel.eval`` and a greedy answer decoded on the device (``LlamaModel.decode``);
  ``generate``  the host-driven token loop, logits of every step back to the host (``LlamaModel.generate``);
  ``prompt``    a prompt alone (``LlamaModel.eval``);
  ``resume``    decoding at the end of a filled context, one of several conversations that take turns on a model
                (``LlamaModel.select_sequence`` and ``decode``);
  ``batch``     sequences decoded in lockstep (``LlamaModel.decode_batch``).

Widths are those of LLaMa2-7B and 13B, the architectures of this repository's configurations; models that only repeat a layer
are kept shorter than 32 or 40 blocks where the call's time is proportional to the depth. Weights are seeded N(0, 0.02),
prompts random token ids. Every result is required to be the same bits: the kernels follow the CPU backend's arithmetic
operation by operation, because the network re-quantizes its activations in front of every matrix and amplifies any
difference.
"""
import os
import tempfile
from collections import OrderedDict

import numpy as np
import torch

from spy_b200 import backend as B
from spy_b200 import gguf_io, quants

TYPES = {"q4_0": quants.Q4_0, "q8_0": quants.Q8_0, "q4_k": quants.Q4_K, "q6_k": quants.Q6_K}
BITS = {"q4_0": 18 * 8 / 32, "q8_0": 34 * 8 / 32, "q4_k": 144 * 8 / 256, "q6_k": 210 * 8 / 256, "f32": 32.0}
HEAD_DIM = 128
WEIGHT_SEED = 1234     # a model's weights are the file a user has; prompts come from the case's seed
SLOTS = 8              # conversations that take turns on a model of the "resume" kind


def _model(kind, name, wtype, n_layer, n_head, n_ff, n_ctx, n_vocab=32000, **more):
    return dict(kind=kind, name=name, wtype=wtype, n_layer=n_layer, n_head=n_head, n_ff=n_ff, n_vocab=n_vocab, n_ctx=n_ctx, **more)


def listed():
    return [
        # the smallest call: one activation column against an attention projection, where the launch weighs as much as the bytes
        dict(kind="matmul", name="matmul q8_0 5120x5120 b1", wtype="q8_0", rows=5120, k=5120, cols=1),
        # a few columns (a short prompt, a small batch) against an FFN matrix of a K-quant file
        dict(kind="matmul", name="matmul q4_k 11008x4096 b4", wtype="q4_k", rows=11008, k=4096, cols=4),
        # a batch of sixteen against the output head, the largest matrix of the model
        dict(kind="matmul", name="matmul q4_0 32000x4096 b16", wtype="q4_0", rows=32000, k=4096, cols=16),
        # the backend as a plain drop-in: Spy's scheduler submits a decode step operator by operator
        dict(kind="layer", name="layer ops q4_0 past 200", wtype="q4_0", n_head=32, n_ff=11008, tokens=1, past=200, n_ctx=512),
        # the headline workload: LLaMa2-7B Q4_0, 8 prompt ids, 32 greedy tokens, context 512
        _model("reply", "reply 7b q4_0 8+32", "q4_0", 32, 32, 11008, 512, prompt=8, steps=32),
        # the same model behind a host-side sampler: every step's logits come back; a prompt of odd length
        _model("generate", "generate 7b q4_0 21+12", "q4_0", 32, 32, 11008, 512, prompt=21, steps=12),
        # a full prompt before the first answer token
        _model("prompt", "prompt 7b q4_0 448", "q4_0", 32, 32, 11008, 512, prompt=448),
        # mixed K-quant files (Q6_K for attn_v, ffn_down and the head, Q4_K elsewhere): answer and prompt
        _model("reply", "reply q4_k_m 8+32", "q4_k_m", 8, 32, 11008, 1024, prompt=8, steps=32),
        _model("prompt", "prompt q4_k_m 512", "q4_k_m", 8, 32, 11008, 1024, prompt=512),
        # a document-sized prompt: attention over thousands of positions beside the matrices
        _model("prompt", "prompt q8_0 3968", "q8_0", 8, 32, 11008, 4096, prompt=3968),
        # a long conversation goes on: the KV cache is read with the weights at every token
        _model("resume", "resume q8_0 3968+32", "q8_0", 8, 32, 11008, 4096, prompt=3968, steps=32),
        # 13B widths, 32 requests decoded together
        _model("batch", "batch 13b q4_0 32 seq", "q4_0", 4, 40, 13824, 512, prompt=8, steps=16, n_seq=32),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "layer", "reply", "generate", "prompt", "prompt", "resume", "batch"])
    if kind == "matmul":
        wtype = rng.choice(["q4_0", "q8_0", "q4_k", "q6_k"])
        unit = 256 if wtype in ("q4_k", "q6_k") else 32
        return dict(kind=kind, wtype=wtype, rows=4 * _log(rng, 256, 8000), k=unit * _log(rng, 1536 // unit, 11264 // unit), cols=_log(rng, 1, 160))
    if kind == "layer":
        n_head = rng.randint(4, 40)
        n_ctx = 4 * rng.randint(32, 256)
        tokens = _log(rng, 1, 24)
        return dict(kind=kind, wtype=rng.choice(["q4_0", "q8_0"]), n_head=n_head, n_ff=32 * rng.randint(6 * n_head, 11 * n_head), tokens=tokens,
                    past=rng.randint(0, n_ctx - tokens), n_ctx=n_ctx)
    wtype = rng.choice(["q4_0", "q8_0", "q4_k_m"])
    n_head = 2 * rng.randint(2, 20)
    unit = 256 if wtype == "q4_k_m" else 32
    n_ff = unit * rng.randint(6 * n_head * 32 // unit, 11 * n_head * 32 // unit)
    shape = dict(kind=kind, wtype=wtype, n_layer=rng.randint(1, 5), n_head=n_head, n_ff=n_ff, n_vocab=4 * _log(rng, 500, 8000))
    if kind == "prompt":
        prompt = _log(rng, 9, 1600)
        return dict(shape, n_ctx=4 * (prompt // 4 + rng.randint(1, 300)), prompt=prompt)
    if kind == "resume":
        prompt, steps = _log(rng, 64, 3000), rng.randint(4, 24)
        return dict(shape, n_ctx=4 * ((prompt + steps) // 4 + rng.randint(1, 200)), prompt=prompt, steps=steps)
    prompt, steps = _log(rng, 1, 60), rng.randint(4, 24)
    n_ctx = 4 * ((prompt + steps) // 4 + rng.randint(1, 300))
    if kind == "batch":
        return dict(shape, n_ctx=n_ctx, prompt=prompt, steps=steps, n_seq=_log(rng, 2, 40))
    return dict(shape, n_ctx=n_ctx, prompt=prompt, steps=steps)


# ---------------------------------------------------------------------------------------------- models and files
def _scratch_dir():
    return "/dev/shm" if os.path.isdir("/dev/shm") and os.access("/dev/shm", os.W_OK) else None


class _Gguf:
    """A synthetic GGUF file of this architecture, unlinked while it is open: it is gone with the object or the process."""

    def __init__(self, cfg, seed):
        fd, path = tempfile.mkstemp(suffix=".gguf", dir=_scratch_dir())
        os.close(fd)
        try:
            gguf_io.make_llama_gguf_cuda(path, cfg, seed=seed)
            self.fd = os.open(path, os.O_RDONLY)
        finally:
            os.unlink(path)
        torch.cuda.empty_cache()
        self.path = f"/proc/self/fd/{self.fd}"

    def tensors(self):
        return {name: (ne, wtype, np.array(raw)) for name, (ne, wtype, raw) in gguf_io.read_gguf(self.path)[1].items()}

    def __del__(self):
        if hasattr(self, "fd"):
            os.close(self.fd)


def _config(case):
    mixed = case["wtype"] == "q4_k_m"
    return gguf_io.LlamaConfig(
        n_layer=case["n_layer"], d_model=HEAD_DIM * case["n_head"], n_head=case["n_head"], n_ff=case["n_ff"], n_vocab=case["n_vocab"],
        wtype=quants.Q4_K if mixed else TYPES[case["wtype"]],
        embd_type=quants.Q4_K if mixed else quants.Q8_0,
        overrides={"attn_v": quants.Q6_K, "ffn_down": quants.Q6_K, "output": quants.Q6_K} if mixed else {})


class _Session:
    """A backend and the model it serves; the model goes before its backend."""

    model = None

    def __init__(self, file, n_ctx, n_seq=0):
        self.backend = B.B200Backend(0)
        self.model = B.LlamaModel(self.backend, file.path, n_ctx=n_ctx)
        if n_seq:
            self.model.set_sequences(n_seq)
        self.free_slots = list(range(n_seq))

    def __del__(self):
        if self.model is not None:
            self.model.close()
            self.backend.close()


_MOST_KEPT = 6
_kept = OrderedDict()          # models that several states share and the file that batch states load theirs from; the least recently used goes first


def _keep(key, make):
    if key in _kept:
        _kept.move_to_end(key)
    else:
        while len(_kept) >= _MOST_KEPT:
            _kept.popitem(last=False)
        _kept[key] = make()
    return _kept[key]


def _shape(case):
    return tuple(case[k] for k in ("wtype", "n_layer", "n_head", "n_ff", "n_vocab"))


def _session(case, n_seq=0):
    return _keep(_shape(case) + (case["n_ctx"], n_seq), lambda: _Session(_Gguf(_config(case), WEIGHT_SEED), case["n_ctx"], n_seq))


def _file(case):
    return _keep(_shape(case), lambda: _Gguf(_config(case), WEIGHT_SEED))


# ---------------------------------------------------------------------------------------------- states
class _Matmul:
    def __init__(self, case, seed):
        rows, k, cols = case["rows"], case["k"], case["cols"]
        wtype = TYPES[case["wtype"]]
        w = _Gguf(gguf_io.LlamaConfig(n_layer=0, d_model=k, n_head=1, n_vocab=rows, wtype=wtype, embd_type=wtype), seed).tensors()["output.weight"][2]
        self.backend = B.B200Backend(0)
        weight = self.backend.upload_constant("output.weight", w, wtype, (k, rows))
        gen = torch.Generator(device="cuda").manual_seed(seed)
        self.x = torch.randn((cols, k), generator=gen, device="cuda")
        self.out = torch.empty((cols, rows), device="cuda")
        d = B.OpDesc()
        d.op_type, d.num_input = B.OP["MatMul"], 2
        d.input[0] = B.make_tensor(weight, wtype, (k, rows), None, B.NODE_CONSTANT)
        d.input[1] = B.make_tensor(self.x.data_ptr(), B.FP32, (k, cols))
        d.output = B.make_tensor(self.out.data_ptr(), B.FP32, (rows, cols))
        self.desc = d

    def run(self):
        self.backend.submit(self.desc)
        return self.out


class _Layer:
    """One decoder layer as the reference's graph lists its operators, every operand in device memory except the token
    positions and the causal mask, which Spy keeps in host vectors."""

    def __init__(self, case, seed):
        h, ff, t, past, n_ctx = case["n_head"], case["n_ff"], case["tokens"], case["past"], case["n_ctx"]
        d, n_kv = h * HEAD_DIM, past + t
        wtype = TYPES[case["wtype"]]
        tensors = _Gguf(gguf_io.LlamaConfig(n_layer=1, d_model=d, n_head=h, n_ff=ff, n_vocab=32, wtype=wtype), seed).tensors()
        be = self.backend = B.B200Backend(0)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        self.x = torch.randn((t, d), generator=gen, device="cuda")
        self.k_cache = torch.randn((n_ctx, d), generator=gen, device="cuda").half()
        self.v_cache = torch.randn((d, n_ctx), generator=gen, device="cuda").half()
        self.k_cache[past:] = 0
        self.v_cache[:, past:] = 0
        self.positions = np.arange(past, n_kv, dtype=np.int32)
        self.mask = np.where(np.arange(n_ctx)[None, :] <= self.positions[:, None], np.float32(0), np.float32(-np.inf)).astype(np.float32)
        self.buffers, self.descs = [], []

        def weight(name):
            ne, number_type, raw = tensors[name]
            return B.make_tensor(be.upload_constant(name, raw, number_type, ne), number_type, ne, None, B.NODE_CONSTANT)

        def buffer(*ne):
            b = torch.empty(tuple(reversed(ne)), device="cuda")
            self.buffers.append(b)
            return B.make_tensor(b.data_ptr(), B.FP32, ne)

        def op(name, inputs, output):
            o = B.OpDesc()
            o.op_type, o.num_input, o.output = B.OP[name], len(inputs), output
            for i, x in enumerate(inputs):
                o.input[i] = x
            o.norm_eps, o.softmax_scale = 1e-5, float(np.float32(1.0) / np.sqrt(np.float32(HEAD_DIM)))
            if name == "Rope":
                r = o.rope
                r.mode, r.num_past, r.num_dim, r.num_context, r.num_origin_context = 0, past, HEAD_DIM, n_ctx, n_ctx
                r.freq_base, r.freq_scale, r.extend_factor, r.attention_factor = 10000.0, 1.0, 0.0, 1.0
            self.descs.append(o)
            return output

        def view(tensor, ne, nb, offset=0):
            return B.make_tensor(tensor.data + offset, tensor.number_type, ne, nb, tensor.node_type)

        p = "blk.0."
        x = B.make_tensor(self.x.data_ptr(), B.FP32, (d, t))
        kc = B.make_tensor(self.k_cache.data_ptr(), B.FP16, (n_ctx * d,), None, B.NODE_CACHE)
        vc = B.make_tensor(self.v_cache.data_ptr(), B.FP16, (n_ctx * d,), None, B.NODE_CACHE)
        pos = B.make_tensor(self.positions.ctypes.data, B.INT32, (t,), None, B.NODE_IO)
        mask = B.make_tensor(self.mask.ctypes.data, B.FP32, (n_ctx, t), None, B.NODE_IO)

        def normed(v, norm):
            return op("Mul", [op("NormRMS", [v], buffer(d, t)), weight(p + norm)], buffer(d, t))

        xn = normed(x, "attn_norm.weight")
        q = op("MatMul", [weight(p + "attn_q.weight"), xn], buffer(d, t))
        k = op("MatMul", [weight(p + "attn_k.weight"), xn], buffer(d, t))
        v = op("MatMul", [weight(p + "attn_v.weight"), xn], buffer(d, t))
        heads = (HEAD_DIM, h, t)
        q = op("Rope", [view(q, heads, (4, 4 * HEAD_DIM, 4 * d)), pos], buffer(*heads))
        k = op("Rope", [view(k, heads, (4, 4 * HEAD_DIM, 4 * d)), pos], buffer(*heads))
        op("Copy", [k, view(kc, (d * t,), (2, 2 * d * t), 2 * d * past)], B.make_tensor(None, B.FP16, (d * t,)))
        op("Copy", [view(v, (t, d), (4 * d, 4)), view(vc, (t, d), (2, 2 * n_ctx), 2 * past)], B.make_tensor(None, B.FP16, (t, d)))
        scores = op("MatMul", [view(kc, (HEAD_DIM, n_kv, h), (2, 2 * d, 2 * HEAD_DIM)), view(q, (HEAD_DIM, t, h), (4, 4 * d, 4 * HEAD_DIM))], buffer(n_kv, t, h))
        probs = op("Softmax", [scores, mask], buffer(n_kv, t, h))
        att = op("MatMul", [view(vc, (n_kv, HEAD_DIM, h), (2, 2 * n_ctx, 2 * HEAD_DIM * n_ctx)), probs], buffer(HEAD_DIM, t, h))
        att = op("Contiguous", [view(att, heads, (4, 4 * HEAD_DIM * t, 4 * HEAD_DIM))], buffer(d, t))
        x = op("Add", [op("MatMul", [weight(p + "attn_output.weight"), att], buffer(d, t)), x], buffer(d, t))
        xn = normed(x, "ffn_norm.weight")
        up = op("MatMul", [weight(p + "ffn_up.weight"), xn], buffer(ff, t))
        gate = op("MatMul", [weight(p + "ffn_gate.weight"), xn], buffer(ff, t))
        act = op("Mul", [up, op("Silu", [gate], buffer(ff, t))], buffer(ff, t))
        op("Add", [op("MatMul", [weight(p + "ffn_down.weight"), act], buffer(d, t)), x], buffer(d, t))
        self.out = self.buffers[-1]

    def run(self):
        submit = self.backend.submit
        for o in self.descs:
            submit(o)
        return {"x": self.out, "k_cache": self.k_cache, "v_cache": self.v_cache}


def _ids(case, seed, n, salt=0):
    return np.random.default_rng((int(seed), salt)).integers(3, case["n_vocab"], size=n).astype(np.int32)


class _Prompt:
    def __init__(self, case, seed):
        self.session = _session(case)
        self.ids = _ids(case, seed, case["prompt"])

    def run(self):
        return self.session.model.eval(self.ids, 0)


class _Reply(_Prompt):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        self.steps = case["steps"]

    def run(self):
        logits = self.session.model.eval(self.ids, 0)
        ids, _ = self.session.model.decode(int(np.argmax(logits)), len(self.ids), self.steps)
        return {"logits": logits, "ids": ids}


class _Generate(_Reply):
    def run(self):
        ids, logits = self.session.model.generate(self.ids, self.steps)
        return {"logits": logits, "ids": ids}


class _Resume:
    """A conversation with its context in one of the model's KV caches."""

    slot = None

    def __init__(self, case, seed):
        self.session = _session(case, SLOTS)
        self.slot = self.session.free_slots.pop()
        self.past, self.steps = case["prompt"], case["steps"]
        model = self.session.model
        model.select_sequence(self.slot)
        self.first = int(np.argmax(model.eval(_ids(case, seed, self.past), 0)))

    def __del__(self):
        if self.slot is not None:
            self.session.free_slots.append(self.slot)

    def run(self):
        model = self.session.model
        model.select_sequence(self.slot)
        return model.decode(self.first, self.past, self.steps)[0]


class _Batch:
    def __init__(self, case, seed):
        self.session = _Session(_file(case), case["n_ctx"], case["n_seq"])
        self.past, self.steps = case["prompt"], case["steps"]
        model, self.first = self.session.model, []
        for c in range(case["n_seq"]):
            model.select_sequence(c)
            self.first.append(int(np.argmax(model.eval(_ids(case, seed, self.past, 1 + c), 0))))

    def run(self):
        return self.session.model.decode_batch(self.first, self.past, self.steps)[0]


_KINDS = {"matmul": _Matmul, "layer": _Layer, "prompt": _Prompt, "reply": _Reply, "generate": _Generate, "resume": _Resume, "batch": _Batch}


def prepare(case, seed):
    return _KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _layer_weights(d, ff):
    return 4 * d * d + 3 * d * ff


def _sequence_work(case, tokens, first, passes):
    """`tokens` tokens of one sequence, at positions `first` on, in `passes` passes over the weights that give a row of logits each."""
    d, ff, layers = HEAD_DIM * case["n_head"], case["n_ff"], case["n_layer"]
    if case["wtype"] == "q4_k_m":
        layer_bits, head_bits = (3 * d * d + 2 * d * ff) * BITS["q4_k"] + (d * d + d * ff) * BITS["q6_k"], BITS["q6_k"]
    else:
        layer_bits, head_bits = _layer_weights(d, ff) * BITS[case["wtype"]], BITS[case["wtype"]]
    weights = passes * (layers * layer_bits + d * case["n_vocab"] * head_bits) / 8
    pairs = tokens * first + tokens * (tokens + 1) // 2                    # (query, key) pairs
    rows_read = pairs if passes == tokens else first + tokens              # a pass reads the cache rows it sees once
    own = layers * (rows_read + tokens) * 4 * d + 4 * case["n_vocab"] * passes
    return {"bytes": weights + own, "own": own, "flops": 2 * tokens * layers * _layer_weights(d, ff) + layers * pairs * 4 * d + 2 * passes * d * case["n_vocab"]}


def work(case):
    kind = case["kind"]
    if kind == "matmul":
        rows, k, cols = case["rows"], case["k"], case["cols"]
        return {"bytes": rows * k * BITS[case["wtype"]] / 8 + 4 * cols * (rows + k), "flops": 2 * rows * k * cols}
    if kind == "layer":
        d, t, past = HEAD_DIM * case["n_head"], case["tokens"], case["past"]
        pairs, weights = t * past + t * (t + 1) // 2, _layer_weights(d, case["n_ff"])
        return {"bytes": weights * BITS[case["wtype"]] / 8 + (past + 2 * t) * 4 * d + 8 * t * d, "flops": 2 * t * weights + pairs * 4 * d}
    parts = []
    if kind in ("prompt", "reply", "generate"):
        parts.append(_sequence_work(case, case["prompt"], 0, 1))
    if kind != "prompt":
        steps = case["steps"] - (kind == "generate")                       # generate() takes its first token from the prompt's logits
        parts.append(_sequence_work(case, steps, case["prompt"], steps))
    if kind == "batch":                                                    # the sequences share a step's weights, not their caches and logits
        one, n = parts.pop(), case["n_seq"]
        parts.append({"bytes": one["bytes"] + (n - 1) * one["own"], "flops": n * one["flops"]})
    return {m: sum(p[m] for p in parts) for m in ("bytes", "flops")}


def tolerance(case):
    return "exact"
