"""Workloads whose time is followed from change to change, run through the engine's public calls.

    decode    the next tokens of a batch of sequences: `Engine.run_io` once per token, faces in, tokens out
    prefill   a prompt whose ids lie on the device: `gehtp_cuda_run_dev`, logits of every position left on the device
    delta     one gated delta-rule layer over a sequence
    session   a request to a model served through row-count runlists: the prompt, then tokens one by one (`Session.feed`)

A case is a dict of plain values; `prepare` makes its inputs from a seed, `run` is one pass, `exact` states in 64 bits what
the pass computes. The engine is one per process, so the weights and the cached context of a case belong to a handle that
every prepared input of that case shares, as the requests to one served model do.
"""
import ctypes

import numpy as np
import torch

import gehtp_b200
from gehtp_b200 import runlists
from gehtp_b200.checkpoint import ArrayTensors
from gehtp_b200.registry import SHAPES, Model
from gehtp_b200.session import Session
from gehtp_b200.wtop import OP, Engine

SMALL, LARGE = "qwen3-0.6b-shape", "qwen3-4b-shape"
DESIGN_SIZES = {1024: (3072, 16), 2560: (9728, 32)}      # width -> feed-forward, heads
DESIGN_VOCAB = 32768
CONV_TAPS, CHUNK, DELTA_HEADS, DELTA_DIM, DELTA_HIDDEN, DELTA_CHANNELS = 4, 64, 16, 128, 1024, 4096


def _decode(name, shape, layers, batch, context, steps, quant="w4"):
    return dict(name=name, kind="decode", shape=shape, layers=layers, batch=batch, context=context, steps=steps, quant=quant)


def _prefill(name, shape, layers, tokens, quant="w4"):
    return dict(name=name, kind="prefill", shape=shape, layers=layers, tokens=tokens, quant=quant)


def _session(name, design, width, prompt, steps, dtype="bfloat16"):
    return dict(name=name, kind="session", design=design, width=width, prompt=prompt, steps=steps, dtype=dtype)


def listed():
    return [
        # one user's chat with the small model: launches and latency
        _decode("decode-small-b1", SMALL, 28, 1, 4096, 8),
        # odd batch and context, weights as the emitter leaves them (fp16)
        _decode("decode-small-b3-f16", SMALL, 8, 3, 1001, 8, "f16"),
        # the serving batch of the benchmark, part of its layers with the whole vocabulary
        _decode("decode-large-b8", LARGE, 8, 8, 8192, 8),
        # a full batch over long contexts
        _decode("decode-large-b64", LARGE, 4, 64, 8192, 4),
        # an ordinary prompt of the small model, all layers
        _prefill("prefill-small-512", SMALL, 28, 512),
        # a prompt whose length is on no tile, fp16 weights
        _prefill("prefill-small-333-f16", SMALL, 8, 333, "f16"),
        # a long prompt of the large model
        _prefill("prefill-large-2048", LARGE, 4, 2048),
        # a linear-attention layer over a long sequence
        dict(name="delta-2048", kind="delta", tokens=2048),
        # latent attention and channel-decay delta rule: a long prompt; a short request answered token by token
        _session("ripidra-prompt-2048", "Ripidra", 1024, 2048, 0),
        _session("ripidra-answer", "Ripidra", 2560, 77, 24),
        # window attention and looped layers: a long prompt; a short request in fp32
        _session("supevik-prompt-2048", "Supevik", 2560, 2048, 0),
        _session("supevik-answer-f32", "Supevik", 1024, 150, 12, "float32"),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "session", "session", "session", "delta"])
    if kind == "decode":
        shape = rng.choice([SMALL, LARGE])
        quant = "f16" if shape == SMALL and rng.random() < 0.4 else "w4"
        layers = rng.randint(4, 8) if shape == LARGE or quant == "f16" else _log(rng, 4, 28)
        batch = _log(rng, 1, 64)
        context = _log(rng, 256, min(8192, 8192 * 256 // (batch * layers)))
        return dict(kind=kind, shape=shape, layers=layers, batch=batch, context=context, steps=rng.randint(4, 8), quant=quant)
    if kind == "prefill":
        shape = rng.choice([SMALL, LARGE])
        quant = "f16" if shape == SMALL and rng.random() < 0.4 else "w4"
        layers = rng.randint(2, 4) if shape == LARGE else rng.randint(4, 8) if quant == "f16" else _log(rng, 4, 28)
        return dict(kind=kind, shape=shape, layers=layers, tokens=_log(rng, 32, 2048 if layers <= 8 else 640), quant=quant)
    if kind == "delta":
        return dict(kind=kind, tokens=CHUNK * _log(rng, 2, 32))
    design, width = rng.choice(["Ripidra", "Supevik"]), rng.choice([1024, 2560])
    dtype = "float32" if width == 1024 and rng.random() < 0.3 else "bfloat16"
    prompt = _log(rng, 16, 300 if dtype == "float32" else 2000)
    return dict(kind=kind, design=design, width=width, prompt=prompt, steps=rng.choice([0, rng.randint(1, 24)]), dtype=dtype)


# ------------------------------------------------------------------------------------------------- handles
class _View:
    """Device memory of the engine as a torch tensor."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, data=(ptr, False), version=2)


class _Handle:
    """What a program keeps of a model: the engine with its weights, and the cached context where there is one."""
    key, now = None, None

    def __init__(self, case):
        self.lib = gehtp_b200.lib()
        getattr(self, "_" + case["kind"])(case)

    def temp(self, tid, shape, typestr="<f2"):
        return torch.as_tensor(_View(self.lib.gehtp_cuda_temp_dev(tid), shape, typestr), device="cuda")

    def run_dev(self, face, out_temp):
        if self.lib.gehtp_cuda_run_dev(ctypes.byref(self.engine.blob), face.data_ptr(), None, out_temp, self.err, 256) != 0:
            raise RuntimeError(self.err.value.decode())

    def _load(self, c, built):
        """The engine of a decoder's blob, with the case's weights in the place of the builder's."""
        blob, self.man = built
        self.engine = Engine(self.lib, blob)
        b, at = self.engine.blob, 0
        for i in range(b.n_ops):
            op = b.ops[i]
            if op.opcode not in (OP.MATMUL_W4A16, OP.MATMUL_F16) or not op.args[1] & 0x8000:
                continue
            bits = _slot_bits(_weight(c, at, op.args[4], op.args[5]), op.opcode)
            sl = b.slots[op.args[1] & 0x7FFF]
            if bits.size != sl.len:
                raise ValueError("weight %d: slot of %d bytes, %d made" % (at, sl.len, bits.size))
            first = b.weight_off + sl.offset
            self.engine.buf[first:first + sl.len] = bits
            at += 1

    def _decode(self, c):
        cfg = SHAPES[c["shape"]]
        self._load(c, runlists.build_decode_runlist(cfg, c["batch"], c["context"], quant=c["quant"], n_layers=c["layers"]))
        self.past = c["context"] - c["steps"]
        self.err = ctypes.create_string_buffer(256)
        elems = c["batch"] * cfg.kv_heads * cfg.head_dim
        for i in range(c["layers"]):
            ring = _ring(c, i)
            torch.cuda.synchronize()
            if self.lib.gehtp_cuda_state_load(ctypes.byref(self.engine.blob), i, ring.data_ptr(), ring.numel() * 2, 1, elems, self.past, self.err, 256):
                raise RuntimeError(self.err.value.decode())
        self.tokens = np.zeros(c["batch"], np.int32)
        self.engine.run_io(_faces(c, self.man, 0)[0], self.man["token_temp"], self.tokens)
        self.logits = self.temp(self.man["logits_temp"], (c["batch"], cfg.vocab))

    def _prefill(self, c):
        cfg = SHAPES[c["shape"]]
        self._load(c, runlists.build_prefill_runlist(cfg, c["tokens"], quant=c["quant"], n_layers=c["layers"]))
        self.err = ctypes.create_string_buffer(256)
        self.engine.run_io(np.zeros(c["tokens"], np.int32), self.man["hidden_temp"])
        self.logits = self.temp(self.man["logits_temp"], (c["tokens"], cfg.vocab))

    def _delta(self, c):
        blob, self.man = runlists.build_gdn_runlist(c["tokens"], DELTA_HIDDEN, DELTA_CHANNELS, CONV_TAPS, DELTA_HEADS, DELTA_DIM, CHUNK)
        self.engine, self.err = Engine(self.lib, blob), ctypes.create_string_buffer(256)
        self.engine.run_io(np.zeros(c["tokens"] * DELTA_HIDDEN, np.float16), self.man["conv_temp"])
        self.outputs = [self.temp(self.man["conv_temp"], (c["tokens"], DELTA_CHANNELS))]
        self.outputs += [self.temp(t, (CHUNK, DELTA_HIDDEN)) for t in self.man["chunk_out"]]

    def _session(self, c):
        cfg, tensors = _design(c)
        bits = {k: v.cpu().view(torch.int16).numpy().view(np.uint16) for k, v in tensors.items()}
        self.session = Session(Model(cfg, ArrayTensors(bits)), c["dtype"], max_tokens=max(2048, c["prompt"] + c["steps"]))
        self.engine = self.session.engine


def _handle(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _Handle.key != key:
        if _Handle.now is not None:
            _Handle.now.engine.shutdown()
        _Handle.key, _Handle.now = None, None
        _Handle.now, _Handle.key = _Handle(case), key
    return _Handle.now


# -------------------------------------------------------------------------------------------------- inputs
def _gen(*parts):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(np.random.default_rng([int(p) for p in parts]).integers(1 << 62)))
    return g


def _weight(c, at, K, N):
    """Projection `at` of a decoder (in the runlist's order), (q, scales) on the device: what quantising normal weights of
    deviation K^-1/2 in groups of 64 leaves - levels about 8 on both sides, scales around one size."""
    g = _gen(72, at, K, N)
    q = torch.empty(K, N, device="cuda", dtype=torch.uint8)
    for k in range(0, K, 512):
        q[k:k + 512] = (torch.randn(min(512, K - k), N, device="cuda", generator=g) * 2.6 + 8.0).round_().clamp_(0, 15).byte()
    return q, ((torch.rand(K // 64, N, device="cuda", generator=g) * 0.6 + 0.7) * (K ** -0.5 / 2.6)).half()


def _values(weight):
    """fp16((q - 8) scale), [K, N]."""
    q, sc = weight
    return torch.cat([((q[k:k + 64].float() - 8.0) * sc[k // 64].float()).half() for k in range(0, q.shape[0], 64)])


def _slot_bits(weight, opcode):
    q, sc = weight
    if opcode == OP.MATMUL_F16:
        return _values(weight).T.contiguous().view(torch.uint8).cpu().numpy().reshape(-1)
    nib = (q[:, 0::2] | q[:, 1::2] << 4).cpu().numpy().reshape(-1)
    return np.concatenate([nib, sc.view(torch.uint8).cpu().numpy().reshape(-1)])


def _ring(c, layer):
    """Cached keys and values ~ N(0, 1), [context][K face | V face]."""
    cfg = SHAPES[c["shape"]]
    return torch.randn(c["context"], 2, c["batch"], cfg.kv_heads, cfg.head_dim, device="cuda", dtype=torch.float16, generator=_gen(71, layer))


def _ids(c, seed):
    rng = np.random.default_rng([int(seed), 17])
    if c["kind"] == "decode":
        return rng.integers(0, SHAPES[c["shape"]].vocab, (c["steps"], c["batch"]))
    if c["kind"] == "prefill":
        return rng.integers(0, SHAPES[c["shape"]].vocab, c["tokens"]).astype(np.int32)
    return rng.integers(0, DESIGN_VOCAB, c["prompt"] + c["steps"])


def _faces(c, man, seed):
    cfg = SHAPES[c["shape"]]
    past = c["context"] - c["steps"]
    return [runlists.decode_face(man, ids, past + s, cfg.head_dim, cfg.rope_theta) for s, ids in enumerate(_ids(c, seed))]


def _hidden(c, seed):
    return torch.randn(c["tokens"], DELTA_HIDDEN, device="cuda", dtype=torch.float16, generator=_gen(seed, 18))


def _design(c):
    """(config.json, tensors in bf16 on the device) of a model of four layer runs, two of each mixer or window."""
    width, (ff, H), G = c["width"], DESIGN_SIZES[c["width"]], 8
    gen, t = _gen(c["width"], 19), {}

    def mat(name, *shape, scale=None):
        t[name] = (torch.randn(shape, device="cuda", generator=gen) * (shape[-1] ** -0.5 if scale is None else scale)).bfloat16()
    mat("embed", DESIGN_VOCAB, width, scale=1.0)
    if c["design"] == "Supevik":
        rot = dict(base=1e6, dims=128, scaling=dict(factor=4.0, fast=32.0, slow=1.0, original=2048))
        layers = [dict(type="attention", mlp=dict(kind="dense", ff=ff),
                       mixer=dict(heads=H, kv_heads=G, dim=128, vdim=128, mask=dict(size=n), rot=rot, scale=128 ** -0.5)) for n in (1024, 8192, 1024)]
        cfg = dict(architecture="Supevik", vocab=DESIGN_VOCAB, width=width, norm=dict(eps=1e-6), embedding=dict(scale=4.0), layers=layers,
                   loop=dict(start=1, stop=2, times=2))

        def norm(name):
            mat(name, width, scale=1.0)
            mat(name + ".b", width, scale=0.1)
            t[name + ".alpha"] = torch.full((1,), 0.5, device="cuda", dtype=torch.bfloat16)
        mat("head", DESIGN_VOCAB, width)
        mat("loop.in", width, 2 * width)
        norm("final.norm")
        for i in range(len(layers)):
            p, q = "l%d." % i, "l%d.mix." % i
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                norm(p + n)
            for n, r in (("q", H), ("k", G), ("v", G), ("g", H)):
                mat(q + n, r * 128, width)
                if n != "g":
                    mat(q + n + ".b", r * 128, scale=0.1)
            mat(q + "q.norm", 128, scale=1.0)
            mat(q + "k.norm", 128, scale=1.0)
            mat(q + "o", width, H * 128)
            mat(p + "mlp.gate", ff, width)
            mat(p + "mlp.up", ff, width)
            mat(p + "mlp.down", width, ff)
        return cfg, t
    lat = dict(heads=H, dim=128, rot_dim=64, vdim=128, kv_rank=512, rot=dict(base=1e6, dims=64), scale=192 ** -0.5)
    dlt = dict(heads=H, kv_heads=H, dim=128, vdim=128, conv=4)
    kinds = [("channel_delta", dlt), ("latent_attention", lat)] * 2
    cfg = dict(architecture="Ripidra", vocab=DESIGN_VOCAB, width=width, norm=dict(eps=1e-6),
               layers=[dict(type=k, mixer=m, mlp=dict(kind="dense", ff=ff)) for k, m in kinds])
    mat("final.norm", width, scale=0.1)
    for i, (k, _) in enumerate(kinds):
        p, q = "l%d." % i, "l%d.mix." % i
        mat(p + "norm1", width, scale=0.1)
        mat(p + "norm2", width, scale=0.1)
        mat(p + "mlp.up", ff, width)
        mat(p + "mlp.down", width, ff)
        mat(q + "o", width, H * 128)
        if k == "latent_attention":
            for n, r, w in (("q", H * 192, width), ("dkv", 576, width), ("uk", H * 128, 512), ("uv", H * 128, 512), ("g", H, width)):
                mat(q + n, r, w)
            mat(q + "dkv.norm", 512, scale=1.0)
            continue
        for n in "qkv":
            mat(q + n, H * 128, width)
            mat(q + n + ".conv", H * 128, 4, scale=0.5)
        for n, r, w in (("b", H, width), ("a1", 128, width), ("a2", H * 128, 128), ("g1", 128, width), ("g2", H * 128, 128)):
            mat(q + n, r, w)
        mat(q + "A_log", H, scale=0.5)
        mat(q + "norm", 128, scale=1.0)
        mat(q + "dt_bias", H * 128, scale=1.0)
    return cfg, t


def prepare(case, seed):
    h = _handle(case)
    s = dict(handle=h, kind=case["kind"])
    if case["kind"] == "decode":
        s["faces"], s["layers"] = _faces(case, h.man, seed), case["layers"]
    elif case["kind"] == "prefill":
        s["ids"] = torch.from_numpy(_ids(case, seed)).cuda()
    elif case["kind"] == "delta":
        s["hidden"] = _hidden(case, seed)
    else:
        ids = _ids(case, seed)
        s["prompt"], s["answer"] = ids[:case["prompt"]], ids[case["prompt"]:]
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------------------------------- runs
def run(state):
    return _RUN[state["kind"]](state["handle"], state)


def _run_decode(h, s):
    """Takes the rings back to the context the sequences share and decodes. Each step's tokens come to the host, where a
    program would sample or stream them; what is returned is the last step's logits, since the choice between two all but
    equal logits is no measure of anything."""
    for i in range(s["layers"]):
        h.lib.gehtp_cuda_state_set_count(i, h.past)
    for face in s["faces"]:
        h.engine.run_io(face, h.man["token_temp"], h.tokens)
    return h.logits


def _run_prefill(h, s):
    h.run_dev(s["ids"], h.man["logits_temp"])
    return h.logits


def _run_delta(h, s):
    h.engine.state_reset()
    h.run_dev(s["hidden"], h.man["conv_temp"])
    return h.outputs


def _run_session(h, s):
    h.session.reset()
    logits = [h.session.feed(s["prompt"], want=(len(s["prompt"]) - 1,))]
    for t in s["answer"]:
        logits.append(h.session.feed([t], want=(0,)))
    return logits


_RUN = dict(decode=_run_decode, prefill=_run_prefill, delta=_run_delta, session=_run_session)


# ---------------------------------------------------------------------------------------------------- work
def work(case):
    by, fl = dict(decode=_work_decode, prefill=_work_prefill, delta=_work_delta, session=_work_session)[case["kind"]](case)
    return {"bytes": float(by), "flops": float(fl)}


def _matrices(cfg):
    """(K, N) of the projections of one layer."""
    q, kv = cfg.n_heads * cfg.head_dim, cfg.kv_heads * cfg.head_dim
    return [(cfg.hidden, q + 2 * kv), (q, cfg.hidden), (cfg.hidden, cfg.ffn), (cfg.hidden, cfg.ffn), (cfg.ffn, cfg.hidden)]


def _weight_bytes(K, N, quant):
    return K * N // 2 + 2 * (K // 64) * N if quant == "w4" else 2 * K * N


def _work_decode(c):
    cfg, B = SHAPES[c["shape"]], c["batch"]
    mats = _matrices(cfg) * c["layers"] + [(cfg.hidden, cfg.vocab)]
    by = sum(_weight_bytes(K, N, c["quant"]) for K, N in mats) + 2 * B * cfg.vocab
    fl = sum(2 * B * K * N for K, N in mats)
    by += c["layers"] * B * c["context"] * cfg.kv_heads * cfg.head_dim * 4
    fl += c["layers"] * B * c["context"] * cfg.n_heads * cfg.head_dim * 4
    return by * c["steps"], fl * c["steps"]


def _work_prefill(c):
    cfg, T = SHAPES[c["shape"]], c["tokens"]
    mats = _matrices(cfg) * c["layers"] + [(cfg.hidden, cfg.vocab)]
    by = sum(_weight_bytes(K, N, c["quant"]) for K, N in mats) + 2 * T * cfg.vocab
    fl = sum(2 * T * K * N for K, N in mats) + c["layers"] * 2 * T * (T + 1) * cfg.n_heads * cfg.head_dim
    return by, fl


def _work_delta(c):
    T, inner = c["tokens"], DELTA_HEADS * DELTA_DIM
    by = sum(_weight_bytes(K, N, "w4") for K, N in ((DELTA_HIDDEN, DELTA_CHANNELS), (inner, DELTA_HIDDEN)))
    by += 2 * T * (2 * DELTA_HIDDEN + DELTA_CHANNELS + 3 * inner) + 8 * inner * DELTA_DIM
    fl = 2 * T * (DELTA_HIDDEN * DELTA_CHANNELS + inner * DELTA_HIDDEN) + 2 * CONV_TAPS * T * DELTA_CHANNELS + 6 * T * inner * DELTA_DIM
    return by, fl


def _work_session(c):
    width, (ff, H) = c["width"], DESIGN_SIZES[c["width"]]
    P, S = c["prompt"], c["steps"]
    es = 4 if c["dtype"] == "float32" else 2
    pairs, inner = P * (P + 1) / 2 + sum(P + i + 1 for i in range(S)), H * 128
    if c["design"] == "Supevik":
        mats = ([(width, 2 * inner + 2048), (inner, width), (width, 2 * ff), (ff, width)]) * 4 + [(2 * width, width)] * 2
        fl = 4 * pairs * inner * 4          # windows reach past these contexts or save less than half
        rows = 4 * 2048 * es
    else:
        mats = [(width, 3 * inner + H + 256), (128, inner), (128, inner), (inner, width), (width, ff), (ff, width)] * 2
        mats += [(width, H * 192 + 576 + H), (512, 2 * inner), (inner, width), (width, ff), (ff, width)] * 2
        fl = 2 * (2 * pairs * H * (192 + 128)) + 2 * (P + S) * 6 * inner * 128
        rows = 2 * 576 * es
    params = sum(K * N for K, N in mats)
    fl += 2 * params * (P + S) + 2 * DESIGN_VOCAB * width * (1 + S)
    by = 2 * (params + DESIGN_VOCAB * width) * (1 + S) + rows * (P + sum(P + i + 1 for i in range(S))) + 4 * DESIGN_VOCAB * (1 + S)
    return by, fl


def tolerance(case):
    """About four times the distance to `exact` that was seen: fp16 or bf16 roundings between the ops of several layers (2e-3 to
    8e-3), of one delta-rule layer (3e-4), sums of 32 bits (7e-7 to 2e-6)."""
    if case["kind"] == "delta":
        return {"rel": 2e-3}
    return {"rel": 1e-5} if case.get("dtype") == "float32" else {"rel": 2.5e-2}


# --------------------------------------------------------------------------------------------------- exact
def _f64(a):
    return (torch.from_numpy(a) if isinstance(a, np.ndarray) else a).cuda().double()


def _w4(pair):
    """Weights [K, N] of a (nibbles, scales) pair: fp16((q - 8) scale)."""
    nib, sc = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in pair)
    q = torch.stack([nib & 15, nib >> 4], -1).reshape(nib.shape[0], -1).float() - 8.0
    return (q * sc.float().repeat_interleave(64, 0)).half().double()


def _rms(x, gamma, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * gamma


def _halves(x, cos, sin):
    h = x.shape[-1] // 2
    return x * cos + torch.cat([-x[..., h:], x[..., :h]], -1) * sin


def _tables(cfg, pos):
    """fp16 cosines and sines, as the faces and slots hold them."""
    ang = np.asarray(pos, np.float64)[:, None] * (1.0 / cfg.rope_theta ** (np.arange(0, cfg.head_dim, 2) / cfg.head_dim))[None]
    return [_f64(np.concatenate([f(ang), f(ang)], 1).astype(np.float16)) for f in (np.cos, np.sin)]


def _gammas(root, layer, cfg):
    """The two norms' weights the builders draw for a layer: the first numbers of its generator."""
    rng = runlists.part_rng(root, layer)
    return [_f64(rng.normal(1.0, 0.1, cfg.hidden).astype(np.float16)) for _ in range(2)]


def _exact_decoder(c, seed):
    """Both shapes of a decoder: T new positions of B sequences behind `past` cached ones. Logits of every new position."""
    cfg = SHAPES[c["shape"]]
    decode = c["kind"] == "decode"
    ids = _ids(c, seed) if decode else _ids(c, seed)[:, None]            # [T, B]
    T, B = ids.shape
    past = c["context"] - T if decode else 0
    root = 1004 if decode else 1003                                      # default weight seeds of the two builders
    nh, kvh, hd, H = cfg.n_heads, cfg.kv_heads, cfg.head_dim, cfg.hidden
    rep = nh // kvh
    block = runlists.synth_embedding(runlists.part_rng(root, runlists.EMB_PART), 1024, H)
    x = _f64(block[ids % 1024])                                          # the table repeats its first 1024 rows
    cos, sin = (t[:, None, None] for t in _tables(cfg, past + np.arange(T)))
    scale = float(np.float16(1.0 / np.sqrt(hd)))
    see = torch.ones(T, T, device="cuda").tril().bool()
    mats = _matrices(cfg)

    def product(a, at, K, N):
        w = _values(_weight(c, at, K, N))
        return torch.cat([a @ w[:, n:n + 16384].double() for n in range(0, N, 16384)], -1)
    for li in range(c["layers"]):
        gammas = _gammas(root, li, cfg)
        y = product(_rms(x, gammas[0]), 5 * li, *mats[0])
        q, k, v = y.split([nh * hd, kvh * hd, kvh * hd], -1)
        q, k, v = _halves(q.reshape(T, B, nh, hd), cos, sin), _halves(k.reshape(T, B, kvh, hd), cos, sin), v.reshape(T, B, kvh, hd)
        ring = _ring(c, li)[:past] if decode else None
        out = torch.empty(T, B, nh, hd, device="cuda", dtype=torch.float64)
        for b in range(B):
            for j in range(kvh):
                qq = q[:, b, j * rep:(j + 1) * rep].transpose(0, 1)      # [rep, T, hd]
                s = (qq @ k[:, b, j].T * scale).masked_fill(~see, -torch.inf)
                vv = v[:, b, j]
                if decode:
                    s = torch.cat([qq @ ring[:, 0, b, j].double().T * scale, s], -1)
                    vv = torch.cat([ring[:, 1, b, j].double(), vv])
                out[:, b, j * rep:(j + 1) * rep] = (torch.softmax(s, -1) @ vv).transpose(0, 1)
        x = x + product(out.reshape(T, B, nh * hd), 5 * li + 1, *mats[1])
        h = _rms(x, gammas[1])
        gate = product(h, 5 * li + 2, *mats[2])
        x = x + product(gate * torch.sigmoid(gate) * product(h, 5 * li + 3, *mats[3]), 5 * li + 4, *mats[4])
    gamma = runlists.part_rng(root, runlists.HEAD_PART).normal(1.0, 0.1, H).astype(np.float16)
    return product(_rms(x[-1] if decode else x[:, 0], _f64(gamma)), 5 * c["layers"], H, cfg.vocab)


def _exact_delta(c, seed):
    T, H, D = c["tokens"], DELTA_HEADS, DELTA_DIM
    part = lambda p: runlists.part_rng(1005, p)  # noqa: E731
    x = _hidden(c, seed).double() @ _w4(runlists.rand_w4(part(0), DELTA_HIDDEN, DELTA_CHANNELS))
    taps = _f64(part(1).normal(0.0, 0.5, (CONV_TAPS, DELTA_CHANNELS)).astype(np.float16))
    rows = torch.cat([x.new_zeros(CONV_TAPS - 1, DELTA_CHANNELS), x])
    rows[T:] = 0                            # the op reads input rows 0 .. T - taps
    out = [sum(rows[j:j + T] * taps[j] for j in range(CONV_TAPS))]
    w_out = _w4(runlists.rand_w4(part(2), H * D, DELTA_HIDDEN))
    S = x.new_zeros(H, D, D)                # [key, value]
    for ci in range(T // CHUNK):
        rng = part(10 + ci)
        k = rng.standard_normal((H, CHUNK, D)).astype(np.float32)
        k = _f64((k / np.linalg.norm(k, axis=-1, keepdims=True)).astype(np.float16))
        v, q = (_f64(rng.standard_normal((H, CHUNK, D)).astype(np.float16)) for _ in range(2))
        beta = _f64((1.0 / (1.0 + np.exp(-rng.standard_normal((H, CHUNK))))).astype(np.float16))
        g = _f64(np.log(1.0 / (1.0 + np.exp(-rng.standard_normal((H, CHUNK))))).astype(np.float16))
        y = torch.empty_like(v)
        for t in range(CHUNK):
            S = S * torch.exp(g[:, t])[:, None, None]
            u = beta[:, t, None] * (v[:, t] - (k[:, t, None] @ S)[:, 0])
            S = S + k[:, t, :, None] * u[:, None]
            y[:, t] = (q[:, t, None] @ S)[:, 0] * D ** -0.5
        out.append(y.transpose(0, 1).reshape(CHUNK, H * D) @ w_out)
    return out


def _pairs(x, pos, base):
    n = x.shape[-1]
    a = pos[:, None] * base ** (-torch.arange(0, n, 2, device="cuda", dtype=torch.float64) / n)
    c, s = torch.cos(a), torch.sin(a)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)


def _channel_delta(h, m, p, eps):
    T, H, D = h.shape[0], m["heads"], m["dim"]
    silu = torch.nn.functional.silu

    def conv(n):
        x, w = h @ p(n).T, p(n + ".conv")
        xp = torch.cat([x.new_zeros(w.shape[1] - 1, x.shape[1]), x])
        return silu(sum(xp[j:j + T] * w[:, j] for j in range(w.shape[1]))).reshape(T, H, D)
    q, k, v = conv("q"), conv("k"), conv("v")
    q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
    q = q * D ** -0.5
    beta = torch.sigmoid(h @ p("b").T)
    a = (h @ p("a1").T @ p("a2").T + p("dt_bias")).reshape(T, H, D)
    g = torch.exp(-torch.exp(p("A_log"))[None, :, None] * torch.nn.functional.softplus(a, threshold=700.0))
    S, o = h.new_zeros(H, D, D), torch.empty_like(v)
    for t in range(T):
        S = S * g[t, :, :, None]
        u = beta[t, :, None] * (v[t] - (k[t, :, None] @ S)[:, 0])
        S = S + k[t, :, :, None] * u[:, None]
        o[t] = (q[t, :, None] @ S)[:, 0]
    gate = torch.sigmoid(h @ p("g1").T @ p("g2").T).reshape(T, H, D)
    return (_rms(o, p("norm"), eps) * gate).reshape(T, H * D) @ p("o").T


def _latent(h, m, p, eps):
    T, H, D, R, V, C = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    pos = torch.arange(T, device="cuda", dtype=torch.float64)
    q = (h @ p("q").T).reshape(T, H, D + R).transpose(0, 1)
    d = h @ p("dkv").T
    c, kr = _rms(d[:, :C], p("dkv.norm"), eps), _pairs(d[:, C:], pos, m["rot"]["base"])
    kn, v = ((c @ p(n).T).reshape(T, H, -1).transpose(0, 1) for n in ("uk", "uv"))
    s = (q[..., :D] @ kn.transpose(1, 2) + _pairs(q[..., D:], pos, m["rot"]["base"]) @ kr.T) * m["scale"]
    s = s.masked_fill(~torch.ones(T, T, device="cuda").tril().bool(), -torch.inf)
    o = torch.softmax(s, -1) @ v * torch.sigmoid(h @ p("g").T).T[:, :, None]
    return o.transpose(0, 1).reshape(T, H * V) @ p("o").T


def _exact_ripidra(cfg, t, ids):
    x, eps = t["embed"][ids], cfg["norm"]["eps"]
    for i, layer in enumerate(cfg["layers"]):
        pre = "l%d." % i
        mixer = _channel_delta if layer["type"] == "channel_delta" else _latent
        x = x + _rms(mixer(x, layer["mixer"], lambda n: t[pre + "mix." + n], eps), 1.0 + t[pre + "norm1"], eps)
        y = torch.relu(x @ t[pre + "mlp.up"].T) ** 2 @ t[pre + "mlp.down"].T
        x = x + _rms(y, 1.0 + t[pre + "norm2"], eps)
    return _rms(x, 1.0 + t["final.norm"], eps), t["embed"]


def _yarn(rot):
    """(angle per position of every pair, factor on cosine and sine)."""
    n, base, s = rot["dims"], rot["base"], rot["scaling"]
    f = base ** (-np.arange(0, n, 2) / n)
    at = lambda turns: n * np.log(s["original"] / (2 * np.pi * turns)) / (2 * np.log(base))  # noqa: E731
    lo, hi = max(np.floor(at(s["fast"])), 0), min(np.ceil(at(s["slow"])), n - 1)
    r = np.clip((np.arange(n // 2) - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    return f * (r / s["factor"] + 1.0 - r), 0.1 * np.log(s["factor"]) + 1.0


def _window(h, m, p, eps):
    T, H, G, D = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
    f, mag = _yarn(m["rot"])
    ang = np.arange(T)[:, None] * f[None]
    cos, sin = (_f64(np.concatenate([z, z], 1)) * mag for z in (np.cos(ang), np.sin(ang)))
    q, k, v = ((h @ p(n).T + p(n + ".b")).reshape(T, r, D).transpose(0, 1) for n, r in (("q", H), ("k", G), ("v", G)))
    q, k = _halves(_rms(q, p("q.norm"), eps), cos, sin), _halves(_rms(k, p("k.norm"), eps), cos, sin)
    gap = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]
    see, out = (gap >= 0) & (gap < m["mask"]["size"]), torch.empty(T, H, D, device="cuda", dtype=torch.float64)
    for i in range(H):
        j = i // (H // G)
        out[:, i] = torch.softmax((q[i] @ k[j].T * m["scale"]).masked_fill(~see, -torch.inf), -1) @ v[j]
    return (out.reshape(T, H * D) * torch.sigmoid(h @ p("g").T)) @ p("o").T


def _exact_supevik(cfg, t, ids):
    eps = cfg["norm"]["eps"]
    norm = lambda n, x: torch.tanh(t[n + ".alpha"] * x) * t[n] + t[n + ".b"]  # noqa: E731
    x0 = x = t["embed"][ids] * cfg["embedding"]["scale"]
    for i, enter in ((0, False), (1, True), (1, True), (2, False)):
        layer, pre = cfg["layers"][i], "l%d." % i
        if enter:
            x = torch.cat([x, x0], -1) @ t["loop.in"].T
        y = _window(norm(pre + "norm1", x), layer["mixer"], lambda n: t[pre + "mix." + n], eps)
        x = x + norm(pre + "norm1b", y)
        h = norm(pre + "norm2", x)
        y = (torch.nn.functional.gelu(h @ t[pre + "mlp.gate"].T, approximate="tanh") * (h @ t[pre + "mlp.up"].T)) @ t[pre + "mlp.down"].T
        x = x + norm(pre + "norm2b", y)
    return norm("final.norm", x), t["head"]


def _exact_session(c, seed):
    cfg, t = _design(c)
    ids = torch.from_numpy(_ids(c, seed)).cuda()
    x, head = (_exact_supevik if c["design"] == "Supevik" else _exact_ripidra)(cfg, {k: v.double() for k, v in t.items()}, ids)
    return [(x[i:i + 1] @ head.T).cpu().numpy() for i in range(c["prompt"] - 1, c["prompt"] + c["steps"])]


def exact(case, seed):
    return dict(decode=_exact_decoder, prefill=_exact_decoder, delta=_exact_delta, session=_exact_session)[case["kind"]](case, seed)
