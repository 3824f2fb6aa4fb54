"""What this framework is timed on: calls that its users make, over the sizes they make them with.

Six kinds of case:
  quantize   weights of a checkpoint to the bundle's codes, scales and zero points (ops.quantize_affine)
  attention  decode attention over a quantized cache that a host schedules itself (ops.TurboQuant.attention)
  decode     steps of a quantized Llama / Qwen3 model, one sequence or several in lockstep (CudaInference.decode_step)
  prefill    a prompt through such a model (CudaInference.prefill)
  prompt     a prompt through a model given as a list of layers (CudaInference.prefill)
  serve      such a model serving several prompts of different lengths: every sequence is added, all are decoded together,
             then they leave (add_sequence, batch_decode_step, remove_sequence)
Tokens are forced, so that the logits of every step can be compared.  Widths, heads and feed-forwards are those of bench.py
(Llama-3-8B and Qwen3-0.6B shapes, w2048 and w4096), with fewer layers and a vocabulary of 32768 where loading a whole model
would only repeat the same layer; weights are random, quantized in groups of 128 with AWQ scales where the option is on.

exact() restates each of them in plain torch, in 64 bits and without any of the roundings in between."""
import math
import zlib

import numpy as np
import torch

from ironmill_b200 import ops
from ironmill_b200.architectures import config_from_json
from ironmill_b200.bundle import ModelConfig, WeightTensor
from ironmill_b200.engine import CudaConfig, CudaInference

GROUP = 128
HEAD = 128
F64 = torch.float64


# ------------------------------------------------------------------------------------------------ the cases
def _model(shape, layers, wbits=4, kv=8, awq=True):
    """Llama-3-8B widths, Qwen3-0.6B widths (with its norms of queries and keys), or w2048 of the layer-list workload."""
    s = {"l8": dict(width=4096, ff=14336, heads=32, kv_heads=8, vocab=32768, qk_norm=False, theta=5e5),
         "q06": dict(width=1024, ff=3072, heads=16, kv_heads=8, vocab=151936, qk_norm=True, theta=1e6),
         "w2048": dict(width=2048, ff=8192, heads=16, kv_heads=8, vocab=32768, qk_norm=False, theta=5e5)}[shape]
    return dict(s, layers=layers, wbits=wbits, kv=kv, awq=awq)


def listed():
    return [
        # a gate or up projection of an 8B model on its way into a bundle
        dict(name="quantize_gate", kind="quantize", rows=14336, cols=4096, bits=4, awq=True),
        # a scheduler's decode attention: 16 sequences of different lengths, 8-bit cache
        dict(name="attention_16_seqs", kind="attention", heads=32, kv_heads=8, seqs=16, ctx=8192, bits=8, ragged=True),
        # interactive use of the smallest model: latency and launches
        dict(name="decode_small_b1", kind="decode", batch=1, ctx=512, steps=4, **_model("q06", 28, awq=False)),
        # interactive use at 8B widths
        dict(name="decode_8b_b1", kind="decode", batch=1, ctx=2048, steps=4, **_model("l8", 4)),
        # a few users at once
        dict(name="decode_8b_b4", kind="decode", batch=4, ctx=1024, steps=2, **_model("l8", 4)),
        # a server's batch: from 16 rows on the projections are contractions
        dict(name="decode_8b_b24", kind="decode", batch=24, ctx=600, steps=2, **_model("l8", 4)),
        # the prompt of the same model
        dict(name="prefill_8b_2048", kind="prefill", tokens=2048, **_model("l8", 4)),
        # a long document with the unquantized cache, in several portions of odd length
        dict(name="prefill_long_fp16kv", kind="prefill", tokens=5003, **_model("w2048", 4, kv=16)),
        # prompts of the two designs given as lists of layers
        dict(name="gizizen_prompt", kind="prompt", design="gizizen", size="w2048", dtype="bfloat16", tokens=2048),
        dict(name="luvatar_prompt", kind="prompt", design="luvatar", size="w2048", dtype="bfloat16", tokens=3001),
        # the same designs serving: many short requests, and one user
        dict(name="gizizen_serve_16", kind="serve", design="gizizen", size="w2048", dtype="bfloat16", seqs=16, prompt=90, steps=16),
        dict(name="luvatar_serve_1", kind="serve", design="luvatar", size="w2048", dtype="bfloat16", seqs=1, prompt=300, steps=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["quantize", "attention", "decode", "decode", "decode", "prefill", "prefill", "prompt", "serve"])
    if kind == "quantize":
        # odd row lengths too: a tensor whose rows are no multiple of the group keeps a short last group
        return dict(kind=kind, rows=_log(rng, 96, 14336), cols=rng.choice([1024, 2048, 3072, 4096, _log(rng, 300, 4000)]), bits=rng.choice([4, 4, 8]),
                    awq=rng.random() < 0.5)
    if kind == "attention":
        seqs = _log(rng, 1, 32)
        return dict(kind=kind, heads=rng.choice([16, 32]), kv_heads=8, seqs=seqs, ctx=_log(rng, 60, min(65536, 131072 // seqs)), bits=rng.choice([8, 8, 4]),
                    ragged=rng.random() < 0.5)
    if kind in ("decode", "prefill"):
        m = _model(rng.choice(["l8", "w2048", "w2048"]), rng.randint(2, 4), wbits=rng.choice([4, 4, 4, 8]), kv=rng.choice([8, 8, 4, 16]), awq=rng.random() < 0.7)
        if kind == "decode":
            batch = rng.choice([1, 1, _log(rng, 2, 15), _log(rng, 16, 64)])
            return dict(kind=kind, batch=batch, ctx=_log(rng, 16, 4000 if batch == 1 else 600), steps=2, **m)
        return dict(kind=kind, tokens=_log(rng, 17, 2040), **m)
    design = rng.choice(["gizizen", "luvatar"])
    # true 32-bit runs are how a port is checked: short ones
    dtype = "float32" if rng.random() < 0.12 else "bfloat16"
    if kind == "prompt":
        return dict(kind=kind, design=design, size="w2048", dtype=dtype, tokens=_log(rng, 20, 150 if dtype == "float32" else 3000))
    seqs = _log(rng, 1, 4 if dtype == "float32" else 16)
    return dict(kind=kind, design=design, size="w2048", dtype=dtype, seqs=seqs, prompt=_log(rng, 16, 60 if dtype == "float32" else 400 if seqs < 4 else 100), steps=8)


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed, name):
    return torch.Generator(device="cuda").manual_seed((seed * 7919 + zlib.crc32(name.encode())) % (1 << 62))


def _randn(seed, name, *shape):
    return torch.randn(shape, generator=_gen(seed, name), device="cuda")


def _tokens(seed, name, vocab, *shape):
    return np.random.Generator(np.random.PCG64([seed, zlib.crc32(name.encode())])).integers(0, vocab, shape).astype(np.uint32)


def _lengths(seed, n, top, ragged=True):
    """Lengths of n sequences, the longest `top`."""
    r = np.random.Generator(np.random.PCG64([seed, 17]))
    return [top if i == 0 or not ragged else int(r.integers(max(1, top // 8), top + 1)) for i in range(n)]


def _quantize(w, bits):
    """Codes, scales and zero points of w [N, K], K a multiple of the group, as a bundle holds them."""
    g = w.float().view(w.shape[0], -1, GROUP)
    lo, hi = g.amin(-1), g.amax(-1)
    s = (hi - lo) / (2 ** bits - 1)
    z = torch.round(-lo / s)
    q = torch.clamp(torch.round(g / s[..., None] + z[..., None]), 0, 2 ** bits - 1).to(torch.uint8).view(w.shape)
    return q, s.half(), z.half()


def _matrix_shapes(c):
    kv = c["kv_heads"] * HEAD
    q = c["heads"] * HEAD
    return {"self_attn.q_proj": (q, c["width"]), "self_attn.k_proj": (kv, c["width"]), "self_attn.v_proj": (kv, c["width"]), "self_attn.o_proj": (c["width"], q),
            "mlp.gate_proj": (c["ff"], c["width"]), "mlp.up_proj": (c["ff"], c["width"]), "mlp.down_proj": (c["width"], c["ff"])}


class _Weights:
    """Tensors of a quantized model by their checkpoint names, drawn from the seed."""

    def __init__(self, c, seed):
        self.c, self.seed = c, seed
        self.cfg = ModelConfig(architecture="qwen3" if c["qk_norm"] else "llama", hidden_size=c["width"], intermediate_size=c["ff"],
                               num_hidden_layers=c["layers"], num_attention_heads=c["heads"], num_key_value_heads=c["kv_heads"], head_dim=HEAD,
                               vocab_size=c["vocab"], max_position_embeddings=8192, rms_norm_eps=1e-6 if c["qk_norm"] else 1e-5, rope_theta=c["theta"],
                               tie_word_embeddings=True)

    def config(self):
        return self.cfg

    def has_tensor(self, name):
        return name != "lm_head.weight"

    def quantized(self, name):
        """(codes, scale, zero, awq or None) on the GPU."""
        parts = name.split(".")
        N, K = _matrix_shapes(self.c)[".".join(parts[3:5])]
        awq = None
        group = {"q_proj": "in", "k_proj": "in", "v_proj": "in", "o_proj": "o", "gate_proj": "ffn", "up_proj": "ffn", "down_proj": "down"}[parts[4]]
        if self.c["awq"]:   # shared by the projections that read the same activations
            awq = (torch.rand(K, generator=_gen(self.seed, "awq%s.%s" % (parts[2], group)), device="cuda") * 1.5 + 0.5).half()
        w = (_randn(self.seed, name, N, K) * 0.02).half()
        if awq is not None:
            w = w.float() * awq.float()
        return _quantize(w, self.c["wbits"]) + (awq,)

    def dense(self, name):
        if name == "model.embed_tokens.weight":   # of the size of what the layers add to it, as in a trained model
            return (_randn(self.seed, name, self.c["vocab"], self.c["width"]) * 0.25).half()
        return torch.ones(HEAD if "self_attn" in name else self.c["width"], dtype=torch.float16, device="cuda")

    def tensor(self, name):
        if "_proj" not in name:
            t = self.dense(name)
            return WeightTensor(t.cpu().numpy(), tuple(t.shape), "float16")
        q, s, z, awq = self.quantized(name)
        shape = tuple(q.shape)
        if self.c["wbits"] == 4:
            q = q.view(-1, 2)
            q = q[:, 0] | (q[:, 1] << 4)
        return WeightTensor(q.reshape(-1).cpu().numpy(), shape, "uint8", s.cpu().numpy(), z.cpu().numpy(), self.c["wbits"], GROUP, 1,
                            None if awq is None else awq.cpu().numpy())


def _rotation(seed):
    """The signs and the projection that a host hands to the quantized cache."""
    r = np.random.Generator(np.random.PCG64([seed, 23]))
    return (r.integers(0, 2, HEAD) * 2 - 1).astype(np.float32), r.standard_normal((HEAD, HEAD)).astype(np.float32)


def _quantized_engine(c, seed, batch, max_seq):
    cfg = CudaConfig(max_seq_len=max_seq, max_batch=batch)
    if c["kv"] == 16:
        cfg.without_turboquant()
    else:
        cfg.with_turboquant(c["kv"])
    eng = CudaInference(cfg)
    signs, qjl = _rotation(seed)
    if c["kv"] == 16:
        eng.load_weights(_Weights(c, seed))
    else:
        eng.load_weights(_Weights(c, seed), tq_signs=signs, tq_qjl=qjl)
    return eng


def _stack_json(c):
    """Eight layer passes of a design at the sizes of bench.py's layer-list workload."""
    z = {"w2048": dict(width=2048, ff=8192, heads=16, vocab=32768), "w4096": dict(width=4096, ff=14336, heads=32, vocab=32768)}[c["size"]]
    mlp = {"kind": "dense", "ff": z["ff"]}
    if c["design"] == "luvatar":
        gla = {"type": "gla", "mlp": mlp, "mixer": {"heads": z["heads"], "dim": 128, "vdim": 128, "tau": 16.0}}
        mixer = {"heads": z["heads"], "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 8192},
                 "rot": {"dims": 128, "base": 5e5, "scaling": {"factor": 4.0}}}
        att, shared1, shared5 = ({"type": "attention", "mlp": mlp, "mixer": dict(mixer, **more)} for more in ({}, {"kv_from": 1}, {"kv_from": 5}))
        return {"architecture": "Luvatar", "vocab": z["vocab"], "width": z["width"], "norm": {"eps": 1e-6}, "embedding": {"scale": z["width"] ** 0.5},
                "layers": [gla, att, gla, shared1, gla, att, gla, shared5]}
    lat = {"type": "latent_attention", "mlp": mlp,
           "mixer": {"heads": z["heads"], "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
                     "rot": {"dims": 64, "base": 5e5, "scaling": {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}}}}
    lin = {"type": "lightning", "mlp": mlp,
           "mixer": {"heads": z["heads"], "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-3 - 6 * i / z["heads"]) for i in range(z["heads"])]}}
    return {"architecture": "Gizizen", "vocab": z["vocab"], "width": z["width"], "norm": {"eps": 1e-6}, "layers": [lat, lat, lin, lat],
            "loop": {"start": 0, "stop": 2, "times": 3}, "logit_softcap": 30.0}


class _StackWeights:
    """bf16 tensors of a list-of-layers model; matrices are scaled to keep activations near one."""

    def __init__(self, c, seed):
        self.cfg, self.seed = config_from_json(_stack_json(c)), seed
        self.cfg.complete(lambda name: (16,))
        self.shapes = self.cfg.tensors()

    def config(self):
        return self.cfg

    def has_tensor(self, name):
        return name in self.shapes

    def value(self, name):
        shape = self.shapes[name]
        w = torch.ones(shape, device="cuda") if name.endswith(("norm", "norm1", "norm2")) else _randn(self.seed, name, *shape) * shape[-1] ** -0.5
        return w.to(torch.bfloat16)

    def tensor(self, name):
        return WeightTensor(self.value(name).view(torch.uint16).cpu().numpy(), self.shapes[name], "bfloat16")


def prepare(case, seed):
    c = case
    if c["kind"] == "quantize":
        awq = (torch.rand(c["cols"], generator=_gen(seed, "awq"), device="cuda") * 1.5 + 0.5).half() if c["awq"] else None
        return dict(case=c, w=(_randn(seed, "w", c["rows"], c["cols"]) * 0.02).half(), awq=awq)
    if c["kind"] == "attention":
        dev = ops.Device(0)
        signs, qjl = _rotation(seed)
        tq = ops.TurboQuant(dev, HEAD, c["bits"], signs, qjl)
        ctx, n, g = c["ctx"], c["seqs"], c["kv_heads"]
        cache = {}
        for part in "kv":   # keys and values of all positions, appended by the encoder as a host would have done
            rows = _randn(seed, part, n * ctx, g, HEAD).half()
            cache[part] = torch.zeros((n, g, ctx, HEAD * c["bits"] // 8), dtype=torch.uint8, device="cuda")
            cache[part + "s"] = torch.zeros((n, g, ctx), device="cuda")
            cache[part + "r"] = torch.zeros((n, g, ctx), device="cuda") if part == "k" else None
            tq.encode(rows, part == "k", cache[part], cache[part + "s"], cache[part + "r"], g, ctx, 0, nseq=n)
        lengths = _lengths(seed, n, ctx, c["ragged"])
        return dict(case=c, dev=dev, tq=tq, cache=cache, q=_randn(seed, "q", n, c["heads"], HEAD).half(),
                    pos=torch.tensor([x - 1 for x in lengths], dtype=torch.int32, device="cuda"))
    if c["kind"] == "decode":
        B, ctx, steps = c["batch"], c["ctx"], c["steps"]
        eng = _quantized_engine(c, seed, B, ctx + steps + 8)
        prompts = _tokens(seed, "prompt", c["vocab"], B, ctx)
        if B == 1:
            eng.prefill(prompts[0])
        else:
            for p in prompts:
                eng.add_sequence(p)
        return dict(case=c, eng=eng, fed=_tokens(seed, "fed", c["vocab"], steps, B))
    if c["kind"] == "prefill":
        return dict(case=c, eng=_quantized_engine(c, seed, 1, c["tokens"] + 8), prompt=_tokens(seed, "prompt", c["vocab"], c["tokens"]))
    seqs, steps = c.get("seqs", 1), c.get("steps", 0)
    top = c["tokens"] if c["kind"] == "prompt" else c["prompt"]
    eng = CudaInference(CudaConfig(max_seq_len=top + steps + 8, max_batch=seqs, dtype=c["dtype"]))
    eng.load_weights(_StackWeights(c, seed))
    vocab = _stack_json(c)["vocab"]
    prompts = [_tokens(seed, "prompt%d" % i, vocab, n) for i, n in enumerate(_lengths(seed, seqs, top))]
    return dict(case=c, eng=eng, prompts=prompts, fed=_tokens(seed, "fed", vocab, steps, seqs))


def run(state):
    c = state["case"]
    if c["kind"] == "quantize":
        return dict(zip(("codes", "scales", "zeros"), ops.quantize_affine(state["w"], GROUP, c["bits"], state["awq"])))
    if c["kind"] == "attention":
        k = state["cache"]
        return state["tq"].attention(state["q"], k["k"], k["v"], k["ks"], k["vs"], k["kr"], HEAD ** -0.5, c["heads"], c["kv_heads"], c["ctx"], 0,
                                     nseq=c["seqs"], pos_dev=state["pos"])
    eng = state["eng"]
    if c["kind"] == "decode":
        eng.truncate_to(c["ctx"])
        return [eng.decode_step(int(t[0]) if c["batch"] == 1 else t) for t in state["fed"]]
    if c["kind"] in ("prefill", "prompt"):
        eng.reset()
        return eng.prefill(state["prompt"] if c["kind"] == "prefill" else state["prompts"][0])
    ids = [eng.add_sequence(p) for p in state["prompts"]]
    out = []
    for t in state["fed"]:
        out.append([logits for _, logits in eng.batch_decode_step(dict(zip(ids, t.tolist())))])
    for i in ids:
        eng.remove_sequence(i)
    return [np.stack(step) for step in out]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _quantized_work(c, passes, rows, ctx_reads, score_flops, logit_rows):
    """passes: forward passes that read the weights; rows: token rows in all; ctx_reads: cached positions read per layer and KV head."""
    params = sum(n * k for n, k in _matrix_shapes(c).values())
    kv_row = {8: 268, 4: 140, 16: 512}[c["kv"]]
    per_pass = c["layers"] * (params * c["wbits"] / 8 + params / GROUP * 4) + 2 * c["vocab"] * c["width"]
    kv = c["layers"] * c["kv_heads"] * kv_row * (ctx_reads + rows)
    return {"bytes": passes * per_pass + kv + 2 * rows * c["width"] + 4 * logit_rows * c["vocab"],
            "flops": 2 * rows * params * c["layers"] + 2 * logit_rows * c["vocab"] * c["width"] + score_flops}


def _stack_sizes(c):
    """[(matrix elements, attention flops per seen position, state elements, cached elements per position)] of every layer pass, and
    the elements of distinct weights outside the head."""
    j = _stack_json(c)
    w = _StackWeights.__new__(_StackWeights)
    w.cfg = config_from_json(j)
    w.cfg.complete(lambda name: (16,))
    shapes = w.cfg.tensors()
    loop = j.get("loop") or {"start": 0, "stop": 0, "times": 0}
    order = list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], len(j["layers"])))
    out = []
    for i in order:
        m, kind = j["layers"][i]["mixer"], j["layers"][i]["type"]
        elems = sum(s[0] * s[1] for n, s in shapes.items() if n.startswith("l%d." % i) and len(s) == 2)
        if kind == "latent_attention":
            out.append((elems, 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), 0, m["kv_rank"] + m["rot_dim"]))
        elif kind == "attention":
            out.append((elems, 2 * m["heads"] * (m["dim"] + m["vdim"]), 0, m["kv_heads"] * (m["dim"] + m["vdim"])))
        else:
            out.append((elems, 0, m["heads"] * m["dim"] * m["vdim"], 0))
    return out, loop["times"] * 2 * j["width"] ** 2, j["vocab"] * j["width"]


def work(case):
    c = case
    if c["kind"] == "quantize":
        n, groups = c["rows"] * c["cols"], c["rows"] * -(-c["cols"] // GROUP)
        return {"bytes": 2 * n + n * c["bits"] / 8 + 8 * groups + (2 * c["cols"] if c["awq"] else 0), "flops": 4 * n}
    if c["kind"] == "attention":
        # lengths of ragged sequences are drawn with the seed: their mean
        seen = c["ctx"] * (1 + (c["seqs"] - 1) * (0.5625 if c["ragged"] else 1.0))
        return {"bytes": seen * c["kv_heads"] * (2 * HEAD * c["bits"] / 8 + 12) + 4 * c["seqs"] * c["heads"] * HEAD, "flops": seen * c["heads"] * 6 * HEAD}
    if c["kind"] == "decode":
        rows, seen = c["batch"] * c["steps"], c["batch"] * sum(c["ctx"] + i + 1 for i in range(c["steps"]))
        return _quantized_work(c, c["steps"], rows, seen, c["layers"] * seen * c["heads"] * 4 * HEAD, rows)
    if c["kind"] == "prefill":
        t = c["tokens"]
        return _quantized_work(c, 1, t, t, c["layers"] * t * (t + 1) / 2 * c["heads"] * 4 * HEAD, 1)
    sizes, loop, head = _stack_sizes(c)
    es = 4 if c["dtype"] == "float32" else 2
    seqs, steps = c.get("seqs", 1), c.get("steps", 0)
    mean = c["tokens"] if c["kind"] == "prompt" else c["prompt"] * (1 + (seqs - 1) * 0.5625) / seqs
    rows, passes = seqs * (mean + steps), (seqs if c["kind"] == "serve" else 1) + steps
    logit_rows = seqs * (1 + steps)
    weights = sum(s[0] for s in sizes) + loop + head
    seen = seqs * (mean * (mean + 1) / 2 + steps * (mean + steps / 2))
    nbytes = passes * weights * es + seqs * steps * sum(2 * 4 * s[2] + es * s[3] * (mean + steps / 2) for s in sizes) + 4 * logit_rows * 32768
    flops = 2 * rows * (sum(s[0] + 2 * s[2] for s in sizes) + loop) + 2 * logit_rows * head + seen * sum(s[1] for s in sizes)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    c = case
    if c["kind"] == "quantize":
        return "exact"
    if c["kind"] == "attention":
        # f16 operands and results, f32 sums
        return {"rel": 3e-3, "max": 0.04}
    if c["kind"] in ("decode", "prefill"):
        # f16 activations; with a quantized cache a last bit can turn into a step of its codebook
        return {"rel": 0.02 if c["kv"] != 16 else 0.008, "max": 0.3 if c["kv"] != 16 else 0.1}
    if c["dtype"] == "float32":
        return {"rel": 1e-4, "max": 2e-3}
    return {"rel": 0.03, "max": 0.4}   # bf16 activations, eight layer passes


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _normal_quantile(p):
    t = p - 0.5

    def poly(coef, x):
        v = 0.0
        for k in coef:
            v = v * x + k
        return v

    if abs(t) <= 0.42:
        return t * poly([2.5066282746310002, 18.6150006252966, 41.39119773534996, 25.44106049637689], t * t) / poly(
            [14.382029373388, 63.690613, 84.681, 40.304, 1.0], t * t)
    s = math.sqrt(-math.log(p if t < 0 else 1.0 - p)) - 1.6
    r = poly([0.000124818987, 0.0227061845, 0.2728688, 1.3058437, 2.7580128, 2.2311569, 0.6462025, 0.001612], s) / poly(
        [0.000038746, 0.00745102, 0.09234118, 0.4710441, 1.0507501, 1.0, 0.2127601, 1.0], s)
    return -r if t < 0 else r


def _erf(x):
    """The five-term form that the table is defined with."""
    t, v = 1.0 / (1.0 + 0.3275911 * abs(x)), 0.0
    for k in (1.061405429, -1.453152027, 1.421413741, -0.284496736, 0.254829592):
        v = (v + k) * t
    return math.copysign(1.0 - (v * math.exp(-x * x) if math.isfinite(x) else 0.0), x)


def _codebook(bits):
    """Levels and boundaries of the cache's code for components of a unit vector (the format's fixed table)."""
    n, sigma = 1 << bits, 1.0 / math.sqrt(HEAD)
    cdf = lambda x: 0.5 * (1.0 + _erf(x / math.sqrt(2.0)))  # noqa: E731
    pdf = lambda x: 0.0 if math.isinf(x) else math.exp(-0.5 * x * x) / math.sqrt(2.0 * math.pi)  # noqa: E731
    lv = [sigma * _normal_quantile((i + 0.5) / n) for i in range(n)]
    for _ in range(200):
        edge = [-math.inf] + [(a + b) / 2 for a, b in zip(lv, lv[1:])] + [math.inf]
        new = []
        for lo, hi in zip(edge, edge[1:]):
            mass = cdf(hi / sigma) - cdf(lo / sigma)
            if mass < 1e-30:
                new.append(hi if math.isinf(lo) else lo if math.isinf(hi) else (lo + hi) / 2)
            else:
                new.append(sigma * (pdf(lo / sigma) - pdf(hi / sigma)) / mass)
        moved = max(abs(a - b) for a, b in zip(lv, new))
        lv = new
        if moved < 1e-10:
            break
    f32 = lambda a: torch.tensor(np.asarray(a, dtype=np.float32)).to("cuda", F64)  # noqa: E731
    return f32(lv), f32([(a + b) / 2 for a, b in zip(lv, lv[1:])])


class _Cache64:
    """The quantized cache: what it gives back for rows written to it, and queries on its terms."""

    def __init__(self, bits, seed):
        signs, qjl = _rotation(seed)
        self.signs, self.qjl = torch.tensor(signs).to("cuda", F64), torch.tensor(qjl).to("cuda", F64)
        self.kcb, self.kbd = _codebook(bits - 1)
        self.vcb, self.vbd = _codebook(bits)
        h = torch.ones((1, 1), dtype=F64, device="cuda")
        while h.shape[0] < HEAD:
            h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
        self.h = h / math.sqrt(HEAD)

    def rotate(self, x):
        return (x * self.signs) @ self.h * self.signs

    def _index(self, u, bounds):
        """The last boundary not above u decides (the tables are not sorted)."""
        out = torch.zeros(u.shape, dtype=torch.int64, device=u.device)
        for b in range(bounds.numel()):
            out[u >= bounds[b]] = b + 1
        return out

    def keys(self, k):
        x = self.rotate(k)
        norm = x.norm(dim=-1, keepdim=True)
        u = x / norm
        c = self.kcb[self._index(u, self.kbd)]
        res = u - c
        sign = torch.where(res @ self.qjl.T >= 0, 1.0, -1.0).to(F64)
        w = res.norm(dim=-1, keepdim=True) * (math.sqrt(2.0 / 3.14159265) / HEAD)
        return (c + w * (sign @ self.qjl)) * norm   # q . this = q . c + w (S q) . sign

    def values(self, v):
        x = self.rotate(v)
        norm = x.norm(dim=-1, keepdim=True)
        return self.vcb[self._index(x / norm, self.vbd)] * norm


def _attend(q, k, v, scale, first=0, start=None, sink=None):
    """Causal attention of one head: q [T, d] at positions first .., k and v [n, d]; start: first position seen, per query."""
    s = q @ k.T * scale
    at = torch.arange(first, first + q.shape[0], device=q.device)[:, None]
    j = torch.arange(k.shape[0], device=q.device)[None]
    hide = j > at
    if start is not None:
        hide = hide | (j < start[:, None])
    s = s.masked_fill(hide, -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.expand(s.shape[0], 1)], 1)
    p = torch.softmax(s, -1)
    return p[:, :k.shape[0]] @ v


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _quantized_forward(c, seed, seqs, last):
    """Logits of the last `last` positions of every sequence of tokens."""
    w = _Weights(c, seed)
    eps = w.cfg.rms_norm_eps
    cache = _Cache64(c["kv"], seed) if c["kv"] != 16 else None
    embed = w.dense("model.embed_tokens.weight").to(F64)
    xs = [embed[torch.from_numpy(np.asarray(s, dtype=np.int64)).cuda()] for s in seqs]
    inv = c["theta"] ** (-torch.arange(0, HEAD, 2, device="cuda", dtype=F64) / HEAD)

    def turn(x):  # [T, heads, d], halves paired; the table is kept in f16
        a = torch.arange(x.shape[0], device="cuda", dtype=F64)[:, None] * inv
        co, si = torch.cos(a).half().to(F64)[:, None], torch.sin(a).half().to(F64)[:, None]
        lo, hi = x[..., :HEAD // 2], x[..., HEAD // 2:]
        return torch.cat([lo * co - hi * si, lo * si + hi * co], -1)

    for i in range(c["layers"]):
        m = {}
        for n, shape in _matrix_shapes(c).items():
            q, s, z, awq = w.quantized("model.layers.%d.%s.weight" % (i, n))
            full = ((q.to(F64).view(shape[0], -1, GROUP) - z.to(F64)[..., None]) * s.to(F64)[..., None]).view(shape)
            m[n.split(".")[1][0]] = full if awq is None else full / awq.to(F64)   # q k v o g u d
        for b, x in enumerate(xs):
            n, T = _rms(x, eps), x.shape[0]
            q, k, v = (n @ m[t].T for t in "qkv")
            q, k, v = q.view(T, -1, HEAD), k.view(T, -1, HEAD), v.view(T, -1, HEAD)
            if c["qk_norm"]:
                q, k = _rms(q, eps), _rms(k, eps)
            q, k = turn(q), turn(k)
            if cache:
                q, k, v = cache.rotate(q), cache.keys(k), cache.values(v)
            per = c["heads"] // c["kv_heads"]
            o = torch.stack([_attend(q[:, h], k[:, h // per], v[:, h // per], HEAD ** -0.5) for h in range(c["heads"])], 1)
            if cache:
                o = cache.rotate(o)
            x = x + o.reshape(T, -1) @ m["o"].T
            n = _rms(x, eps)
            xs[b] = x + (torch.nn.functional.silu(n @ m["g"].T) * (n @ m["u"].T)) @ m["d"].T
        del m
    return [_rms(x[-last:], eps) @ embed.T for x in xs]


def _rope_pairs(x, freqs, amp=1.0):
    """x [T, ..., d], neighbours paired, the first 2 len(freqs) of them turned."""
    a = torch.arange(x.shape[0], device="cuda", dtype=F64)[:, None] * freqs
    a = a.view((x.shape[0],) + (1,) * (x.dim() - 2) + (len(freqs),))
    co, si = torch.cos(a) * amp, torch.sin(a) * amp
    n = 2 * len(freqs)
    u, v = x[..., 0:n:2], x[..., 1:n:2]
    return torch.cat([torch.stack([u * co - v * si, v * co + u * si], -1).flatten(-2), x[..., n:]], -1)


def _frequencies(rot):
    d, base, sc = rot["dims"], float(rot["base"]), rot.get("scaling")
    f = base ** (-2.0 * torch.arange(d // 2, device="cuda", dtype=F64) / d)
    if not sc:
        return f, 1.0
    if "original" not in sc:
        return f / sc["factor"], 1.0
    at = lambda turns: d * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), d - 1)
    ramp = ((torch.arange(d // 2, device="cuda", dtype=F64) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def _latent64(h, W, m, eps, shared):
    H, d, vd, r = m["heads"], m["dim"], m["vdim"], m["kv_rank"]
    f, amp = _frequencies(m["rot"])
    q = (h @ W("q").T).view(len(h), H, -1)
    q = torch.cat([q[..., :d], _rope_pairs(q[..., d:], f, amp)], -1)
    dkv = h @ W("dkv").T
    lat = _rms(dkv[:, :r], eps) * W("dkv.norm")
    kr = _rope_pairs(dkv[:, r:], f, amp)
    k, v = (lat @ W("uk").T).view(len(h), H, d), (lat @ W("uv").T).view(len(h), H, vd)
    sink = W("sink")
    o = torch.stack([_attend(q[:, i], torch.cat([k[:, i], kr], -1), v[:, i], m["scale"], sink=sink[i]) for i in range(H)], 1)
    return o.flatten(1) @ W("o").T


def _recurrence(q, k, v, decay):
    """decay [T or 1, H, d]: S <- decay S + k v^T, o = S^T q."""
    S = torch.zeros((q.shape[1], q.shape[2], v.shape[2]), dtype=F64, device="cuda")
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = decay[t % len(decay)][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.bmm(q[t][:, None], S)[:, 0]
    return out


def _lightning64(h, W, m, eps, shared):
    silu = torch.nn.functional.silu
    H, T = m["heads"], len(h)
    q, k, v = (silu(h @ W(n).T).view(T, H, -1) for n in "qkv")
    dec = torch.tensor(m["decay"], dtype=F64, device="cuda")[None, :, None].expand(1, H, m["dim"])
    o = _rms(_recurrence(q, k, v, dec).flatten(1), eps) * W("norm") * torch.sigmoid(h @ W("g").T)
    return o @ W("o").T


def _grouped64(h, W, m, eps, shared):
    H, G, T = m["heads"], m["kv_heads"], len(h)
    f, _ = _frequencies(m["rot"])
    q = _rope_pairs(_rms((h @ W("q").T).view(T, H, -1), eps) * W("q.norm"), f)
    if m.get("kv_from") is None:
        shared["now"] = (_rope_pairs(_rms((h @ W("k").T).view(T, G, -1), eps) * W("k.norm"), f), (h @ W("v").T).view(T, G, -1))
    k, v = shared["now"] if m.get("kv_from") is None else shared[m["kv_from"]]
    start = torch.arange(T, device="cuda") // m["mask"]["size"] * m["mask"]["size"]
    sink = W("sink")
    o = torch.stack([_attend(q[:, i], k[:, i // (H // G)], v[:, i // (H // G)], m["scale"], start=start, sink=sink[i]) for i in range(H)], 1)
    return (o.flatten(1) * torch.sigmoid(h @ W("g").T)) @ W("o").T


def _gated64(h, W, m, eps, shared):
    H, d, T = m["heads"], m["dim"], len(h)
    q, k, v = (h @ W("q").T).view(T, H, d) / math.sqrt(d), (h @ W("k").T).view(T, H, d), (h @ W("v").T).view(T, H, -1)
    a = (torch.sigmoid(h @ W("a1").T @ W("a2").T + W("a2.b")) ** (1.0 / m["tau"])).view(T, H, d)
    o = (_rms(_recurrence(q, k, v, a), eps) * W("norm")).flatten(1) * torch.nn.functional.silu(h @ W("g").T)
    return o @ W("o").T


def _stack_forward(c, seed, tokens, last):
    j, w = _stack_json(c), _StackWeights(c, seed)
    get = lambda name: w.value(name).to(F64)  # noqa: E731
    eps = j["norm"]["eps"]
    mix = {"latent_attention": _latent64, "lightning": _lightning64, "attention": _grouped64, "gla": _gated64}
    post = c["design"] == "luvatar"
    x = get("embed")[torch.from_numpy(tokens.astype(np.int64)).cuda()]
    x = x * j["embedding"]["scale"] if post else _rms(x, eps) * get("embed.norm")
    x0, shared = x, {}
    loop = j.get("loop") or {"start": 0, "stop": 0, "times": 0}
    order = [(i, -1) for i in range(loop["start"])] + [(i, p) for p in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
    order += [(i, -1) for i in range(loop["stop"], len(j["layers"]))]
    for i, p in order:
        if p >= 0 and i == loop["start"]:
            x = torch.cat([x, x0], -1) @ get("loop.in").T + get("loop.step")[p]
        L = j["layers"][i]
        h = x if post else _rms(x, eps) * get("l%d.norm1" % i)
        y = mix[L["type"]](h, lambda n: get("l%d.mix.%s" % (i, n)), L["mixer"], eps, shared)
        shared[i] = shared.get("now")
        if post:
            x = h = x + _rms(y, eps) * get("l%d.norm1" % i)
        act = torch.nn.functional.silu(h @ get("l%d.mlp.gate" % i).T) if post else torch.nn.functional.gelu(h @ get("l%d.mlp.gate" % i).T, approximate="tanh")
        f = (act * (h @ get("l%d.mlp.up" % i).T)) @ get("l%d.mlp.down" % i).T
        x = x + _rms(f, eps) * get("l%d.norm2" % i) if post else x + y + f
    z = (_rms(x[-last:], eps) * get("final.norm")) @ get("embed" if post else "head").T
    cap = j.get("logit_softcap")
    return cap * torch.tanh(z / cap) if cap else z


def exact(case, seed):
    c = case
    if c["kind"] == "quantize":
        s = prepare(c, seed)
        x = s["w"].to(F64) * (s["awq"].to(F64) if c["awq"] else 1.0)
        G = -(-c["cols"] // GROUP)
        lo, hi = (torch.stack([fn(p, -1) for p in x.split(GROUP, 1)], 1) for fn in (torch.amin, torch.amax))
        scale = (hi - lo) / (2 ** c["bits"] - 1)
        # the zero point is a rounded value, the codes are whole: no nearer value exists
        return {"codes": None, "scales": scale.view(c["rows"], G), "zeros": None}
    if c["kind"] == "attention":
        t, ctx, n, g = _Cache64(c["bits"], seed), c["ctx"], c["seqs"], c["kv_heads"]
        k = _randn(seed, "k", n * ctx, g, HEAD).half().to(F64).view(n, ctx, g, HEAD)
        v = _randn(seed, "v", n * ctx, g, HEAD).half().to(F64).view(n, ctx, g, HEAD)
        q = t.rotate(_randn(seed, "q", n, c["heads"], HEAD).half().to(F64))
        out = torch.empty((n, c["heads"], HEAD), dtype=F64, device="cuda")
        for i, length in enumerate(_lengths(seed, n, ctx, c["ragged"])):
            for h in range(g):
                kk, vv = t.keys(k[i, :length, h]), t.values(v[i, :length, h])
                for r in range(c["heads"] // g):
                    a = h * (c["heads"] // g) + r
                    out[i, a] = _attend(q[i, a][None], kk, vv, HEAD ** -0.5, first=length - 1)[0]
        return t.rotate(out)
    if c["kind"] == "decode":
        prompts, fed = _tokens(seed, "prompt", c["vocab"], c["batch"], c["ctx"]), _tokens(seed, "fed", c["vocab"], c["steps"], c["batch"])
        rows = _quantized_forward(c, seed, [np.concatenate([prompts[b], fed[:, b]]) for b in range(c["batch"])], c["steps"])
        return [rows[0][i] if c["batch"] == 1 else torch.stack([r[i] for r in rows]) for i in range(c["steps"])]
    if c["kind"] == "prefill":
        return _quantized_forward(c, seed, [_tokens(seed, "prompt", c["vocab"], c["tokens"])], 1)[0][0]
    if c["kind"] == "prompt":
        return _stack_forward(c, seed, _tokens(seed, "prompt0", 32768, c["tokens"]), 1)[0]
    fed = _tokens(seed, "fed", 32768, c["steps"], c["seqs"])
    rows = [_stack_forward(c, seed, np.concatenate([_tokens(seed, "prompt%d" % i, 32768, n), fed[:, i]]), c["steps"])
            for i, n in enumerate(_lengths(seed, c["seqs"], c["prompt"]))]
    return [torch.stack([r[i] for r in rows]) for i in range(c["steps"])]
