"""Workloads of the compressed KV cache that its performance is judged on.

Every case goes through the package's public entry points the way a program that uses them does.  `listed()`
names the fixed ones, `draw(rng)` gives further cases of the same kinds and ranges.  A case is a dict of plain
values; its "op" selects the path:

  step        one decode step of one layer, issued from Python: KVCacheManager.append of one token, then attend
  graph       the same step for all layers of a decoder, recorded once as a CUDA graph (position and length on the
              device) and replayed per token
  decode      decode attention through a prepared call (attention.prepare_decode), as a serving loop keeps it
  attention   attention.compressed_attention on a finished cache, with or without the key sketch
  prefill     attention.prefill_attention: a chunk of query positions against a longer cache
  prompt      a prompt's first pass through one layer: KVCacheManager.append of all its tokens, then causal attend
  compress    quantizer.compress of a key tensor (with its residual sketch) and of a value tensor
  decompress  compressor.decompress of a whole cache to float16
  bridge      the llama.cpp bridge's calls for one token of one layer: compress the new key and value, rotate the
              query, attend, rotate back
  bridge_compress   the bridge's compress of a prompt's keys

Keys and values are normal with a log-normal scale per channel and two channels ten times larger, as measured
KV tensors look; queries are normal.
"""

from __future__ import annotations

import functools
import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "polarquant-kv_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(1, _PACKAGE)

from polarquant_kv import attention, compressor, llama_bridge, quantizer  # noqa: E402
from polarquant_kv.codebook import build_lloyd_max_codebook  # noqa: E402
from polarquant_kv.inference import KVCacheManager, PolarQuantConfig  # noqa: E402
from polarquant_kv.qjl import generate_jl_matrix  # noqa: E402
from polarquant_kv.rotation import device_plan, generate_rotation_matrix  # noqa: E402

DEVICE = "cuda"
ROTATION_SEED, JL_SEED = 42, 1


def listed():
    return [
        # The smallest call there is: a chat of one user with a small model (14 query and 2 KV heads of 64), one
        # token, one layer.  Latency of three kernels and of the host code around them.
        {"name": "one token, one layer", "op": "step", "batch": 1, "kv_heads": 2, "q_heads": 14, "head_dim": 64,
         "seq": 511, "capacity": 1024, "k_bits": 4, "v_bits": 4},
        # A decode step of a batch of 64 over all layers' caches as generate_graph replays it.
        {"name": "graph step, 16 layers", "op": "graph", "layers": 16, "batch": 64, "kv_heads": 2, "q_heads": 14,
         "head_dim": 64, "seq": 4096, "capacity": 4352, "k_bits": 4, "v_bits": 4},
        # The benchmark's headline: an 8B-class model (32 query, 8 KV heads of 128), 32 sequences of 8192 tokens.
        {"name": "decode 32 x 8192", "op": "decode", "batch": 32, "kv_heads": 8, "q_heads": 32, "head_dim": 128,
         "seq": 8192, "capacity": 8192, "k_bits": 4, "v_bits": 4},
        # One very long sequence, eight query heads per KV head (a 70B-class model reading a book).
        {"name": "decode 1 x 131072", "op": "decode", "batch": 1, "kv_heads": 8, "q_heads": 64, "head_dim": 128,
         "seq": 131072, "capacity": 131072, "k_bits": 4, "v_bits": 4},
        # The facade with everything switched on: key sketch, 2-bit values, a length off every tile boundary.
        {"name": "sketched attention 4 x 4099", "op": "attention", "batch": 4, "kv_heads": 8, "q_heads": 32,
         "head_dim": 128, "seq_q": 1, "seq": 4099, "capacity": 4099, "k_bits": 4, "v_bits": 2, "jl_dim": 128},
        # A chunk of a long prompt (chunked prefill), 2 sequences x 512 positions against 4096 tokens.
        {"name": "prefill chunk 512 of 4096", "op": "prefill", "batch": 2, "kv_heads": 8, "q_heads": 32,
         "head_dim": 128, "seq_q": 512, "seq": 4096, "capacity": 4096, "k_bits": 4, "v_bits": 4, "causal": True},
        # Verification of a handful of drafted tokens (speculative decoding), ragged length.
        {"name": "verify 5 drafted tokens", "op": "prefill", "batch": 8, "kv_heads": 8, "q_heads": 32,
         "head_dim": 128, "seq_q": 5, "seq": 3001, "capacity": 4096, "k_bits": 4, "v_bits": 4, "causal": True},
        # First pass over 16 prompts of 4096 tokens, one layer of the small model.
        {"name": "prompt 16 x 4096", "op": "prompt", "batch": 16, "kv_heads": 2, "q_heads": 14, "head_dim": 64,
         "seq": 4096, "capacity": 4352, "k_bits": 4, "v_bits": 4},
        # Bulk compression of keys with the 128-projection sketch and of values.
        {"name": "compress 2^21 keys and values", "op": "compress", "batch": 16, "kv_heads": 8, "seq": 16384,
         "head_dim": 128, "k_bits": 4, "v_bits": 4, "jl_dim": 128},
        # A cache handed back as float16 (what the Hugging Face adapter does on every update).
        {"name": "decompress 2^20 vectors", "op": "decompress", "batch": 16, "kv_heads": 8, "seq": 8192,
         "head_dim": 128, "k_bits": 4},
        # llama.cpp: one token of one layer of an 8B-class model at 32768 tokens of context ...
        {"name": "bridge token at 32768", "op": "bridge", "kv_heads": 8, "q_heads": 32, "head_dim": 128, "seq": 32768},
        # ... and the keys of a prompt of 16384 tokens.
        {"name": "bridge prompt 16384", "op": "bridge_compress", "kv_heads": 8, "head_dim": 128, "seq": 16384},
    ]


# ----------------------------------------------------------------------------------------------- drawn cases
_OPS = ["step", "step", "graph", "decode", "decode", "decode", "attention", "attention", "prefill", "prefill", "prompt",
        "compress", "decompress", "bridge", "bridge_compress"]
_CACHE_BYTES = 300e6          # most compressed bytes of one attention call, as the largest listed one
_ATTENTION_FLOPS = 200e9      # most multiply-adds x 2 of one prefill call
_VECTORS = 1 << 21            # most vectors per tensor of a compress call


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _token_bytes(c):
    return (c["head_dim"] // 32) * ((2 + 4 * c["k_bits"]) + (2 + 4 * c["v_bits"]))


def draw(rng):
    op = rng.choice(_OPS)
    c = {"op": op, "kv_heads": rng.choice([1, 2, 4, 8]), "head_dim": rng.choice([64, 128, 128])}
    group = rng.choice([1, 2, 3, 4, 4, 5, 7, 8])
    if op in ("bridge", "bridge_compress"):
        c["kv_heads"] = rng.choice([2, 4, 8])
        if op == "bridge":
            c["q_heads"] = c["kv_heads"] * rng.choice([1, 4, 4, 8])
            c["seq"] = _log(rng, 200, 65536)
        else:
            c["seq"] = _log(rng, 16, 32768)
        return c
    c["k_bits"] = rng.choice([4, 4, 4, 2])
    if op == "decompress":
        c["batch"] = _log(rng, 1, 32)
        c["seq"] = _log(rng, 16, max(17, (1 << 20) // (c["batch"] * c["kv_heads"])))
        return c
    c["v_bits"] = rng.choice([4, 4, 2]) if c["k_bits"] == 4 else 2
    if op == "compress":
        c["batch"] = _log(rng, 1, 32)
        c["seq"] = _log(rng, 1, max(2, _VECTORS // (c["batch"] * c["kv_heads"])))
        c["jl_dim"] = rng.choice([0, 64, 128])
        return c
    c["q_heads"] = c["kv_heads"] * group
    c["batch"] = _log(rng, 1, 64)
    rows = c["batch"] * c["kv_heads"]
    longest = int(_CACHE_BYTES / (rows * _token_bytes(c)))
    if op == "graph":
        c["layers"] = rng.randint(2, 16)
        longest = min(longest, int(8 * _CACHE_BYTES / (3 * c["layers"] * rows * _token_bytes(c))))
    c["seq"] = _log(rng, 64, max(65, min(131072 if op == "decode" else 16384, longest)))
    if op in ("prefill", "prompt", "attention"):
        # (query positions, cache length) within the arithmetic limit
        c["seq"] = min(c["seq"], 8192)
        unit = 4.0 * c["batch"] * c["q_heads"] * c["head_dim"]
        if op == "prompt":
            c["seq"] = max(2, min(c["seq"], int(math.sqrt(2 * _ATTENTION_FLOPS / unit))))
        else:
            most = max(2, min(c["seq"], 2048, int(_ATTENTION_FLOPS / (unit * c["seq"]))))
            c["seq_q"] = _log(rng, 2, most) if op == "prefill" or rng.random() < 0.5 else 1
            c["causal"] = op == "prefill" and rng.random() < 0.8
        if op == "attention":
            c["jl_dim"] = rng.choice([0, 64, 128]) if c["seq_q"] == 1 else 0
    # caches are reserved in advance, in whole pages of 256 tokens with room for more, or hold exactly one prompt
    c["capacity"] = c["seq"] if rng.random() < 0.3 else (c["seq"] // 256 + 1) * 256
    if op in ("step", "graph"):
        c["capacity"] = (c["seq"] // 256 + 1) * 256
    return c


# ----------------------------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _rotation(d):
    return generate_rotation_matrix(d, seed=ROTATION_SEED)


@functools.lru_cache(maxsize=None)
def _projection(m, d):
    return generate_jl_matrix(m, d, seed=JL_SEED)


@functools.lru_cache(maxsize=None)
def _bridge_constants(d):
    codebook = torch.from_numpy(build_lloyd_max_codebook(d, 4)[0]).to(DEVICE)
    return torch.from_numpy(_rotation(d)).to(device=DEVICE, dtype=torch.float32).contiguous(), codebook


class _Inputs:
    """Tensors drawn on the device from one seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEVICE)
        self.gen.manual_seed(seed)

    def normal(self, *shape):
        return torch.randn(shape, generator=self.gen, device=DEVICE)

    def channels(self, d):
        scale = torch.exp(self.normal(d))
        scale[torch.randperm(d, generator=self.gen, device=DEVICE)[:2]] *= 10.0
        return scale

    def kv(self, *shape, dtype=torch.float16):
        scale = self.channels(shape[-1])
        out = torch.empty(shape, dtype=dtype, device=DEVICE)
        flat = out.view(-1, shape[-1])
        for lo in range(0, flat.shape[0], 1 << 19):
            hi = min(flat.shape[0], lo + (1 << 19))
            flat[lo:hi] = self.normal(hi - lo, shape[-1]) * scale
        return out

    def query(self, *shape):
        return self.normal(*shape).to(torch.float16)

    def cache(self, c, bits, jl_dim=0):
        """A filled cache of c's shape, compressed from this generator's keys or values."""
        R = _rotation(c["head_dim"])
        P = _projection(jl_dim, c["head_dim"]) if jl_dim else None
        out = quantizer.allocate_cache(c["batch"], c["kv_heads"], c["capacity"], c["head_dim"], bits, jl_dim, DEVICE)
        x = self.kv(c["batch"], c["kv_heads"], c["seq"], c["head_dim"])
        return quantizer.compress(x, R, bits, jl_matrix=P, out=out, position=0)

    def manager(self, c, tokens):
        config = PolarQuantConfig(n_bits=c["k_bits"], v_bits=c["v_bits"])
        m = KVCacheManager(config, c["capacity"], c["batch"], c["kv_heads"], c["head_dim"], DEVICE, ROTATION_SEED)
        if tokens:
            shape = (c["batch"], c["kv_heads"], tokens, c["head_dim"])
            m.append(self.kv(*shape), self.kv(*shape))
        return m


def prepare(case, seed):
    c, x = case, _Inputs(seed)
    op = c["op"]
    s = {"op": op}
    if op in ("step", "prompt"):
        new = 1 if op == "step" else c["seq"]
        s["kept"] = c["seq"] if op == "step" else 0
        s["manager"] = x.manager(c, s["kept"])
        s["k"] = x.kv(c["batch"], c["kv_heads"], new, c["head_dim"])
        s["v"] = x.kv(c["batch"], c["kv_heads"], new, c["head_dim"])
        s["q"] = x.query(c["batch"], c["q_heads"], new, c["head_dim"])
    elif op == "graph":
        managers = [x.manager(c, c["seq"]) for _ in range(c["layers"])]
        k = [x.kv(c["batch"], c["kv_heads"], 1, c["head_dim"]) for _ in managers]
        v = [x.kv(c["batch"], c["kv_heads"], 1, c["head_dim"]) for _ in managers]
        q = [x.query(c["batch"], c["q_heads"], 1, c["head_dim"]) for _ in managers]
        position = torch.full((1,), c["seq"], dtype=torch.int64, device=DEVICE)
        length = position + 1

        def step():
            outs = []
            for i, m in enumerate(managers):
                m.append(k[i], v[i], position=position)
                outs.append(m.attend(q[i], seq_len_tensor=length))
            return outs

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
        torch.cuda.current_stream().wait_stream(side)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            outs = step()
        appended = [cache.blocks[:, :, c["seq"]] for m in managers for cache in m.get_kv()]
        s["out"] = {"attention": outs, "appended": appended}
        s["keep"] = (managers, k, v, q, position, length)
    elif op == "decode":
        ck, cv = x.cache(c, c["k_bits"]), x.cache(c, c["v_bits"])
        q = x.query(c["batch"], c["q_heads"], c["head_dim"])
        s["call"] = attention.prepare_decode(q, ck, cv, device_plan(_rotation(c["head_dim"]), DEVICE))
    elif op == "attention":
        s["ck"], s["cv"] = x.cache(c, c["k_bits"], c["jl_dim"]), x.cache(c, c["v_bits"])
        s["q"] = x.query(c["batch"], c["q_heads"], c["seq_q"], c["head_dim"])
        s["R"] = _rotation(c["head_dim"])
        s["P"] = _projection(c["jl_dim"], c["head_dim"]) if c["jl_dim"] else None
    elif op == "prefill":
        s["ck"], s["cv"] = x.cache(c, c["k_bits"]), x.cache(c, c["v_bits"])
        s["q"] = x.query(c["batch"], c["q_heads"], c["seq_q"], c["head_dim"])
        s["plan"] = device_plan(_rotation(c["head_dim"]), DEVICE)
        s["causal"] = c["causal"]
    elif op == "compress":
        shape = (c["batch"], c["kv_heads"], c["seq"], c["head_dim"])
        s["k"], s["v"] = x.kv(*shape), x.kv(*shape)
        s["R"], s["k_bits"], s["v_bits"] = _rotation(c["head_dim"]), c["k_bits"], c["v_bits"]
        s["P"] = _projection(c["jl_dim"], c["head_dim"]) if c["jl_dim"] else None
    elif op == "decompress":
        s["cache"] = x.cache(dict(c, capacity=c["seq"]), c["k_bits"])
        s["R"] = _rotation(c["head_dim"])
    elif op == "bridge":
        s["R"], s["codebook"] = _bridge_constants(c["head_dim"])
        d, s["slot"], s["scale"] = c["head_dim"], c["seq"] - 1, 1.0 / math.sqrt(c["head_dim"])
        for name in ("k", "v"):
            radius, packed = llama_bridge.compress(x.kv(c["kv_heads"] * c["seq"], d, dtype=torch.float32), s["R"], s["codebook"])
            s[name + "_radius"] = radius.view(c["kv_heads"], c["seq"])
            s[name + "_packed"] = packed.view(c["kv_heads"], c["seq"], d // 2)
            s[name] = x.kv(c["kv_heads"], d, dtype=torch.float32)
        s["q"] = x.normal(c["q_heads"], d)
    elif op == "bridge_compress":
        s["R"], s["codebook"] = _bridge_constants(c["head_dim"])
        s["k"] = x.kv(c["kv_heads"] * c["seq"], c["head_dim"], dtype=torch.float32)
    else:
        raise ValueError(f"unknown op {op!r}")
    return s


# ----------------------------------------------------------------------------------------------- one pass
def run(state):
    s = state
    op = s["op"]
    if op in ("step", "prompt"):
        m = s["manager"]
        m.reset()
        m.advance(s["kept"])                 # the tokens before this pass are in place
        m.append(s["k"], s["v"])
        out = m.attend(s["q"], causal=True)
        ck, cv = m.get_kv()
        return {"attention": out, "keys": ck.blocks, "values": cv.blocks}
    if op == "graph":
        s["graph"].replay()
        return s["out"]
    if op == "decode":
        return s["call"]()
    if op == "attention":
        return attention.compressed_attention(s["q"], s["ck"], s["cv"], s["R"], s["P"])
    if op == "prefill":
        return attention.prefill_attention(s["q"], s["ck"], s["cv"], s["plan"], causal=s["causal"])
    if op == "compress":
        k = quantizer.compress(s["k"], s["R"], s["k_bits"], jl_matrix=s["P"])
        v = quantizer.compress(s["v"], s["R"], s["v_bits"])
        return {"keys": k.blocks, "signs": k.qjl_signs, "norms": k.residual_norms, "values": v.blocks}
    if op == "decompress":
        return compressor.decompress(s["cache"], s["R"])
    if op == "bridge":
        R, codebook, slot = s["R"], s["codebook"], s["slot"]
        for name in ("k", "v"):
            radius, packed = llama_bridge.compress(s[name], R, codebook)
            s[name + "_radius"][:, slot] = radius
            s[name + "_packed"][:, slot] = packed
        q = llama_bridge.rotate_query(s["q"], R)
        out = llama_bridge.fused_attention(q, s["k_packed"], s["k_radius"], s["v_packed"], s["v_radius"], codebook, s["scale"])
        return {"attention": llama_bridge.inverse_rotate(out, R), "keys": s["k_packed"], "key radii": s["k_radius"],
                "values": s["v_packed"], "value radii": s["v_radius"]}
    if op == "bridge_compress":
        radius, packed = llama_bridge.compress(s["k"], s["R"], s["codebook"])
        return {"radius": radius, "packed": packed}
    raise ValueError(f"unknown op {op!r}")


# ----------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    """What one pass cannot do without: stored or given bytes read once, results written once; the arithmetic of
    the attention scores and sums, and of the rotations of what is stored or handed back."""
    c = case
    op, d, kv = c["op"], c["head_dim"], c["kv_heads"]
    if op == "bridge_compress":
        n = kv * c["seq"]
        return {"bytes": n * (4 * d + d // 2 + 4) + 4 * d * d, "flops": 2 * n * d * d}
    if op == "bridge":
        stored, hq = 2 * kv * c["seq"] * (d // 2 + 4), c["q_heads"]
        return {"bytes": stored + 2 * kv * (4 * d + d // 2 + 4) + 2 * hq * 4 * d + 4 * d * d,
                "flops": 4 * hq * c["seq"] * d + 2 * (2 * kv + 2 * hq) * d * d}
    blocks = d // 32
    kb = blocks * (2 + 4 * c["k_bits"])
    rows = c["batch"] * kv
    if op == "decompress":
        n = rows * c["seq"]
        return {"bytes": n * (kb + 2 * d), "flops": 2 * n * d * d}
    vb = blocks * (2 + 4 * c["v_bits"])
    if op == "compress":
        n, jl = rows * c["seq"], c["jl_dim"]
        return {"bytes": n * (4 * d + kb + vb + (jl // 8 + 2 if jl else 0)), "flops": n * (4 * d * d + 2 * d * jl)}
    hq, layers = c["batch"] * c["q_heads"], c.get("layers", 1)
    if op in ("step", "graph"):
        attended, positions, appended = c["seq"] + 1, 1, 1
        pairs = attended
    elif op == "prompt":
        attended = positions = appended = c["seq"]
        pairs = attended * (attended + 1) // 2
    else:
        attended, positions, appended = c["seq"], c.get("seq_q", 1), 0
        pairs = attended * positions
        if c.get("causal"):
            seen_by_last = min(positions, attended)
            pairs = seen_by_last * (2 * attended - seen_by_last + 1) // 2
    sketch = (c["jl_dim"] // 8 + 2) if c.get("jl_dim") else 0
    per_token = kb + vb + sketch
    flops = 4 * hq * pairs * d + 4 * hq * positions * d * d + 4 * rows * appended * d * d
    if sketch:
        flops += 2 * hq * (pairs + positions * d) * c["jl_dim"]
    data = rows * attended * per_token + 6 * hq * positions * d + rows * appended * 4 * d
    return {"bytes": layers * data, "flops": layers * flops}


def tolerance(case):
    """Attention accumulates in float32 over operands carried with about 22 bits or more, and its softmax turns an
    absolute error of a score into a relative one of a weight.  Stored bytes come from comparisons of float32 numbers
    with decision boundaries and from float16 roundings: two correct summation orders differ at ties only."""
    op = case["op"]
    if op == "decompress":
        return {"rel": 5e-4, "max": 2e-3}                  # one rounding to float16
    if op == "compress":
        return {"rel": 5e-4, "max": 2e-3, "differ": 1e-4}   # norms are float16
    if op == "bridge_compress":
        return {"rel": 2e-6, "max": 2e-5, "differ": 1e-4}
    if op in ("prefill", "prompt", "attention"):
        return {"rel": 5e-5, "max": 2e-3, "differ": 1e-4}
    return {"rel": 2e-5, "max": 1e-3, "differ": 1e-4}
