"""The work a user of this library has it do, as cases that can be timed.

A case is one submission of a model's forward pass: a single projection, the projections of a dense layer at decode,
verify or prefill width, a mixture-of-experts block, an output head, a feed-forward block in a 4-bit codebook format.
Shapes are those of the benchmark: a dense 27B-class layer (hidden 5120, attention width 6144, feed-forward 17408,
Q4_K with a Q6_K down projection) and a 35B-A3B-class expert block (hidden 2048, 256 experts of width 512, top 8).

What a decoding program records once and replays for every token -- a step of a few activation rows -- is a captured
graph here too; prompt-sized work is enqueued call by call.
"""
import math

import torch

from ferrum_b200 import surface as S

Q8_0, Q4_K, Q5_K, Q6_K, IQ4_NL, IQ4_XS = 8, 12, 13, 14, 20, 23
BLOCK = {Q8_0: (32, 34), Q4_K: (256, 144), Q5_K: (256, 176), Q6_K: (256, 210), IQ4_NL: (32, 18), IQ4_XS: (256, 136)}
EPS = 1e-6
VOCAB = 4096  # rows of the embedding table the steps look their tokens up in


def listed():
    dense = {"hidden": 5120, "attn": 6144, "kv": 1024, "ffn": 17408, "fmt": Q4_K, "down": Q6_K}
    moe = {"hidden": 2048, "experts": 256, "used": 8, "ffn": 512}
    return [
        # One projection of a 4096-wide model, enqueued by itself: what a call costs.
        {"name": "call_q4k_m1", "kind": "call", "rows": 4096, "cols": 4096, "fmt": Q4_K, "m": 1},
        # A decode step of one sequence: the embedding lookup and two layers' projections, norms and feed-forward blocks.
        {"name": "decode_m1", "kind": "step", "layers": 2, "m": 1, **dense},
        # The same layers verifying a draft of eight and of sixteen tokens (or decoding that many sequences).
        {"name": "verify_m8", "kind": "step", "layers": 2, "m": 8, **dense},
        {"name": "verify_m16", "kind": "step", "layers": 2, "m": 16, **dense},
        # A prompt through one layer's projections in bf16: a full chunk, and the ragged rest of a shorter prompt.
        {"name": "prefill_bf16_2048", "kind": "prefill", "m": 2048, **dense},
        {"name": "prefill_bf16_509", "kind": "prefill", "m": 509, **dense},
        # A prompt through one layer in F32, the hybrid engine's own activation type.
        {"name": "prefill_f32_512", "kind": "prefill_f32", "m": 512, **dense},
        # A mixture-of-experts block: one token, a small ragged batch, a prompt chunk.
        {"name": "moe_t1", "kind": "moe", "m": 1, **moe},
        {"name": "moe_t21", "kind": "moe", "m": 21, **moe},
        {"name": "moe_t1024", "kind": "moe", "m": 1024, **moe},
        # Greedy sampling of one token: the final norm, a Q8_0 output head over the whole vocabulary, the argmax.
        {"name": "head_q8_m1", "kind": "head", "rows": 151936, "cols": 2048, "fmt": Q8_0, "m": 1},
        # A feed-forward block of a model stored in IQ4_XS, four sequences decoding together.
        {"name": "ffn_iq4xs_m4", "kind": "ffn", "hidden": 5120, "ffn": 17408, "fmt": IQ4_XS, "down": IQ4_XS, "m": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    wide = lambda lo, hi: 256 * max(1, int(round(_log(rng, lo, hi) / 256)))  # a whole number of superblocks
    kind = rng.choice(["call", "call", "step", "step", "prefill", "prefill_f32", "moe", "moe", "head", "ffn"])
    if kind == "call":
        return {"kind": kind, "rows": _log(rng, 1024, 32768), "cols": wide(1024, 12288),
                "fmt": rng.choice([Q4_K, Q4_K, Q6_K, Q6_K, Q5_K, Q8_0, IQ4_XS, IQ4_NL]), "m": rng.choice([1, 1, 1, _log(rng, 2, 16)])}
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 32000, 151936), "cols": wide(1024, 5120), "fmt": rng.choice([Q8_0, Q6_K]),
                "m": rng.choice([1, 1, _log(rng, 2, 8)])}
    if kind == "ffn":
        fmt = rng.choice([IQ4_XS, IQ4_NL])
        return {"kind": kind, "hidden": wide(1024, 5120), "ffn": wide(2816, 17408), "fmt": fmt, "down": fmt, "m": _log(rng, 1, 16)}
    if kind == "moe":
        used = rng.choice([4, 8])
        return {"kind": kind, "m": rng.choice([1, _log(rng, 2, 1024)]), "hidden": wide(1024, 2048), "experts": rng.choice([64, 128, 256]),
                "used": used, "ffn": wide(256, 768)}
    hidden = wide(1024, 5120)
    fmt = rng.choice([Q4_K, Q4_K, Q4_K, Q5_K, Q6_K])
    dense = {"hidden": hidden, "attn": wide(1024, 6144), "kv": rng.choice([256, 512, 1024]), "ffn": wide(2816, 17408), "fmt": fmt, "down": Q6_K}
    if kind == "step":
        return {"kind": kind, "layers": rng.choice([1, 2]), "m": rng.choice([1, _log(rng, 2, 16)]), **dense}
    return {"kind": kind, "m": _log(rng, 17, 2048 if kind == "prefill" else 640), **dense}


# ---------------------------------------------------------------- weights and handles

_device = None


def device():
    """The process's one handle, on its own stream (graphs are captured there)."""
    global _device
    if _device is None:
        _device = S.Device(0, use_torch_stream=False)
    return _device


def packed(gen, fmt, values):
    """Blocks whose decoded weights are centred with a deviation of about 0.02, as a model's are: uniform quants and
    sub-scales, the superblock scales spread over a factor of three, the minimums at half of the quants' range."""
    elems, size = BLOCK[fmt]
    n = values // elems
    out = torch.randint(0, 256, (n, size), dtype=torch.uint8, device="cuda", generator=gen)
    spread = torch.rand(n, device="cuda", generator=gen) + 0.5
    half = lambda v: v.to(torch.float16).view(torch.uint8).reshape(n, 2)
    if fmt == Q4_K or fmt == Q5_K:
        d = spread * (1.4e-4 if fmt == Q4_K else 7e-5)
        out[:, 0:2], out[:, 2:4] = half(d), half(d * (7.5 if fmt == Q4_K else 15.5))
    elif fmt == Q6_K:
        out[:, 208:210] = half(spread * 1.5e-5)
    elif fmt == Q8_0:
        out[:, 0:2] = half(spread * 2.7e-4)
        q = out[:, 2:]
        q[q == 128] = 127  # -128 is outside the format
    else:
        out[:, 0:2] = half(spread * (2.7e-4 if fmt == IQ4_NL else 1.5e-5))
    return out.reshape(-1).cpu().numpy()


def matrix(gen, fmt, rows, cols, experts=1):
    return S.Matrix.from_packed(device(), rows, cols, experts, fmt, packed(gen, fmt, rows * cols * experts))


def nbytes(fmt, rows, cols):
    elems, size = BLOCK[fmt]
    return rows * cols // elems * size


def dense_shapes(c):
    """The matrices of one layer: name -> (rows, cols, format)."""
    h, a, kv, f = c["hidden"], c["attn"], c["kv"], c["ffn"]
    return {"q": (a, h, c["fmt"]), "k": (kv, h, c["fmt"]), "v": (kv, h, c["fmt"]), "o": (h, a, c["fmt"]),
            "gate": (f, h, c["fmt"]), "up": (f, h, c["fmt"]), "down": (h, f, c["down"])}


# ---------------------------------------------------------------- one pass

def prepare(case, seed):
    c, dev = dict(case), device()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 1000003 + 17)
    m = c["m"]
    randn = lambda *shape: torch.randn(shape, device="cuda", generator=gen)
    zeros = lambda *shape: torch.zeros(shape, device="cuda")
    weight = lambda n: 1.0 + 0.1 * torch.randn(n, device="cuda", generator=gen)
    s = {"c": c, "kind": c["kind"], "m": m}
    if c["kind"] == "call":
        s["w"] = matrix(gen, c["fmt"], c["rows"], c["cols"])
        s["x"], s["y"] = randn(m, c["cols"]), zeros(m, c["rows"])
    elif c["kind"] == "head":
        s["w"] = matrix(gen, c["fmt"], c["rows"], c["cols"])
        s["x"], s["norm"], s["n"], s["y"] = randn(m, c["cols"]), weight(c["cols"]), zeros(m, c["cols"]), zeros(m, c["rows"])
        s["token"] = torch.zeros(m, dtype=torch.int32, device="cuda")
    elif c["kind"] == "ffn":
        s["gate"], s["up"] = matrix(gen, c["fmt"], c["ffn"], c["hidden"]), matrix(gen, c["fmt"], c["ffn"], c["hidden"])
        s["down"] = matrix(gen, c["down"], c["hidden"], c["ffn"])
        s["x"], s["scratch"], s["y"] = randn(m, c["hidden"]), zeros(3 * m * c["ffn"]), zeros(m, c["hidden"])
    elif c["kind"] == "moe":
        h, e, f = c["hidden"], c["experts"], c["ffn"]
        s["moe"] = S.MoeFfn(matrix(gen, Q8_0, e, h), matrix(gen, Q4_K, f, h, e), matrix(gen, Q4_K, f, h, e), matrix(gen, Q6_K, h, f, e),
                            matrix(gen, Q4_K, f, h), matrix(gen, Q4_K, f, h), matrix(gen, Q6_K, h, f), 0.02 * randn(h), e, c["used"], h, f, f,
                            False, True)
        s["x"], s["y"] = randn(m, h), zeros(m, h)
        s["scratch"] = zeros(S.moe_ffn_scratch_elems(dev, s["moe"], m))
    elif c["kind"] == "prefill":
        s["w"] = {n: matrix(gen, f, r, k) for n, (r, k, f) in dense_shapes(c).items()}
        s["y"] = {n: torch.zeros(m, r, dtype=torch.bfloat16, device="cuda") for n, (r, _, _) in dense_shapes(c).items()}
        s["x"] = {n: randn(m, k).to(torch.bfloat16) for n, k in (("h", c["hidden"]), ("a", c["attn"]), ("f", c["ffn"]))}
    else:  # step, prefill_f32
        h, a = c["hidden"], c["attn"]
        s["embed"] = matrix(gen, Q6_K, VOCAB, h)
        s["ids"] = torch.randint(0, VOCAB, (m,), dtype=torch.int32, device="cuda", generator=gen)
        s["layers"] = [{"w": {n: matrix(gen, f, r, k) for n, (r, k, f) in dense_shapes(c).items()},
                        "norm1": weight(h), "norm2": weight(h),
                        "attn": randn(m, a),  # what attention hands to the output projection
                        "q": zeros(m, a), "k": zeros(m, c["kv"]), "v": zeros(m, c["kv"]), "o": zeros(m, h), "h": zeros(m, h), "f": zeros(m, h),
                        "out": zeros(m, h)} for _ in range(c.get("layers", 1))]
        s["x"], s["n"], s["scratch"] = zeros(m, h), zeros(m, h), zeros(3 * m * c["ffn"])
        s["final"], s["last"] = weight(h), zeros(m, h)
    # A step of a few rows is recorded once and replayed; a single call and a prompt are enqueued.
    s["graph"] = None
    if c["kind"] in ("step", "head", "ffn") or (c["kind"] == "moe" and m <= 32):
        torch.cuda.synchronize()
        dev.capture_begin()
        enqueue(dev, s)
        s["graph"] = dev.capture_end()
    return s


def enqueue(dev, s):
    m, kind = s["m"], s["kind"]
    if kind == "call":
        S.project(dev, s["w"], s["x"], m, s["y"])
    elif kind == "head":
        S.rmsnorm_project_many(dev, [s["w"]], s["x"], s["norm"], EPS, m, [s["y"]], s["n"])
        S.argmax(dev, s["y"], s["w"].rows, m, s["token"])
    elif kind == "ffn":
        S.dense_ffn(dev, s["gate"], s["up"], s["down"], s["x"], m, s["scratch"], s["y"])
    elif kind == "moe":
        S.moe_ffn(dev, s["moe"], s["x"], m, s["scratch"], s["y"])
    elif kind == "prefill":
        w, x, y = s["w"], s["x"], s["y"]
        S.project_many(dev, [w["q"], w["k"], w["v"]], x["h"], m, [y["q"], y["k"], y["v"]])
        S.project(dev, w["o"], x["a"], m, y["o"])
        S.project_many(dev, [w["gate"], w["up"]], x["h"], m, [y["gate"], y["up"]])
        S.project(dev, w["down"], x["f"], m, y["down"])
    else:
        S.get_rows(dev, s["embed"], s["ids"], s["x"])
        x, f = s["x"], None
        for l in s["layers"]:
            w, qkv = l["w"], [l["q"], l["k"], l["v"]]
            if f is None:
                S.rmsnorm_project_many(dev, [w["q"], w["k"], w["v"]], x, l["norm1"], EPS, m, qkv, s["n"])
            else:
                S.add_rmsnorm(dev, x, f, l["norm1"], EPS, m, l["out"], s["n"])
                x = l["out"]
                S.project_many(dev, [w["q"], w["k"], w["v"]], s["n"], m, qkv)
            S.project(dev, w["o"], l["attn"], m, l["o"])
            S.add_rmsnorm(dev, x, l["o"], l["norm2"], EPS, m, l["h"], s["n"])
            S.dense_ffn(dev, w["gate"], w["up"], w["down"], s["n"], m, s["scratch"], l["f"])
            x, f = l["h"], l["f"]
        S.add_rmsnorm(dev, x, f, s["final"], EPS, m, s["last"], s["n"])


def run(s):
    dev = device()
    if s["graph"] is not None:
        s["graph"].launch()
    else:
        enqueue(dev, s)
    kind = s["kind"]
    if kind == "head":
        return [s["y"], s["token"]]
    if kind == "prefill":
        return s["y"]
    if kind in ("step", "prefill_f32"):
        return [[l[n] for n in ("q", "k", "v", "o", "h", "f")] for l in s["layers"]] + [s["last"], s["n"]]
    return s["y"]


# ---------------------------------------------------------------- what a pass cannot do without

def work(c):
    m, kind = c["m"], c["kind"]
    if kind in ("call", "head"):
        r, k = c["rows"], c["cols"]
        return {"bytes": nbytes(c["fmt"], r, k) + 4 * m * (r + k), "flops": 2 * m * r * k}
    if kind == "ffn":
        h, f = c["hidden"], c["ffn"]
        return {"bytes": 2 * nbytes(c["fmt"], f, h) + nbytes(c["down"], h, f) + 8 * m * h, "flops": 6 * m * h * f}
    if kind == "moe":
        h, e, f, used = c["hidden"], c["experts"], c["ffn"], c["used"]
        expert = 2 * nbytes(Q4_K, f, h) + nbytes(Q6_K, h, f)
        met = e * (1.0 - (1.0 - used / e) ** m)  # experts that at least one token is routed to, at random
        return {"bytes": (met + 1) * expert + nbytes(Q8_0, e, h) + 8 * m * h, "flops": 2 * m * ((used + 1) * 3 * h * f + e * h)}
    shapes = list(dense_shapes(c).values())
    weights, flops = sum(nbytes(f, r, k) for r, k, f in shapes), sum(2 * m * r * k for r, k, _ in shapes)
    if kind == "prefill":
        return {"bytes": weights + 2 * m * (c["hidden"] + c["attn"] + c["ffn"] + sum(r for r, _, _ in shapes)), "flops": flops}
    layers = c.get("layers", 1)
    io = 4 * m * (2 * c["attn"] + 2 * c["kv"] + 3 * c["hidden"])  # the attention output in; q, k, v and the residuals out
    return {"bytes": layers * (weights + io) + nbytes(Q6_K, m, c["hidden"]) + 8 * m * c["hidden"], "flops": layers * flops}


def tolerance(c):
    kind = c["kind"]
    if kind == "prefill":
        return {"rel": 1e-2}  # bf16 operands and results
    if kind == "moe" and c["m"] * c["used"] > 256:
        # Expert products on fp16 weights; and among this many tokens one may have its last two experts so close
        # that another order of summation in the router picks the other one.
        return {"rel": 1e-2, "max": 0.99}
    if kind == "head":
        return {"rel": 1e-4, "differ": 0.01}  # the token may differ where two logits tie
    # Activations carried to 16 bits of their superblock's maximum: 4e-5 a projection, and the chain of a layer.
    return {"rel": 1e-4} if kind == "call" else {"rel": 4e-4}
