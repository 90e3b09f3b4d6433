"""The workloads this framework's speed is judged by.

Every case goes through the public entry points of ``nnlib_jl_b200`` exactly as a user's program calls them:
``dot_product_attention`` (prefill, encoder, cross attention, one decode step, with and without the scores),
``dot_product_attention_pullback`` (one training step of the layer: output and all gradients), ``batched_mul`` and
``softmax`` / ``logsoftmax`` with their pullbacks.  Inputs are N(0, 1) (biases N(0, 0.5)), what normalised
activations look like; padded batches have lengths uniform in [L/2, L].

``listed()`` are the named cases, ``draw(rng)`` gives further ones of the same ranges: odd lengths, other head
sizes, every element type, each mask form, with and without bias and dropout.
"""
import math

import torch

import nnlib_jl_b200 as nb

_DTYPE = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32, "tf32": torch.float32}
_BYTES = {"bf16": 2, "f16": 2, "f32": 4, "tf32": 4}


def _attn(name, kind, dtype, d, H, Lq, Lkv, B, mask="none", bias="none", dropout=0.0):
    """kind: forward (x), scores (x and α), train (x and gradients).  dtype "tf32": Float32 arrays in fast math
    mode.  mask: none, causal, pad (key padding, one length per sample), window (causal, the last quarter of the
    keys; a Bool matrix).  bias: none, full (one value per score), heads (shared by the batch)."""
    return {"name": name, "kind": kind, "dtype": dtype, "d": d, "H": H, "Lq": Lq, "Lkv": Lkv, "B": B, "mask": mask,
            "bias": bias, "dropout": dropout}


def listed():
    return [
        # the reference's own default: Float32 arrays, a layer small enough to be tried out at the REPL, scores kept
        _attn("f32_small_scores", "scores", "f32", 64, 8, 128, 128, 4),
        # training such a Float32 model as it is, without opting into reduced precision
        _attn("f32_train_causal", "train", "f32", 64, 8, 512, 512, 8, mask="causal"),
        # a Float32 decoder layer whose user allows TF32 (CUDA.jl's FAST_MATH)
        _attn("tf32_prefill", "forward", "tf32", 128, 32, 4096, 4096, 2, mask="causal"),
        # BERT-base sized encoder layer over a padded batch, attention weights returned
        _attn("encoder_scores", "scores", "bf16", 64, 12, 512, 512, 32, mask="pad"),
        # prefill of a 7B-sized decoder layer
        _attn("prefill_4k", "forward", "bf16", 128, 32, 4096, 4096, 8, mask="causal"),
        # long-context prefill, the largest call
        _attn("prefill_32k", "forward", "bf16", 128, 16, 32768, 32768, 8, mask="causal"),
        # cross attention with an additive bias and attention dropout
        _attn("cross_bias_dropout", "forward", "f16", 64, 16, 256, 2048, 16, bias="full", dropout=0.1),
        # one generated token for each of eight sequences against an 8k history
        _attn("decode_8k", "forward", "bf16", 128, 32, 1, 8192, 8, mask="causal"),
        # one training step of the 7B-sized decoder layer
        _attn("train_4k", "train", "bf16", 128, 32, 4096, 4096, 8, mask="causal"),
        # one training step of an encoder-decoder's cross attention: lengths and head size of no particular
        # roundness, padded keys, dropout
        _attn("train_ragged", "train", "f16", 80, 8, 1000, 777, 6, mask="pad", dropout=0.1),
        # attention put together by hand from the building blocks: the logits batched_mul(kᵀ, q) of 64 heads
        {"name": "bmm_logits", "kind": "bmm", "dtype": "bf16", "M": 2048, "N": 2048, "K": 64, "batch": 64,
         "ta": True, "tb": False},
        # the loss side of a language model: logsoftmax over a vocabulary and its pullback
        {"name": "logsoftmax_vocab", "kind": "softmax", "dtype": "bf16", "log": True, "inner": 1, "n": 32000,
         "outer": 4096},
    ]


# --------------------------------------------------------------------------------------------------- drawn cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """Spread over the logarithm of the range; half of the lengths are multiples of 64, the others fall anywhere."""
    n = _log_int(rng, lo, hi)
    return max(64, n // 64 * 64) if rng.random() < 0.5 and hi >= 64 else n


# largest forward work (flops) of a drawn case: Float32 in exact arithmetic is what one does with small models
_CAP = {"bf16": 1.5e12, "f16": 1.5e12, "tf32": 2e11, "f32": 1e10}


def _fit(c):
    """Fewer sequences, then fewer heads, then shorter ones, until the case is within its range."""
    def too_much():
        scores = c["Lq"] * c["Lkv"] * c["H"] * c["B"]
        big = scores * _BYTES[c["dtype"]] if (c["kind"] == "scores" or c["bias"] == "full") else 0
        kv = (c["Lq"] + c["Lkv"]) * c["H"] * c["d"] * c["B"] * _BYTES[c["dtype"]]
        flops = 4 * c["d"] * scores * (4 if c["kind"] == "train" else 1)
        return flops > _CAP[c["dtype"]] or big > 1 << 30 or kv > 2 << 30
    while too_much():
        if c["B"] > 1:
            c["B"] //= 2
        elif c["H"] > 2:
            c["H"] //= 2
        else:
            c["Lq"], c["Lkv"] = max(1, c["Lq"] * 3 // 4), c["Lkv"] * 3 // 4
    return c


def _draw_attention(rng, kind):
    dtype = rng.choice(["bf16", "bf16", "bf16", "f16", "f16", "f32", "tf32"])
    d = rng.choice([64, 64, 64, 128, 128, 128, 32, 40, 80, 96])
    H = rng.choice([4, 8, 12, 16, 32])
    B = _log_int(rng, 1, 32)
    mask = rng.choice(["none", "causal", "causal", "pad", "window"])
    bias = rng.choice(["none", "none", "none", "none", "full", "heads"])
    dropout = rng.choice([0.0, 0.0, 0.0, 0.1])
    Lq = Lkv = _length(rng, 32, 8192)
    if mask in ("none", "pad") and rng.random() < 0.4:
        Lkv = _length(rng, 32, 8192)
    return _fit(_attn("", kind, dtype, d, H, Lq, Lkv, B, mask, bias, dropout))


def _draw_decode(rng):
    dtype = rng.choice(["bf16", "bf16", "f16", "tf32", "f32"])
    Lkv = _length(rng, 256, 32768)
    return _fit(_attn("", "forward", dtype, rng.choice([64, 128]), rng.choice([8, 16, 32]), rng.choice([1, 1, 1, 4, 16]),
                      Lkv, _log_int(rng, 1, 32), mask="causal"))


def _draw_bmm(rng):
    dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
    M, N, K = (_length(rng, 32, 4096) for _ in range(3))
    batch = _log_int(rng, 1, 64)
    cap = 1e10 if dtype == "f32" else 1.1e12
    while 2.0 * M * N * K * batch > cap and batch > 1:
        batch //= 2
    while 2.0 * M * N * K * batch > cap:
        M, N, K = M * 3 // 4, N * 3 // 4, K * 3 // 4
    return {"kind": "bmm", "dtype": dtype, "M": M, "N": N, "K": K, "batch": batch, "ta": rng.random() < 0.5,
            "tb": rng.random() < 0.5}


def _draw_softmax(rng):
    n = _length(rng, 10, 65536)
    total = _log_int(rng, 1e4, 2e8)
    inner = rng.choice([1, 1, 1, _log_int(rng, 8, 512)])
    return {"kind": "softmax", "dtype": rng.choice(["bf16", "f16", "f32"]), "log": rng.random() < 0.5, "inner": inner,
            "n": n, "outer": max(1, total // (n * inner))}


def draw(rng):
    what = rng.choice(["forward", "forward", "forward", "scores", "scores", "train", "train", "train", "decode", "decode",
                       "bmm", "softmax"])
    if what == "decode":
        c = _draw_decode(rng)
    elif what == "bmm":
        c = _draw_bmm(rng)
    elif what == "softmax":
        c = _draw_softmax(rng)
    else:
        c = _draw_attention(rng, what)
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------------------ inputs and runs
def _normal(gen, shape, dtype, std=1.0):
    """Column-major array of normally distributed values (drawn in slices, so that no large Float32 copy exists)."""
    t = torch.empty(shape[::-1], dtype=dtype, device="cuda")
    t.normal_(0.0, std, generator=gen)
    return t.permute(*range(len(shape) - 1, -1, -1))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = _DTYPE[case["dtype"]]
    s = {"case": case, "seed": int(seed)}
    if case["kind"] == "bmm":
        M, N, K, nb_ = case["M"], case["N"], case["K"], case["batch"]
        s["A"] = _normal(gen, (K, M, nb_) if case["ta"] else (M, K, nb_), dt)
        s["B"] = _normal(gen, (N, K, nb_) if case["tb"] else (K, N, nb_), dt)
        return s
    if case["kind"] == "softmax":
        shape = (case["inner"], case["n"], case["outer"]) if case["inner"] > 1 else (case["n"], case["outer"])
        s["x"] = _normal(gen, shape, dt, 2.0)
        s["dy"] = _normal(gen, shape, dt)
        return s
    d, H, Lq, Lkv, B = (case[k] for k in ("d", "H", "Lq", "Lkv", "B"))
    s["q"], s["k"], s["v"] = _normal(gen, (d * H, Lq, B), dt), _normal(gen, (d * H, Lkv, B), dt), _normal(gen, (d * H, Lkv, B), dt)
    s["bias"] = None
    if case["bias"] != "none":
        s["bias"] = _normal(gen, (Lkv, Lq, H, B) if case["bias"] == "full" else (Lkv, Lq, H), dt, 0.5)
    s["mask"] = None
    if case["mask"] == "causal":
        # the square matrix as long as a program would hold one; new queries against a history and very long
        # sequences use the sentinel
        s["mask"] = nb.make_causal_mask(s["q"]) if Lq == Lkv and Lq <= 8192 else nb.CausalMask(Lkv - Lq)
    elif case["mask"] == "pad":
        n = torch.randint((Lkv + 1) // 2, Lkv + 1, (B,), generator=gen, device="cuda")
        keep = torch.arange(Lkv, device="cuda")[None, :] < n[:, None]          # (B, Lkv) row-major
        s["mask"] = keep.reshape(B, 1, 1, Lkv).permute(3, 2, 1, 0)
    elif case["mask"] == "window":
        j, i = torch.arange(Lkv, device="cuda"), torch.arange(Lq, device="cuda")
        back = i[:, None] - j[None, :]
        s["mask"] = ((back >= 0) & (back < max(1, Lkv // 4))).t()              # (Lkv, Lq), column-major
    if case["kind"] == "train":
        s["dx"] = _normal(gen, (d * H, Lq, B), dt)
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "bmm":
        A = nb.batched_transpose(s["A"]) if case["ta"] else s["A"]
        B = nb.batched_transpose(s["B"]) if case["tb"] else s["B"]
        return nb.batched_mul(A, B)
    if case["kind"] == "softmax":
        dims = 1 if case["inner"] == 1 else 2
        fwd, back = ((nb.softmax.logsoftmax, nb.softmax.logsoftmax_pullback) if case["log"] else
                     (nb.softmax.softmax, nb.softmax.softmax_pullback))
        y = fwd(s["x"], dims=dims)
        return y, back(s["dy"], y, dims=dims)
    # the two switches are process-wide settings of the framework, so a program that mixes uses sets them per use
    nb.set_math_mode("fast" if case["dtype"] == "tf32" else "default")
    nb.set_scores_mode("eager" if case["kind"] == "scores" else "lazy")
    fdrop = nb.PhiloxDropout(case["dropout"], seed=s["seed"]) if case["dropout"] > 0 else nb.identity
    if case["kind"] == "train":
        x, _, back = nb.dot_product_attention_pullback(s["q"], s["k"], s["v"], s["bias"], fdrop=fdrop, mask=s["mask"],
                                                       nheads=case["H"])
        dq, dk, dv, dbias = back(s["dx"])
        return (x, dq, dk, dv) if dbias is None else (x, dq, dk, dv, dbias)
    x, alpha = nb.dot_product_attention(s["q"], s["k"], s["v"], s["bias"], fdrop=fdrop, mask=s["mask"], nheads=case["H"])
    return (x, alpha) if case["kind"] == "scores" else x


# ------------------------------------------------------------------------------------------- work and tolerances
def _pairs(case):
    """Scores one (head, sample) unit cannot do without."""
    Lq, Lkv = case["Lq"], case["Lkv"]
    if case["mask"] == "causal":
        return Lq * (Lkv - Lq) + Lq * (Lq + 1) // 2
    if case["mask"] == "window":
        w = max(1, Lkv // 4)
        return w * (w + 1) // 2 + (Lq - w) * w
    return Lq * Lkv * 3 // 4 if case["mask"] == "pad" else Lq * Lkv


def work(case):
    z = _BYTES[case["dtype"]]
    if case["kind"] == "bmm":
        M, N, K, n = case["M"], case["N"], case["K"], case["batch"]
        return {"bytes": z * n * (M * K + K * N + M * N), "flops": 2.0 * M * N * K * n}
    if case["kind"] == "softmax":
        # forward: x in, y out; pullback: y and dy in, dx out (y is needed again only after it was written)
        n = case["inner"] * case["n"] * case["outer"]
        return {"bytes": 5 * z * n, "flops": 8.0 * n}
    d, H, Lq, Lkv, B = (case[k] for k in ("d", "H", "Lq", "Lkv", "B"))
    P = _pairs(case) * H * B
    scores = Lq * Lkv * H * B
    arrays = z * d * H * B * (2 * Lq + 2 * Lkv)                     # q, x and k, v
    bias = 0 if case["bias"] == "none" else z * (scores if case["bias"] == "full" else Lq * Lkv * H)
    mask = {"none": 0, "causal": 0, "pad": Lkv * B, "window": Lq * Lkv}[case["mask"]]
    if case["kind"] == "train":
        # two products forward, five backward; every array and its gradient once, the bias and its gradient
        return {"bytes": 2 * arrays + 2 * bias + mask, "flops": 2.0 * d * P * 7}
    alpha = z * scores if case["kind"] == "scores" else 0
    return {"bytes": arrays + bias + mask + alpha, "flops": 4.0 * d * P}


def tolerance(case):
    # four times the largest relative error (2-norm) seen against the same computation in Float64 over 180 drawn
    # cases: attention 2.4e-3 / 2.9e-4 / 1.9e-6 / 4.6e-4 (bf16 / f16 / f32 / tf32), its gradients 2.7e-3 / 3.3e-4 /
    # 9.9e-7 (they carry the rounding of P and dS as well; TF32 rounds like f16, so its gradients are as much above
    # its forward as those of f16), batched_mul 1.7e-3 / 2.1e-4 / 6.3e-7, softmax 1.7e-3 / 2.1e-4 / 9.3e-7
    if case["kind"] == "train":
        rel = {"bf16": 1.1e-2, "f16": 1.3e-3, "f32": 8e-6, "tf32": 2.4e-3}
    elif case["kind"] in ("forward", "scores"):
        rel = {"bf16": 1e-2, "f16": 1.2e-3, "f32": 8e-6, "tf32": 2e-3}
    else:
        rel = {"bf16": 7e-3, "f16": 9e-4, "f32": 3e-6 if case["kind"] == "bmm" else 4e-6}
    return {"rel": rel[case["dtype"]]}
