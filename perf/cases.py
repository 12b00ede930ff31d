"""The work this engine is used for, as timed cases: every Linear of a nanochat model under the MXFP8 recipe in
training (forward and backward) and in evaluation (forward only, weights quantized once), the chunked lm_head loss, the
fused residual step in front of the merged q/k/v projection, and the refresh of a model's quantized weights after an
optimizer step. Each pass goes through the public functions of nanochat_cpp_b200.engine as a training or evaluation
loop calls them.

Sizes are those of the depth-4 to depth-26 models (embedding 64 x depth, MLP hidden 4 x, vocabulary 32768), with token
counts from one 128-row tile up to the 8 x 2048 tokens of a training micro-batch, odd multiples of 128 among them.

A case is {"kind": ...} and:
  linear_eval   tokens, cin, cout                       fp8_matmul without grad, weight kept quantized by a cache
  linear        tokens, cin, cout, weight               fp8_matmul forward + backward; fp32 (straight into .grad) or bf16 weight
  qkv           tokens, embd, kv, fused                 fp8_qkv forward + backward; fused: behind residual_norm_mx
  mlp           tokens, embd, micro                     fp8_relu_square_mlp forward + backward over `micro` micro-batches,
                                                        whose weight gradients accumulate
  lm_head       tokens, embd, vocab, padded, chunk      softcap_cross_entropy (mean) forward + backward
  lm_head_eval  tokens, embd, vocab, padded, chunk      softcap_cross_entropy per token, without grad
  weights       layers, embd                            quantize_mx_batch_into of every block matrix of a model
"""
import math

import torch

import nanochat_cpp_b200 as nc

SOFTCAP = 15.0
GATE_COLS = 12
VOCAB = 32768


def listed():
    return [
        # one 128-token tile through a d12 attention-output projection: a short evaluation prompt
        {"name": "linear_eval_128", "kind": "linear_eval", "tokens": 128, "cin": 768, "cout": 768},
        # one 2048-token sequence through the d24 MLP's first projection in evaluation
        {"name": "linear_eval_d24", "kind": "linear_eval", "tokens": 2048, "cin": 1536, "cout": 6144},
        # a training step's d12 MLP projection on one sequence: forward and both gradients
        {"name": "linear_d12", "kind": "linear", "tokens": 2048, "cin": 768, "cout": 3072, "weight": "fp32"},
        # d26 attention output (13 x 128 wide) on an odd number of tokens, weight kept in bf16
        {"name": "linear_d26_odd", "kind": "linear", "tokens": 3968, "cin": 1664, "cout": 1664, "weight": "bf16"},
        # merged q/k/v of a d12 block with fewer key/value heads on a short odd batch
        {"name": "qkv_d12_odd", "kind": "qkv", "tokens": 1152, "embd": 768, "kv": 256, "fused": False},
        # the d24 block's input: residual add, blend and norm emitting MX, then q/k/v, on a training micro-batch
        {"name": "residual_qkv_d24", "kind": "qkv", "tokens": 16384, "embd": 1536, "kv": 1536, "fused": True},
        # the d12 MLP on one sequence
        {"name": "mlp_d12", "kind": "mlp", "tokens": 2048, "embd": 768, "micro": 1},
        # the d24 MLP over an optimizer step of two micro-batches
        {"name": "mlp_d24", "kind": "mlp", "tokens": 16384, "embd": 1536, "micro": 2},
        # the loss of a d12 model on one sequence
        {"name": "lm_head_d12", "kind": "lm_head", "tokens": 2048, "embd": 768, "vocab": VOCAB, "padded": VOCAB, "chunk": 2048},
        # the loss of a d24 model on a training micro-batch, in chunks of 2048 rows: the largest call
        {"name": "lm_head_d24", "kind": "lm_head", "tokens": 16384, "embd": 1536, "vocab": VOCAB, "padded": VOCAB, "chunk": 2048},
        # validation loss per token, vocabulary not a multiple of the padding, last chunk short
        {"name": "lm_head_eval_d24", "kind": "lm_head_eval", "tokens": 4992, "embd": 1536, "vocab": 32500, "padded": VOCAB, "chunk": 2048},
        # every block matrix of a d12 model re-quantized after an optimizer step
        {"name": "weights_d12", "kind": "weights", "layers": 12, "embd": 768},
    ]


def _log_tokens(rng, low, high):
    """A multiple of 128 between low and high, even over the logarithm."""
    return 128 * max(1, round(math.exp(rng.uniform(math.log(low), math.log(high))) / 128))


def draw(rng):
    kind = rng.choice(["linear_eval", "linear", "qkv", "mlp", "lm_head", "lm_head_eval", "weights"])
    embd = 64 * rng.choice(range(4, 27, 2))
    tokens = _log_tokens(rng, 128, 16384)
    if kind == "weights":
        return {"kind": kind, "layers": rng.randint(1, 24), "embd": embd}
    if kind in ("linear_eval", "linear"):
        cin, cout = rng.choice([(embd, embd), (embd, 4 * embd), (4 * embd, embd), (embd, 3 * embd)])
        case = {"kind": kind, "tokens": tokens, "cin": cin, "cout": cout}
        if kind == "linear":
            case["weight"] = rng.choice(["fp32", "fp32", "fp32", "bf16"])
        return case
    if kind == "qkv":
        kv = 128 * rng.randint(1, embd // 128)
        return {"kind": kind, "tokens": tokens, "embd": embd, "kv": rng.choice([embd, kv]), "fused": rng.random() < 0.5}
    if kind == "mlp":
        return {"kind": kind, "tokens": tokens, "embd": embd, "micro": rng.choice([1, 1, 2])}
    embd = min(embd, 1536)
    padded = 128 * rng.choice([32, 64, 100, 256, 256, 256])
    vocab = padded - rng.choice([0, 0, rng.randint(1, 127)])
    return {"kind": kind, "tokens": tokens, "embd": embd, "vocab": vocab, "padded": padded, "chunk": rng.choice([1024, 2048])}


# ---------------------------------------------------------------------------------------------------- inputs

class _Draws:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def randn(self, *shape, std=1.0, dtype=torch.bfloat16):
        return torch.randn(shape, generator=self.gen, device="cuda").mul_(std).to(dtype)

    def weight(self, out_features, in_features, dtype=torch.float32):
        w = self.randn(out_features, in_features, std=in_features ** -0.5, dtype=dtype)
        return w.requires_grad_(True)

    def rand(self, n):
        return torch.rand(n, generator=self.gen, device="cuda")


def prepare(case, seed):
    d, kind = _Draws(seed), case["kind"]
    state = {"kind": kind}
    if kind == "weights":
        # fp32 master weights, and the buffers their quantized copies live in; one buffer per part, a matrix is a view
        embd = case["embd"]
        shapes = [(3 * embd, embd), (embd, embd), (4 * embd, embd), (embd, 4 * embd)] * case["layers"]
        total = sum(n * k for n, k in shapes)
        flat = d.randn(total, std=embd ** -0.5, dtype=torch.float32)
        parts = [torch.empty(total, dtype=torch.uint8, device="cuda") for _ in range(2)]
        parts += [torch.empty(total // 32, dtype=torch.uint8, device="cuda") for _ in range(2)]
        jobs, at = [], 0
        for n, k in shapes:
            data = [p[at:at + n * k].view(torch.float8_e4m3fn) for p in parts[:2]]
            scale = [p[at // 32:(at + n * k) // 32].view(torch.float8_e8m0fnu) for p in parts[2:]]
            jobs.append((flat[at:at + n * k].view(n, k), nc.mx_out(data[0].view(n, k), scale[0]),
                         nc.mx_out(data[1].view(k, n), scale[1])))
            at += n * k
        state.update(jobs=jobs, parts=parts)
    elif kind in ("linear_eval", "linear"):
        tokens, cin, cout = case["tokens"], case["cin"], case["cout"]
        state["x"] = d.randn(tokens, cin)
        state["w"] = d.weight(cout, cin, torch.bfloat16 if case.get("weight") == "bf16" else torch.float32)
        if kind == "linear":
            state["dy"] = d.randn(tokens, cout, std=1e-3)
            state["x"].requires_grad_(True)
        else:
            state["cache"] = nc.Fp8WeightCache(True)
            nc.quantize_fp8_weight(state["w"], state["cache"])
    elif kind == "qkv":
        tokens, embd = case["tokens"], case["embd"]
        sizes = (embd, case["kv"], case["kv"])
        state["x"] = d.randn(tokens, embd)
        state["w"] = [d.weight(n, embd) for n in sizes]
        state["dy"] = [d.randn(tokens, n, std=1e-3) for n in sizes] + [d.randn(tokens, GATE_COLS, std=1e-3)]
        if case["fused"]:
            state.update(r=d.randn(tokens, embd, std=0.5), x0=d.randn(tokens, embd), lr=d.rand(4) + 0.5, l0=d.rand(4) * 0.3)
        else:
            state["x"].requires_grad_(True)
    elif kind == "mlp":
        tokens, embd = case["tokens"], case["embd"]
        state["x"] = [d.randn(tokens, embd).requires_grad_(True) for _ in range(case["micro"])]
        state["dy"] = [d.randn(tokens, embd, std=1e-3) for _ in range(case["micro"])]
        state["w"] = [d.weight(4 * embd, embd), d.weight(embd, 4 * embd)]
    else:
        # hidden states with the heavy tails that reach the lm_head (Student-t, 3 degrees of freedom, halved)
        tokens, embd = case["tokens"], case["embd"]
        chi2 = sum(d.randn(tokens, embd, dtype=torch.float32).square_() for _ in range(3))
        state["x"] = (d.randn(tokens, embd, dtype=torch.float32) / (chi2 / 3).sqrt_()).mul_(0.5).to(torch.bfloat16)
        state["w"] = d.weight(case["padded"], embd)
        state["targets"] = torch.randint(0, case["vocab"], (tokens,), generator=d.gen, device="cuda")
        state["targets"][d.rand(tokens) < 0.03] = -1  # padding tokens carry no loss
        state["args"] = (case["vocab"], SOFTCAP, case["chunk"])
        if kind == "lm_head":
            state["x"].requires_grad_(True)
        else:
            state["cache"] = nc.Fp8WeightCache(True)
            nc.quantize_fp8_weight(state["w"], state["cache"])
    return state


# ---------------------------------------------------------------------------------------------------- passes

def run(state):
    return _RUN[state["kind"]](state)


def _run_linear_eval(s):
    with torch.no_grad():
        return nc.fp8_matmul(s["x"], s["w"], s["cache"])


def _run_linear(s):
    x, w = s["x"], s["w"]
    x.grad = w.grad = None
    y = nc.fp8_matmul(x, w)
    y.backward(s["dy"])
    return y, x.grad, w.grad


def _run_qkv(s):
    ws = s["w"]
    for w in ws:
        w.grad = None
    if "r" in s:
        res, n, n_mx, rstd, kept = nc.residual_norm_mx(s["x"], s["r"], s["x0"], s["lr"], s["l0"], 2, GATE_COLS)
        n.requires_grad_(True)
        out = nc.fp8_qkv(n, *ws, gate_cols=GATE_COLS, x_mx=n_mx)
        more = (res, rstd, kept)
    else:
        n, more = s["x"], ()
        n.grad = None
        out = nc.fp8_qkv(n, *ws, gate_cols=GATE_COLS)
    torch.autograd.backward(out, s["dy"])
    return (*out, n.grad, *(w.grad for w in ws), *more)


def _run_mlp(s):
    w_fc, w_proj = s["w"]
    w_fc.grad = w_proj.grad = None
    fc_cache, proj_cache = nc.Fp8WeightCache(True), nc.Fp8WeightCache(True)  # the step's weights, quantized once
    out = []
    for x, dy in zip(s["x"], s["dy"]):
        x.grad = None
        y = nc.fp8_relu_square_mlp(x, w_fc, w_proj, fc_cache, proj_cache)
        y.backward(dy)
        out += [y, x.grad]
    return (*out, w_fc.grad, w_proj.grad)


def _run_lm_head(s):
    x, w = s["x"], s["w"]
    x.grad = w.grad = None
    loss = nc.softcap_cross_entropy(x, w, s["targets"], *s["args"])
    loss.backward()
    return loss, x.grad, w.grad


def _run_lm_head_eval(s):
    with torch.no_grad():
        return nc.softcap_cross_entropy(s["x"], s["w"], s["targets"], *s["args"], reduction="none", cache=s["cache"])


def _run_weights(s):
    nc.quantize_mx_batch_into(s["jobs"])
    return s["parts"]


_RUN = {"linear_eval": _run_linear_eval, "linear": _run_linear, "qkv": _run_qkv, "mlp": _run_mlp,
        "lm_head": _run_lm_head, "lm_head_eval": _run_lm_head_eval, "weights": _run_weights}


# ---------------------------------------------------------------------------------------------------- what a pass is

def work(case):
    """Inputs read once, outputs written once; 2 M N K operations per matrix product."""
    kind, mx = case["kind"], 1 + 1 / 32  # bytes of a quantized value with its share of the scale
    if kind == "weights":
        return {"bytes": case["layers"] * 12 * case["embd"] ** 2 * (4 + 2 * mx), "flops": 0}
    n = case["tokens"]
    if kind == "linear_eval":
        i, o = case["cin"], case["cout"]
        return {"bytes": 2 * n * (i + o) + mx * i * o, "flops": 2 * n * i * o}
    if kind == "linear":
        i, o = case["cin"], case["cout"]
        return {"bytes": 4 * n * (i + o) + 2 * i * o * (4 if case["weight"] == "fp32" else 2), "flops": 6 * n * i * o}
    c = case["embd"]
    if kind == "qkv":
        o = c + 2 * case["kv"]
        residual = (2 * n * c * 4 + 4 * n) if case["fused"] else 0  # r, x0 in; the new stream and the kept sum out
        return {"bytes": 4 * n * (c + o) + 8 * c * o + residual, "flops": 6 * n * c * o}
    if kind == "mlp":
        return {"bytes": case["micro"] * 8 * n * c + 2 * 8 * c * 4 * c, "flops": case["micro"] * 12 * n * c * 4 * c}
    v = case["padded"]
    if kind == "lm_head":
        return {"bytes": 4 * n * c + 8 * n + 8 * c * v, "flops": 6 * n * c * v}
    return {"bytes": 2 * n * c + 12 * n + mx * c * v, "flops": 2 * n * c * v}


def tolerance(case):
    if case["kind"] == "weights":
        return "exact"
    if case["kind"] in ("linear_eval", "linear"):
        return {"rel": 4e-3}  # one bf16 rounding (2^-9) per value of y and dx
    if case["kind"] == "lm_head_eval":
        return {"rel": 1e-3}  # fp32 losses of order log(vocab) from logits rounded to bf16
    return {"rel": 1e-2}      # bf16 values that are rounded again to e4m3 on the way
