"""What a user of the W4A16 projection library has it do, as measurable cases.

A case is a dict of plain values.  Its "path" names the form in which a program uses the
library; the other values are sizes and options:

  linear    one projection call, `int4_gemv_bf16` for one row, `batch_int4_gemv_bf16` for more
  step      one decode step of a stack of decoder layers, issued layer by layer with the calls
            an engine makes (shared-input projections together, projection + residual,
            gate/up + silu, down + residual)
  group     one decode step's independent projections as one `LinearGroup`
  cohort    batched decode through the MLPs of all layers: one group of gate and up
            projections, one of down projections
  token     the vocabulary projection with the token pick, with or without sampling
  prefill   the rows of a prompt through one layer's projections
  quantize  bf16 weights to packed int4 and scales (model conversion)

The model sizes are those of the 24-layer hybrid stack of the benchmark (18 DeltaNet-style and
6 full-attention layers, hidden size 1024, MLP 3584, vocabulary 248,320) and generic ones.
"""
import math

import torch

import cudalm_agent_b200 as eng

HIDDEN, MLP, MIXER = 1024, 3584, 2048   # hidden size, MLP width, width of a mixer's output
DELTANET_IN = 6144                      # DeltaNet in-projection
ATTN_Q, ATTN_KV = 4096, 512             # query + gate, key, value
VOCAB = 248320


def _is_attention(layer):
    """Every fourth layer of the stack is a full-attention layer."""
    return layer % 4 == 3


def listed():
    return [
        # the smallest call: a key or value projection of one decoded token
        {"name": "linear_512x1024_m1", "path": "linear", "N": 512, "K": 1024, "M": 1},
        # a projection of a larger model, one token
        {"name": "linear_8192x8192_m1", "path": "linear", "N": 8192, "K": 8192, "M": 1},
        # a ragged batch on ragged sizes (N a prime, an odd number of quantisation groups)
        {"name": "linear_5003x2944_m13", "path": "linear", "N": 5003, "K": 2944, "M": 13},
        # one token of one sequence through all layers, issued call by call
        {"name": "step_m1", "path": "step", "layers": 24, "M": 1},
        # the same for small and for full batches of sequences
        {"name": "step_m8", "path": "step", "layers": 24, "M": 8},
        {"name": "step_m48", "path": "step", "layers": 24, "M": 48},
        # all 132 projections of one token in one launch (the headline benchmark)
        {"name": "group_m1", "path": "group", "layers": 24, "M": 1},
        # batched decode of a full cohort
        {"name": "cohort_m64", "path": "cohort", "layers": 24, "M": 64},
        # next token of one sequence, greedy
        {"name": "token_m1_greedy", "path": "token", "N": VOCAB, "K": HIDDEN, "M": 1, "top_k": 50,
         "sampled": False},
        # next tokens of a batch, sampled with temperature, top-k and top-p
        {"name": "token_m32_sampled", "path": "token", "N": VOCAB, "K": HIDDEN, "M": 32, "top_k": 50,
         "sampled": True},
        # a long prompt through one layer
        {"name": "prefill_2048", "path": "prefill", "M": 2048, "hidden": HIDDEN, "mlp": MLP},
        # converting the largest matrix of the model
        {"name": "quantize_248320x1024", "path": "quantize", "N": VOCAB, "K": HIDDEN},
    ]


def _log_int(rng, lo, hi):
    """An integer of lo..hi, spread evenly over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    path = rng.choice(["linear", "linear", "linear", "step", "group", "cohort", "token", "token",
                       "prefill", "prefill", "quantize"])
    if path == "linear":
        K = 128 * _log_int(rng, 1, 64)
        N = _log_int(rng, 16, min(32768, 8192 * 8192 // K))
        return {"path": path, "N": N, "K": K, "M": _log_int(rng, 1, 64)}
    if path == "step":
        return {"path": path, "layers": _log_int(rng, 2, 24), "M": _log_int(rng, 1, 64)}
    if path == "group":
        return {"path": path, "layers": _log_int(rng, 2, 24), "M": _log_int(rng, 1, 16)}
    if path == "cohort":
        return {"path": path, "layers": _log_int(rng, 2, 24), "M": _log_int(rng, 2, 64)}
    if path == "token":
        return {"path": path, "N": _log_int(rng, 4096, VOCAB), "K": HIDDEN, "M": _log_int(rng, 1, 32),
                "top_k": rng.choice([1, 8, 20, 50, 64]), "sampled": rng.random() < 0.5}
    if path == "prefill":
        return {"path": path, "M": _log_int(rng, 65, 2048), "hidden": 128 * rng.randint(4, 8),
                "mlp": 128 * rng.randint(8, 28)}
    K = 128 * _log_int(rng, 1, 64)
    return {"path": path, "N": _log_int(rng, 16, VOCAB * HIDDEN // K), "K": K}


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
def _weights(gen, N, K):
    """A projection as the converter makes it: bf16 ~N(0, 0.02), quantized per 128 of k."""
    w = torch.randn((N, K), generator=gen, device="cuda", dtype=torch.float32).mul_(0.02)
    return eng.W4A16Linear(*eng.quantize_w4a16(w.to(torch.bfloat16)))


def _acts(gen, M, K, outliers=False):
    """bf16 activations ~N(0, 1); batched decode has 1 % of entries twenty times as large."""
    x = torch.randn((M, K), generator=gen, device="cuda", dtype=torch.float32)
    if outliers:
        x[torch.rand((M, K), generator=gen, device="cuda") < 0.01] *= 20.0
    return x.to(torch.bfloat16)


def _empty(*shape):
    return torch.empty(shape, device="cuda", dtype=torch.bfloat16)


def _layer(gen, layer):
    """One layer's projections: the mixer's inputs, the mixer's output, gate, up, down."""
    ins = [ATTN_Q, ATTN_KV, ATTN_KV] if _is_attention(layer) else [DELTANET_IN]
    return {"ins": [_weights(gen, n, HIDDEN) for n in ins], "out": _weights(gen, HIDDEN, MIXER),
            "gate": _weights(gen, MLP, HIDDEN), "up": _weights(gen, MLP, HIDDEN),
            "down": _weights(gen, HIDDEN, MLP)}


def prepare(case, seed):
    path = case["path"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st = {"case": case}
    if path == "linear":
        M, N, K = case["M"], case["N"], case["K"]
        st["lin"] = _weights(gen, N, K)
        x = _acts(gen, M, K, outliers=M > 1)
        st["x"], st["y"] = (x[0], _empty(N)) if M == 1 else (x, _empty(M, N))
    elif path == "step":
        M = case["M"]
        st["layers"] = [_layer(gen, i) for i in range(case["layers"])]
        st["h0"] = _acts(gen, M, HIDDEN)          # the step's embeddings
        # what the parts of a layer that are not this library's hand to the projections: the
        # norms before the mixer and before the MLP, and the mixer (DeltaNet or attention)
        L = case["layers"]
        st["x_mixer"] = [_acts(gen, M, HIDDEN, outliers=True) for _ in range(L)]
        st["x_mlp"] = [_acts(gen, M, HIDDEN, outliers=True) for _ in range(L)]
        st["mixed"] = [_acts(gen, M, MIXER) for _ in range(L)]
        st["mixer_in"] = [[_empty(M, lin.N) for lin in ly["ins"]] for ly in st["layers"]]
        st["mid"], st["act"], st["h"] = _empty(M, HIDDEN), _empty(M, MLP), _empty(M, HIDDEN)
    elif path == "group":
        M, items = case["M"], []
        x1, x2, x3 = _acts(gen, M, HIDDEN), _acts(gen, M, MIXER), _acts(gen, M, MLP)
        layers = [_layer(gen, i) for i in range(case["layers"])]
        lins = [(lin, x) for ly in layers
                for lin, x in [(v, x1) for v in ly["ins"]] + [(ly["out"], x2), (ly["gate"], x1),
                                                              (ly["up"], x1), (ly["down"], x3)]]
        st["y"] = _empty(sum(lin.N for lin, _ in lins) * M)
        at = 0
        for lin, x in lins:
            items.append((lin, x, st["y"][at:at + M * lin.N].view(M, lin.N)))
            at += M * lin.N
        st["group"] = eng.LinearGroup(items)
    elif path == "cohort":
        M, L = case["M"], case["layers"]
        x, act = _acts(gen, M, HIDDEN, outliers=True), _acts(gen, M, MLP, outliers=True)
        st["gate"], st["up"], st["down"] = _empty(L, M, MLP), _empty(L, M, MLP), _empty(L, M, HIDDEN)
        gate_up, down = [], []
        for i in range(L):
            gate_up.append((_weights(gen, MLP, HIDDEN), x, st["gate"][i]))
            gate_up.append((_weights(gen, MLP, HIDDEN), x, st["up"][i]))
            down.append((_weights(gen, HIDDEN, MLP), act, st["down"][i]))
        st["groups"] = [eng.LinearGroup(gate_up), eng.LinearGroup(down)]
    elif path == "token":
        M, K = case["M"], case["K"]
        st["head"] = eng.LmHead(_weights(gen, case["N"], K), top_k=case["top_k"], max_rows=M,
                                keep_logits=True)
        x = torch.randn((M, K), generator=gen, device="cuda", dtype=torch.float32)
        st["x"] = (x / x.square().mean(dim=1, keepdim=True).sqrt()).to(torch.bfloat16)
        st["rng"] = torch.randint(-2 ** 62, 2 ** 62, (M,), generator=gen, device="cuda", dtype=torch.int64)
        st["token"] = torch.empty(M, device="cuda", dtype=torch.int32)
    elif path == "prefill":
        M, H, F = case["M"], case["hidden"], case["mlp"]
        st["h0"], st["mixed"] = _acts(gen, M, H), _acts(gen, M, 2 * H)
        st["x_mixer"], st["x_mlp"] = _acts(gen, M, H, outliers=True), _acts(gen, M, H, outliers=True)
        st["in"], st["out"] = _weights(gen, 6 * H, H), _weights(gen, H, 2 * H)
        st["gate"], st["up"], st["down"] = _weights(gen, F, H), _weights(gen, F, H), _weights(gen, H, F)
        st["proj"], st["mid"], st["act"], st["h"] = _empty(M, 6 * H), _empty(M, H), _empty(M, F), _empty(M, H)
    else:
        w = torch.empty((case["N"], case["K"]), device="cuda", dtype=torch.bfloat16)
        for lo in range(0, case["N"], 65536):   # in pieces: no fp32 copy of the whole matrix
            part = w[lo:lo + 65536]
            part.copy_(torch.randn(part.shape, generator=gen, device="cuda", dtype=torch.float32).mul_(0.02))
        st["w"] = w
    return st


# ---------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------
def run(st):
    path = st["case"]["path"]
    if path == "linear":
        lin = st["lin"]
        if st["case"]["M"] == 1:
            return eng.int4_gemv_bf16(lin.weight, lin.scale, st["x"], st["y"])
        return eng.batch_int4_gemv_bf16(lin.weight, lin.scale, st["x"], st["y"])
    if path == "step":
        h, mid, act = st["h0"], st["mid"], st["act"]
        for i, ly in enumerate(st["layers"]):
            ins, ys = ly["ins"], st["mixer_in"][i]
            x_mixer, x_mlp = st["x_mixer"][i], st["x_mlp"][i]
            if len(ins) == 1:
                eng.batch_int4_gemv_bf16(ins[0].weight, ins[0].scale, x_mixer, ys[0])
            else:
                eng.linear_multi([(lin, x_mixer, y) for lin, y in zip(ins, ys)])
            eng.linear_residual_bf16(ly["out"], st["mixed"][i], h, y=mid)
            eng.gate_up_silu_bf16(ly["gate"], ly["up"], x_mlp, out=act)
            h = eng.linear_residual_bf16(ly["down"], act, mid, y=st["h"])
        return {"h": h, "mixer_in": [y for ys in st["mixer_in"] for y in ys]}
    if path == "group":
        st["group"].run()
        return st["y"]
    if path == "cohort":
        for g in st["groups"]:
            g.run()
        return st["gate"], st["up"], st["down"]
    if path == "token":
        head = st["head"]
        argmax, idx, val = head.forward(st["x"])
        out = {"logits": head.logits, "argmax": argmax, "idx": idx, "val": val}
        if st["case"]["sampled"]:
            out["token"] = eng.sample_topk(idx, val, 0.8, st["case"]["top_k"], 0.95, st["rng"], st["token"])
            out["rng"] = st["rng"]
        return out
    if path == "prefill":
        proj = eng.batch_int4_gemv_bf16(st["in"].weight, st["in"].scale, st["x_mixer"], st["proj"])
        mid = eng.linear_residual_bf16(st["out"], st["mixed"], st["h0"], y=st["mid"])
        act = eng.gate_up_silu_bf16(st["gate"], st["up"], st["x_mlp"], out=st["act"])
        h = eng.linear_residual_bf16(st["down"], act, mid, y=st["h"])
        return {"proj": proj, "mid": mid, "act": act, "h": h}
    return eng.quantize_w4a16(st["w"])


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _linear_work(N, K, M):
    """Weights, scales, inputs and outputs of one projection once; two operations per weight and row."""
    return N * K // 2 + N * (K // 128) * 2 + M * K * 2 + M * N * 2, 2 * N * K * M


def _shapes(case):
    """The projections (N, K) of a pass."""
    path = case["path"]
    if path == "linear":
        return [(case["N"], case["K"])]
    if path == "cohort":
        return [(MLP, HIDDEN), (MLP, HIDDEN), (HIDDEN, MLP)] * case["layers"]
    if path == "prefill":
        H, F = case["hidden"], case["mlp"]
        return [(6 * H, H), (H, 2 * H), (F, H), (F, H), (H, F)]
    out = []
    for i in range(case["layers"]):
        ins = [ATTN_Q, ATTN_KV, ATTN_KV] if _is_attention(i) else [DELTANET_IN]
        out += [(n, HIDDEN) for n in ins] + [(HIDDEN, MIXER), (MLP, HIDDEN), (MLP, HIDDEN), (HIDDEN, MLP)]
    return out


def work(case):
    path = case["path"]
    if path == "quantize":
        n = case["N"] * case["K"]
        return {"bytes": 2 * n + n // 2 + n // 64, "flops": 0}
    if path == "token":
        b, f = _linear_work(case["N"], case["K"], case["M"])  # the logits are an output
        return {"bytes": b + case["M"] * (4 + 6 * case["top_k"]), "flops": f}
    parts = [_linear_work(n, k, case["M"]) for n, k in _shapes(case)]
    bytes_ = sum(b for b, _ in parts)
    if path in ("step", "prefill"):
        # two residuals per layer are read besides; gate and up share their input and leave one
        # product of the MLP's width instead of two outputs
        layers, H, F = (case["layers"], HIDDEN, MLP) if path == "step" else (1, case["hidden"], case["mlp"])
        bytes_ += layers * case["M"] * 2 * (2 * H - H - F)
    return {"bytes": bytes_, "flops": sum(f for _, f in parts)}


def _outputs(case):
    """Values of the smallest output of a pass."""
    path = case["path"]
    if path in ("linear", "token"):
        return case["N"] * case["M"]
    return case["M"] * min(n for n, _ in _shapes(case))


def tolerance(case):
    """The outputs are bf16 roundings of fp32 sums.  Sums in another order fall either side of a
    rounding boundary now and then.  Against 64-bit sums rounded the same way the 2-norm was off
    by up to 3e-5 on projections, 1e-4 where a rounded activation is projected again and 7e-4
    where a residual runs through a whole stack; one value by a step of bf16 (2^-7), two where
    roundings follow one another.  A small output that holds one such value is off by the step
    over the root of its size.  Of the picked ids, one changed logit moves a few."""
    path = case["path"]
    if path == "quantize":
        return "exact"
    rel = {"step": 2.8e-3, "prefill": 4e-4}.get(path, 1.2e-4)
    return {"rel": max(rel, 0.016 / math.sqrt(_outputs(case))),
            "max": 6e-2 if path in ("step", "prefill") else 3e-2, "differ": 0.01}
