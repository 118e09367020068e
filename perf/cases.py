"""The work a user has this package do, as a list of cases that can be timed and compared.

A case is one call pattern of one Prism layer:

* ``forward``: ``cute_mma_b200.forward`` (serving through the functional API),
* ``step``:    ``cute_mma_b200.forward`` + ``backward`` (a training step that brings its own autograd),
* ``infer``:   ``PrismLinear`` under ``torch.no_grad()`` (serving through the module),
* ``train``:   ``PrismLinear`` forward and ``loss.backward()`` (training through autograd),

with its sizes (tokens ``M``, features ``K`` -> ``N``, ``gs`` outputs per group, ``rs``-wide rotation blocks), its
data type and the options in use.  ``listed()`` names the common ones, ``draw()`` gives others of the same ranges.
"""
import math

import torch

import cute_mma_b200 as cp

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
ACTS = {"plain": None, "silu": "silu_gate", "sigmoid": "sigmoid_gate"}

# What most calls leave off: output bias, internal bias (gated modes), dropout probability (gated modes, with the
# seeds in hand), input shuffle (module, rs 16), fp32 parameter gradients (functional backward).
DEFAULTS = {"bias": False, "ib": False, "p": 0.0, "shuffle": False, "f32_grads": False}

MOST_WORK = 16384.0 * 4096 * 14336   # M * K * N of the largest listed case


def _case(name, call, M, K, N, gs, rs, dtype, act, **options):
    return dict(DEFAULTS, name=name, call=call, M=M, K=K, N=N, gs=gs, rs=rs, dtype=dtype, act=act, **options)


def listed():
    return [
        # one token of one sequence through the wide layer of a decoder: the latency of a generated token
        _case("decode_1", "forward", 1, 4096, 14336, 256, 16, "bf16", "silu"),
        # a batch of 20 sequences, one token each, through the module in fp16
        _case("decode_20_module", "infer", 20, 1024, 16384, 256, 8, "fp16", "silu", bias=True),
        # a short prompt (or a large decode batch): between the streaming and the compute-bound regime
        _case("prompt_128", "forward", 128, 4096, 14336, 256, 16, "bf16", "silu"),
        # a prompt of ordinary length through the module
        _case("prompt_2048_module", "infer", 2048, 4096, 14336, 256, 16, "bf16", "silu", bias=True),
        # the smallest training step: launches and host work count
        _case("step_1024_small", "step", 1024, 256, 1024, 256, 8, "fp16", "silu"),
        # sizes off every tile edge, narrow groups, the other gate, internal bias and fp32 parameter gradients
        _case("step_1000_ragged", "step", 1000, 1000, 1440, 96, 8, "bf16", "sigmoid", ib=True, f32_grads=True),
        # fine-tuning (frozen weight, trained rotation) of a small transformer's MLP up-projection: 16 sequences
        _case("finetune_mlp", "train", 16384, 768, 3072, 256, 8, "bf16", "plain", bias=True),
        # the same model's attention projection on a single sequence
        _case("finetune_proj", "train", 1024, 768, 768, 256, 8, "bf16", "plain", bias=True),
        # one GPU's share of a data-parallel training step of a wide layer, fp16
        _case("step_8192_wide", "step", 8192, 1024, 16384, 256, 8, "fp16", "silu"),
        # training from scratch with dropout and internal bias
        _case("step_4096_dropout", "step", 4096, 1024, 4096, 256, 16, "bf16", "silu", ib=True, p=0.1),
        # training a layer whose groups see shuffled inputs, through the module
        _case("train_4096_shuffle", "train", 4096, 1024, 4096, 256, 16, "bf16", "silu", bias=True, ib=True, shuffle=True),
        # the full training step of the large layer, the benchmark's workload
        _case("step_16384_large", "step", 16384, 4096, 14336, 256, 16, "bf16", "silu"),
    ]


def _spread(rng, low, high):
    """A whole number from low to high, even in its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    call = rng.choice(["forward", "step", "infer", "train"])
    act = rng.choice(["plain", "silu", "silu", "sigmoid"])
    gated = act != "plain"
    c = dict(DEFAULTS, call=call, act=act, dtype=rng.choice(["bf16", "bf16", "fp16"]))
    c["shuffle"] = call in ("infer", "train") and gated and rng.random() < 0.2
    c["rs"] = 16 if c["shuffle"] else rng.choice([8, 8, 16, 16, 32, 64])
    if call == "step" and gated and c["rs"] <= 16 and rng.random() < 0.2:
        c["p"] = round(rng.uniform(0.05, 0.5), 3)
    c["bias"] = call in ("infer", "train") and rng.random() < 0.7
    c["ib"] = gated and rng.random() < 0.3
    c["f32_grads"] = call == "step" and rng.random() < 0.25
    special = c["shuffle"] or c["p"] > 0     # these options cost several times the plain layer
    step = 64 if c["shuffle"] else c["rs"]
    c["K"] = step * max(1, _spread(rng, 64, 2048 if special else 4096) // step)
    c["gs"] = rng.choice([32, 64, 96, 128, 128, 256, 256, 256, 512])
    c["N"] = c["gs"] * max(1, _spread(rng, 256, 4096 if special else 16384) // c["gs"])
    c["M"] = _spread(rng, 1 if call in ("forward", "infer") else 64, 4096 if special else 16384)
    c["M"] = max(1, min(c["M"], int(MOST_WORK / (c["K"] * c["N"]))))
    return c


def _rotation(c, gen, dev):
    """R as a layer holds it: skew-symmetric blocks at the gated layer's initial scale, orthogonal blocks (the Cayley
    transform of small skew-symmetric ones) in plain mode."""
    G, K, rs = c["N"] // c["gs"], c["K"], c["rs"]
    X = torch.randn(G, K // rs, rs, rs, device=dev, generator=gen)
    if c["act"] == "plain":
        S = (X - X.mT) * 0.05
        eye = torch.eye(rs, device=dev).expand_as(S)
        X = torch.linalg.solve(eye - S, eye + S)
    else:
        X = (X - X.mT) * (4.0 / math.sqrt(2 * (rs - (2 if c["ib"] else 1))))
    return X.permute(0, 2, 1, 3).reshape(G * rs, K).to(DTYPES[c["dtype"]]).contiguous()


def prepare(case, seed):
    c, dev = case, torch.device("cuda")
    dt, act = DTYPES[c["dtype"]], ACTS[c["act"]]
    M, K, N, gs, rs = c["M"], c["K"], c["N"], c["gs"], c["rs"]
    gen = torch.Generator(device=dev).manual_seed(seed)
    A = torch.randn(M, K, device=dev, generator=gen).to(dt)
    dC = None
    if c["call"] in ("step", "train"):
        dC = (torch.randn(M, N, device=dev, generator=gen) * (0.1 if c["dtype"] == "fp16" else 1.0)).to(dt)
    state = {"case": c, "A": A, "dC": dC}
    if c["call"] in ("forward", "step"):
        state["B"] = (torch.randn(N, K, device=dev, generator=gen) * K ** -0.5).to(dt)
        state["R"] = _rotation(c, gen, dev)
        state["fwd"] = {"activation": act}
        state["bwd"] = {"activation": act}
        if c["ib"]:
            ib = (torch.randn(N // gs, K, device=dev, generator=gen) / math.sqrt(rs - 1)).to(dt)
            state["fwd"]["internal_bias"] = state["bwd"]["internal_bias"] = ib
        if c["p"] > 0:
            seeds = torch.randint(1, 1 << 62, (N // gs,), dtype=torch.int64, device=dev, generator=gen)
            state["fwd"].update(dropout_seeds=seeds, dropout_p=c["p"], training=True)
            state["bwd"].update(dropout_seeds=seeds, dropout_p=c["p"])
        if c["f32_grads"]:
            state["bwd"].update(dR_dtype=torch.float32, dB_dtype=torch.float32)
        return state
    torch.manual_seed(seed)
    with torch.device("cpu" if c["shuffle"] else dev):   # the shuffle's masks are built bit by bit on the host
        layer = cp.PrismLinear(K, N, group_size=gs, reconn_sz=rs, bias=c["bias"], activation=act,
                               input_shuffle=c["shuffle"], internal_bias=c["ib"])
    layer = layer.to(dev)
    if act is None:
        with torch.no_grad():   # a rotation that has been trained away from the identity
            layer.reconn.normal_(0.0, 0.05, generator=gen)
    layer = layer.to(dt)
    state["layer"] = layer.train() if c["call"] == "train" else layer.eval()
    state["A"].requires_grad_(c["call"] == "train")
    return state


def run(state):
    c, A, dC = state["case"], state["A"], state["dC"]
    if c["call"] in ("forward", "step"):
        B, R = state["B"], state["R"]
        C, _ = cp.forward(A, B, R, c["gs"], c["rs"], **state["fwd"])
        if c["call"] == "forward":
            return C
        dA, dR, dB, d_ib = cp.backward(dC, A, B, R, c["gs"], c["rs"], **state["bwd"])
        return C, dA, dR, dB, d_ib
    layer = state["layer"]
    if c["call"] == "infer":
        with torch.no_grad():
            return layer(A)
    A.grad = None
    layer.zero_grad(set_to_none=True)
    y = layer(A)
    y.backward(dC)
    return [y.detach(), A.grad] + [p.grad for p in layer.parameters() if p.requires_grad]


def work(case):
    """Each input read once and each output written once; the dense products (two floating-point operations per
    multiply-add) and the block-diagonal ones.  The rotation that a backward recomputes is not counted."""
    c = case
    M, K, N, G = c["M"], c["K"], c["N"], c["N"] // c["gs"]
    gated, back = c["act"] != "plain", c["call"] in ("step", "train")
    grad = 4 if c["f32_grads"] else 2
    dense, rot = 2.0 * M * N * K, 2.0 * M * K * c["rs"] * G
    params = 2.0 * (N * K + G * c["rs"] * K + (N if c["bias"] else 0) + (G * K if c["ib"] else 0))
    nbytes, flops = params + 2.0 * M * (K + N), dense + rot
    if back:
        # the backward reads dC, A and the parameters and writes dA and the trained parameters' gradients
        nbytes += params + 2.0 * M * (N + 2 * K) + grad * G * c["rs"] * K + 2.0 * ((N if c["bias"] else 0) + (G * K if c["ib"] else 0))
        flops += dense + 2 * rot
        if gated:
            nbytes += grad * N * K
            flops += dense
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Four times the largest error against the same formulas in float64, over the listed cases and 24 drawn ones:
    bf16 0.0030 relative (2-norm) and 0.022 of one value; fp16, whose gate is evaluated in fp16 pairs, 0.00098 and
    0.0145."""
    return {"rel": 0.012, "max": 0.09} if case["dtype"] == "bf16" else {"rel": 0.004, "max": 0.06}


def _splitmix(x):
    """splitmix64 on int64 tensors (the arithmetic wraps; the shifts are logical)."""
    x = x + (0x9E3779B97F4A7C15 - (1 << 64))
    x = (x ^ ((x >> 30) & ((1 << 34) - 1))) * (0xBF58476D1CE4E5B9 - (1 << 64))
    x = (x ^ ((x >> 27) & ((1 << 37) - 1))) * (0x94D049BB133111EB - (1 << 64))
    return x ^ ((x >> 31) & ((1 << 33) - 1))


def _kept(seed, M, K, p, dev):
    """The dropout mask of one group, over 1 - p: element (m, k) stays if its 24-bit hash is at least p."""
    h = _splitmix(_splitmix(seed + 0xDEADBEEF) ^ _splitmix(torch.arange(M * K, device=dev))) >> 40 & ((1 << 24) - 1)
    return ((h.float() / (1 << 24)) >= p).double().view(M, K) / (1.0 - p)


def _shuffled(masks, K):
    """Where each of a group's features is taken from: pairs of features change places by two rounds of swaps in each
    chunk of 64, one mask bit a pair of segments."""
    G, chunks, rounds = masks.shape
    seg = torch.arange(32, device=masks.device).expand(G, chunks, 32).clone()
    for r, delta in enumerate((8, 16)):
        low = torch.tensor([i for i in range(32) if not i & delta], device=masks.device)
        swap = (masks[:, :, r, None] >> torch.arange(16, device=masks.device) & 1).bool()
        a, b = seg[..., low].clone(), seg[..., low + delta].clone()
        seg[..., low], seg[..., low + delta] = torch.where(swap, b, a), torch.where(swap, a, b)
    at = torch.arange(0, K, 64, device=masks.device)[None, :, None, None] + 2 * seg[..., None]
    return (at + torch.arange(2, device=masks.device)).reshape(G, K)


def exact(case, seed):
    """The formulas in float64, group by group, with autograd for the gradients."""
    state, c = prepare(case, seed), case
    M, K, N, gs, rs, G = c["M"], c["K"], c["N"], c["gs"], c["rs"], c["N"] // c["gs"]
    back, layer = c["call"] in ("step", "train"), state.get("layer")
    B, R, ib = (state["B"], state["R"], state["fwd"].get("internal_bias")) if layer is None else (
        layer.weight, layer.reconn, layer._internal_bias)
    A, dC = state["A"].detach().double().requires_grad_(back), state["dC"]
    P = [None if t is None else t.detach().double().requires_grad_(back) for t in (B, R, ib)]
    perm = _shuffled(layer._shuffle_masks, K) if c["shuffle"] else None
    y, grads, dA = torch.empty(M, N, dtype=torch.float64, device=A.device), [[], [], []], torch.zeros_like(A)
    for g in range(G):
        b, r, i = (None if t is None else t.view(G, -1, K)[g] for t in P)
        r = r.reshape(rs, K // rs, rs).transpose(0, 1)
        if layer is not None and c["act"] == "plain":   # the module holds the Cayley parameter
            s, eye = r - r.mT, torch.eye(rs, dtype=torch.float64, device=A.device)
            r = torch.linalg.solve(eye - s, eye + s)
        a = A if perm is None else A[:, perm[g]]
        s = torch.einsum("mbj,bij->mbi", a.view(M, K // rs, rs), r).reshape(M, K)
        s = s if i is None else s + i
        h = {"plain": lambda: s, "silu": lambda: a * s * torch.sigmoid(s), "sigmoid": lambda: 2 * a * torch.sigmoid(s)}[c["act"]]()
        if c["p"] > 0:
            h = h * _kept(state["fwd"]["dropout_seeds"][g], M, K, c["p"], A.device)
        out = h @ b.mT
        y[:, g * gs:(g + 1) * gs] = out.detach()
        if back:
            got = torch.autograd.grad(out, [A] + [t for t in P if t is not None], dC[:, g * gs:(g + 1) * gs].double())
            dA += got[0]
            for k, t in enumerate(got[1:]):   # a view's gradient is zero outside its group
                grads[k].append(t.view(G, -1, K)[g].clone())
    if layer is not None and layer.bias is not None:
        y += layer.bias.detach().double()
    if not back:
        return y
    dB, dR, d_ib = (torch.cat(t) if t else None for t in grads)
    if layer is None:
        return y, dA, dR, None if c["act"] == "plain" else dB, d_ib
    gain = {"plain": 1.0, "silu": 1.437, "sigmoid": 1.15}[c["act"]]   # the layer divides its gradients by this, its bias's not
    out = [y, dA / gain] + ([] if c["act"] == "plain" else [dB / gain]) + [dR / gain]
    return out + ([dC.double().sum(0)] if c["bias"] else []) + ([] if d_ib is None else [d_ib / gain])
