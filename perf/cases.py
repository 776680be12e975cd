"""Performance cases of the attention operators: what a model that is built on them calls, over the sizes it calls them with.

A case is one attention layer: the forward alone (sampling), the forward and the backward (training), or a training step
that the program has captured once as a CUDA graph (`llsa_b200.capture_fwd_bwd`) and replays.  Its keys:

    op      llsa_l1 | llsa_l2 | llsa_l1_rope | llsa_l2_rope | llsa_l1_rms_rope | llsa_l2_rms_rope
    pass    fwd | train | captured
    B, H, N batch, heads, tokens (head dimension 64, blocks of 16 tokens)
    topk    selected blocks per query block, the same at every level
    dtype   bf16 | fp32
    layout  bhnd: contiguous [B,H,N,D] | bnhd: [B,H,N,D] views of [B,N,H,D] storage, what a projection layer hands over

Inputs are N(0,1) plus a smooth 2-D field over the Morton-ordered tokens, so that neighbouring blocks select alike blocks as
image tokens do.  Upstream gradients are N(0,1).
"""
import math

import torch

import llsa_b200

D, BLOCK = 64, 16
EPS = 1e-5
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


def _case(op, mode, B, H, N, topk=8, dtype="bf16", layout="bhnd", name=None):
    c = {"op": op, "pass": mode, "B": B, "H": H, "N": N, "topk": topk, "dtype": dtype, "layout": layout}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call of a training program: 32 x 32 tokens, two heads, in the precision that a numerics check runs in
        _case("llsa_l1", "train", 1, 2, 1024, dtype="fp32", name="l1 32x32 fp32 train"),
        # one denoising step of one image on a 32 x 32 latent: the smallest call of a sampling program
        _case("llsa_l1_rope", "fwd", 1, 6, 1024, layout="bnhd", name="l1 32x32 sample"),
        # a training layer at 64 x 64 tokens, the rotation of q and k fused in front
        _case("llsa_l1_rope", "train", 4, 6, 4096, name="l1 64x64 train"),
        # a sequence that is no power of two, odd batch and head counts, too short for the top pooled level
        _case("llsa_l2", "train", 3, 5, 5376, name="l2 ragged 5376 train"),
        # one denoising step of one image at 128 x 128 tokens, the whole q / k preparation of the block fused in front
        _case("llsa_l2_rms_rope", "fwd", 1, 6, 16384, layout="bnhd", name="l2 128x128 sample"),
        # the attention of a pixel-space training step at 128 x 128 tokens as the model calls it
        _case("llsa_l2_rms_rope", "train", 4, 6, 16384, layout="bnhd", name="l2 128x128 block train"),
        # the same size with eight images and the step captured: the benchmark's workload
        _case("llsa_l2", "captured", 8, 6, 16384, name="l2 128x128 captured"),
        # one-level attention at 128 x 128 tokens: 1024 pooled keys per row
        _case("llsa_l1", "train", 2, 4, 16384, name="l1 128x128 train"),
        # a wide selection (top-16) over 160 level-2 keys, odd batch and heads
        _case("llsa_l2", "train", 1, 5, 40960, topk=16, name="l2 ragged 40960 top16 train"),
        # sampling at 256 x 256 tokens with two levels
        _case("llsa_l2", "fwd", 2, 4, 65536, name="l2 256x256 sample"),
        # one-level attention at 256 x 256 tokens: 4096 pooled keys per row, the heaviest forward
        _case("llsa_l1", "fwd", 2, 4, 65536, name="l1 256x256 sample"),
        # a training layer at 512 x 512 tokens, one image
        _case("llsa_l2", "train", 1, 6, 262144, name="l2 512x512 train"),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _tokens(rng, levels, lo, hi):
    """A sequence length that the operators take (pooled levels long enough to be attended come in whole tiles of 32 keys);
    now and then the power of two below it."""
    n = _spread(rng, lo, hi)
    if rng.random() < 0.35:
        return 1 << (n.bit_length() - 1)
    unit = 512 if levels == 1 else (256 if n < 16384 else 8192)
    return max(lo, n // unit * unit)


def _cost(c):
    w = work(c)
    return max(w["bytes"] / 6e12, w["flops"] / (3e13 if c["dtype"] == "fp32" else 4e14))


def draw(rng):
    most = {"bf16": max(_cost(c) for c in listed()), "fp32": 1e-3}
    while True:
        dtype = "fp32" if rng.random() < 0.1 else "bf16"
        levels = rng.choice((1, 2))
        front = rng.choice(("", "", "_rope", "_rms_rope"))
        mode = rng.choice(("fwd", "train", "train", "captured"))
        N = _tokens(rng, levels, *((1024, 65536) if levels == 1 else (2048, 262144)))
        topk = rng.choice((8, 8, 8, 4, 16))
        if levels == 2 and topk > N // 256:
            topk = 8
        c = _case("llsa_l%d%s" % (levels, front), mode, _spread(rng, 1, 16), _spread(rng, 1, 12), N, topk, dtype, rng.choice(("bhnd", "bnhd")))
        if _cost(c) <= most[dtype] and c["B"] * c["H"] * N <= 8 * 6 * 16384 * 2:
            return c


def _levels(case):
    return 1 if case["op"].startswith("llsa_l1") else 2


def _fronted(case):
    """(rotation in front, normalisation in front)"""
    return "rope" in case["op"], "rms" in case["op"]


def _grid(N, device):
    """Row and column of every token: the odd and even bits of its index (Morton order)."""
    n = torch.arange(N, device=device)
    row, col = torch.zeros_like(n), torch.zeros_like(n)
    for i in range((N.bit_length() + 1) // 2):
        col |= ((n >> (2 * i)) & 1) << i
        row |= ((n >> (2 * i + 1)) & 1) << i
    return row.double(), col.double()


def _field_modes(N, device):
    """Four smooth functions of the token's place, unit root mean square: [4, N]."""
    row, col = _grid(N, device)
    y, x = (row + 0.5) / (row.max() + 1), (col + 0.5) / (col.max() + 1)
    modes = torch.stack([torch.cos(math.pi * y), torch.cos(math.pi * x), torch.cos(math.pi * y) * torch.cos(math.pi * x),
                         torch.cos(2 * math.pi * y) + torch.cos(2 * math.pi * x)])
    return (modes / modes.square().mean(1, keepdim=True).sqrt()).float()


def _table(N, dtype, device):
    """The [N, D] sin / cos table of 2-D positions: 16 frequencies for the row, 16 for the column."""
    omega = 10000.0 ** (-torch.arange(0, 32, 2, device=device, dtype=torch.float64) / 32)
    parts = [torch.stack([torch.sin(p[:, None] * omega), torch.cos(p[:, None] * omega)], -1).reshape(N, 32) for p in _grid(N, device)]
    return torch.cat(parts, -1).to(dtype).contiguous()


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    B, H, N, dtype = case["B"], case["H"], case["N"], DTYPES[case["dtype"]]
    modes = _field_modes(N, dev)

    def tensor(amplitude):
        out = torch.empty((B, H, N, D), dtype=dtype, device=dev)
        if case["layout"] == "bnhd":
            out = torch.empty((B, N, H, D), dtype=dtype, device=dev).transpose(1, 2)
        for b in range(B):      # one batch element at a time: the fp32 values of a large case need not be there at once
            x = torch.randn((H, N, D), generator=gen, device=dev)
            if amplitude:
                coef = 0.5 * torch.randn((H, D, 4), generator=gen, device=dev)
                x += amplitude * torch.matmul(coef, modes).transpose(1, 2)
            out[b] = x
        return out

    s = {"case": case, "leaves": [tensor(0.5) for _ in range(3)]}
    train = case["pass"] != "fwd"
    if train:
        s["do"] = tensor(0.0)
    rope, rms = _fronted(case)
    if rms:      # learned scales of the two norms
        s["leaves"] += [1 + 0.1 * torch.randn(D, generator=gen, device=dev) for _ in range(2)]
    s["table"] = _table(N, dtype, dev) if rope else None
    if case["pass"] == "train":
        s["leaves"] = [t.requires_grad_(True) for t in s["leaves"]]
    if case["pass"] == "captured":
        q, k, v = s["leaves"][:3]
        s["graph"], s["outputs"] = llsa_b200.capture_fwd_bwd(lambda q, k, v: _layer(s, [q, k, v] + s["leaves"][3:]), q, k, v, s["do"])
    return s


def _layer(s, leaves):
    case, table = s["case"], s["table"]
    fn, levels, (rope, rms) = getattr(llsa_b200, case["op"]), _levels(case), _fronted(case)
    args = list(leaves) + ([table] if rope else []) + ([EPS] if rms else [])
    return fn(*args, *[case["topk"]] * levels, BLOCK)


def run(s):
    """A sampling pass returns o; a training pass o and the gradient of every input."""
    mode = s["case"]["pass"]
    if mode == "captured":
        s["graph"].replay()
        return s["outputs"]
    if mode == "fwd":
        with torch.no_grad():
            return _layer(s, s["leaves"])
    o = _layer(s, s["leaves"])
    return (o,) + torch.autograd.grad(o, s["leaves"], s["do"])


def work(case):
    """Bytes: q, k, v (and d_o) read once, o (and dq, dk, dv) written once, and the table.  Operations: the products of the
    attended keys (scores and P.V forward; scores, dP, dQ, dV, dK backward) and of the selection."""
    slices, N, topk = case["B"] * case["H"], case["N"], case["topk"]
    size, levels = (4 if case["dtype"] == "fp32" else 2), _levels(case)
    n1, n2 = N // BLOCK, N // BLOCK ** 2
    keys = topk * BLOCK + ((n1 if n1 >= 64 else 0) if levels == 1 else topk * BLOCK + (n2 if n2 >= 64 else 0))
    select = 2 * D * (n1 * n1 if levels == 1 else n2 * n2 + n1 * topk * BLOCK)
    train = case["pass"] != "fwd"
    rope, _ = _fronted(case)
    return {"bytes": (8 if train else 4) * slices * N * D * size + (N * D * size if rope else 0),
            "flops": slices * ((14 if train else 4) * N * keys * D + select)}


def tolerance(case):
    """bf16 operands and results with fp32 sums; fp32 throughout."""
    return {"rel": 1e-5, "max": 1e-3} if case["dtype"] == "fp32" else {"rel": 1e-2}
