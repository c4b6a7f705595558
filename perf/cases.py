"""The work that users of this package have it do, as cases that can be timed and whose outputs can be compared.

Three kinds of programs call the package: molecule models (2-simplicial attention on padded batches of molecules, with
and without the geometry operands), periodic-crystal models (neighbour search, block list, radius and local-window
attention) and the EDM trunk around both (a training step, a sampling run).  Shapes and distributions are those of the
package's synthetic workloads and tests: QM9-sized molecules of 9-29 atoms, drug-sized molecules of 20-181 atoms padded
to 192, crystals of up to 4096 atoms; d_model 512 with 8 heads of 64 channels, bf16 with fp32 accumulation, and fp32
calls at a head size of 32.

Atom counts are spread evenly over the range of a case and dealt to the molecules in an order that depends on the seed,
so that two seeds do the same amount of work.
"""
from __future__ import annotations

import math

import torch

import matterformer_b200 as mfb
from matterformer_b200.dp import GraphedTrainStep, build_edm_net
from matterformer_b200.sampler import GraphedDenoiser, build_pad_mask, edm_sample
from matterformer_b200.trunk import EDMLoss

ATOM_TYPES = (0.51, 0.35, 0.06, 0.07, 0.01)  # H, C, N, O, F
CRYSTAL_CUTOFF = 6.0  # Angstrom
LIQUID_DENSITY = 4096 / 35.0**3  # atoms per cubic Angstrom of the 35 Angstrom cell with 4096 atoms


def _simplicial(batch, tokens, lo, dtype="bf16", head_dim=64, bias=False, rank=0, backward=True, hi=None):
    return {"kind": "simplicial", "batch": batch, "tokens": tokens, "lo": lo, "hi": hi or tokens, "heads": 8,
            "head_dim": head_dim, "dtype": dtype, "bias": bias, "rank": rank, "backward": backward}  # fmt: skip


def _crystal(kind, batch, tokens, lo, **more):
    return {"kind": kind, "batch": batch, "tokens": tokens, "lo": lo, "hi": tokens, **more}


def listed():
    return [
        # the attention call of a training step on drug-sized molecules: the package's headline workload
        {"name": "drug_train", **_simplicial(64, 192, 20, hi=181)},
        # the same call while sampling or evaluating: forward only, a smaller batch padded to its own odd maximum
        {"name": "drug_forward", **_simplicial(16, 131, 20, backward=False)},
        # small fp32 batch (parity runs, debugging): the smallest call, launches and the host path count
        {"name": "small_fp32", **_simplicial(8, 29, 9, dtype="f32", head_dim=32)},
        # factorized geometry bias, the default geometry mode of the molecule models, at QM9 and at drug size
        {"name": "qm9_bias", **_simplicial(256, 29, 9, bias=True)},
        {"name": "drug_bias", **_simplicial(64, 192, 20, bias=True, hi=181)},
        # bias plus the optional low-rank angle and message residuals at their default rank of 16
        {"name": "qm9_residual", **_simplicial(64, 29, 9, bias=True, rank=16)},
        # one attention layer of a crystal model over the atoms within 6 Angstrom, forward and backward
        {"name": "crystal_radius", **_crystal("radius", 16, 1024, 1024, sorted=True)},
        # what such a model builds once per step from positions and lattice: cell sort and block list, ragged cells
        {"name": "crystal_blocks", **_crystal("blocks", 8, 500, 300)},
        # band attention over large cells, forward and backward
        {"name": "cell_local", **_crystal("local", 32, 4096, 4096, window=64)},
        # neighbour lists of large cells
        {"name": "cell_knn", **_crystal("knn", 32, 4096, 4096, k=16)},
        # a training step of the 12-layer trunk on 1024 small molecules: loss, gradients, clipping, AdamW
        {"name": "trunk_train", "kind": "train", "batch": 1024, "tokens": 29, "lo": 9, "hi": 29},
        # a sampling run of the same model: 10 Heun steps, 19 evaluations of the denoiser on 64 molecules
        {"name": "trunk_sample", "kind": "sample", "batch": 64, "tokens": 29, "lo": 9, "hi": 29, "steps": 10},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    """One more call of the listed ranges; every kind of call is as likely as it is listed."""
    pick = rng.choice(["bf16", "forward", "f32", "bias_small", "bias", "residual", "radius", "blocks", "local", "knn",
                       "train", "sample"])  # fmt: skip
    if pick in ("bf16", "forward"):
        n = _log(rng, 9, 192)
        batch = _log(rng, 1, 1024 if n <= 32 else 64)
        return _simplicial(batch, n, rng.randint(max(1, n // 8), n), backward=pick == "bf16")
    if pick == "f32":
        n = _log(rng, 9, 64)
        return _simplicial(_log(rng, 1, 16), n, rng.randint(max(1, n // 3), n), dtype="f32", head_dim=rng.choice([32, 64]))
    if pick == "bias_small":
        n = rng.randint(9, 32)
        return _simplicial(_log(rng, 16, 512), n, rng.randint(max(1, n // 3), n), bias=True)
    if pick == "bias":
        n = rng.randint(33, 192)
        return _simplicial(_log(rng, 4, 64), n, rng.randint(n // 8, n), bias=True)
    if pick == "residual":
        n = _log(rng, 9, 48)
        return _simplicial(_log(rng, 4, 64), n, rng.randint(max(1, n // 3), n), bias=rng.random() < 0.5,
                           rank=rng.choice([8, 16, 16, 32]))  # fmt: skip
    if pick == "radius":
        n = _log(rng, 64, 1024)
        return _crystal("radius", _log(rng, 1, 16), n, rng.randint(n // 2, n), sorted=rng.random() < 0.5)
    if pick == "blocks":
        n = _log(rng, 64, 1024)
        return _crystal("blocks", _log(rng, 1, 16), n, rng.randint(n // 2, n))
    if pick == "local":
        n = _log(rng, 200, 4096)
        return _crystal("local", _log(rng, 1, 32), n, rng.randint(n // 2, n), window=rng.choice([32, 64, 64, 128]))
    if pick == "knn":
        n = _log(rng, 100, 4096)
        return _crystal("knn", _log(rng, 1, 32), n, rng.randint(n // 2, n), k=rng.choice([8, 16, 16, 32]))
    n = rng.randint(20, 32)
    if pick == "train":
        return {"kind": "train", "batch": _log(rng, 64, 1024), "tokens": n, "lo": rng.randint(5, 15), "hi": n}
    return {"kind": "sample", "batch": _log(rng, 16, 256), "tokens": n, "lo": rng.randint(5, 15), "hi": n, "steps": 5}


def _counts(case):
    """Atom counts spread evenly over [lo, hi], the largest first."""
    lo, hi, b = case["lo"], case["hi"], case["batch"]
    return [hi] if b == 1 else [round(hi - (hi - lo) * i / (b - 1)) for i in range(b)]


def _dealt(case, g):
    n = torch.tensor(_counts(case), dtype=torch.int32, device="cuda")
    return n[torch.randperm(case["batch"], generator=g, device="cuda")]


def _randn(g, *shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _prepare_simplicial(case, g):
    """Projected heads N(0,1)/sqrt(D) with suffix padding, geometry operands as the package's bias workload draws them."""
    B, H, N, D, R = case["batch"], case["heads"], case["tokens"], case["head_dim"], case["rank"]
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    n = _dealt(case, g)
    leaves = [_randn(g, B, H, N, D, scale=D**-0.5, dtype=dtype) for _ in range(5)]
    s = {"heads": leaves, "grad": _randn(g, B, H, N, D, dtype=dtype), "backward": case["backward"],
         "valid": torch.arange(N, device="cuda")[None, :] < n[:, None], "bias": None, "angle": None, "message": None}  # fmt: skip
    if case["bias"]:
        s["bias"] = (*(_randn(g, B, H, N, N, scale=0.5) for _ in range(3)), _randn(g, B, H, N))
    if R:
        s["angle"] = (_randn(g, B, H, N, N, R), _randn(g, B, H, N, N, R), _randn(g, B, H, N))
        s["message"] = (_randn(g, B, H, N, N, R), _randn(g, B, H, N, N, R), _randn(g, H, R, D, scale=R**-0.5))
    s["leaves"] = [*leaves, *(t for group in (s["bias"], s["angle"], s["message"]) if group for t in group)]
    if case["backward"]:
        for t in s["leaves"]:
            t.requires_grad_(True)
    return s


def _run_simplicial(s):
    with torch.set_grad_enabled(s["backward"]):
        out = mfb.simplicial_attention_cuda(*s["heads"], query_valid=s["valid"], pair_key_valid=s["valid"],
                                            factorized_bias=s["bias"], angle_residual=s["angle"],
                                            message_residual=s["message"])  # fmt: skip
    return [out, *torch.autograd.grad(out, s["leaves"], s["grad"])] if s["backward"] else out


def _triclinic(batch, g):
    """Latents [log a, log b, log c, cos alpha, cos beta, cos gamma] of cells with edges of 15-30 Angstrom, 70-110 degrees."""
    lat = torch.rand(batch, 6, generator=g, device="cuda")
    lat[:, :3] = torch.log(15.0 + 15.0 * lat[:, :3])
    lat[:, 3:] = torch.cos(torch.deg2rad(70.0 + 40.0 * lat[:, 3:]))
    return lat


def _crystal_positions(batch, n, g):
    """Atoms near the sites of a simple lattice (fractional), so that no two of them coincide."""
    m = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    site = torch.stack([torch.randperm(m**3, generator=g, device="cuda")[:n] for _ in range(batch)])
    site = torch.stack([site // (m * m), site // m % m, site % m], dim=-1)
    return (site + 0.2 + 0.6 * torch.rand(batch, n, 3, generator=g, device="cuda")) / m


def _prepare_crystal(case, g):
    B, N = case["batch"], case["tokens"]
    s = {"n": _dealt(case, g)}
    if case["kind"] == "knn":
        edge = (N / LIQUID_DENSITY) ** (1.0 / 3.0)
        s.update(k=case["k"], pos=torch.rand(B, N, 3, generator=g, device="cuda"),
                 lattice=torch.tensor([math.log(edge)] * 3 + [0.0] * 3, device="cuda").repeat(B, 1))  # fmt: skip
        return s
    if case["kind"] in ("radius", "blocks"):
        s.update(pos=_crystal_positions(B, N, g), lattice=_triclinic(B, g))
    if case["kind"] == "radius":
        s.update(blocks=mfb.build_radius_blocks(s["pos"], s["lattice"], s["n"], CRYSTAL_CUTOFF), sorted=case["sorted"])
    if case["kind"] in ("radius", "local"):
        s["window"] = case.get("window")
        s["qkv"] = [_randn(g, B, 8, N, 64, scale=1 / 8, dtype=torch.bfloat16).requires_grad_(True) for _ in range(3)]
        s["grad"] = _randn(g, B, 8, N, 64, dtype=torch.bfloat16)
    return s


def _run_radius(s):
    out = mfb.radius_block_sparse_attention(*s["qkv"], s["blocks"], sorted_inputs=s["sorted"])
    return [out, *torch.autograd.grad(out, s["qkv"], s["grad"])]


def _run_local(s):
    out = mfb.local_window_attention(*s["qkv"], s["n"], window=s["window"])
    return [out, *torch.autograd.grad(out, s["qkv"], s["grad"])]


def _run_blocks(s):
    blocks = mfb.build_radius_blocks(s["pos"], s["lattice"], s["n"], CRYSTAL_CUTOFF)
    return [blocks.perm, blocks.block_count, blocks.block_cols, blocks.block_mask]


def _run_knn(s):
    return mfb.knn_topk(s["pos"], s["lattice"], s["n"], k=s["k"])


def _network(seed):
    """The 12-layer network some way into training: the layers that start at zero (modulation, pair head) are not zero."""
    net = build_edm_net(seed=seed).cuda()
    with torch.no_grad():
        for p in net.parameters():
            if not p.any():
                p.normal_(std=0.02)
    return net


def _molecules(case, g):
    B, N = case["batch"], case["tokens"]
    n = _dealt(case, g)
    valid = torch.arange(N, device="cuda")[None, :] < n[:, None]
    p = torch.tensor(ATOM_TYPES, device="cuda").repeat(B, 1)
    types = torch.multinomial(p, N, replacement=True, generator=g) * valid
    coords = _randn(g, B, N, 3, scale=1.5) * valid[..., None]
    coords = (coords - coords.sum(1, keepdim=True) / n[:, None, None]) * valid[..., None]
    return n, {"atom_types": types, "coords": coords, "pad_mask": ~valid}


def _prepare_train(case, g, seed):
    """Parameters and AdamW's moments live in flat buffers, one stretch for each role of a parameter (the same weight of
    all layers), as a program that checkpoints or shards them keeps them; the step is captured once, then the training
    state is put back to its beginning."""
    _, batch = _molecules(case, g)
    net = _network(seed)
    roles = {}
    for name, p in net.named_parameters():
        layer = [x for x in name.split(".") if x.isdigit()][:1] if ".blocks." in name else []
        kind = net.model.trunk.blocks[int(layer[0])].attn_type + "." + name.split(layer[0], 1)[1][1:] if layer else name
        roles.setdefault(kind, []).append(p)
    padded = lambda p: -(-p.numel() // 128) * 128  # noqa: E731
    flat, m, v = (torch.zeros(sum(padded(p) for ps in roles.values() for p in ps), device="cuda") for _ in range(3))
    opt = torch.optim.AdamW(net.parameters(), lr=1e-4, fused=True, capturable=True)
    at, moments, steps = 0, {}, []
    for kind, ps in roles.items():
        begin = at
        for p in ps:
            place = lambda t: t[at : at + p.numel()].view(p.shape)  # noqa: E731
            place(flat).copy_(p.data)
            p.data = place(flat)
            steps.append(torch.zeros((), device="cuda"))
            opt.state[p] = {"step": steps[-1], "exp_avg": place(m), "exp_avg_sq": place(v)}
            at += padded(p)
        moments[kind] = m[begin:at]
    first = flat.clone()
    step = GraphedTrainStep(net, EDMLoss(sigma_data=1.0), opt, batch, warmup=3)
    flat.copy_(first)
    for t in (m, v, *steps):
        t.zero_()
    torch.manual_seed(seed)
    return {"step": step, "batch": batch, "net": net, "opt": opt, "params": flat, "moments": moments}


def _run_train(s):
    loss = s["step"](s["batch"])
    return {"loss": loss, "params": s["params"], "exp_avg": s["moments"]}


def _prepare_sample(case, g, seed):
    n, _ = _molecules(case, g)
    net = _network(seed).eval()
    pad = build_pad_mask(n)
    B, N = pad.shape
    with torch.no_grad():
        denoiser = GraphedDenoiser(net, torch.zeros(B, N, 6, device="cuda"), torch.zeros(B, N, 3, device="cuda"), pad, None,
                                   torch.bfloat16)  # fmt: skip
    torch.manual_seed(seed)
    return {"net": net, "n": n, "denoiser": denoiser, "steps": case["steps"]}


def _run_sample(s):
    atoms, coords, _ = edm_sample(s["net"], s["n"], num_steps=s["steps"], autocast_dtype=torch.bfloat16,
                                  denoiser=s["denoiser"])  # fmt: skip
    return [atoms, coords]


_RUN = {"simplicial": _run_simplicial, "radius": _run_radius, "blocks": _run_blocks, "local": _run_local,
        "knn": _run_knn, "train": _run_train, "sample": _run_sample}  # fmt: skip


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "simplicial":
        s = _prepare_simplicial(case, g)
    elif case["kind"] in ("train", "sample"):
        s = (_prepare_train if case["kind"] == "train" else _prepare_sample)(case, g, seed)
    else:
        s = _prepare_crystal(case, g)
    s["run"] = _RUN[case["kind"]]
    return s


def run(state):
    return state["run"](state)


def work(case):
    """Bytes: every input once and every output once, padding included where it has to be read or written.  FLOPs: on
    valid atoms only."""
    n, B, N = _counts(case), case["batch"], case["tokens"]
    s1, s3 = float(sum(n)), float(sum(x**3 for x in n))
    if case["kind"] == "simplicial":
        H, D, R = case["heads"], case["head_dim"], case["rank"]
        rows = B * H * N * D * (2 if case["dtype"] == "bf16" else 4)
        pairs = 4 * B * H * (N * N * ((3 if case["bias"] else 0) + 4 * R) + N)
        flops = H * s3 * (4 * D + 4 * R)  # logits and values, angle logits and message coefficients
        if not case["backward"]:
            return {"bytes": 6 * rows + pairs, "flops": flops}
        return {"bytes": 12 * rows + 2 * pairs, "flops": 3.5 * flops}
    if case["kind"] == "radius":
        # a cell of 15-30 Angstrom edges has a mean inverse volume of about (ln 2 / 15)**3 * 1.08
        near = min(1.0, (math.log(2) / 15) ** 3 * 1.08 * 4 / 3 * math.pi * CRYSTAL_CUTOFF**3)
        pairs = sum(x * x for x in n) * near
        return {"bytes": 12 * B * 8 * N * 64 * 2 + B * N * N / 4, "flops": 14.0 * 64 * 8 * pairs}
    if case["kind"] == "local":
        return {"bytes": 12 * B * 8 * N * 64 * 2, "flops": 14.0 * 64 * 8 * s1 * min(case["window"], N)}
    if case["kind"] == "blocks":
        t = -(-N // 32)
        return {"bytes": B * (16 * N + 36 + 4 * t + 4 * t * t * 33), "flops": 0}
    if case["kind"] == "knn":
        return {"bytes": B * N * (12 + 8 * case["k"]), "flops": 0}
    # 12 layers, half of them simplicial, d_model 512: Linear layers, attention cores, modulation
    d, s2 = 512, float(sum(x * x for x in n))
    forward = s1 * 312 * d * d + 6 * 4 * s3 * d + 6 * 4 * s2 * d + B * 144 * d * d
    weights = 60.8e6
    if case["kind"] == "train":  # fp32 parameters and two moments read and written
        return {"bytes": 24 * weights, "flops": 3 * forward}
    return {"bytes": (2 * case["steps"] - 1) * 2 * weights, "flops": (2 * case["steps"] - 1) * forward}


def tolerance(case):
    """fp32 attention: sums of 32-bit products, softmax and its differences in the backward pass.  bf16 attention: operands,
    probabilities and results rounded to 8 bits.  Training step: gradients through twelve layers of bf16 arithmetic (two
    choices of kernels differ by 1e-3 to 3e-3).  Sampling: the network moves the samples by small steps, which dilutes
    its rounding (2e-4).  Neighbour lists and block lists are compared bit for bit, as the package promises."""
    if case["kind"] in ("blocks", "knn"):
        return "exact"
    if case["kind"] == "train":
        return {"rel": 1e-2, "max": 0.3}
    if case["kind"] == "sample":
        return {"rel": 2e-3, "max": 0.05}
    return {"rel": 2e-5} if case.get("dtype") == "f32" else {"rel": 1e-2}
