"""Cases that performance work on the attention operator is measured on.

Four kinds of pass, all through the public entry points:

  rebuild   MaskedStepDeploy.step() that rebuilds the structure (projection, clustering, selection, plan,
            attention, residual) from warm centroids: every call at mask_refresh = 1, one in mask_refresh
            steps otherwise
  reuse     MaskedStepDeploy.step() on a stored structure, with the activations of a later denoising step
  first     the first sparse call of a layer in a request: init_state() and the rebuild behind it
  request   the same through the serving backend, T2TAttentionImpl.forward on [1, N, H, 128] tensors: both
            guidance branches of the first sparse step of a new request (two initialisations, one rebuild,
            one reuse)

Inputs are the 3D locality mixture of token2tile_b200/synth.py, drawn on the device.
"""
from __future__ import annotations

import math

import torch

from token2tile_b200 import t2t_attn
from token2tile_b200.deploy_step import MaskedStepDeploy

C, D, R = 2048, 128, 32          # key clusters, head dimension, rank of the projected space


def listed():
    return [
        # the benchmark's layer: 720p latent grid (21 x 45 x 80), 40 heads on one GPU, 1.5 % budget
        dict(name="rebuild_720p_40h", kind="rebuild", H=40, N=75600, CQ=512, s_frac=0.015, width=80, height=45,
             token_major=False, pin_tail=0),
        # the same layer on the seven of eight steps that reuse the structure
        dict(name="reuse_720p_40h", kind="reuse", H=40, N=75600, CQ=512, s_frac=0.015, width=80, height=45,
             token_major=False, pin_tail=0),
        # first sparse call of that layer: initialisation and rebuild
        dict(name="first_720p_40h", kind="first", H=40, N=75600, CQ=512, s_frac=0.015, width=80, height=45,
             token_major=False, pin_tail=0),
        # one rank's share of it on 8 GPUs, read and written in the host's token-major layout
        dict(name="rebuild_720p_5h", kind="rebuild", H=5, N=75600, CQ=512, s_frac=0.015, width=80, height=45,
             token_major=True, pin_tail=0),
        dict(name="reuse_720p_5h", kind="reuse", H=5, N=75600, CQ=512, s_frac=0.015, width=80, height=45,
             token_major=True, pin_tail=0),
        # 480p latent grid (21 x 30 x 52) at the benchmark's larger budget, 5 %
        dict(name="rebuild_480p_40h", kind="rebuild", H=40, N=32760, CQ=256, s_frac=0.05, width=52, height=30,
             token_major=False, pin_tail=0),
        dict(name="reuse_480p_12h", kind="reuse", H=12, N=32760, CQ=256, s_frac=0.032, width=52, height=30,
             token_major=True, pin_tail=0),
        # the serving backend with a built-in profile: first sparse step of a request, 480p, 12 heads
        dict(name="request_480p_12h", kind="request", H=12, N=32760, CQ=256, s_frac=0.032, width=52, height=30,
             token_major=True, pin_tail=0, profile="auto"),
        # one head chunk of the packed [video | context] documents: ragged length, pinned context keys
        dict(name="packed_28h", kind="rebuild", H=28, N=18413, CQ=144, s_frac=0.05, width=40, height=24,
             token_major=False, pin_tail=397),
        # the smallest configuration of the tests and the benchmark: launches and latency
        dict(name="rebuild_small", kind="rebuild", H=2, N=4096, CQ=32, s_frac=0.05, width=32, height=32,
             token_major=False, pin_tail=0),
        dict(name="reuse_small", kind="reuse", H=2, N=4096, CQ=32, s_frac=0.05, width=32, height=32,
             token_major=False, pin_tail=0),
        dict(name="first_small", kind="first", H=2, N=4096, CQ=32, s_frac=0.05, width=32, height=32,
             token_major=False, pin_tail=0),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """Head counts 1..40, sequence lengths from the smallest allowed (2048) to 720p, odd ones among them, about
    one query cluster per 100..250 rows, budgets of 1..8 %, both layouts, all four kinds."""
    kind = rng.choice(("rebuild", "rebuild", "reuse", "first", "request"))
    # the largest listed case runs a rebuild on all of these rows and pairs; the attention's cost grows with
    # heads x tokens x budget, everything else with heads x tokens
    rows, pairs = 40 * 75600, 40 * 75600 * 75600 * 0.015
    if kind in ("first", "request"):      # an initialisation (or two) on top
        rows, pairs = rows // 2, pairs / 2
    while True:
        n = int(_log_uniform(rng, 2048, 75600.99))
        h = rng.choice((12, 40)) if kind == "request" else int(_log_uniform(rng, 1, 40.99))
        s = round(_log_uniform(rng, 0.01, 0.08), 4)
        if h * n <= rows and h * n * n * s <= pairs:
            break
    width = rng.choice((32, 40, 52, 64, 80))
    case = dict(kind=kind, H=h, N=n, CQ=max(8, int(n / rng.uniform(100, 250))), s_frac=s, width=width,
                height=rng.randint(width // 2, width), token_major=kind == "request" or rng.random() < 0.5, pin_tail=0)
    if kind == "request":
        case["profile"] = "manual"
    elif rng.random() < 0.25 and n >= 4096:
        case["pin_tail"] = rng.randint(1, n // 16)
    return case


# -- inputs --------------------------------------------------------------------------------------------------
def _activations(case, gen, count=1):
    """`count` triples q, k, v [H, N, 128] bfloat16 that share their centres, as those of neighbouring denoising
    steps do: tokens on a row-major (t, y, x) grid, one of 512 centres per 1 x 4 x 4 block and head, noise 0.3
    around it, standard normal values.  token_major stores them [N, H, 128] and hands out the [H, N, 128] view."""
    H, N, X, Y = case["H"], case["N"], case["width"], case["height"]
    dev = "cuda"
    i = torch.arange(N, device=dev)
    x, y, t = i % X, (i // X) % Y, i // (X * Y)
    bx, by = (X + 3) // 4, (Y + 3) // 4
    block = (t * by + y // 4) * bx + x // 4
    nblocks = (-(-N // (X * Y))) * by * bx
    sets = []
    for _ in range(count):
        one = []
        for _ in range(3):
            if case["token_major"]:
                one.append(torch.empty(N, H, D, device=dev, dtype=torch.bfloat16).transpose(0, 1))
            else:
                one.append(torch.empty(H, N, D, device=dev, dtype=torch.bfloat16))
        sets.append(one)
    normal = lambda *shape: torch.randn(*shape, device=dev, generator=gen)
    for h in range(H):
        centres = normal(512, D)
        base = centres[torch.randint(0, 512, (nblocks,), device=dev, generator=gen)[block]]
        for q, k, v in sets:
            k[h] = torch.add(base, normal(N, D), alpha=0.3)
            q[h] = torch.add(base, normal(N, D), alpha=0.3)
            v[h] = normal(N, D)
    return sets


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, H, N, CQ = case["kind"], case["H"], case["N"], case["CQ"]
    if kind == "request":
        branches = [[t.transpose(0, 1).unsqueeze(0) for t in qkv] for qkv in _activations(case, gen, 2)]
        impl = t2t_attn.T2TAttentionImpl(H, D, False, D ** -0.5, prefix="blocks.7.attn1")
        options = dict(profile_name="auto")
        if case["profile"] == "manual":
            options = dict(profile_name="manual", ns_base=max(1, int(case["s_frac"] * N)), dense_prefix_steps=12, cq=CQ,
                           ck=C, step_profile=(1.0,) * 4, layer_profile=(1.0,) * 6, cfg_mult=(1.0, 1.0))
        return dict(kind=kind, impl=impl, branches=branches, options=options)
    op = MaskedStepDeploy(H, N, CQ, s_frac=case["s_frac"], mask_refresh=4 if kind == "reuse" else 1,
                          pin_tail=case["pin_tail"])
    earlier, now = _activations(case, gen, 2) if kind != "first" else (None, _activations(case, gen)[0])
    out = torch.empty_like(now[0])      # keeps the layout of q
    s = dict(kind=kind, op=op, qkv=now, out=out)
    if kind != "first":
        # the previous denoising step: its centroids warm-start this one, its structure is the one to reuse
        q, k, v = earlier
        s["state"] = op.init_state(q, k, warm_iters=4, seed=0)
        if kind == "reuse":
            op.set_cfg_call(0, key=0, step=0)
        op.step(q, k, v, s["state"])
        torch.cuda.synchronize()
    return s


def run(s):
    if s["kind"] == "request":
        # a request brings its own cache; the previous one stays referenced until this one is in place
        cache = t2t_attn.T2TRequestCache()
        s["cache"] = cache
        meta = t2t_attn.T2TAttentionMetadataBuilder().build(12, 50, cache, mask_refresh=4, **s["options"])
        return [s["impl"].forward(q, k, v, meta) for q, k, v in s["branches"]]
    op, (q, k, v) = s["op"], s["qkv"]
    if s["kind"] == "first":
        # the factors are defined up to the signs of their columns, so the state itself is not compared
        return op.step(q, k, v, op.init_state(q, k, warm_iters=4, seed=0), out=s["out"])
    if s["kind"] == "reuse":
        op.set_cfg_call(0, key=0, step=1)
        return op.step(q, k, v, s["state"], out=s["out"])
    state = dict(s["state"])      # step() puts the new centroids into the dict: every pass starts from the same ones
    out = op.step(q, k, v, state, out=s["out"])
    return dict(out=out, ck=state["ck"], cq=state["cq"])


# -- what a pass cannot do without ---------------------------------------------------------------------------
def work(case):
    """q, k, v read once and the output written once; products of every stage, the exact attention counted over
    the token budget alone (the union of a query cluster, which every one of its rows attends to, is larger and
    depends on the data)."""
    H, N, CQ = case["H"], case["N"], case["CQ"]
    rows = float(H) * N
    ns = max(1, int(case["s_frac"] * N))
    attend = rows * (4.0 * D * ns + C * (2.0 * R + 2.0 * D))
    project = rows * 2.0 * D * R
    rebuild = 2 * project + rows * 2.0 * R * (2 * CQ + C) + rows * 2.0 * R * C + attend
    reuse = project + attend
    init = rows * 2 * 2.0 * D * D + 2 * project + 4 * rows * 2.0 * R * (CQ + C)
    flops = {"rebuild": rebuild, "reuse": reuse, "first": init + rebuild, "request": 2 * init + rebuild + reuse}
    qkvo = 4.0 * rows * D * 2
    bytes_ = {"rebuild": qkvo + 4.0 * H * (C + CQ) * R, "reuse": qkvo, "first": qkvo, "request": 2 * qkvo}
    return {"bytes": bytes_[case["kind"]], "flops": flops[case["kind"]]}


def tolerance(case):
    """Summing every product over the 128 dimensions in another order (q, k and the projections permuted alike) moves
    the output by at most 2.6e-4 and the centroids by 1.3e-4 (a few rows change their cluster; largest single
    difference 0.044).  The bfloat16 rounding of the attention weights, which that experiment keeps, is relative to
    whatever row maximum an implementation refers them to: 2^-9 / sqrt(3) each, 1.6e-3 between two of them."""
    return {"rel": 0.004, "max": 0.2}
