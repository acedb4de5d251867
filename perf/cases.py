"""Performance cases of the operators: what is timed, on which inputs, and how results compare.

Every case goes through the package's Python operators, as a model calls them. ``mode`` "train"
is one forward and one backward with the gradients of all differentiable inputs; "infer" is the
forward under ``torch.no_grad()``. Inputs are made on the GPU from the seed alone.

  msda    multi_scale_deformable_attn: encoder, decoder and bird's-eye-view attention
  fused   multi_scale_deformable_attn_fused: the same, fed by reference points, offsets, logits
  gka     geometric_kernel_attention: integer pixel locations around a projected point
  da      deformable_aggregation: multi-camera key-point sampling
  dcn     deform_conv2d / modulated_deform_conv2d in a backbone
  stem    npu_max_pool2d of a frozen stem, then npu_add_relu of a residual block with its gradient
"""
import math

import torch

import drivingsdk_b200 as sdk

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
DETR_LEVELS = "100x134,50x67,25x34,13x17"
SCA_LEVELS = "116x200,58x100,29x50,15x25"


def listed():
    return [
        # the repository's small attention configuration: launches and host work count
        dict(name="msda_toy_f32", op="msda", mode="train", dtype="f32", B=1, Q=1000, H=8, D=32,
             levels="32x32,16x16,8x8,4x4", P=4, where="uniform", lo=-0.1, hi=1.1),
        # decoder cross-attention of a detector being served: a few hundred queries, no gradient
        dict(name="msda_decoder_infer_f16", op="msda", mode="infer", dtype="f16", B=1, Q=900, H=8,
             D=32, levels=DETR_LEVELS, P=4, where="uniform", lo=0.0, hi=1.0),
        # encoder self-attention: one query per pixel, samples a few pixels around it
        dict(name="msda_encoder_f32", op="msda", mode="train", dtype="f32", B=2, Q=17821, H=8, D=32,
             levels=DETR_LEVELS, P=4, where="grid", spread=3.0),
        # spatial cross-attention over six cameras: the headline workload, in both types
        dict(name="msda_sca_f32", op="msda", mode="train", dtype="f32", B=6, Q=2500, H=8, D=32,
             levels=SCA_LEVELS, P=8, where="uniform", lo=-0.05, hi=1.05),
        dict(name="msda_sca_bf16", op="msda", mode="train", dtype="bf16", B=6, Q=2500, H=8, D=32,
             levels=SCA_LEVELS, P=8, where="uniform", lo=-0.05, hi=1.05),
        # temporal self-attention over two stacked bird's-eye-view grids, one level
        dict(name="msda_tsa_bf16", op="msda", mode="train", dtype="bf16", B=2, Q=40000, H=8, D=32,
             levels="200x200", P=4, where="grid", spread=3.0),
        # wide heads, large batch: the largest call
        dict(name="msda_wide_bf16", op="msda", mode="train", dtype="bf16", B=8, Q=20000, H=8, D=128,
             levels="64x176,32x88,16x44,8x22", P=4, where="uniform", lo=-0.1, hi=1.1),
        # the operator that takes over the module's softmax and location arithmetic
        dict(name="fused_sca_f32", op="fused", mode="train", dtype="f32", B=6, Q=2500, H=8, D=32,
             levels=SCA_LEVELS, P=8, where="uniform", spread=4.0),
        # map-vector kernel attention, the shape of the operator's test: 3 x 5 pixels per query
        dict(name="gka_map_f32", op="gka", mode="train", dtype="f32", B=24, Q=7156, H=4, D=64, L=1,
             height=15, width=25, P=15, loc="float"),
        # key points of 900 anchors in six cameras at four scales; under half are in view
        dict(name="da_f32", op="da", mode="train", dtype="f32", B=6, C=256, G=8, anchors=900, pts=13,
             cams=6, maps="64x176,32x88,16x44,8x22"),
        # backbone stage with modulated deformable 3x3 convolution, the shape of the operator's test
        dict(name="dcn_f32", op="dcn", mode="train", dtype="f32", N=18, C=512, Co=512, height=29,
             width=50, stride=1, groups=1, deform_groups=1, modulated=True),
        # frozen stem pooling, then the first residual addition
        dict(name="stem_f32", op="stem", mode="train", dtype="f32", N=6, C=64, height=464, width=800),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pyramid(rng, top, levels):
    h, w = _log(rng, 8, top), _log(rng, 8, top)
    got = []
    for _ in range(levels):
        got.append("%dx%d" % (h, w))
        h, w = max(1, (h + 1) // 2), max(1, (w + 1) // 2)
    return ",".join(got)


def _keys(levels):
    return sum(h * w for h, w in _sizes(levels))


def draw(rng):
    op = rng.choice(["msda", "msda", "msda", "fused", "gka", "da", "dcn", "stem"])
    dtype = rng.choice(["f32", "f32", "bf16", "f16"])
    mode = rng.choice(["train", "train", "infer"])
    c = dict(op=op, mode=mode, dtype=dtype)
    if op in ("msda", "fused"):
        levels = rng.randint(1, 5)
        c.update(B=rng.randint(1, 8), Q=_log(rng, 100, 40000), H=rng.choice([4, 8, 8]),
                 # mostly powers of two; 24 and 48 are heads of models with 192 and 384 channels
                 D=rng.choice([16, 24, 32, 32, 32, 48, 64, 128]), levels=_pyramid(rng, 200, levels),
                 P=rng.choice([1, 2, 4, 4, 5, 8] if levels > 3 else [3, 4, 4, 8]))
        if op == "fused":
            c["P"] = min(c["P"], 32 // levels)
            c.update(where=rng.choice(["uniform", "grid"]), spread=rng.choice([2.0, 4.0]))
        elif rng.random() < 0.5:
            c.update(where="grid", spread=rng.choice([1.0, 3.0]))
        else:
            c.update(where="uniform", lo=-0.05, hi=1.05)
        # no more samples or keys than the largest listed call
        row = c["H"] * c["D"]
        while c["B"] > 1 and c["B"] * _keys(c["levels"]) * row > 120_000_000:
            c["B"] -= 1
        most = 2_000_000_000 // (c["B"] * row * levels * c["P"] * (1 if dtype != "f32" else 2))
        c["Q"] = max(50, min(c["Q"], most))
    elif op == "gka":
        c.update(B=rng.randint(1, 24), Q=_log(rng, 100, 8000), H=rng.choice([4, 8]),
                 D=rng.choice([32, 64]), L=rng.choice([1, 1, 2]), height=_log(rng, 8, 60),
                 width=_log(rng, 8, 100), P=rng.choice([9, 15, 15]), loc=rng.choice(["float", "int64"]))
    elif op == "da":
        scales = rng.randint(2, 4)
        c.update(B=rng.randint(1, 6), C=rng.choice([128, 256, 256]), G=8, anchors=_log(rng, 50, 900),
                 pts=rng.randint(5, 13), cams=rng.randint(4, 7), maps=_pyramid(rng, 120, scales))
    elif op == "dcn":
        c.update(N=rng.randint(1, 12), C=rng.choice([64, 128, 256, 512]), height=_log(rng, 12, 60),
                 width=_log(rng, 12, 100), stride=rng.choice([1, 1, 2]), groups=rng.choice([1, 1, 1, 2]),
                 deform_groups=rng.choice([1, 1, 4]), modulated=rng.choice([True, True, False]))
        c["Co"] = c["C"]
    else:
        c.update(N=rng.randint(1, 12), C=rng.choice([32, 64]), height=_log(rng, 100, 464),
                 width=_log(rng, 100, 800))
    return c


def _sizes(levels):
    return [tuple(int(v) for v in s.split("x")) for s in levels.split(",")]


def _level_tensors(sizes):
    shapes = torch.tensor(sizes, dtype=torch.int64)
    keys = shapes[:, 0] * shapes[:, 1]
    starts = torch.cat([keys.new_zeros(1), keys.cumsum(0)[:-1]])
    return shapes.cuda(), starts.cuda()


def _centres(g, where, B, Q):
    """Reference points [B, Q, 2] in (0, 1): anywhere, or the cells of a grid in row order."""
    if where == "uniform":
        return torch.rand(B, Q, 2, generator=g, device="cuda")
    side = max(1, int(math.ceil(math.sqrt(Q))))
    q = torch.arange(Q, device="cuda")
    at = torch.stack([(q % side + 0.5) / side, (q // side + 0.5) / side], -1)
    return at.expand(B, Q, 2).contiguous()


def _attention_inputs(c, g, dtype):
    sizes = _sizes(c["levels"])
    shapes, starts = _level_tensors(sizes)
    B, Q, H, D, L, P = c["B"], c["Q"], c["H"], c["D"], len(sizes), c["P"]
    K = _keys(c["levels"])
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    value = rand(B, K, H, D).to(dtype)
    logits = rand(B, Q, H, L, P)
    wh = shapes.flip(-1).float()[None, None, None, :, None, :]
    if c["op"] == "fused":
        ref = _centres(g, c["where"], B, Q)[:, :, None, :].expand(B, Q, L, 2).contiguous()
        off = rand(B, Q, H, L, P, 2) * c["spread"]
        diff = [value, ref.to(dtype), off.to(dtype), logits.to(dtype)]
    else:
        if c["where"] == "grid":
            loc = (_centres(g, "grid", B, Q)[:, :, None, None, None, :]
                   + rand(B, Q, H, L, P, 2) * c["spread"] / wh)
        else:
            loc = torch.rand(B, Q, H, L, P, 2, generator=g, device="cuda")
            loc = loc * (c["hi"] - c["lo"]) + c["lo"]
        attn = logits.flatten(3).softmax(-1).view(B, Q, H, L, P)
        diff = [value, loc.to(dtype), attn.to(dtype)]
    return shapes, starts, diff, rand(B, Q, H * D).to(dtype)


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype = DTYPES[c["dtype"]]
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    op = c["op"]
    if op in ("msda", "fused"):
        shapes, starts, diff, grad = _attention_inputs(c, g, dtype)
        fn = sdk.multi_scale_deformable_attn if op == "msda" else sdk.multi_scale_deformable_attn_fused
        call = lambda value, *rest: fn(value, shapes, starts, *rest)  # noqa: E731
    elif op == "gka":
        B, Q, H, D, L, P = c["B"], c["Q"], c["H"], c["D"], c["L"], c["P"]
        h, w = c["height"], c["width"]
        shapes, starts = _level_tensors([(h, w)] * L)
        # a window of pixels around a projected point, the same for all heads; points can
        # fall a little outside the image, where they are clamped
        rows = 3
        p = torch.arange(P, device="cuda")
        window = torch.stack([p // rows - P // rows // 2, p % rows - rows // 2], -1)
        centre = torch.rand(B, Q, 1, L, 1, 2, generator=g, device="cuda")
        centre = (centre * torch.tensor([w + 4.0, h + 4.0], device="cuda") - 2).floor().long()
        loc = (centre + window).expand(B, Q, H, L, P, 2).contiguous()
        loc = loc if c["loc"] == "int64" else loc.to(dtype)
        value = rand(B, h * w * L, H, D).to(dtype)
        attn = rand(B, Q, H, L * P).softmax(-1).view(B, Q, H, L, P).to(dtype)
        diff, grad = [value, attn], rand(B, Q, H * D).to(dtype)
        call = lambda v, a: sdk.geometric_kernel_attention(v, shapes, starts, loc, a)  # noqa: E731
    elif op == "da":
        B, A, pts, cams, G = c["B"], c["anchors"], c["pts"], c["cams"], c["G"]
        sizes = _sizes(c["maps"])
        shapes = torch.tensor([sizes] * cams, dtype=torch.int32)
        counts = (shapes[..., 0] * shapes[..., 1]).reshape(-1)
        starts = (counts.cumsum(0) - counts).to(torch.int32).view(cams, len(sizes)).cuda()
        shapes = shapes.cuda()
        feat = rand(B, int(counts.sum()), c["C"]).to(dtype)
        loc = (torch.rand(B, A, pts, cams, 2, generator=g, device="cuda") * 1.5 - 0.25).to(dtype)
        wts = rand(B, A, pts * cams * len(sizes), G).softmax(2)
        wts = wts.view(B, A, pts, cams, len(sizes), G).to(dtype)
        diff, grad = [feat, loc, wts], rand(B, A, c["C"]).to(dtype)
        call = lambda f, l, w: sdk.deformable_aggregation(f, shapes, starts, l, w)  # noqa: E731
    elif op == "dcn":
        N, C, Co, h, w, s = c["N"], c["C"], c["Co"], c["height"], c["width"], c["stride"]
        ho, wo, dg, gr = (h - 1) // s + 1, (w - 1) // s + 1, c["deform_groups"], c["groups"]
        x, weight = rand(N, C, h, w).to(dtype), (rand(Co, C // gr, 3, 3) / math.sqrt(9 * C // gr)).to(dtype)
        offset = (rand(N, dg * 18, ho, wo) * 1.5).to(dtype)
        grad = rand(N, Co, ho, wo).to(dtype)
        if c["modulated"]:
            diff = [x, offset, rand(N, dg * 9, ho, wo).sigmoid().to(dtype), weight]
            call = lambda x, o, m, k: sdk.modulated_deform_conv2d(x, o, m, k, None, s, 1, 1, gr, dg)  # noqa: E731
        else:
            diff = [x, offset, weight]
            call = lambda x, o, k: sdk.deform_conv2d(x, o, k, s, 1, 1, gr, dg)  # noqa: E731
    else:
        N, C, h, w = c["N"], c["C"], c["height"], c["width"]
        x = rand(N, C, h, w).to(dtype)
        diff = [rand(N, C, (h + 1) // 2, (w + 1) // 2).to(dtype)]
        grad = torch.randn(diff[0].shape, generator=g, device="cuda").to(dtype)
        call = lambda y: sdk.npu_add_relu(sdk.npu_max_pool2d(x, 3, 2, 1), y)  # noqa: E731
    if c["mode"] == "train":
        diff = [t.requires_grad_() for t in diff]
    return {"call": call, "diff": diff, "grad": grad, "train": c["mode"] == "train"}


def run(state):
    if not state["train"]:
        with torch.no_grad():
            return state["call"](*state["diff"])
    out = state["call"](*state["diff"])
    return (out, *torch.autograd.grad(out, state["diff"], state["grad"]))


def work(case):
    """Bytes: inputs and results once per direction. Operations: the multiply-adds of the path."""
    c = case
    e = 4 if c["dtype"] == "f32" else 2
    train = c["mode"] == "train"
    op = c["op"]
    if op in ("msda", "fused", "gka"):
        if op == "gka":
            K, L = c["height"] * c["width"] * c["L"], c["L"]
        else:
            K, L = _keys(c["levels"]), len(_sizes(c["levels"]))
        v = c["B"] * K * c["H"] * c["D"]
        s = c["B"] * c["Q"] * c["H"] * L * c["P"]
        o = c["B"] * c["Q"] * c["H"] * c["D"]
        corners = 1 if op == "gka" else 4
        r = 2 * c["B"] * c["Q"] * L if op == "fused" else 0
        le = 8 if c.get("loc") == "int64" else e   # bytes of one coordinate
        fwd = e * (v + s + r + o) + 2 * le * s
        bwd = e * (2 * v + 2 * s + 2 * r + o) + 2 * le * s * (1 if op == "gka" else 2)
        flops = 2 * corners * s * c["D"]
        return {"bytes": fwd + (bwd if train else 0), "flops": flops * (3 if train else 1)}
    if op == "da":
        F = c["cams"] * sum(h * w for h, w in _sizes(c["maps"]))
        p = c["B"] * c["anchors"] * c["pts"] * c["cams"]
        S = len(_sizes(c["maps"]))
        f, w, o = c["B"] * F * c["C"], p * S * c["G"], c["B"] * c["anchors"] * c["C"]
        fwd, bwd = e * (f + 2 * p + w + o), e * (2 * f + 4 * p + 2 * w + o)
        flops = 2 * 4 * p * S * c["C"] * 4 / 9   # the share of points in view
        return {"bytes": fwd + (bwd if train else 0), "flops": flops * (3 if train else 1)}
    if op == "dcn":
        s = c["stride"]
        m = c["N"] * ((c["height"] - 1) // s + 1) * ((c["width"] - 1) // s + 1)
        x, o = c["N"] * c["C"] * c["height"] * c["width"], m * c["Co"]
        w = c["Co"] * c["C"] // c["groups"] * 9
        t = m * c["deform_groups"] * (27 if c["modulated"] else 18)
        fwd, bwd = e * (x + w + t + o), e * (2 * x + 2 * w + 2 * t + o)
        return {"bytes": fwd + (bwd if train else 0), "flops": 2 * m * w * (3 if train else 1)}
    x = c["N"] * c["C"] * c["height"] * c["width"]
    y = c["N"] * c["C"] * ((c["height"] + 1) // 2) * ((c["width"] + 1) // 2)
    # the pooled tensor passes between two operators: written by one and read by the other
    return {"bytes": e * (x + 4 * y + (3 * y if train else 0)), "flops": 10 * y}


def tolerance(case):
    if case["op"] == "stem":
        return "exact"
    if case["dtype"] == "f32":
        # sums of a few hundred (dcn: a few thousand, from split operands) 32-bit products; location
        # gradients cancel, which "max" leaves room for
        return {"rel": 2e-5 if case["op"] == "dcn" else 1e-5, "max": 1e-3}
    return {"rel": 1e-2}
