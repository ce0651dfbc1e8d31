"""Performance cases of the MoE layer: the calls a user's program makes, over the range of sizes it makes them with.

Every case is one rank (the whole expert set local), seeded and synthetic:
  forward   build_schedule + forward: an inference step, BF16 or MXFP8 routed weights
  train     build_schedule + forward + backward: a training step that drives the functional API itself
  autograd  route_and_schedule + moe_experts + torch.autograd.grad: a training step of a model that leaves routing and
            gradients to the package
  quantise  mxfp8_quantize of a weight stack in both layouts: what an MXFP8 trainer does after each optimiser step
  schedule  the slot tables of one rank of an expert-parallel group, from the gathered routes of all of its ranks
Token counts, hidden and intermediate sizes are multiples of 256 (the layer's own rule); expert counts, top-k and
routing skew are free.
"""
import importlib
import math
import os
import sys

import torch
import torch.distributed as dist

# the package's folder has a dash in its name, so it is reached the way the tests reach it
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mixture-of-kittens_b200"))
mok = importlib.import_module("mok")
F, ops = mok.functional, mok.ops
nn = importlib.import_module("mok.nn")

MACROBATCH, MINIBATCH = 262144, 4096


def _layer(name, kind, T, H, I, E, K, *, mxfp8=False, zipf=0.0, limit=0.0, macrobatch=MACROBATCH):
    return {"name": name, "kind": kind, "T": T, "H": H, "I": I, "E": E, "K": K, "mxfp8": mxfp8, "zipf": zipf,
            "limit": limit, "macrobatch": macrobatch}


def listed():
    return [
        # the smallest layer the package accepts: launches and host time are all there is
        _layer("forward_smallest", "forward", 512, 256, 256, 4, 2),
        # a decode-sized batch on the benchmark's layer: a few tokens per expert, so reading the weights is the work
        _layer("forward_few_tokens", "forward", 512, 2048, 768, 128, 8),
        # the benchmark's inference step (prefill): many small experts, near-uniform routing
        _layer("forward_prefill", "forward", 16384, 2048, 768, 128, 8),
        # a small training step with the clamped SwiGLU
        _layer("train_small", "train", 1024, 512, 768, 8, 4, limit=3.0),
        # an ordinary fine-tuning step with sizes that divide into nothing evenly, router included
        _layer("autograd_ragged", "autograd", 2816, 1792, 1280, 24, 5),
        # skewed routing and a schedule of several windows: rows go through the combine buffer, backward replays forward
        _layer("train_skewed_windows", "train", 8192, 2048, 1024, 32, 4, zipf=1.2, macrobatch=16384),
        # the benchmark's training step: one GPU's share of the eight-rank BF16 workload
        _layer("train_large", "train", 16384, 4096, 1536, 8, 6),
        # MXFP8: a small training step, an inference step with moderate batch, and the benchmark's training step
        _layer("mxfp8_train_small", "train", 1024, 1024, 512, 16, 4, mxfp8=True),
        _layer("mxfp8_forward", "forward", 2048, 7168, 2048, 32, 8, mxfp8=True),
        _layer("mxfp8_train_large", "train", 16384, 7168, 2048, 32, 8, mxfp8=True),
        # one of the three weight stacks of that layer, quantised again after an optimiser step
        {"name": "quantise_weights", "kind": "quantise", "E": 32, "M": 2048, "N": 7168},
        # the tables of one of eight ranks at that layer's sizes
        {"name": "schedule_eight_ranks", "kind": "schedule", "W": 8, "T": 16384, "K": 8, "El": 32},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["forward", "forward", "train", "train", "autograd", "quantise", "schedule"])
    if kind == "quantise":
        return {"kind": kind, "E": rng.randint(1, 32), "M": 128 * int(_log_uniform(rng, 2, 17)), "N": 128 * int(_log_uniform(rng, 2, 57))}
    if kind == "schedule":
        return {"kind": kind, "W": rng.choice([1, 2, 4, 8]), "T": 256 * int(_log_uniform(rng, 2, 65)), "K": rng.randint(1, 8),
                "El": int(_log_uniform(rng, 2, 129))}
    T, H, I = 256 * int(_log_uniform(rng, 2, 65)), 256 * int(_log_uniform(rng, 1, 29)), 256 * int(_log_uniform(rng, 1, 9))
    K = rng.randint(1, 8)
    E = max(K, int(_log_uniform(rng, 4, 129)))
    while E * H * I > 20 * 7168 * 2048:                 # no more bytes than the largest listed layer moves
        E = max(K, E // 2)
        if E == K:
            H = max(256, H // 512 * 256)
    mxfp8 = kind != "autograd" and rng.random() < 0.4
    windows = rng.random() < 0.2                        # a schedule that does not fit one window
    return {"kind": kind, "T": T, "H": H, "I": I, "E": E, "K": K, "mxfp8": mxfp8,
            "zipf": round(rng.uniform(0.5, 1.3), 3) if rng.random() < 0.3 else 0.0,
            "limit": round(rng.uniform(2.5, 7.0), 2) if rng.random() < 0.3 else 0.0,
            "macrobatch": max(MINIBATCH, T * K // 2 // MINIBATCH * MINIBATCH) if windows else MACROBATCH}


# ------------------------------------------------------------------------------------------------------ inputs
def _group():
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    return dist.group.WORLD


def _randn(gen, *shape, std=1.0, dtype=torch.bfloat16):
    t = torch.empty(*shape, dtype=dtype, device="cuda")
    for part in (t if t.ndim == 3 else [t]):            # a slice at a time: no 32-bit copy of a whole weight stack
        part.copy_(torch.randn(part.shape, generator=gen, device="cuda") * std)
    return t


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "quantise":
        return {"w": _randn(gen, case["E"], case["M"], case["N"], std=case["N"] ** -0.5)}
    if case["kind"] == "schedule":
        logits = torch.rand(case["W"] * case["T"], case["W"] * max(case["El"], case["K"]), generator=gen, device="cuda")
        return {"topk": logits.topk(case["K"], dim=1).indices.int().view(case["W"], case["T"], case["K"])}
    T, H, I, E, K = (case[n] for n in "THIEK")
    logits = torch.randn(T, E, generator=gen, device="cuda") * 0.9
    if case["zipf"]:
        order = torch.randperm(E, generator=gen, device="cuda")
        logits -= case["zipf"] * torch.log(order.float() + 1.0)
    weights = [_randn(gen, I, H, std=H ** -0.5), _randn(gen, I, H, std=H ** -0.5), _randn(gen, H, I, std=I ** -0.5),
               _randn(gen, E, I, H, std=H ** -0.5), _randn(gen, E, I, H, std=H ** -0.5), _randn(gen, E, H, I, std=I ** -0.5)]
    got = {"x": _randn(gen, T, H), "logits": logits, "weights": weights}
    if case["kind"] != "forward":
        got["d_out"] = _randn(gen, T, H)
    top, experts = logits.topk(K, dim=1)
    got["experts"], got["rw"] = experts, torch.softmax(top, dim=1)
    return got


def prepare(case, seed):
    got = _inputs(case, seed)
    got["kind"] = case["kind"]
    if case["kind"] == "quantise":
        return got
    if case["kind"] == "schedule":
        rows = case["W"] * case["T"] * case["K"]
        got["capacity"] = (max(rows // case["W"] * 2, rows // 2) + 256 * case["El"] + 255) // 256 * 256
        got["El"], got["rank"] = case["El"], case["W"] // 2
        return got
    T, H, E, K = (case[n] for n in "THEK")
    need = T * K + 255 * E                              # every expert's rows are padded to 256
    got["config"] = F.MoKConfig(minibatch_size=MINIBATCH, macrobatch_size=case["macrobatch"],
                                schedule_capacity_multiplier=float(max(2, -(-need // (T * K)))),
                                all_gather_top_experts_chunk_bytes=1024)
    got["workspace"] = F.create_workspace(got["config"], _group(), device=torch.device("cuda", torch.cuda.current_device()),
                                          num_local_tokens=T, hidden_size=H, topk=K)
    got["E"], got["limit"] = E, case["limit"] or None
    shared, routed = got["weights"][:3], got["weights"][3:]
    got["fwd_weights"] = got["bwd_weights"] = got["weights"]
    if case["mxfp8"]:
        both = case["kind"] != "forward"
        g, u, d = (ops.mxfp8_quantize(w, True, both) for w in routed)
        got["fwd_weights"] = shared + [(g[0], g[1]), (u[0], u[1]), (d[0], d[1])]
        got["bwd_weights"] = shared + [tuple(g), tuple(u), (d[2], d[3])]
        del got["weights"]
    if case["kind"] == "autograd":
        got["leaves"] = [t.requires_grad_(True) for t in (got["x"], got["logits"], *got["weights"])]
    return got


# ------------------------------------------------------------------------------------------------------ the calls
def run(s):
    if s["kind"] == "quantise":
        return [t.view(torch.uint8) for t in ops.mxfp8_quantize(s["w"], True, True)]
    if s["kind"] == "schedule":
        return list(ops.schedule(s["topk"], s["El"], s["capacity"], s["rank"]))
    config, ws = s["config"], s["workspace"]
    if s["kind"] == "autograd":
        schedule, _, rw = F.route_and_schedule(ws, config, s["logits"], num_local_experts=s["E"])
        out = nn.moe_experts(config, ws, schedule, s["x"], rw, *s["weights"], swiglu_limit=s["limit"])
        return [out, *torch.autograd.grad(out, s["leaves"], s["d_out"])]
    schedule = F.build_schedule(ws, config, s["experts"], num_local_experts=s["E"])
    out, ctx = F.forward(config, ws, schedule, s["x"], s["rw"], *s["fwd_weights"], swiglu_limit=s["limit"])
    if s["kind"] == "forward":
        return [out]
    return [out, *F.backward(config, ws, schedule, ctx, s["d_out"], s["x"], s["rw"], *s["bwd_weights"], swiglu_limit=s["limit"])]


def work(case):
    if case["kind"] == "quantise":
        n = case["E"] * case["M"] * case["N"]
        return {"bytes": 2 * n + 2 * (n + n // 32), "flops": 0}
    if case["kind"] == "schedule":
        rows = case["W"] * case["T"] * case["K"]
        capacity = (max(rows // case["W"] * 2, rows // 2) + 256 * case["El"] + 255) // 256 * 256
        return {"bytes": 4 * rows + 8 * capacity + 4 * case["El"] + 4, "flops": 0}
    T, H, I, E, K = (case[n] for n in "THIEK")
    back = case["kind"] != "forward"
    act, shared, routed = 2 * T * H, 6 * H * I, 3 * E * H * I
    one = 33 / 32 if case["mxfp8"] else 2.0             # bytes of a routed weight
    b = 2 * act + 12 * T * K + shared + one * routed    # x, output, routes and their weights, the expert weights
    if back:                                            # grad_output and d_x, weight gradients, the weights once more
        b += 2 * act + 8 * T * K + 2 * shared + 2 * routed + one * routed
    return {"bytes": b, "flops": 6.0 * (T + T * K) * H * I * (3 if back else 1)}


def tolerance(case):
    if case["kind"] in ("quantise", "schedule"):
        return "exact"
    # BF16: products are rounded to bf16 between the GEMMs (2^-9 each).  MXFP8: gate, up, hidden and their gradients are
    # rounded to 3-bit mantissas between the GEMMs, so a sum in another order moves single values by 2^-4
    return {"rel": 2e-2} if case["mxfp8"] else {"rel": 1e-2}


# ------------------------------------------------------------------------------------------------------ 64 bits
def _ffn(x, wg, wu, limit):
    g, u = x @ wg.T, x @ wu.T
    gc, uc = (g.clamp(max=limit), u.clamp(-limit, limit)) if limit else (g, u)
    sig = torch.sigmoid(gc)
    return g, u, gc, uc, sig, gc * sig * uc


def _ffn_back(d_hid, f, limit):
    g, u, gc, uc, sig, _ = f
    dg, du = d_hid * uc * sig * (1 + gc * (1 - sig)), d_hid * gc * sig
    return (dg * (g <= limit), du * (u.abs() <= limit)) if limit else (dg, du)


def exact(case, seed):
    """The layer in 64 bits from the same inputs.  MXFP8 cases are compared with the unquantised layer."""
    if case["kind"] in ("quantise", "schedule"):
        return None
    s = _inputs(case, seed)
    limit, back = case["limit"] or None, case["kind"] != "forward"
    f64 = lambda t: t.double()  # noqa: E731
    x, experts, T, E, K = f64(s["x"]), s["experts"], case["T"], case["E"], case["K"]
    top = f64(s["logits"]).gather(1, experts)
    rw = torch.softmax(top, dim=1) if case["kind"] == "autograd" else f64(s["rw"])
    sg, su, sd = (f64(w) for w in s["weights"][:3])
    d_out = f64(s["d_out"]) if back else None
    f = _ffn(x, sg, su, limit)
    out = f[5] @ sd.T
    if back:
        dg, du = _ffn_back(d_out @ sd, f, limit)
        d_x = dg @ sg + du @ su
        d_shared = [dg.T @ x, du.T @ x, d_out.T @ f[5]]
        d_rw = torch.zeros_like(rw)
        d_routed = [torch.zeros(w.shape, dtype=torch.float64, device="cuda") for w in s["weights"][3:]]
    del f
    for e in range(E):
        wg, wu, wd = (f64(w[e]) for w in s["weights"][3:])
        tok, k = (experts == e).nonzero(as_tuple=True)
        w, xe = rw[tok, k].unsqueeze(1), x[tok]
        f = _ffn(xe, wg, wu, limit)
        y = f[5] @ wd.T
        out.index_add_(0, tok, w * y)
        if back:
            d_y = d_out[tok]
            d_rw[tok, k] = (d_y * y).sum(1)
            dg, du = _ffn_back((w * d_y) @ wd, f, limit)
            d_x.index_add_(0, tok, dg @ wg + du @ wu)
            for grad, value in zip(d_routed, (dg.T @ xe, du.T @ xe, (w * d_y).T @ f[5])):
                grad[e] = value
        del f
    if not back:
        return [out]
    if case["kind"] == "autograd":
        d_logits = torch.zeros(T, E, dtype=torch.float64, device="cuda")
        d_logits.scatter_(1, experts, rw * (d_rw - (rw * d_rw).sum(1, keepdim=True)))
        return [out, d_x, d_logits, *d_shared, *d_routed]
    return [out, d_x, d_rw, *d_routed, *d_shared]
