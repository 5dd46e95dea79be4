"""Performance cases of the multislice mixed-probe ptychography path.

Each case is one call (or one differentiable step) that a program built on this package
makes through its public entry points: gradient steps of the reconstruction at every built
probe window, the forward simulation, the analytic update, a multi-dataset step, the
optional object and probe constraints, and the learned initialiser's network.  ``exact``
restates every path in 64-bit PyTorch.
"""
import math

import numpy as np
import torch

from quantem_b200 import engine, multi, ops
from quantem_b200.core.ml.cnn import CNN2d, mse_loss
from quantem_b200.diffractive_imaging import ptycho_utils

DEVICE = "cuda"
ENERGY_LAMBDA = 0.019687489   # electron wavelength at 300 kV [A]
PIXEL = 0.2                   # real-space pixel [A]
DZ = 20.0                     # slice thickness [A]


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the single-slice, single-mode iteration: the smallest call, 256 positions of 64^2
        # replayed from a CUDA graph with its Adam steps (latency and launches)
        {"name": "iteration_64_graphed", "kind": "graph", "n": 64, "slices": 1, "modes": 1, "rows": 16, "cols": 16,
         "step": 4, "batch": 256, "loss": "l2_amplitude", "positions": False},
        # an ordinary mini-batch of the headline geometry (8 slices, 4 modes, 128^2)
        {"name": "gradient_128_minibatch", "kind": "gradient", "n": 128, "slices": 8, "modes": 4, "rows": 32,
         "cols": 32, "step": 6, "batch": 256, "loss": "l2_amplitude", "positions": False},
        # the headline iteration: a full batch of the 64 x 64 raster
        {"name": "gradient_128_full", "kind": "gradient", "n": 128, "slices": 8, "modes": 4, "rows": 64, "cols": 64,
         "step": 6, "batch": 4096, "loss": "l2_amplitude", "positions": False},
        # 96^2 windows, ragged scan and batch, Poisson likelihood, scan positions refined
        {"name": "gradient_96_refine", "kind": "gradient", "n": 96, "slices": 3, "modes": 2, "rows": 27, "cols": 31,
         "step": 5, "batch": 701, "loss": "poisson", "positions": True},
        # 256^2 windows on thread-block clusters: the large multislice geometry, a mini-batch
        {"name": "gradient_256_minibatch", "kind": "gradient", "n": 256, "slices": 16, "modes": 6, "rows": 12,
         "cols": 12, "step": 6, "batch": 64, "loss": "l2_amplitude", "positions": False},
        # forward simulation of a 32 x 32 crop: the training data of the learned initialiser
        {"name": "forward_128", "kind": "forward", "n": 128, "slices": 8, "modes": 4, "rows": 32, "cols": 32,
         "step": 6, "batch": 1024},
        # the analytic (autograd=False) update directions of a batch
        {"name": "analytic_128", "kind": "analytic", "n": 128, "slices": 4, "modes": 2, "rows": 20, "cols": 20,
         "step": 6, "batch": 400},
        # six datasets of uneven size with 96^2 and 128^2 windows in one multi-dataset step
        {"name": "multi_dataset", "kind": "multi",
         "sets": "24:1:96 32:2:128 40:3:96 48:5:128 56:6:96 64:8:128", "step": 4},
        # the optional object constraints (blur, Butterworth low-pass, TV) and their gradient
        {"name": "object_constraints", "kind": "object", "type": "complex", "slices": 8, "height": 510, "width": 516,
         "sigma": 1.0, "lowpass": 1.0},
        # the probe constraints (orthogonalisation, centring, TV) and their gradient
        {"name": "probe_constraints", "kind": "probe", "n": 128, "modes": 4},
        # one training step of the learned initialiser: 16 objects of 32 x 32 positions
        {"name": "network_train", "kind": "train", "cin": 1024, "cout": 36, "filters": 32, "levels": 5, "batch": 16,
         "side": 32},
        # its inference on a 64 x 64 scan
        {"name": "network_infer", "kind": "infer", "cin": 1024, "cout": 36, "filters": 32, "levels": 5, "batch": 1,
         "side": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gradient"] * 5 + ["graph", "forward", "analytic", "multi", "object", "probe", "train", "infer"])
    if kind in ("gradient", "graph", "forward", "analytic"):
        n = 64 if kind == "graph" else rng.choice([64, 96, 128, 256] if kind in ("gradient", "forward") else [64, 96, 128])
        c = {"kind": kind, "n": n, "slices": _log(rng, 1, 12), "modes": _log(rng, 1, 6), "step": rng.randint(3, 8)}
        # keep a drawn case below the cost of the full headline batch
        most = 4096 * 8 * 4 * 128 ** 2 / (c["slices"] * c["modes"] * n * n) / (6 if n == 256 else 1.5)
        batch = max(5, min(_log(rng, 5, 3000), int(most)))
        side = max(3, math.ceil(math.sqrt(batch)) + rng.randint(0, 3))
        c.update(rows=side, cols=side + rng.randint(0, 4), batch=batch)
        if kind in ("gradient", "graph"):
            c["loss"] = rng.choice(["l2_amplitude", "l2_amplitude", "l2_intensity", "poisson"])
            c["positions"] = kind == "gradient" and n != 256 and rng.random() < 0.3
        return c
    if kind == "multi":
        return {"kind": "multi", "step": rng.randint(3, 6), "sets": " ".join(
            "%d:%d:%d" % (_log(rng, 5, 36), rng.randint(1, 6), rng.choice([64, 96, 128])) for _ in range(rng.randint(2, 4)))}
    if kind == "object":
        return {"kind": "object", "type": rng.choice(["complex", "complex", "potential"]), "slices": _log(rng, 1, 10),
                "height": rng.randint(150, 560), "width": rng.randint(150, 560),
                "sigma": round(rng.uniform(0.5, 2.0), 2), "lowpass": round(rng.uniform(0.6, 2.0), 2)}
    if kind == "probe":
        return {"kind": "probe", "n": rng.choice([64, 96, 128, 256]), "modes": rng.randint(1, 8)}
    side = rng.choice([32, 64]) if kind == "infer" else 32
    return {"kind": kind, "cin": rng.choice([64, 256, 1024]), "cout": rng.choice([1, 9, 25, 36]),
            "filters": rng.choice([16, 32]), "levels": rng.randint(2, 5), "batch": _log(rng, 1, 16), "side": side}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) % (1 << 31))


def _smooth(shape, gen, width):
    """Band-limited Gaussian noise of unit variance per slice."""
    x = torch.randn(shape, generator=gen, device=DEVICE)
    qr = torch.fft.fftfreq(shape[-2], device=DEVICE)[:, None]
    qc = torch.fft.rfftfreq(shape[-1], device=DEVICE)[None]
    y = torch.fft.irfft2(torch.fft.rfft2(x) * torch.exp(-2 * (math.pi * width) ** 2 * (qr ** 2 + qc ** 2)), s=shape[-2:])
    return y / y.std(dim=(-2, -1), keepdim=True)


def _amplitude(shape, gen):
    """Amplitudes of an iterate on both sides of the clamp at 1, a little away from its edge."""
    u = 0.15 * torch.rand(shape, generator=gen, device=DEVICE) - 0.12
    return 1.0 + u + 0.001 * torch.sign(u)


def _modes(n, P, gen):
    """P probe modes: a 20 mrad aperture at 200 A defocus, each mode with its own smooth phase."""
    k = torch.fft.fftfreq(n, PIXEL, device=DEVICE)
    k2 = k[:, None] ** 2 + k[None] ** 2
    edge = 0.020 / ENERGY_LAMBDA
    ap = torch.sigmoid((edge - k2.sqrt()) * n * PIXEL * 2)
    chi = math.pi * ENERGY_LAMBDA * 200.0 * k2
    c = torch.randn((P, 3), generator=gen, device=DEVICE)
    ph = chi[None] + (c[:, 0, None, None] * k[None, :, None] + c[:, 1, None, None] * k[None, None, :]) * 4.0 / edge
    ph = ph + c[:, 2, None, None] * (k2 / edge ** 2)[None]
    p = torch.fft.ifft2(torch.polar(ap.expand(P, n, n).contiguous(), ph))
    w = torch.tensor([0.6 ** i for i in range(P)], device=DEVICE)
    w = w / w.sum()
    return (p * torch.sqrt(w / p.abs().square().sum(dim=(-2, -1)))[:, None, None]).to(torch.complex64)


def _dataset(n, S, P, rows, cols, step, gen, counts=1e5, intensities=False):
    """Current object and probe iterates, propagators, positions and measured data."""
    Ho, Wo = (rows - 1) * step + n + 6, (cols - 1) * step + n + 7
    phase = 0.15 * _smooth((S, Ho, Wo), gen, 1.5)
    rr, cc = torch.meshgrid(torch.arange(rows, device=DEVICE), torch.arange(cols, device=DEVICE), indexing="ij")
    pos = torch.stack([rr.reshape(-1), cc.reshape(-1)], -1) * float(step) + n // 2 + 3
    pos = (pos + torch.rand(pos.shape, generator=gen, device=DEVICE) - 0.5).float().contiguous()
    probe = _modes(n, P, gen) * math.sqrt(counts)
    # measured patterns: the projected object, Poisson noise
    proj = torch.polar(torch.ones_like(phase[0]), phase.sum(0))
    f = torch.fft.fftfreq(n, 1.0 / n, device=DEVICE).round().long()
    data = torch.empty((pos.shape[0], n, n), device=DEVICE)
    for s in range(0, pos.shape[0], 256):
        r0 = pos[s:s + 256].round().long()
        pat = proj[((r0[:, 0, None] + f) % Ho)[:, :, None], ((r0[:, 1, None] + f) % Wo)[:, None, :]]
        inten = torch.zeros(pat.shape, device=DEVICE)
        for m in range(P):
            inten += torch.fft.fft2(pat * probe[m], norm="ortho").abs().square()
        data[s:s + 256] = torch.poisson(torch.fft.fftshift(inten, dim=(-2, -1)), generator=gen)
    mean = float(data.double().sum() / data.shape[0])
    obj = torch.polar(_amplitude((S, Ho, Wo), gen),
                      0.5 * phase + 0.02 * torch.randn((S, Ho, Wo), generator=gen, device=DEVICE))
    probe = probe * (1 + 0.05 * torch.randn(probe.shape, generator=gen, device=DEVICE))
    k = torch.fft.fftfreq(n, PIXEL, dtype=torch.float64)
    fac = torch.polar(torch.ones(S - 1, n, dtype=torch.float64),
                      (-math.pi * ENERGY_LAMBDA * DZ * k ** 2)[None].expand(S - 1, n).contiguous())
    fac = fac.to(torch.complex64).to(DEVICE)
    return {"obj": obj.to(torch.complex64).contiguous(), "probe": probe.to(torch.complex64).contiguous(),
            "prop": (fac, fac.clone()), "pos": pos, "data": data if intensities else data.sqrt(), "mean": mean,
            "mask": torch.ones((n, n), device=DEVICE)}


def _single(case, seed):
    g = _gen(seed)
    d = _dataset(case["n"], case["slices"], case["modes"], case["rows"], case["cols"], case["step"], g,
                 intensities=case.get("loss", "l2_amplitude") in ("poisson", "l2_intensity"))
    d["idx"] = torch.randperm(d["pos"].shape[0], generator=g, device=DEVICE)[:case["batch"]].contiguous()
    return d


def _sets(case):
    return [tuple(int(v) for v in s.split(":")) for s in case["sets"].split()]


def _many(case, seed):
    g = _gen(seed)
    out = []
    for scan, S, n in _sets(case):
        d = _dataset(n, S, 1, scan, scan, case["step"], g)
        d["idx"] = torch.randperm(d["pos"].shape[0], generator=g, device=DEVICE)
        out.append(d)
    return out


def _object(case, seed):
    g = _gen(seed)
    shape = (case["slices"], case["height"], case["width"])
    ph = 0.2 * _smooth(shape, g, 1.0) + 0.02 * torch.randn(shape, generator=g, device=DEVICE)
    up = torch.complex(torch.randn(shape, generator=g, device=DEVICE), torch.randn(shape, generator=g, device=DEVICE))
    if case["type"] == "potential":
        return {"obj": (ph + 0.4).contiguous(), "up": up * 1e-2}
    return {"obj": torch.polar(_amplitude(shape, g), ph).to(torch.complex64).contiguous(), "up": up * 1e-2}


def _probes(case, seed):
    g = _gen(seed)
    p = _modes(case["n"], case["modes"], g) * 300.0
    p = torch.roll(p, (2, -3), dims=(-2, -1))
    p = (p * (1 + 0.1 * torch.randn(p.shape, generator=g, device=DEVICE))).to(torch.complex64).contiguous()
    up = torch.randn(p.shape, generator=g, device=DEVICE, dtype=torch.complex64)
    return {"probe": p, "up": up}


def _layers(case):
    """(name, kind, in, out) of every layer of the network, in the order of its flat parameters."""
    L, f = case["levels"], case["filters"]

    def block(prefix, ci, co):
        for j in range(2):
            yield f"{prefix}.block.{3 * j}", "conv", ci if j == 0 else co, co
            yield f"{prefix}.block.{3 * j + 2}", "bn", co, co

    ci = case["cin"]
    for l in range(L):
        co = f << l
        yield from block(f"down_conv_blocks.{l}", ci, co)
        ci = co
    yield from block("bottleneck", ci, 2 * ci)
    ci = 2 * ci
    for u in range(L):
        co = f if u == L - 1 else ci // 2
        yield f"upsample_blocks.{u}.upsample2x", "up", ci, ci
        yield f"upsample_blocks.{u}.conv", "one", ci, co
        yield f"upsample_blocks.{u}.bn", "bn", co, co
        yield from block(f"up_conv_blocks.{u}", ci, co)
        ci = co
    yield "final_conv.block.0", "conv", f, case["cout"]


def _weights(case, gen):
    sd = {}
    for name, kind, ci, co in _layers(case):
        if kind == "bn":
            sd[name + ".weight"] = 1 + 0.1 * torch.randn(co, generator=gen, device=DEVICE)
            sd[name + ".bias"] = 0.1 * torch.randn(co, generator=gen, device=DEVICE)
            sd[name + ".running_mean"] = 0.3 + 0.05 * torch.randn(co, generator=gen, device=DEVICE)
            sd[name + ".running_var"] = 0.3 + 0.1 * torch.rand(co, generator=gen, device=DEVICE)
            continue
        shape = {"conv": (co, ci, 3, 3), "up": (ci, co, 3, 3), "one": (co, ci, 1, 1)}[kind]
        fan = ci * (1 if kind == "one" else 9)
        sd[name + ".weight"] = torch.randn(shape, generator=gen, device=DEVICE) / math.sqrt(fan)
        sd[name + ".bias"] = 0.1 * torch.randn(co, generator=gen, device=DEVICE)
    return {k: v.cpu() for k, v in sd.items()}


def _network(case, seed):
    g = _gen(seed)
    sd = _weights(case, g)
    B, s = case["batch"], case["side"]
    # binned patterns of neighbouring scan positions resemble each other: smooth maps plus noise
    x = _smooth((B * case["cin"], s, s), g, 1.5) + 0.3 * torch.randn((B * case["cin"], s, s), generator=g, device=DEVICE)
    x = x.view(B, case["cin"], s * s).permute(0, 2, 1).reshape(B * s * s, case["cin"]).to(torch.bfloat16).contiguous()
    t = 0.3 * torch.randn((B, case["cout"], s, s), generator=g, device=DEVICE)
    return sd, x, t


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": dict(case)}
    if kind in ("gradient", "graph"):
        d = _single(case, seed)
        pt = engine.ProblemTensors(
            obj=d["obj"].requires_grad_(True), probe=d["probe"].requires_grad_(True), prop=d["prop"],
            positions=d["pos"].requires_grad_(bool(case["positions"])), targets=d["data"].contiguous(),
            mask=d["mask"], mean_intensity=d["mean"], upsample_factor=float(case["step"]), loss_type=case["loss"])
        state.update(pt=pt, idx=d["idx"])
        if kind == "graph":
            state["graph"] = engine.GraphedIteration(pt, lr_obj=1e-3, lr_probe=1e-3, batch_idx=d["idx"]).capture(warmup=1)
    elif kind in ("forward", "analytic"):
        d = _single(case, seed)
        # the constrained object and the orthogonalised probe of the current iterate
        with torch.no_grad():
            d["obj"] = ops.constrained_object(d["obj"])
            d["probe"] = ptycho_utils.orthogonalize_probes(d["probe"])
        state.update(d)
    elif kind == "multi":
        state["problems"] = [
            multi.Problem(d["obj"].requires_grad_(True), d["probe"].requires_grad_(True), d["prop"], d["pos"],
                          d["data"].contiguous(), d["mask"], d["mean"], float(case["step"]), batch_idx=d["idx"])
            for d in _many(case, seed)]
        state["grids"] = multi.default_grids(state["problems"])
    elif kind == "object":
        d = _object(case, seed)
        d["obj"].requires_grad_(True)
        state.update(d)
        state["constraints"] = {"gaussian_sigma": case["sigma"], "q_lowpass": case["lowpass"], "butterworth_order": 4}
    elif kind == "probe":
        d = _probes(case, seed)
        d["probe"].requires_grad_(True)
        state.update(d)
    else:
        sd, x, t = _network(case, seed)
        net = CNN2d(case["cin"], case["cout"], start_filters=case["filters"], num_layers=case["levels"], device=DEVICE)
        net.load_state_dict(sd)
        net.train(kind == "train")
        state.update(net=net, x=x, target=t, rows=(case["batch"], case["side"], case["side"]))
    return state


def run(state):
    kind = state["kind"]
    if kind == "gradient":
        pt = state["pt"]
        pt.obj.grad = pt.probe.grad = pt.positions.grad = None
        loss = engine.batch_step(pt, state["idx"])
        out = {"loss": loss, "obj": pt.obj.grad, "probe": pt.probe.grad}
        if pt.positions.grad is not None:
            out["positions"] = pt.positions.grad
        return out
    if kind == "graph":
        loss = state["graph"].replay()
        pt = state["pt"]
        return {"loss": loss, "obj": pt.obj, "probe": pt.probe}
    if kind == "forward":
        s = state
        out = ops.batch_forward(s["obj"], s["probe"], s["prop"], s["pos"], s["idx"], s["data"], s["mask"],
                                s["pos"].shape[0], s["mean"])
        return {"loss": out["loss"], "intensity": out["intensity"]}
    if kind == "analytic":
        s = state
        loss, g_obj, g_probe = ops.batch_analytic(s["obj"], s["probe"], s["prop"], s["pos"], s["idx"], s["data"],
                                                  s["mask"], s["pos"].shape[0], s["mean"])
        return {"loss": loss, "obj": g_obj, "probe": g_probe}
    if kind == "multi":
        for p in state["problems"]:
            p.obj.grad = p.probe.grad = None
        losses = multi.multi_losses(state["problems"], state["grids"])
        losses.sum().backward()
        return {"losses": losses.detach(), "obj": [p.obj.grad for p in state["problems"]],
                "probe": [p.probe.grad for p in state["problems"]]}
    if kind == "object":
        obj, ty = state["obj"], state["case"]["type"]
        obj.grad = None
        out = ops.constrained_object_ext(obj, ty, state["constraints"], sampling=(PIXEL, PIXEL))
        soft = ops.soft_constraint_loss(out, ty, tv_weight_z=0.01, tv_weight_xy=0.01)
        t = ops.transmission_of(out)
        torch.autograd.backward([t, soft], [state["up"], torch.ones_like(soft)])
        return {"transmission": t.detach(), "soft": soft.detach(), "obj": obj.grad}
    if kind == "probe":
        probe = state["probe"]
        probe.grad = None
        out = ptycho_utils.center_probe(ptycho_utils.orthogonalize_probes(probe))
        tv = ptycho_utils.probe_tv_loss(out, 0.1)
        torch.autograd.backward([out, tv], [state["up"], torch.ones_like(tv)])
        return {"probe": out.detach(), "tv": tv.detach(), "grad": probe.grad}
    net = state["net"]
    if kind == "infer":
        with torch.no_grad():
            return {"out": net(state["x"], rows=state["rows"])}
    net.flat.grad = None
    pred = net(state["x"], rows=state["rows"])
    loss = mse_loss(pred, state["target"])
    loss.backward()
    return {"loss": loss.detach(), "out": pred.detach(), "grad": net.flat.grad}


# ---------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------
def _pty_work(n, S, P, rows, cols, step, B, backward):
    hw, obj = n * n, S * ((rows - 1) * step + n + 6) * ((cols - 1) * step + n + 7)
    fl = B * P * S * (2 * 5 * hw * math.log2(hw) + 20 * hw) * (2 if backward else 1)
    by = 4 * hw * B + 8 * obj + 8 * P * hw
    return fl, by + (8 * obj + 8 * P * hw if backward else 4 * hw * B)


def work(case):
    kind = case["kind"]
    if kind in ("gradient", "graph", "forward", "analytic"):
        fl, by = _pty_work(case["n"], case["slices"], case["modes"], case["rows"], case["cols"], case["step"],
                           case["batch"], kind != "forward")
        if kind == "graph":  # Adam: moments read and written, parameters written
            by += 5 * 8 * case["slices"] * ((case["rows"] - 1) * case["step"] + case["n"] + 6) * \
                ((case["cols"] - 1) * case["step"] + case["n"] + 7)
    elif kind == "multi":
        parts = [_pty_work(n, S, 1, scan, scan, case["step"], scan * scan, True) for scan, S, n in _sets(case)]
        fl, by = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "object":
        size = case["slices"] * case["height"] * case["width"]
        taps = 2 * math.ceil(3 * case["sigma"]) + 1
        fl = size * (4 * 5 * math.log2(case["height"] * case["width"]) + 2 * 2 * 4 * taps + 100)
        by = size * (8 * 3 + (8 if case["type"] == "complex" else 4))
    elif kind == "probe":
        hw, P = case["n"] ** 2, case["modes"]
        fl = hw * P * (4 * 5 * math.log2(hw) + 16 * P + 100)
        by = 4 * 8 * hw * P
    else:
        fl, by, lvl = 0.0, 0.0, 0
        B, side, L = case["batch"], case["side"], case["levels"]
        for name, k, ci, co in _layers(case):
            if name.startswith("down_conv_blocks"):
                lvl = int(name.split(".")[1])
            elif name.startswith("bottleneck"):
                lvl = L
            elif name.startswith(("upsample_blocks", "up_conv_blocks")):
                lvl = L - 1 - int(name.split(".")[1]) + (1 if k == "up" else 0)
            else:
                lvl = 0
            if k != "bn":
                taps = 1 if k == "one" else 9
                fl += 2.0 * B * (side >> lvl) ** 2 * taps * ci * co * (3 if kind == "train" else 1)
                by += 4.0 * taps * ci * co * (2 if kind == "train" else 1)
        by += B * side * side * (2 * case["cin"] + 4 * case["cout"])
    return {"bytes": float(by), "flops": float(fl)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _constrain64(o):
    ph = torch.angle(o)
    return torch.polar(torch.clamp(o.abs(), 0, 1), ph - ph.mean())


def _ortho64(p):
    norms = torch.sqrt((p.real ** 2 + p.imag ** 2).sum(dim=(-2, -1)))
    out = []
    for i in range(p.shape[0]):
        u = p[i]
        for q in out:
            u = u - (q.conj() * u).sum() * q
        out.append(u / torch.sqrt((u.real ** 2 + u.imag ** 2).sum()).clamp_min(1e-12))
    o = torch.stack(out) * norms[:, None, None]
    return o[torch.argsort((o.real ** 2 + o.imag ** 2).sum(dim=(-2, -1)).detach(), descending=True)]


class _Model64:
    """The multislice forward model of one dataset, evaluated in chunks of positions."""

    def __init__(self, d):
        self.n = d["mask"].shape[0]
        self.S, self.Ho, self.Wo = d["obj"].shape
        self.kr, self.kc = (t.to(torch.complex128) for t in d["prop"])
        self.f = torch.fft.fftfreq(self.n, 1.0 / self.n, device=DEVICE).round().long()
        self.q = self.f.double() / self.n
        per = d["probe"].shape[0] * self.S * self.n ** 2 * 16 * 8
        self.chunk = max(1, min(256, int(6e9 / per)))

    def index(self, pos):
        r0 = pos.detach().round().long()
        return (((r0[:, 0, None] + self.f) % self.Ho)[:, :, None] * self.Wo
                + ((r0[:, 1, None] + self.f) % self.Wo)[:, None, :])

    def far(self, obj, probe_hat, pos, keep=None):
        """Far fields (P, b, n, n); ``keep`` collects (index, patch, wave) of every slice."""
        frac = pos - pos.detach().round()
        ramp = torch.polar(torch.ones((), dtype=torch.float64, device=DEVICE),
                           -2 * math.pi * (self.q[None, :, None] * frac[:, 0, None, None]
                                           + self.q[None, None, :] * frac[:, 1, None, None]))
        at = self.index(pos)
        psi = torch.fft.ifft2(probe_hat[:, None] * ramp[None])
        for s in range(self.S):
            patch = obj[s].reshape(-1)[at]
            if keep is not None:
                keep.append((at, patch, psi))
            psi = psi * patch[None]
            if s < self.S - 1:
                psi = torch.fft.ifft2(torch.fft.fft2(psi) * (self.kr[s][:, None] * self.kc[s][None]))
        return torch.fft.fft2(psi, norm="ortho")


def _loss64(far, t, mask, loss, scale, mean):
    inten = torch.fft.fftshift((far.real ** 2 + far.imag ** 2).sum(0), dim=(-2, -1))
    if loss == "l2_amplitude":
        return (((torch.sqrt(inten + 1e-9) - t) * mask) ** 2).sum() * scale
    if loss == "l2_intensity":
        return (((inten - t) * mask) ** 2).sum() * scale
    return (inten - t * torch.log(inten + 1e-6)).sum() / mean


def _gradient64(d, raw_obj, raw_probe, loss, rescale, positions=False):
    """(loss, object gradient, probe gradient, position gradient) of one batch step."""
    m = _Model64(d)
    o = raw_obj.detach().clone().requires_grad_(True)
    p = raw_probe.detach().clone().requires_grad_(True)
    oc, ph = _constrain64(o), torch.fft.fft2(_ortho64(p))
    ol, pl = oc.detach().requires_grad_(True), ph.detach().requires_grad_(True)
    total, gpos = 0.0, torch.zeros(d["pos"].shape, dtype=torch.float64, device=DEVICE)
    scale = d["pos"].shape[0] / d["idx"].numel() / d["mean"]
    mask = d["mask"].double()
    for s in range(0, d["idx"].numel(), m.chunk):
        i = d["idx"][s:s + m.chunk]
        pos = d["pos"].detach()[i].double().requires_grad_(positions)
        v = _loss64(m.far(ol, pl, pos), d["data"][i].double(), mask, loss, scale, d["mean"])
        v.backward()
        total += float(v)
        if positions:
            gpos[i] = pos.grad
    go, = torch.autograd.grad(oc, o, ol.grad)
    gp, = torch.autograd.grad(ph, p, pl.grad)
    return torch.tensor(total, dtype=torch.float64), go * rescale, gp, gpos


def _adam64(x, g, st, lr):
    st["t"] += 1
    xr, gr = torch.view_as_real(x), torch.view_as_real(g)
    st["m"] = 0.9 * st["m"] + 0.1 * gr
    st["v"] = 0.999 * st["v"] + 0.001 * gr * gr
    a = st["m"] / (1 - 0.9 ** st["t"])
    return torch.view_as_complex(xr - lr * a / (torch.sqrt(st["v"] / (1 - 0.999 ** st["t"])) + 1e-8))


def _network64(case, sd, x, training):
    """The network's output and its 64-bit parameters (leaf tensors)."""
    F = torch.nn.functional
    w = {k: v.to(DEVICE).double() for k, v in sd.items()}
    for k in w:
        if not k.endswith(("running_mean", "running_var")):
            w[k].requires_grad_(True)

    def bn(y, name):
        return F.batch_norm(y, w[name + ".running_mean"].clone(), w[name + ".running_var"].clone(),
                            w[name + ".weight"], w[name + ".bias"], training=training, eps=1e-5)

    def conv(y, name):
        return F.conv2d(F.pad(y, (1, 1, 1, 1), mode="circular"), w[name + ".weight"], w[name + ".bias"])

    def block(y, prefix):
        for j in range(2):
            y = bn(F.relu(conv(y, f"{prefix}.block.{3 * j}")), f"{prefix}.block.{3 * j + 2}")
        return y

    B, s = case["batch"], case["side"]
    y = x.double().view(B, s, s, case["cin"]).permute(0, 3, 1, 2)
    skips = []
    for l in range(case["levels"]):
        y = block(y, f"down_conv_blocks.{l}")
        skips.append(y)
        y = F.max_pool2d(y, 2)
    y = block(y, "bottleneck")
    for u in range(case["levels"]):
        p = f"upsample_blocks.{u}"
        y = F.conv_transpose2d(y, w[p + ".upsample2x.weight"], w[p + ".upsample2x.bias"], stride=2, padding=1,
                               output_padding=1)
        y = bn(F.conv2d(y, w[p + ".conv.weight"], w[p + ".conv.bias"]), p + ".bn")
        y = block(torch.cat([y, skips.pop()], dim=1), f"up_conv_blocks.{u}")
    return conv(y, "final_conv.block.0"), w


def _flat64(case, w):
    """Parameter gradients in the order and layout of the network's flat parameter tensor."""
    parts = []

    def put(t):
        t = t.reshape(-1)
        parts.append(torch.nn.functional.pad(t, (0, -t.numel() % 8)))

    for name, kind, _, _ in _layers(case):
        g = w[name + ".weight"].grad
        if kind == "conv":
            g = g.permute(0, 2, 3, 1)
        elif kind == "up":
            g = g.permute(2, 3, 1, 0)
        put(g)
        put(w[name + ".bias"].grad)
    return torch.cat(parts)


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        d = _single(case, seed)
        loss, go, gp, gpos = _gradient64(d, d["obj"].to(torch.complex128), d["probe"].to(torch.complex128),
                                         case["loss"], case["step"] ** 2 / 2, bool(case["positions"]))
        out = {"loss": loss, "obj": go, "probe": gp}
        if case["positions"]:
            out["positions"] = gpos
        return out
    if kind == "graph":  # one warm-up iteration, then the replayed one
        d = _single(case, seed)
        o, p = d["obj"].to(torch.complex128), d["probe"].to(torch.complex128)
        sts = [{"t": 0, "m": 0.0, "v": 0.0} for _ in range(2)]
        for _ in range(2):
            loss, go, gp, _ = _gradient64(d, o, p, case["loss"], case["step"] ** 2 / 2)
            o, p = _adam64(o, go, sts[0], 1e-3), _adam64(p, gp, sts[1], 1e-3)
        return {"loss": loss, "obj": o, "probe": p}
    if kind == "forward":
        d = _single(case, seed)
        with torch.no_grad():
            m = _Model64(d)
            oc = _constrain64(d["obj"].to(torch.complex128))
            ph = torch.fft.fft2(_ortho64(d["probe"].to(torch.complex128)))
            out = torch.empty((d["idx"].numel(), m.n, m.n), dtype=torch.float64, device=DEVICE)
            total, scale = 0.0, d["pos"].shape[0] / d["idx"].numel() / d["mean"]
            for s in range(0, d["idx"].numel(), m.chunk):
                i = d["idx"][s:s + m.chunk]
                far = m.far(oc, ph, d["pos"][i].double())
                out[s:s + m.chunk] = torch.fft.fftshift(far.abs().square().sum(0), dim=(-2, -1))
                total += float(_loss64(far, d["data"][i].double(), d["mask"].double(), "l2_amplitude", scale, d["mean"]))
        return {"loss": torch.tensor(total, dtype=torch.float64), "intensity": out}
    if kind == "analytic":
        return _analytic64(_single(case, seed))
    if kind == "multi":
        got = [_gradient64(d, d["obj"].to(torch.complex128), d["probe"].to(torch.complex128), "l2_amplitude", 1.0)
               for d in _many(case, seed)]
        return {"losses": torch.stack([g[0] for g in got]), "obj": [g[1] for g in got], "probe": [g[2] for g in got]}
    if kind == "object":
        return _object64(case, seed)
    if kind == "probe":
        d = _probes(case, seed)
        n = case["n"]
        p = d["probe"].to(torch.complex128).requires_grad_(True)
        o = _ortho64(p)
        inten = torch.fft.fftshift(o.real ** 2 + o.imag ** 2, dim=(-2, -1))
        y, tot = torch.arange(n, device=DEVICE).double(), inten.sum(dim=(-2, -1))
        cr = (inten * y[:, None]).sum(dim=(-2, -1)) / tot - n // 2
        cc = (inten * y[None]).sum(dim=(-2, -1)) / tot - n // 2
        k = torch.fft.fftfreq(n, dtype=torch.float64, device=DEVICE)
        ang = 2 * math.pi * (k[None, :, None] * cr[:, None, None] + k[None, None, :] * cc[:, None, None])
        out = torch.fft.ifft2(torch.fft.fft2(o) * torch.polar(torch.ones_like(ang), ang))
        tv = 0.1 * (torch.diff(out, dim=-1).abs().mean() + torch.diff(out, dim=-2).abs().mean())
        torch.autograd.backward([out, tv], [d["up"].to(torch.complex128), torch.ones_like(tv)])
        return {"probe": out.detach(), "tv": tv.detach(), "grad": p.grad}
    sd, x, t = _network(case, seed)
    if kind == "infer":
        with torch.no_grad():
            return {"out": _network64(case, sd, x, False)[0]}
    out, w = _network64(case, sd, x, True)
    loss = torch.nn.functional.mse_loss(out, t.double())
    loss.backward()
    if case["levels"] > 3:  # batch statistics over a few bottleneck pixels amplify the BF16 rounding of every layer
        return {"loss": loss.detach(), "out": None, "grad": None}
    return {"loss": loss.detach(), "out": out.detach(), "grad": _flat64(case, w)}


def _analytic64(d):
    with torch.no_grad():
        m = _Model64(d)
        oc = _constrain64(d["obj"].to(torch.complex128))
        po = _ortho64(d["probe"].to(torch.complex128))
        ph = torch.fft.fft2(po)
        P, n = po.shape[0], m.n
        upd = torch.zeros((m.S, m.Ho * m.Wo, 2), dtype=torch.float64, device=DEVICE)
        norm = torch.zeros((m.S, P, m.Ho * m.Wo), dtype=torch.float64, device=DEVICE)
        g_probe = torch.zeros_like(po)
        total, energy, scale = 0.0, 0.0, d["pos"].shape[0] / d["idx"].numel() / d["mean"]
        for s0 in range(0, d["idx"].numel(), m.chunk):
            i = d["idx"][s0:s0 + m.chunk]
            t = d["data"][i].double()
            keep = []
            far = m.far(oc, ph, d["pos"][i].double(), keep)
            total += float(_loss64(far, t, d["mask"].double(), "l2_amplitude", scale, d["mean"]))
            meas = torch.fft.ifftshift(t, dim=(-2, -1))[None]
            if P == 1:
                mod = meas * torch.polar(torch.ones_like(meas), torch.angle(far))
            else:
                est = torch.sqrt((far + 1e-9).abs().square().sum(0))
                mod = torch.where(est == 0, torch.zeros_like(est), meas[0] / est)[None] * far
            g = torch.fft.ifft2(mod - far, norm="ortho")
            for s in reversed(range(m.S)):
                at, patch, psi = keep[s]
                energy = max(energy, float(patch.abs().square().sum(dim=(-2, -1)).max()))
                upd[s].index_add_(0, at.reshape(-1), torch.view_as_real((psi.conj() * g).sum(0)).reshape(-1, 2))
                for q in range(P):
                    norm[s, q].index_add_(0, at.reshape(-1), psi[q].abs().square().reshape(-1))
                g = patch.conj()[None] * g
                if s > 0:
                    k = m.kr[s - 1][:, None] * m.kc[s - 1][None]
                    g = torch.fft.ifft2(torch.fft.fft2(g) * k.conj())
            g_probe += g.sum(1)
        obj = torch.view_as_complex(upd).view(m.S, m.Ho, m.Wo) / norm.amax(-1).sum(-1)[:, None, None]
        ortho = 2.0 * n if P == 1 else 1.0 / (2.0 * n)
        return {"loss": torch.tensor(total, dtype=torch.float64), "obj": -obj, "probe": -g_probe / energy / ortho}


def _object64(case, seed):
    d = _object(case, seed)
    cplx = case["type"] == "complex"
    o = d["obj"].to(torch.complex128 if cplx else torch.float64).requires_grad_(True)
    out = _constrain64(o) if cplx else torch.clamp(o, min=0)
    half = math.ceil(3 * case["sigma"])
    ax = np.arange(-half, half + 1, dtype=np.float32)
    taps = np.exp(-0.5 * (ax / np.float32(case["sigma"])) ** 2).astype(np.float32)
    taps = torch.as_tensor((taps / taps.sum()).astype(np.float64), device=DEVICE)

    def blur(x):
        x = torch.nn.functional.conv2d(x[:, None], taps.view(1, 1, -1, 1), padding=(half, 0))
        return torch.nn.functional.conv2d(x, taps.view(1, 1, 1, -1), padding=(0, half))[:, 0]

    out = torch.complex(blur(out.real), blur(out.imag)) if cplx else blur(out)
    q = [np.fft.fftfreq(v, PIXEL).astype(np.float32) for v in (case["height"], case["width"])]
    r = np.sqrt(q[0][:, None] ** 2 + q[1][None] ** 2).astype(np.float32)
    env = torch.as_tensor((1 / (1 + (r / np.float32(case["lowpass"])) ** 8)).astype(np.float32), device=DEVICE).double()
    mu = out.mean(dim=(-2, -1), keepdim=True)
    y = torch.fft.ifft2(torch.fft.fft2(out - mu) * env)
    out = (y if cplx else y.real) + mu

    def tv(a):
        dims = [k for k in range(3) if a.shape[k] > 1 or k]
        return sum(0.01 * torch.diff(a, dim=k).abs().mean() for k in dims) / len(dims)

    soft = tv(torch.angle(out)) + tv(out.abs()) if cplx else tv(out)
    t = out if cplx else torch.polar(torch.ones_like(out), out)
    torch.autograd.backward([t, soft], [d["up"].to(torch.complex128), torch.ones_like(soft)])
    return {"transmission": t.detach(), "soft": soft.detach(), "obj": o.grad}
