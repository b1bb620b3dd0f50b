"""The work a user of this package has it do, as cases that can be timed.

Every case goes through the package's public entry points (the Model classes,
find_solution, Ensemble, and the surrogate module's network, layers and FD
runs) over the sizes of the package's own configurations and of ordinary use.
A case is a dict of plain values; `kind` selects one of

  step      one model (or a batch of equal instances) on a 2D or 3D grid:
            find_solution over `steps` forward-Euler steps between two saves,
            then the fields copied out as a save point does.  `tune`: the
            program calls autotune once when it sets up, as the benchmark
            does; without it the kernel is the library's own choice.
            `observe`: the save point also reads mass and energy.
  ensemble  independent 2D systems of uneven sizes stepped together.
  fd_batch  surrogate.fd_run: a batch of equal 2D fields put on the solver,
            stepped and read back (training data, the judge, the fallback).
  net       one inference pass of the jump network.
  layer     one convolution layer of the network in training: forward, GELU
            and backward (input, weight and bias gradients).
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

import symphas_b200 as sp
from symphas_b200 import surrogate

MODELS = {"A": sp.model_MA_t, "B": sp.model_MB_t, "C": sp.model_MC_t, "AMK": sp.model_MAMK_t,
          "BMK": sp.model_MBMK_t}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _step(name, model, dims, steps, dtype="f32", form="fused", **kw):
    nx, ny, nz = (tuple(dims) + (1,))[:3]
    c = {"name": name, "kind": "step", "model": model, "dim": len(dims), "nx": nx, "ny": ny,
         "nz": nz, "steps": steps, "dtype": dtype, "form": form, "batch": 1, "wide": False,
         "walls": "", "h": 1.0, "dt": 0.01 if len(dims) == 2 else 0.005, "c1": 1.0, "c2": 1.0,
         "tune": False, "observe": False}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest configuration: model A on 64^2, dx 0.5, dt 0.01, 1000
        # steps in SymPhas's own arithmetic (latency per step counts)
        _step("a2d_64_f64", "A", (64, 64), 1000, "f64", "exact", h=0.5),
        # a 2D run of ordinary, ragged size (about the size of a regional
        # window), set up without tuning
        _step("b2d_804x601_f32", "B", (804, 601), 100),
        # a large 2D run, tuned
        _step("b2d_4096_f32", "B", (4096, 4096), 20, tune=True),
        # 3D with walls in y, SymPhas's default 15-point Laplacian, odd sizes
        _step("a3d_150_walls_f32", "A", (150, 131, 97), 40, wide=True, walls="y", dt=0.02),
        # the headline: Cahn-Hilliard 256^3, FP32
        _step("b3d_256_f32", "B", (256, 256, 256), 50, tune=True),
        # the same in FP64 and SymPhas's term order, with mass and energy read
        _step("b3d_256_f64", "B", (256, 256, 256), 20, "f64", "exact", observe=True),
        # model C, eight 256^3 instances of two fields
        _step("c3d_8x256_f32", "C", (256, 256, 256), 10, batch=8, c1=0.5, tune=True),
        # the parameter sweep: 1024 members of eight sizes and two models
        {"name": "ens_1024_f32", "kind": "ensemble", "count": 1024, "steps": 40, "tune": True},
        # a batch of the surrogate's fields on the solver
        {"name": "fd_256x256_f32", "kind": "fd_batch", "batch": 256, "n": 256, "steps": 32},
        # one jump of the network
        {"name": "net_64x256", "kind": "net", "batch": 64, "n": 256},
        # training: the widest-grid layer, and a deep one with a skip
        {"name": "layer_256_32", "kind": "layer", "batch": 16, "h": 256, "w": 256, "cin": 32,
         "cout": 32, "skip": False},
        {"name": "layer_64_128", "kind": "layer", "batch": 32, "h": 64, "w": 64, "cin": 256,
         "cout": 128, "skip": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step2", "step2", "step3", "step3", "step3", "ensemble", "fd_batch", "net",
                       "layer", "layer"])
    if kind in ("step2", "step3"):
        dim = int(kind[-1])
        dims = tuple(_log(rng, 48, 2048) if dim == 2 else _log(rng, 24, 256) for _ in range(dim))
        if rng.random() < 0.3:  # powers of two are common
            dims = tuple(1 << int(round(math.log2(d))) for d in dims)
        model = rng.choice(["A", "B", "B", "C", "AMK", "BMK"])
        dtype, form = rng.choice([("f32", "fused")] * 3 + [("f64", "exact")] * 2 + [("f64", "fused")])
        wide = model in "ABC" and rng.random() < 0.25
        walls = rng.choice(["", "", "", "x", "y", "xy"])
        sites = math.prod(dims) * (2 if model == "C" else 1)
        steps = max(5, min(200, int(4e8 / sites)))
        c = _step("", model, dims, steps, dtype, form, wide=wide, walls=walls,
                  c1=round(rng.uniform(0.5, 1.2), 3), c2=round(rng.uniform(0.5, 1.2), 3),
                  tune=rng.random() < 0.4,
                  observe=model in ("B", "BMK", "C") and rng.random() < 0.4)  # a mass that is not 0
        del c["name"]
        return c
    if kind == "ensemble":
        return {"kind": kind, "count": _log(rng, 8, 512), "steps": rng.randint(10, 40),
                "tune": rng.random() < 0.5}
    if kind == "fd_batch":
        n = 8 * rng.randint(8, 32)
        return {"kind": kind, "batch": _log(rng, 4, 256), "n": n, "steps": rng.randint(4, 32)}
    if kind == "net":
        return {"kind": kind, "batch": _log(rng, 2, 64), "n": 16 * rng.randint(4, 16)}
    cin, cout = rng.choice([(32, 32), (32, 64), (64, 64), (64, 32), (64, 128), (128, 128),
                            (128, 64), (128, 256), (256, 256), (256, 128)])
    top = 256 * 32 // max(cin, cout)
    return {"kind": kind, "batch": _log(rng, 2, 16), "h": rng.randint(max(8, top // 4), top),
            "w": rng.randint(max(8, top // 4), top), "cin": cin, "cout": cout,
            "skip": rng.random() < 0.3}


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _dims(c):
    return (c["nx"], c["ny"], c["nz"])[: c["dim"]]


def _tdtype(c):
    return torch.float32 if c.get("dtype", "f32") == "f32" else torch.float64


def _fields(c, seed):
    """[field][batch, (z,) y, x]: noise about the mean of the quench."""
    g = _gen(seed)
    shape = (c["batch"],) + tuple(reversed(_dims(c)))
    mean = {"A": 0.0, "AMK": 0.0, "B": -0.2, "BMK": -0.2, "C": 0.1}[c["model"]]
    out = [mean - 0.1 + 0.2 * torch.rand(shape, generator=g, device="cuda", dtype=_tdtype(c))]
    if c["model"] == "C":
        out.append(-0.1 + 0.2 * torch.rand(shape, generator=g, device="cuda", dtype=_tdtype(c)))
    return out


def _smooth(batch, n, seed):
    """Phase-separated fields: domains of about 16 sites with values in [-1, 1]."""
    g = _gen(seed)
    z = torch.randn(batch, 1, n // 8, n // 8, generator=g, device="cuda")
    return torch.tanh(2.0 * F.interpolate(z, size=(n, n), mode="bilinear"))[:, 0].contiguous()


def _members(c):
    return sp.ensemble_members(c["count"], seed=c["count"])


def _member_fields(c, seed):
    """One flat tensor, and each member's slice of it."""
    sides = [m["dims"][0] for m in _members(c)]
    at = np.cumsum([0] + [s * s for s in sides])
    flat = -0.1 + 0.2 * torch.rand(int(at[-1]), generator=_gen(seed), device="cuda")
    return flat, sides, at


CHANNELS = (32, 64, 128, 256)


def _net_weights(seed):
    """The network's layers, encoder to head, as (cin, cout, w, b)."""
    shapes, cin = [], surrogate.CIN
    for ch in CHANNELS:
        shapes += [(cin, ch), (ch, ch)]
        cin = ch
    for k in (2, 1, 0):
        shapes += [(CHANNELS[k + 1], CHANNELS[k]), (CHANNELS[k], CHANNELS[k])]
    shapes.append((CHANNELS[0], 32))
    g = _gen(seed + 1)
    out = []
    for i, (ci, co) in enumerate(shapes):
        w = torch.randn(co, 3, 3, ci, generator=g, device="cuda") * math.sqrt(2.0 / (9 * ci))
        b = 0.05 * torch.randn(co, generator=g, device="cuda")
        if i == len(shapes) - 1:
            # the head: channel 0 is the output, without an offset (a trained
            # network predicts a change of zero mean)
            w[0] -= w[0].mean()
            w[1:], b[:] = 0.0, 0.0
        out.append((w, b))
    return out


def _layer_inputs(c, seed):
    """x, dy, skip (or None), w, b: activations after a GELU, gradients and
    skips of unit scale in bf16, weights in fp32."""
    g = _gen(seed)

    def r(*s):
        return torch.randn(*s, generator=g, device="cuda")

    n, h, w = c["batch"], c["h"], c["w"]
    x = F.gelu(r(n, h, w, c["cin"]), approximate="tanh").bfloat16()
    dy = r(n, h, w, c["cout"]).bfloat16()
    skip = r(n, h, w, c["cout"]).bfloat16() if c["skip"] else None
    wt = r(c["cout"], 3, 3, c["cin"]) * math.sqrt(2.0 / (9 * c["cin"]))
    return x, dy, skip, wt, 0.1 * r(c["cout"])


# ---------------------------------------------------------------------------
# what a program holds before the call
# ---------------------------------------------------------------------------
_solver_stream = None


def _stream():
    """The program's solver stream: one for all its models, as the benchmark has."""
    global _solver_stream
    if _solver_stream is None:
        _solver_stream = torch.cuda.Stream()
    return _solver_stream.cuda_stream


def _boundaries(c):
    P, D = sp.BoundaryType.PERIODIC, sp.BoundaryType.DEFAULT
    return [D if axis in c["walls"] else P for axis in "xyz" for _ in range(2)]


def _model(c):
    if c["dim"] == 2:
        st = sp.Stencil2d2h() if c["wide"] else sp.Stencil2d2h(5, 6, 13)
    else:
        st = sp.Stencil3d2h() if c["wide"] else sp.Stencil3d2h(7, 10, 25)
    params = sp.ProblemParameters(_dims(c), h=c["h"], boundary=_boundaries(c))
    return MODELS[c["model"]](c["dim"], sp.SolverFT(st, form=c["form"]), params,
                              coeff=(c["c1"], c["c2"]), dtype=c["dtype"], batch=c["batch"],
                              dt=c["dt"])


def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] == "step":
        fields = _fields(c, seed)
        torch.cuda.synchronize()  # the models work on a stream of their own
        m = s["model"] = _model(c)
        m.set_stream(_stream())
        for f, v in enumerate(fields):
            m.batch_from_device(f, v.data_ptr(), v.numel() * v.element_size())
        if c["tune"]:
            m.autotune(5)
        m.synchronize()
        s["out"] = fields  # the save point's device buffers
    elif c["kind"] == "ensemble":
        flat, sides, at = _member_fields(c, seed)
        torch.cuda.synchronize()
        m = s["model"] = sp.Ensemble(sp.SolverFT(sp.Stencil2d2h(5, 6, 13), form="fused"),
                                     _members(c), dtype="f32")
        m.set_stream(_stream())
        s["ptrs"] = [(flat.data_ptr() + 4 * int(at[i]), 4 * n * n) for i, n in enumerate(sides)]
        for i, (p, nb) in enumerate(s["ptrs"]):
            m.field_from_device(0, p, nb, inst=i)
        if c["tune"]:
            m.autotune(5)
        m.synchronize()
        s["out"] = flat
    elif c["kind"] == "fd_batch":
        s["psi"] = 0.4 * _smooth(c["batch"], c["n"], seed)
        s["model"] = surrogate.fd_model(c["n"], c["batch"], 0.01)
    elif c["kind"] == "net":
        s["psi"] = _smooth(c["batch"], c["n"], seed)
        net = s["net"] = surrogate.JumpNet(CHANNELS)
        layers = _net_weights(seed)
        net.load({"w": [w for w, _ in layers], "b": [b for _, b in layers], "scale": 0.3})
    else:
        x, dy, skip, w, b = _layer_inputs(c, seed)
        layer = surrogate.ConvLayer(c["cin"], c["cout"], torch.Generator().manual_seed(0))
        layer.w.copy_(w)
        layer.b.copy_(b)
        layer.wb.copy_(layer.w.bfloat16())
        s.update(x=x.requires_grad_(), dy=dy, skip=skip, layer=layer)
        if skip is not None:
            skip.requires_grad_()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    c = state["case"]
    if c["kind"] == "step":
        m = state["model"]
        sp.find_solution(m, c["dt"], c["steps"])
        for f, v in enumerate(state["out"]):
            m.batch_to_device(f, v.data_ptr(), v.numel() * v.element_size())
        if c["observe"]:
            mass, energy = m.reduce()
            return {"fields": state["out"], "mass": mass, "energy": energy}
        return {"fields": state["out"]}
    if c["kind"] == "ensemble":
        m = state["model"]
        m.step(c["steps"])
        for i, (p, nb) in enumerate(state["ptrs"]):
            m.field_to_device(0, p, nb, inst=i)
        return {"fields": state["out"]}
    if c["kind"] == "fd_batch":
        return surrogate.fd_run(state["psi"], c["steps"], 0.01, state["model"])
    if c["kind"] == "net":
        with torch.no_grad():
            return state["net"](state["psi"])
    layer, x, skip = state["layer"], state["x"], state["skip"]
    layer.zero_grad()
    x.grad = None
    if skip is not None:
        skip.grad = None
    y = surrogate.conv_gelu(x, layer, skip)
    y.backward(state["dy"])
    out = {"y": y.detach(), "dx": x.grad, "dw": layer.gw, "db": layer.gb}
    if skip is not None:
        out["dskip"] = skip.grad
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
ON_CHIP = 100e6  # bytes of fields that stay in the L2 between steps


def work(case):
    c = case
    if c["kind"] in ("step", "ensemble", "fd_batch"):
        if c["kind"] == "step":
            nf, esz = (2 if c["model"] == "C" else 1), (4 if c["dtype"] == "f32" else 8)
            sites = math.prod(_dims(c)) * c["batch"]
            lap = {2: (9 if c["wide"] else 5), 3: (15 if c["wide"] else 7)}[c["dim"]] + 1
            per = lap + 5 if c["model"] in ("A", "AMK") else 2 * lap + 6
            per += lap + 12 if c["model"] == "C" else 0
        else:
            nf, esz = 1, 4
            if c["kind"] == "ensemble":
                sites = sum(m["dims"][0] * m["dims"][1] for m in _members(c))
            else:
                sites = c["batch"] * c["n"] ** 2
            per = 6 + 5 if c["kind"] == "ensemble" else 12 + 6
        # every step reads and writes each field once, unless the fields stay
        # on the chip between the steps; a save point reads and writes once
        # more (both in fd_batch: on the way in and out)
        fields = nf * sites * esz
        passes = c["steps"] if 2 * fields > ON_CHIP else 1
        saves = 2 if c["kind"] == "fd_batch" else 1
        return {"bytes": 2 * fields * (passes + saves), "flops": per * sites * c["steps"]}
    if c["kind"] == "net":
        flops, n, b = 0, c["n"], c["batch"]
        nbytes = 2 * 4 * b * n * n
        for lvl, ch in enumerate(CHANNELS):
            s = b * (n >> lvl) ** 2
            below = CHANNELS[lvl - 1] if lvl else 1
            flops += 18 * s * (below * ch + ch * ch)
            if lvl < len(CHANNELS) - 1:
                flops += 18 * s * (CHANNELS[lvl + 1] * ch + ch * ch)
        return {"bytes": nbytes, "flops": flops + 18 * b * n * n * CHANNELS[0]}
    pix = c["batch"] * c["h"] * c["w"]
    acts = pix * (2 * c["cin"] + 3 * c["cout"] + (2 * c["cout"] if c["skip"] else 0))
    wts = 9 * c["cin"] * c["cout"]
    return {"bytes": 2 * acts + 6 * wts, "flops": 3 * 18 * pix * c["cin"] * c["cout"]}


def tolerance(case):
    c = case
    if c["kind"] == "step" and c["dtype"] == "f64":
        return {"rel": 1e-13, "max": 1e-11}
    if c["kind"] in ("step", "ensemble", "fd_batch"):
        return {"rel": 1e-6, "max": 1e-4}
    if c["kind"] == "net":
        return {"rel": 3e-2, "max": 0.35}
    return {"rel": 1e-2, "max": 0.2}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _points(dim, wide):
    """Stencils as {offset (x, y, z): weight} at unit spacing."""
    def face(k):
        return [tuple(s * k if b == a else 0 for b in range(3)) for a in range(dim)
                for s in (-1, 1)]

    o = (0, 0, 0)
    diag = [(i, j, 0) for i in (-1, 1) for j in (-1, 1)]
    if dim == 2:
        if wide:
            lap = {**{p: 1 / 6 for p in diag}, **{p: 4 / 6 for p in face(1)}, o: -20 / 6}
        else:
            lap = {**{p: 1.0 for p in face(1)}, o: -4.0}
        bil = {**{p: 1.0 for p in face(2)}, **{p: 2.0 for p in diag},
               **{p: -8.0 for p in face(1)}, o: 20.0}
        return lap, bil
    corner = [(i, j, k) for i in (-1, 1) for j in (-1, 1) for k in (-1, 1)]
    edge = [p for p in [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)]
            if sum(map(abs, p)) == 2]
    if wide:
        lap = {**{p: 1 / 12 for p in corner}, **{p: 8 / 12 for p in face(1)}, o: -56 / 12}
    else:
        lap = {**{p: 1.0 for p in face(1)}, o: -6.0}
    bil = {**{p: 1.0 for p in face(2)}, **{p: 2.0 for p in edge},
           **{p: -12.0 for p in face(1)}, o: 42.0}
    return lap, bil


def _halo(v, dim, walls, r=2):
    """v grown by r on every axis: periodic images, zero beyond a wall."""
    for a in range(dim):
        d = v.dim() - 1 - a
        lo, hi = v.narrow(d, v.shape[d] - r, r), v.narrow(d, 0, r)
        if "xyz"[a] in walls:
            lo, hi = torch.zeros_like(lo), torch.zeros_like(hi)
        v = torch.cat([lo, v, hi], d)
    return v


def _apply(pts, v, dim, h, r=2):
    out = None
    for off, wt in pts.items():
        s = v
        for a in range(dim):
            d = v.dim() - 1 - a
            s = s.narrow(d, r + off[a], v.shape[d] - 2 * r)
        out = wt * s if out is None else out.add_(s, alpha=wt)
    return out / h


def _euler(model, dim, fields, steps, dt, h, c1, c2, wide=False, walls=""):
    lap_p, bil_p = _points(dim, wide)

    def lap(v):
        return _apply(lap_p, v, dim, h ** 2)

    def bilap(v):
        return _apply(bil_p, v, dim, h ** 4)

    f = [v.double() for v in fields]
    for _ in range(steps):
        p, q = f[0], _halo(f[0], dim, walls)
        if model == "A":
            d = [lap(q) + (c1 - c2 * p * p) * p]
        elif model == "B":
            d = [-bilap(q) + lap(c2 * q ** 3 - c1 * q)]
        elif model == "AMK":
            d = [c1 * (c2 * lap(q) - p ** 3 + p)]
        elif model == "BMK":
            d = [c1 * (lap(q ** 3 - q) - c2 * bilap(q))]
        else:
            e, k = f[1], _halo(f[1], dim, walls)
            d = [-bilap(q) + lap(q ** 3 - q + 2 * c1 * q * k * k),
                 lap(k) + e - e ** 3 - 2 * c1 * p * p * e]
        f = [a.add(b, alpha=dt) for a, b in zip(f, d)]
    return f


def _energy(c, f):
    """Landau free energy with forward differences over the interior and its halo."""
    dim, h = c["dim"], c["h"]
    grown = [_halo(v, dim, c["walls"], 1) for v in f]
    e = 0.0
    for v, g in zip(f, grown):
        g2 = 0.0
        for a in range(dim):
            n = g
            for b in range(dim):
                d = g.dim() - 1 - b
                n = n.narrow(d, 2 if b == a else 1, g.shape[d] - 2)
            g2 = g2 + ((n - v) / h) ** 2
        if c["model"] in ("A", "B"):
            e = e - 0.5 * c["c1"] * v ** 2 + 0.25 * c["c2"] * v ** 4 + 0.5 * g2
        else:
            kappa = 1.0 if c["model"] == "C" else c["c2"]
            e = e - 0.5 * v ** 2 + 0.25 * v ** 4 + 0.5 * kappa * g2
    if c["model"] == "C":
        e = e + c["c1"] * f[0] ** 2 * f[1] ** 2
    return float(e.sum() * h ** dim)


def _conv64(x, w, b):
    """NHWC circular 3x3 convolution; w [cout][3][3][cin]."""
    x = F.pad(x.permute(0, 3, 1, 2), (1, 1, 1, 1), mode="circular")
    return F.conv2d(x, w.permute(0, 3, 1, 2), b).permute(0, 2, 3, 1)


def _gelu(x):
    return F.gelu(x, approximate="tanh")


def _net64(psi, layers):
    """One pass of the network on [n, H, W] fields."""
    x = torch.zeros(psi.shape + (surrogate.CIN,), device="cuda", dtype=torch.float64)
    x[..., 0] = psi
    it, skips = iter(layers), []

    def cg(v, res=None):
        z = _conv64(v, *next(it))
        return _gelu(z if res is None else z + res)

    for lvl in range(4):
        x = cg(cg(x))
        if lvl < 3:
            skips.append(x)
            x = (x[:, ::2, ::2] + x[:, 1::2, ::2] + x[:, ::2, 1::2] + x[:, 1::2, 1::2]) / 4
    for s in reversed(skips):
        x = cg(x.repeat_interleave(2, 1).repeat_interleave(2, 2), s)
        x = cg(x)
    d = _conv64(x, *next(it))[..., 0]
    return 0.3 * (d - d.mean((1, 2), keepdim=True))


def exact(case, seed):
    c = case
    if c["kind"] == "step":
        f = _fields(c, seed)
        parts = [_euler(c["model"], c["dim"], [v[i:i + 1] for v in f], c["steps"], c["dt"], c["h"],
                        c["c1"], c["c2"], c["wide"], c["walls"]) for i in range(c["batch"])]
        f = [torch.cat([p[k] for p in parts]) for k in range(len(f))]
        if c["observe"]:
            return {"fields": f, "mass": float(f[0].sum()), "energy": _energy(c, [v[:1] for v in f])}
        return {"fields": f}
    if c["kind"] == "ensemble":
        flat, sides, at = _member_fields(c, seed)
        members, out = _members(c), torch.empty_like(flat, dtype=torch.float64)
        groups = {}
        for i, m in enumerate(members):
            groups.setdefault((m["model"], sides[i]), []).append(i)
        for (model, n), idx in groups.items():
            def col(v):
                return torch.tensor(v, device="cuda", dtype=torch.float64).view(-1, 1, 1)

            psi = torch.stack([flat[at[i]:at[i + 1]].view(n, n) for i in idx])
            M, kap = (col([members[i]["coeff"][k] for i in idx]) for k in (0, 1))
            # dt differs by member: folded into the mobility
            dt = col([members[i]["dt"] for i in idx])
            psi = _euler(model, 2, [psi], c["steps"], 1.0, 1.0, M * dt, kap)[0]
            for k, i in enumerate(idx):
                out[at[i]:at[i + 1]] = psi[k].reshape(-1)
        return {"fields": out}
    if c["kind"] == "fd_batch":
        psi = 0.4 * _smooth(c["batch"], c["n"], seed)
        return _euler("B", 2, [psi], c["steps"], 0.01, 1.0, 1.0, 1.0)[0]
    if c["kind"] == "net":
        psi = _smooth(c["batch"], c["n"], seed).double()
        layers = [(w.double(), b.double()) for w, b in _net_weights(seed)]
        with torch.no_grad():
            return torch.cat([_net64(p, layers) for p in psi.split(4)])
    x, dy, skip, w, b = _layer_inputs(c, seed)
    w, b = w.double().requires_grad_(), b.double().requires_grad_()
    y, dx, ds = [], [], []
    for k in range(0, c["batch"], 4):  # the gradients of w and b accumulate
        xk = x[k:k + 4].double().requires_grad_()
        z = _conv64(xk, w, b)
        if skip is not None:
            sk = skip[k:k + 4].double().requires_grad_()
            z = z + sk
        yk = _gelu(z)
        yk.backward(dy[k:k + 4].double())
        y.append(yk.detach())
        dx.append(xk.grad)
        if skip is not None:
            ds.append(sk.grad)
    out = {"y": torch.cat(y), "dx": torch.cat(dx), "dw": w.grad, "db": b.grad}
    if skip is not None:
        out["dskip"] = torch.cat(ds)
    return out
