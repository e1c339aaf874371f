"""What a user of the package has it compute, as measurable cases.

Each case is a dict of plain values; ``prepare`` makes what a program holds
before the call (media on the device, subdomains, networks), ``run`` is one
pass through the public entry points.  Media are random sphere packs voxelised
on the device and Gaussian random fields (FFT-filtered white noise).  Voxel
edges are powers of two (unit boxes of 2^k voxels) or not (a scan's 2.25
micrometres, a unit box of 200 voxels).
"""

from __future__ import annotations

import math

import numpy as np
import torch

import pmmoto_gb300 as P
from pmmoto_gb300.filters import connected_components as CC
from pmmoto_gb300.filters import distance as D
from pmmoto_gb300.filters import equilibrium_distribution as ED
from pmmoto_gb300.filters import morphological_operators as M
from pmmoto_gb300.filters import porosimetry as PO

BOUNDARIES = {
    "end": (("end", "end"),) * 3,
    "periodic": (("periodic", "periodic"),) * 3,
    "drain": (("end", "end"), ("wall", "wall"), ("wall", "wall")),
}
# 3x3x3 stride-2 convolutions of the schedule network: (c_in, c_out)
CONVS = ((1, 16), (16, 32), (32, 64), (64, 64))
HEAD = 64


def listed():
    return [
        # distance transform of a small periodic pack (the 128^3, 400-sphere
        # configuration): a single call where launches and latency count
        {"name": "edt_pack128", "kind": "edt", "n0": 128, "n1": 128, "n2": 128, "medium": "pack", "phi": 0.7,
         "r_lo": 3.84, "r_hi": 10.24, "h0": 2.0 ** -7, "h1": 2.0 ** -7, "h2": 2.0 ** -7, "bc": "periodic",
         "entry": "edt3d", "squared": True},
        # distance transform of a cropped scan: odd sides, a slice spacing
        # that differs from the pixel size, no boundary conditions
        {"name": "edt_scan", "kind": "edt", "n0": 301, "n1": 257, "n2": 187, "medium": "grf", "phi": 0.45,
         "sigma": 5.0, "h0": 5.0, "h1": 2.25, "h2": 2.25, "bc": "end", "entry": "edt3d", "squared": False},
        # the large configuration: 1024^3 periodic Gaussian random field
        {"name": "edt_grf1024", "kind": "edt", "n0": 1024, "n1": 1024, "n2": 1024, "medium": "grf", "phi": 0.35,
         "sigma": 4.0, "h0": 1.0, "h1": 1.0, "h2": 1.0, "bc": "periodic", "entry": "edt3d", "squared": True},
        # labelling of a segmented scan with three phases and odd sides
        {"name": "cc_phases", "kind": "cc", "n0": 257, "n1": 200, "n2": 323, "medium": "grf", "phi": 0.3,
         "sigma": 4.0, "h": 2.25, "bc": "end", "phases": 2, "dtype": "u8"},
        # labelling of the large periodic field (seam merge and numbering)
        {"name": "cc_grf1024", "kind": "cc", "n0": 1024, "n1": 1024, "n2": 1024, "medium": "grf", "phi": 0.35,
         "sigma": 4.0, "h": 2.0 ** -10, "bc": "periodic", "phases": 1, "dtype": "u8"},
        # pore space connected to the inlet of the 512^3 drainage pack
        {"name": "select_pack512", "kind": "select", "n0": 512, "n1": 512, "n2": 512, "medium": "pack", "phi": 0.53,
         "r_lo": 10.24, "r_hi": 25.6, "h": 2.0 ** -9, "bc": "drain", "which": "inlet", "phase": 1},
        # opening of a periodic pack of uneven sides (the batch's voxel size)
        {"name": "open_pack256", "kind": "morph", "n0": 256, "n1": 192, "n2": 320, "medium": "pack", "phi": 0.4,
         "r_lo": 5.12, "r_hi": 15.36, "h": 2.0 ** -8, "bc": "periodic", "op": "opening", "radius": 5.5,
         "fft": False},
        # pore size distribution with every default on a periodic unit box
        {"name": "psd_pack200", "kind": "psd", "n0": 200, "n1": 200, "n2": 200, "medium": "pack", "phi": 0.45,
         "r_lo": 5.0, "r_hi": 14.0, "h": 1.0 / 200, "bc": "periodic", "radii": 25, "mode": "hybrid"},
        # drainage of one pack of the batched configuration, medium included
        {"name": "drain_pack", "kind": "drain", "n0": 96, "n1": 160, "n2": 224, "medium": "pack", "phi": 0.4,
         "r_lo": 5.12, "r_hi": 15.36, "h": 2.0 ** -8, "radii": 24, "small": 1.0, "large": 12.0,
         "mode": "distance"},
        # drainage of a scan with the default mode: voxels of no power of two
        {"name": "drain_scan", "kind": "drain", "n0": 150, "n1": 121, "n2": 99, "medium": "grf", "phi": 0.45,
         "sigma": 4.0, "h": 2.25, "radii": 20, "small": 1.0, "large": 8.0, "mode": "hybrid"},
        # the dense exact curve of the 512^3 pack (40 radii), medium included
        {"name": "drain_pack512", "kind": "drain", "n0": 512, "n1": 512, "n2": 512, "medium": "pack", "phi": 0.53,
         "r_lo": 10.24, "r_hi": 25.6, "h": 2.0 ** -9, "radii": 40, "small": 1.0, "large": 20.0,
         "mode": "distance"},
        # forward and backward pass of the schedule network at its training batch
        {"name": "net_grad64", "kind": "net", "batch": 64, "grad": True},
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _medium(rng, side):
    if rng.random() < 0.5:
        # radii well below the smallest side, so that some pore space is left
        r_hi = round(min(rng.uniform(4.0, 26.0), side / 5.0), 2)
        return {"medium": "pack", "phi": round(rng.uniform(0.35, 0.75), 3),
                "r_lo": round(r_hi * rng.uniform(0.3, 0.7), 2), "r_hi": r_hi}
    return {"medium": "grf", "phi": round(rng.uniform(0.3, 0.6), 3), "sigma": rng.choice([2.5, 3.0, 4.0, 5.0, 6.0])}


def draw(rng):
    kind = rng.choice(["edt", "edt", "cc", "select", "morph", "psd", "drain", "drain", "net"])
    if kind == "net":
        return {"kind": "net", "batch": _side(rng, 1, 64), "grad": rng.random() < 0.6}
    hi = {"edt": 512, "cc": 448, "select": 512, "morph": 320, "psd": 200, "drain": 256}[kind]
    case = {"kind": kind, "n0": _side(rng, 48, hi), "n1": _side(rng, 48, hi), "n2": _side(rng, 48, hi)}
    case.update(_medium(rng, min(_shape(case))))
    h = rng.choice([1.0, 2.0 ** -8, 2.25])
    if kind == "edt":
        case.update(h0=h * rng.choice([1.0, 1.0, 2.0]), h1=h, h2=h, bc=rng.choice(["end", "periodic", "drain"]),
                    entry=rng.choice(["edt3d", "edt"]), squared=rng.random() < 0.5)
        return case
    case["h"] = h
    if kind == "cc":
        case.update(bc=rng.choice(["end", "periodic", "drain"]), phases=rng.choice([1, 1, 2]),
                    dtype=rng.choice(["u8", "u8", "i32"]))
    elif kind == "select":
        case.update(bc="drain", which=rng.choice(["inlet", "outlet", "both", "isolated"]),
                    phase=rng.choice([None, 1]))
    elif kind == "morph":
        case.update(bc=rng.choice(["periodic", "drain"]), op=rng.choice(["erode", "dilate", "opening", "closing"]),
                    radius=round(rng.uniform(1.2, 9.0), 2), fft=rng.random() < 0.3)
    elif kind == "psd":
        case.update(bc=rng.choice(["periodic", "drain"]), radii=rng.randint(5, 25),
                    mode=rng.choice(["hybrid", "distance", "morph"]))
    else:
        case.update(radii=rng.randint(8, 40), small=1.0, large=round(rng.uniform(5.0, 14.0), 2),
                    mode=rng.choice(["hybrid", "distance", "morph"]))
    return case


# ---- inputs ------------------------------------------------------------------

def _shape(case):
    return case["n0"], case["n1"], case["n2"]


def _voxel(case):
    return (case["h0"], case["h1"], case["h2"]) if "h0" in case else (case["h"],) * 3


def _subdomain(case, bc):
    vox, h = _shape(case), _voxel(case)
    inlet = ((bc == "drain", False), (False, False), (False, False))
    outlet = ((False, bc == "drain"), (False, False), (False, False))
    return P.initialize(vox, box=tuple((0.0, n * e) for n, e in zip(vox, h)), boundary_types=BOUNDARIES[bc],
                        inlet=inlet, outlet=outlet)


def _spheres(case, rng):
    """Overlapping spheres at uniform centres, as many as leave the porosity
    phi; radii uniform in [r_lo, r_hi] voxels of the smallest edge."""
    vox, h = _shape(case), _voxel(case)
    length = [n * e for n, e in zip(vox, h)]
    a, b = case["r_lo"] * min(h), case["r_hi"] * min(h)
    r3 = (b ** 4 - a ** 4) / (4.0 * (b - a))
    n = max(1, int(round(-math.log(case["phi"]) * math.prod(length) / (4.0 / 3.0 * math.pi * r3))))
    return np.c_[rng.random((n, 3)) * np.array(length), rng.uniform(a, b, n)]


def _field(case, seed):
    """Pore space (1) of a periodic Gaussian random field: white noise under
    a Gaussian of sigma voxels, pore up to its phi-quantile (of a sample)."""
    vox = _shape(case)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed % (1 << 31))
    f = torch.fft.rfftn(torch.randn(vox, generator=g, device="cuda"))
    for d, n in enumerate(vox):
        k = torch.fft.rfftfreq(n, device="cuda") if d == 2 else torch.fft.fftfreq(n, device="cuda")
        view = [1, 1, 1]
        view[d] = -1
        f *= torch.exp(-2.0 * (math.pi * case["sigma"] * k) ** 2).view(view)
    f = torch.fft.irfftn(f, s=vox)
    sample = f.view(-1)[::max(1, f.numel() >> 22)].sort().values
    return (f <= sample[int(case["phi"] * sample.numel())]).to(torch.uint8)


def _on_subdomain(own, sd):
    """Padded image of an own-region image: wrapped halos, solid walls."""
    img = own
    for d in range(3):
        lo, hi = sd.pad[d]
        if lo or hi:
            n = img.shape[d]
            img = img.index_select(d, torch.arange(-lo, n + hi, device=img.device) % n)
    return sd.set_wall_bcs(img.contiguous())


def _image(case, sd, seed):
    """Pore space (1) of the case's medium on the padded subdomain."""
    if case["medium"] == "pack":
        sph = torch.as_tensor(_spheres(case, np.random.default_rng(seed)), device="cuda")
        return P.domain_generation.gen_pm_spheres_domain(sd, sph).img
    return _on_subdomain(_field(case, seed), sd)


def _own_image(case, seed):
    """The same medium without halos."""
    if case["medium"] == "grf":
        return _field(case, seed)
    return _image(case, _subdomain(case, "end"), seed)


def _phases(case, sd, seed):
    """Image of 1 (pore) or of 1 and 2 (two pore phases of one field or
    pack: nested levels, as a wetting film around a pore's core)."""
    img = _image(case, sd, seed)
    if case["phases"] == 2:
        if case["medium"] == "grf":
            wide = dict(case, phi=min(0.9, case["phi"] + 0.25))
            img = img + _image(wide, sd, seed)
        else:
            img = img + (img == 1) * (torch.arange(img.shape[2], device=img.device) // 24 % 2).to(torch.uint8)
    return img.to({"u8": torch.uint8, "i32": torch.int32}[case["dtype"]])


def _net_shapes():
    out = []
    for cin, cout in CONVS:
        out += [(cout, cin, 27), (cout,)]
    return out + [(HEAD, HEAD), (HEAD,), (HEAD, HEAD), (HEAD,)]


def _net_data(case, seed):
    """Weights (flat fp32), inputs (bf16 fields of distances in [0, 1]) and
    targets (saturation curves, non-decreasing in the radius)."""
    rng = np.random.default_rng(seed)
    parts = []
    for s in _net_shapes():
        fan_in = math.prod(s[1:]) if len(s) > 1 else 0
        parts.append(rng.standard_normal(s) * (math.sqrt(2.0 / fan_in) if fan_in else 0.05))
    flat = torch.as_tensor(np.concatenate([p.reshape(-1) for p in parts]).astype(np.float32))
    b = case["batch"]
    coarse = torch.as_tensor(rng.uniform(-0.5, 1.0, (b, 1, 16, 16, 16)).astype(np.float32), device="cuda")
    x = torch.nn.functional.interpolate(coarse, size=(64, 64, 64), mode="trilinear", align_corners=False)
    x = x.clamp_min(0.0).reshape(b, -1).to(torch.bfloat16).contiguous()
    target = torch.as_tensor(np.sort(rng.random((b, HEAD)), axis=1).astype(np.float32), device="cuda")
    return flat, x, target


def prepare(case, seed):
    kind = case["kind"]
    if kind == "net":
        from pmmoto_gb300.learned import ScheduleNet

        flat, x, target = _net_data(case, seed)
        net = ScheduleNet(seed=0)
        net.params.copy_(flat)
        net.pack()
        return {"case": case, "net": net, "x": x, "target": target}
    st = {"case": case}
    if kind == "edt" and case["entry"] == "edt3d":
        st["img"] = _own_image(case, seed)
        return st
    sd = st["sd"] = _subdomain(case, case.get("bc", "drain"))
    st["img"] = _phases(case, sd, seed) if kind == "cc" else _image(case, sd, seed)
    if kind == "drain":
        r = np.linspace(case["small"], case["large"], case["radii"]) * case["h"]
        st["pressures"] = sorted(float(p) for p in 2.0 / r)
    return st


# ---- one pass ----------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "edt":
        if case["entry"] == "edt":
            return D.edt(state["img"], state["sd"])
        per = (case["bc"] == "periodic",) * 3
        return D.edt3d(state["img"], periodic=per, resolution=_voxel(case), squared=case["squared"])
    if kind == "cc":
        labels, count = CC.connect_components(state["img"], state["sd"])
        return {"labels": labels, "count": count}
    if kind == "select":
        fn = {"inlet": CC.inlet_connected_img, "outlet": CC.outlet_connected_img,
              "both": CC.inlet_outlet_connected_img, "isolated": CC.isolated_img}[case["which"]]
        return fn(state["sd"], state["img"], case["phase"])
    if kind == "morph":
        fn = {"erode": M.erode, "dilate": M.dilate, "opening": M.opening, "closing": M.closing}[case["op"]]
        return fn(state["sd"], state["img"], case["radius"] * case["h"], case["fft"])
    if kind == "psd":
        pm = P.domain_generation.gen_pm(state["sd"], state["img"])
        return PO.pore_size_distribution(state["sd"], pm, num_radii=case["radii"], mode=case["mode"])
    if kind == "drain":
        pm = P.domain_generation.gen_pm(state["sd"], state["img"])
        mp = P.domain_generation.gen_mp_constant(pm, 2)
        sat = ED.drainage(mp, state["pressures"], mode=case["mode"])
        return {"saturation": sat, "img": mp.img}
    net = state["net"]
    if not case["grad"]:
        return {"pred": net.predict(state["x"])}
    pred = net.forward(state["x"], state["target"])
    net.backward(state["x"])
    return {"pred": pred, "grads": net.grads}


def work(case):
    """Bytes and operations a pass cannot do without: every input read once,
    every output written once; two operations per multiply-add."""
    kind = case["kind"]
    if kind == "net":
        macs, side, act = 0, 64, 64 ** 3
        for cin, cout in CONVS:
            side //= 2
            macs += side ** 3 * cout * 27 * cin
            act += side ** 3 * cout
        macs += 2 * HEAD * HEAD
        params = sum(math.prod(s) for s in _net_shapes())
        b = case["batch"]
        if not case["grad"]:
            return {"bytes": b * 64 ** 3 * 2 + params * 4 + b * HEAD * 4, "flops": 2 * b * macs}
        # forward, weight gradients, input gradients of all layers but the first
        first = 32 ** 3 * CONVS[0][1] * 27
        return {"bytes": b * 64 ** 3 * 2 + params * 8 + b * HEAD * 8, "flops": 2 * b * (3 * macs - first)}
    pads = [0, 0, 0]
    bc = case.get("bc", "drain")
    if not (kind == "edt" and case["entry"] == "edt3d"):
        pads = {"end": [0, 0, 0], "periodic": [2, 2, 2], "drain": [0, 2, 2]}[bc]
    n = math.prod(s + p for s, p in zip(_shape(case), pads))
    per = {"edt": 1 + 4, "cc": (4 if case.get("dtype") == "i32" else 1) + 8, "select": 1 + 8, "morph": 1 + 1,
           "psd": 1 + 8, "drain": 1 + 1}[kind]
    return {"bytes": n * per, "flops": 0}


# ---- plain 64-bit results ------------------------------------------------------

def _sweep(f, dim, a, periodic):
    """min over v of f(v) + a (x - v)^2 along dim, in place of the envelope."""
    n = f.shape[dim]
    out = f.clone()
    for d in range(1, n):
        if a * d * d >= float(out.max()):
            break
        add = a * d * d
        if periodic:
            out = torch.minimum(out, torch.roll(f, d, dim) + add)
            out = torch.minimum(out, torch.roll(f, -d, dim) + add)
        else:
            hi, lo = out.narrow(dim, d, n - d), out.narrow(dim, 0, n - d)
            hi.copy_(torch.minimum(hi, f.narrow(dim, 0, n - d) + add))
            lo.copy_(torch.minimum(lo, f.narrow(dim, d, n - d) + add))
    return out


def _exact_edt(case, seed):
    if case["entry"] == "edt" or math.prod(_shape(case)) > 1 << 26:
        return None
    img = _own_image(case, seed)
    f = torch.where(img == 0, 0.0, math.inf).to(torch.float64)
    for dim, h in enumerate(_voxel(case)):
        f = _sweep(f, dim, float(np.float64(np.float32(h)) ** 2), case["bc"] == "periodic")
    return f if case["squared"] else f.sqrt()


def _exact_net(case, seed):
    flat, x, target = _net_data(case, seed)
    w, off = [], 0
    for s in _net_shapes():
        n = math.prod(s)
        w.append(flat[off:off + n].reshape(s).to("cuda", torch.float64).requires_grad_(True))
        off += n
    b = case["batch"]
    preds = []
    for i in range(0, b, 8):
        h = x[i:i + 8].to(torch.float64).reshape(-1, 1, 64, 64, 64)
        for k, (cin, cout) in enumerate(CONVS):
            h = torch.relu(torch.nn.functional.conv3d(h, w[2 * k].reshape(cout, cin, 3, 3, 3), w[2 * k + 1], 2, 1))
        h = h.mean(dim=(2, 3, 4))
        h = torch.relu(h @ w[8].T + w[9])
        p = torch.sigmoid(h @ w[10].T + w[11])
        if case["grad"]:
            ((p - target[i:i + 8].to(torch.float64)) ** 2).sum().div(b * HEAD).backward()
        preds.append(p.detach())
    out = {"pred": torch.cat(preds)}
    if case["grad"]:
        out["grads"] = torch.cat([t.grad.reshape(-1) for t in w])
    return out


def exact(case, seed):
    """The distance transforms and the network in 64 bits.  The periodic
    transform imports a truncated set of boundary parabolas by design, so it
    need not equal the true one; the other kinds' outputs are whole numbers, or
    ratios of counts of voxels that follow from the whole sweep."""
    if case["kind"] == "edt":
        return _exact_edt(case, seed)
    if case["kind"] == "net":
        return _exact_net(case, seed)
    return None
