"""The work that users of this framework have it do, as cases to be timed.

A case is one of these calls, through the package's public entry points:

  eval    forces of a plan that is resident on the GPU (Plan.eval): what a
          simulation repeats between rebuilds of its lists
  build   host positions to host forces in one call (build_eval)
  grad    differentiable forces, forward and backward (autograd.gravity)
  step    eight KDK steps with their rebuild, then the new state (Stepper)
  lists   host-built, run-packed lists to host forces (grav_groups_CUDA)
  dropin  the reference's call sequence: one grav_mn_CUDA per group and list

on an isolated Plummer or Hernquist sphere of n bodies (scale radius 1,
softening 0.01), or on a periodic unit box of n1d^3 bodies on a grid displaced
by a Gaussian random field with P(k) ~ k^-2.5 (softening 1/50 of the spacing),
with the Ewald correction.  order is 2 (quadrupoles) or 4.
"""
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "ahotsph-2hot-apps_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

BOX_TOL = 2.5e-6   # MAC tolerance of the periodic boxes


def listed():
    return [
        # the smallest systems: a few thousand bodies, where launches and latency count
        {"name": "eval_plummer_2k", "call": "eval", "ics": "plummer", "n": 2000, "order": 2,
         "tol": 1e-4},
        # the plain force evaluation of a Plummer sphere, order 2
        {"name": "eval_plummer_64k", "call": "eval", "ics": "plummer", "n": 65536, "order": 2,
         "tol": 2e-5},
        # a cusped profile of about a million bodies, order 4, a ragged count
        {"name": "eval_hernquist_1m", "call": "eval", "ics": "hernquist", "n": 1000003, "order": 4,
         "tol": 1e-5},
        # a periodic box that fits in the caches, odd grid
        {"name": "eval_box_61", "call": "eval", "ics": "box", "n1d": 61, "rms": 0.25, "order": 4,
         "tol": BOX_TOL},
        # the largest: a clustered periodic box of four million bodies
        {"name": "eval_box_160", "call": "eval", "ics": "box", "n1d": 160, "rms": 0.5, "order": 4,
         "tol": BOX_TOL},
        # positions to forces in one call: an isolated sphere, and a periodic box
        {"name": "build_plummer_100k", "call": "build", "ics": "plummer", "n": 100003, "order": 2,
         "tol": 2e-5},
        {"name": "build_box_96", "call": "build", "ics": "box", "n1d": 96, "rms": 0.5, "order": 4,
         "tol": BOX_TOL},
        # a loss on accelerations and potentials, differentiated: order 2 isolated, order 4 periodic
        {"name": "grad_plummer_128k", "call": "grad", "ics": "plummer", "n": 131072, "order": 2,
         "tol": 1e-5},
        {"name": "grad_box_32", "call": "grad", "ics": "box", "n1d": 32, "rms": 0.25, "order": 4,
         "tol": BOX_TOL},
        # time stepping of a periodic box, graph-captured steps and a rebuild every eight
        {"name": "step_box_48", "call": "step", "ics": "box", "n1d": 48, "rms": 0.25, "order": 4,
         "tol": BOX_TOL},
        # lists walked on the host, in page-locked memory, to forces in one call
        {"name": "lists_box_40", "call": "lists", "ics": "box", "n1d": 40, "rms": 0.25, "order": 4,
         "tol": BOX_TOL},
        # the drop-in boundary as the reference's walk drives it, full lists of a small sphere
        {"name": "dropin_plummer_8k", "call": "dropin", "ics": "plummer", "n": 8192, "order": 2,
         "tol": 1e-4},
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    """One more case: (call, inputs) as in the list, sizes over the whole range."""
    call, ics = rng.choice([("eval", "plummer"), ("eval", "hernquist"), ("eval", "box"),
                            ("eval", "plummer"), ("eval", "hernquist"), ("eval", "box"),
                            ("build", "plummer"), ("build", "box"), ("grad", "plummer"),
                            ("grad", "box"), ("step", "box"), ("lists", "box"),
                            ("dropin", "plummer")])
    c = {"call": call, "ics": ics}
    if ics == "box":
        hi = {"eval": 150, "build": 110, "grad": 48, "step": 56, "lists": 48}[call]
        lo = {"eval": 20, "build": 20, "grad": 16, "step": 20, "lists": 20}[call]
        c.update(n1d=_log_int(rng, lo, hi), rms=rng.choice([0.25, 0.5]), order=4, tol=BOX_TOL)
    else:
        hi = {"eval": 1000000, "build": 400000, "grad": 250000, "dropin": 16384}[call]
        c.update(n=_log_int(rng, 2000, hi), tol=rng.choice([1e-5, 2e-5, 1e-4]),
                 order=2 if call == "dropin" else rng.choice([2, 4]))
    return c


# ------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _sphere(case, seed):
    """n positions of the profile, truncated at 20 scale radii, isotropic."""
    n, g = case["n"], _generator(seed)
    r = torch.empty(0, dtype=torch.float64, device="cuda")
    while r.numel() < n:
        u = torch.rand(n + 1024, generator=g, dtype=torch.float64, device="cuda")
        u = u[u > 0]
        q = torch.sqrt(u)
        t = 1 / torch.sqrt(u ** (-2.0 / 3.0) - 1) if case["ics"] == "plummer" else q / (1 - q)
        r = torch.cat([r, t[t <= 20.0]])
    r = r[:n]
    c = 2 * torch.rand(n, generator=g, dtype=torch.float64, device="cuda") - 1
    p = 2 * np.pi * torch.rand(n, generator=g, dtype=torch.float64, device="cuda")
    s = torch.sqrt(1 - c * c)
    return torch.stack([r * s * torch.cos(p), r * s * torch.sin(p), r * c], 1)


def _box(case, seed):
    """The n1d^3 grid displaced by the curl-free field of a Gaussian random density."""
    n1, g = case["n1d"], _generator(seed)
    k = torch.fft.fftfreq(n1, dtype=torch.float64, device="cuda") * n1
    kz = torch.fft.rfftfreq(n1, dtype=torch.float64, device="cuda") * n1
    K = torch.meshgrid(k, k, kz, indexing="ij")
    k2 = K[0] ** 2 + K[1] ** 2 + K[2] ** 2
    k2[0, 0, 0] = 1.0
    amp = k2 ** (-2.5 / 4)
    amp[0, 0, 0] = 0.0
    white = torch.randn((n1, n1, n1), generator=g, dtype=torch.float64, device="cuda")
    delta = torch.fft.rfftn(white) * amp
    disp = torch.stack([torch.fft.irfftn(1j * q / k2 * delta, s=(n1, n1, n1)) for q in K], -1)
    disp *= case["rms"] / n1 / torch.sqrt((disp ** 2).sum(-1).mean())
    x = (torch.arange(n1, dtype=torch.float64, device="cuda") + 0.5) / n1
    grid = torch.stack(torch.meshgrid(x, x, x, indexing="ij"), -1)
    return torch.remainder(grid + disp, 1.0).reshape(-1, 3)


def _morton(x, box):
    """The bodies' order along the Z curve of their cube (21 bits per axis)."""
    x = x.double()
    if box > 0:
        origin, side = [0.0] * 3, box
    else:
        lo, hi = x.amin(0).tolist(), x.amax(0).tolist()
        side = max(h - l for l, h in zip(lo, hi)) * (1.0 + 1e-5)
        origin = [0.5 * (l + h) - 0.5 * side for l, h in zip(lo, hi)]
    o = torch.tensor(origin, dtype=torch.float64, device=x.device)
    cell = torch.floor((x - o) * (2.0 ** 21 / side)).long().clamp_(0, 2 ** 21 - 1)
    key = torch.zeros(len(x), dtype=torch.int64, device=x.device)
    for bit in range(20, -1, -1):
        for d in range(3):
            key = key << 1 | cell[:, d] >> bit & 1
    return torch.sort(key, stable=True).indices


def _bodies(case, seed):
    """(n, 4) float32 (x, y, z, m) on the GPU, total mass 1.  Programs that keep
    a plan keep their bodies along the space-filling curve; the calls that take
    positions get them in any order."""
    x = (_box if case["ics"] == "box" else _sphere)(case, seed).float()
    if case["ics"] == "box":
        x[x >= 1.0] = 0.0  # values that round up to the box side
    if case["call"] in ("eval", "lists", "dropin"):
        x = x[_morton(x, 1.0 if case["ics"] == "box" else 0.0)]
    m = torch.full((len(x), 1), 1.0 / len(x), dtype=torch.float32, device="cuda")
    return torch.cat([x, m], 1).contiguous()


def _softening(case):
    return (1.0 / case["n1d"] / 50.0) ** 2 if case["ics"] == "box" else 1e-4


def _weights(n, seed):
    """The loss of a gradient case: L = sum_i w_i . a_i + u_i phi_i."""
    g = _generator(seed + 7919)
    w = torch.randn((n, 3), generator=g, device="cuda")
    return w, torch.randn(n, generator=g, device="cuda")


def _tree_kw(case):
    return dict(leaf_max=16, group_max=32, p2cut=7, p4cut=20 if case["order"] == 4 else 0,
                tol=case["tol"])


class _DeviceArray:
    """A float32 array that its owner keeps on the GPU, for torch.as_tensor."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False),
                                         "version": 3}


# ------------------------------------------------------------ the calls
def prepare(case, seed):
    from pgrav import gravcuda as gc, host
    call = case["call"]
    box = 1.0 if case["ics"] == "box" else 0.0
    eps2, kw = _softening(case), _tree_kw(case)
    b = _bodies(case, seed)
    n = len(b)
    s = {"call": call, "box": box, "eps2": eps2, "kw": kw, "n": n}
    torch.cuda.synchronize()
    if call == "eval":
        s["plan"] = gc.Plan.build(None, None, eps2, box=box, ewald=box > 0, bodies=b, **kw)
        s["out"] = torch.as_tensor(_DeviceArray(s["plan"].output_ptr(), (n, 4), s["plan"]),
                                   device="cuda")
    elif call == "build":
        s["bodies"] = b.cpu().pin_memory().numpy()
        s["out"] = torch.empty((n, 4), dtype=torch.float32).pin_memory().numpy()
    elif call == "grad":
        s["pos"] = b[:, :3].contiguous().requires_grad_(True)
        s["mass"] = b[:, 3].contiguous().requires_grad_(True)
        s["w"], s["u"] = _weights(n, seed)
    elif call == "step":
        from pgrav.step import Stepper
        g = _generator(seed + 104729)
        v = torch.randn((n, 3), generator=g, device="cuda") * 0.01
        s["stepper"] = Stepper(b[:, :3].cpu().numpy(), v.cpu().numpy(), b[:, 3].cpu().numpy(),
                               eps2, box=box, rebuild=8, tree_kw=kw)
    else:
        x, m = b[:, :3].cpu().numpy(), b[:, 3].cpu().numpy()
        t = host.Tree(x, m, box=box, emit_aosoa=call == "dropin", **kw)
        if call == "lists":
            t.pack()
            s["lists"] = gc.pinned_problem(t, packed=True)
        else:
            s["tree"] = t
            s["table"] = gc.body_table(t.sorted_pos, t.points[:n, 3])
            s["packs"] = [(r, sz, t.aosoa[k][0], t.aosoa[k][1])
                          for k, (r, sz) in enumerate((("pMp", 4), ("pQp", 13)))]
            s["first"] = np.ascontiguousarray(t.groups["first"])
            s["count"] = np.ascontiguousarray(t.groups["count"])
    torch.cuda.synchronize()
    return s


def run(s):
    from pgrav import gravcuda as gc
    call = s["call"]
    if call == "eval":
        s["plan"].eval(torch.cuda.current_stream().cuda_stream)
        return {"acc_phi": s["out"]}
    if call == "build":
        return {"acc_phi": gc.build_eval(s["bodies"], s["eps2"], box=s["box"], ewald=s["box"] > 0,
                                         out=s["out"], **s["kw"])}
    if call == "grad":
        from pgrav.autograd import gravity
        kw = dict(s["kw"], box=s["box"], ewald=True) if s["box"] > 0 else s["kw"]
        acc, phi = gravity(s["pos"], s["mass"], s["eps2"], **kw)
        loss = (s["w"] * acc).sum() + (s["u"] * phi).sum()
        gx, gm = torch.autograd.grad(loss, (s["pos"], s["mass"]))
        return {"acc": acc.detach(), "phi": phi.detach(), "grad_pos": gx, "grad_mass": gm}
    if call == "step":
        energies = [r["e"] for r in s["stepper"].run(8, 1e-4)]
        pos, vel = s["stepper"].state()
        return {"energy": energies, "pos": pos, "vel": vel}
    if call == "lists":
        return {"acc_phi": gc.groups_eval_problem(s["lists"], s["eps2"], s["box"], ewald=True)}
    s["table"][:, 7:11] = 0.0
    d = gc.DropIn(s["table"])
    gc.drive_mn(d, s["first"], s["count"], s["packs"], s["eps2"])
    return {"acc": d.btab[:, 7:10], "phi": d.btab[:, 10]}


# ------------------------------------------------------------ work
def work(case):
    """Bytes: every body read once and every result written once (a gradient
    also reads its weights and writes dL/dx, dL/dm; the drop-in reads its
    lists).  Flops: interactions at 23 (point), 66 (quadrupole) or 217 (order
    4) each, their number a fit of the walks' counts over these ranges."""
    if case["ics"] == "box":
        n = case["n1d"] ** 3
        flops = n * min(23.0 * n, 1.2e5 * float(np.log2(n)) - 1.1e6)
    else:
        n = case["n"]
        flops = n * (1.95e4 if case["order"] == 2 else 1.6e4) * float(np.log2(n / 500.0)) * \
            (1e-4 / case["tol"]) ** 0.25
    passes = {"grad": 3.0, "step": 8.0}.get(case["call"], 1.0)
    nbytes = {"grad": 16 + 16 + 16 + 16, "step": 28 + 24, "dropin": 12 + 16 + 8000}
    return {"bytes": float(n * nbytes.get(case["call"], 32)), "flops": float(flops * passes)}


# ------------------------------------------------------------ 64 bits
_ALPHA = 12.0  # of the exact Ewald sum: erfc(6) is below 1e-16 at half the box


def _pairs(xs, x, m, eps2, box):
    """Direct sum over pairs at sinks xs: acc, phi (periodic: the part that is
    short-ranged in real space, on nearest images, softened as 1/sqrt(r^2 + eps2))."""
    d = xs[:, None, :] - x[None, :, :]
    if box > 0:
        d = d - torch.round(d.detach())
    r2 = (d * d).sum(-1)
    s = torch.rsqrt(r2 + eps2)
    phi, f = -s, -s ** 3
    if box > 0:
        near = r2 < 1e-12
        r = torch.sqrt(torch.where(near, torch.full_like(r2, 1e-12), r2))
        e = torch.erf(_ALPHA * r) / r
        g = 2 * _ALPHA / np.sqrt(np.pi)
        phi = phi + torch.where(near, torch.full_like(r, g), e)
        f = f + torch.where(near, torch.full_like(r, g * 2 * _ALPHA ** 2 / 3),
                            (e - g * torch.exp(-(_ALPHA * r) ** 2)) / (r * r))
    return (f[..., None] * d * m[None, :, None]).sum(1), (phi * m[None, :]).sum(1)


def _wave_vectors():
    h = torch.arange(-23, 24, dtype=torch.float64, device="cuda")
    v = torch.stack(torch.meshgrid(h, h, h, indexing="ij"), -1).reshape(-1, 3)
    h2 = (v * v).sum(1)
    half = (v[:, 2] > 0) | ((v[:, 2] == 0) & ((v[:, 1] > 0) | ((v[:, 1] == 0) & (v[:, 0] > 0))))
    v = v[half & (h2 <= 23 ** 2)]
    h2 = (v * v).sum(1)
    return 2 * np.pi * v, 2 * torch.exp(-np.pi ** 2 * h2 / _ALPHA ** 2) / (np.pi * h2)


def _waves(xs, x, m):
    """The periodic sum's smooth part (unit box) at sinks xs."""
    acc, phi = torch.zeros_like(xs), torch.zeros_like(xs[:, 0])
    k, a = _wave_vectors()
    step = max(1, (1 << 26) // max(len(x), len(xs)))
    for lo in range(0, len(k), step):
        kk, aa = k[lo:lo + step], a[lo:lo + step]
        p = x @ kk.T
        c, s = (m[:, None] * torch.cos(p)).sum(0), (m[:, None] * torch.sin(p)).sum(0)
        q = xs @ kk.T
        cq, sq = torch.cos(q), torch.sin(q)
        phi = phi - (aa * (cq * c + sq * s)).sum(1)
        acc = acc + (aa * (cq * s - sq * c)) @ kk
    return acc, phi


def _direct(x, m, eps2, box):
    """acc, phi of every body: direct sum, Ewald-summed in the unit box."""
    n, out = len(x), []
    step = max(1, (1 << 25) // n)
    for lo in range(0, n, step):
        out.append(_pairs(x[lo:lo + step], x, m, eps2, box))
    acc, phi = (torch.cat(v) for v in zip(*out))
    if box > 0:
        a, p = _waves(x, x, m)
        # the neutralising background; a body's own images count as pi / 4 L in place of 2.8373 / L
        acc, phi = acc + a, phi + p + np.pi / _ALPHA ** 2 * m.sum() - m * (2.837297479480620 - np.pi / 4)
    return acc, phi


def _direct_grad(x, m, w, u, eps2, box):
    """dL/dx and dL/dm of L = sum_i w_i . a_i + u_i phi_i, by autograd over chunks of sinks."""
    x, m = x.clone().requires_grad_(True), m.clone().requires_grad_(True)
    step = max(1, (1 << 24) // len(x))
    for lo in range(0, len(x), step):
        a, p = _pairs(x[lo:lo + step], x, m, eps2, box)
        ((w[lo:lo + step] * a).sum() + (u[lo:lo + step] * p).sum()).backward()
    gx, gm = x.grad, m.grad
    if box > 0:  # sum over k of a (cw c + sw s), with the sinks' sums in w and u
        x, m = x.detach(), m.detach()
        k, a = _wave_vectors()
        for lo in range(0, len(k), 2048):
            kk, aa = k[lo:lo + 2048], a[lo:lo + 2048]
            p = x @ kk.T
            c, s, wk = torch.cos(p), torch.sin(p), w @ kk.T
            C, S = (m[:, None] * c).sum(0), (m[:, None] * s).sum(0)
            uc, us = (u[:, None] * c).sum(0), (u[:, None] * s).sum(0)
            wc, ws = (wk * c).sum(0), (wk * s).sum(0)
            # L_k = a (wc S - ws C - uc C - us S)
            gm = gm + ((wc - us) * s - (ws + uc) * c) @ aa
            own = -wk * (s * S + c * C) + u[:, None] * (s * C - c * S)
            src = m[:, None] * ((wc - us) * c + (ws + uc) * s)
            gx = gx + (aa * (own + src)) @ kk
        gm = gm + u.sum() * np.pi / _ALPHA ** 2 - u * (2.837297479480620 - np.pi / 4)
    return gx, gm


def exact(case, seed):
    box = 1.0 if case["ics"] == "box" else 0.0
    n = case["n1d"] ** 3 if box else case["n"]
    if case["call"] == "step" or n > (240000 if box else 400000) or \
            (case["call"] == "grad" and n > 150000):
        return None
    b = _bodies(case, seed)
    x, m = b[:, :3].double(), b[:, 3].double()
    acc, phi = _direct(x, m, _softening(case), box)
    if case["call"] == "dropin":
        return {"acc": acc, "phi": None}  # its quadrupole potential has the reference's sign
    if case["call"] == "grad":
        w, u = _weights(n, seed)
        gx, gm = _direct_grad(x, m, w.double(), u.double(), _softening(case), box)
        return {"acc": acc, "phi": phi, "grad_pos": gx, "grad_mass": gm}
    return {"acc_phi": torch.cat([acc, phi[:, None]], 1)}
