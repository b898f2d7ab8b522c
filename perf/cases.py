"""Performance cases of the woven-field library: what its users have it do, through its public
entry points (fastweavturb_b200.api, .ensemble and .surrogate).

A case is a dict of plain values; its `kind` names the call:

``field``     one whole realisation, as the ensemble and the `tube` program build it: centerlines
              already on the GPU, Context.run() (deposition, Biot-Savart, normalisation, PDFs, S_p)
              and the statistics a caller reads back.  Sizes follow the surrogate family, the
              ensemble family, cfg0, cfg1 and the reference's own WT2 input (fastweavturb_b200.configs,
              tests/golden).
``lines``     the deposition of a set of lines alone (set_centerlines_device + deposit) on the larger
              grids, by tube thickness: levels of the 8-level benchmark family.
``spectral``  from omega to velocity and statistics: Biot-Savart, normalisation, spectra, PDFs, S_p.
``generate``  the fractional-Brownian-bridge generator of the centerlines.
``train``     training steps of the surrogate's network, weights read at the end.
``gradient``  the input gradient of the network's loss: one iteration of the inverse fit.

Inputs are drawn with torch from the seed: the fractional Brownian bridges of the field and
line cases by circulant embedding (the statistics of the library's own generator, another
stream).  exact() is the same quantity in 64 bits by torch alone: the reference's construction
written out for small fields, full FFTs, Philox in integer arithmetic for the generator.

Statistics of a single-precision field are returned in single precision: they carry the
field's rounding, not that of the FP64 sums behind them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fastweavturb_b200 as F
from fastweavturb_b200.ensemble import member_statistics
from fastweavturb_b200.surrogate import MLP, N_IN, N_OUT

PI2 = 2.0 * math.pi
DEV = "cuda"


def listed():
    fam = {"kind": "field", "precision": 32, "sigma0": 0.4, "tubes0": 4.0, "H": 0.7, "gexp": 4.0 / 3.0, "core_ratio": 1.0,
           "nodes_fixed": False, "db_over_sigma": 10.0}
    lines = {"kind": "lines", "N": 512, "H": 0.7, "gexp": 4.0 / 3.0, "db_over_sigma": 10.0}
    return [
        # one training realisation of the surrogate: the smallest call, made thousands of times
        dict(fam, name="surrogate-64", N=64, levels=3, nodes0=64),
        # a middle member of the ensemble: every kernel family meets in one small field
        dict(fam, name="member-192", N=192, levels=5, nodes0=256, tubes0=6.0, H=0.55, gexp=1.35),
        # the reference's shipped input: 73 lines of 148 nodes, cores varying by four along each,
        # on a grid that no tile divides
        dict(fam, name="varying-core-200", N=200, levels=3, nodes0=148, nodes_fixed=True, tubes0=1.0, sigma0=0.0604305,
             core_ratio=4.0, db_over_sigma=40.0),
        # the smallest configuration in double precision
        dict(fam, name="fp64-64", precision=64, N=64, levels=3, nodes0=256, sigma0=0.3),
        # the middle configuration: 256^3, six levels, single precision
        dict(fam, name="six-levels-256", N=256, levels=6, nodes0=256),
        # levels 0-3 of the 1024^3 benchmark on half its grid: tubes 122 to 15 spacings in radius
        dict(lines, name="thick-512", sigma0=0.5, levels=4, tubes0=2.0, nodes0=256, tubes_growth=4),
        # its levels 3 and 4: 15 and 7.6 spacings
        dict(lines, name="middle-512", sigma0=0.0625, levels=2, tubes0=128.0, nodes0=2048, tubes_growth=4),
        # its levels 5 and 6: 3.8 and 1.9 spacings, a share of their tubes
        dict(lines, name="thin-512", sigma0=0.015625, levels=2, tubes0=256.0, nodes0=8192, tubes_growth=1),
        # omega to u and statistics on half the benchmark's grid
        {"name": "spectral-512", "kind": "spectral", "N": 512, "precision": 32, "bins": 201, "order": 6},
        # the centerlines of the middle configuration's first five levels
        {"name": "generate-5-levels", "kind": "generate", "levels": 5, "tubes0": 4, "nodes0": 256, "H": 0.7, "sigma0": 0.4},
        # the surrogate's training loop at its own batch
        {"name": "train-256", "kind": "train", "batch": 256, "steps": 8, "width": 256, "depth": 4},
        # the inverse fit: 64 starts for each of three level counts
        {"name": "gradient-192", "kind": "gradient", "batch": 192, "width": 256, "depth": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    # deposition grids are multiples of four; tiles are 16 x 8 x 8 points, so most are ragged
    kind = rng.choice(["field", "field", "field", "lines", "lines", "lines", "spectral", "generate", "train", "gradient"])
    if kind == "field":
        precision = rng.choice([32, 32, 32, 64])
        varying = rng.random() < 0.25
        N = 4 * _log_int(rng, 8, 24 if precision == 64 else 60)
        case = {"kind": kind, "precision": precision, "N": N, "H": round(rng.uniform(0.3, 0.8), 4),
                "gexp": round(rng.uniform(1.2, 1.5), 4)}
        if varying:
            case.update(levels=rng.randint(1, 3), nodes0=_log_int(rng, 37, 300), nodes_fixed=True, tubes0=1.0,
                        sigma0=round(rng.uniform(0.04, 0.08), 5), core_ratio=rng.choice([2.0, 4.0]), db_over_sigma=40.0)
        else:
            deepest = 3 if precision == 64 or N < 100 else 5
            case.update(levels=rng.randint(2, deepest), nodes0=rng.choice([64, 100, 256]), nodes_fixed=False,
                        tubes0=round(rng.uniform(2.0, 8.0), 3), sigma0=round(rng.uniform(0.25, 0.5), 4), core_ratio=1.0,
                        db_over_sigma=10.0)
        return case
    if kind == "lines":
        N = 4 * _log_int(rng, 32, 128)
        cells = math.exp(rng.uniform(math.log(1.2), math.log(120.0)))   # truncation radius in grid spacings
        sigma = cells * PI2 / N / 3.0
        sigma = min(sigma, 0.5)
        nodes = _log_int(rng, 200, 6000)
        # accepted pairs per node: 10 sigma pi (3 sigma)^2 / dx^3; at most ~6e9 pairs and 3 M nodes
        per_node = 90.0 * math.pi * (sigma * N / PI2) ** 3
        budget = min(math.exp(rng.uniform(math.log(1e8), math.log(6e9))) / per_node, 3e6)
        tubes = max(1.0, min(20000.0, budget / nodes))
        nodes = int(max(32, min(nodes, budget / tubes)))
        return {"kind": kind, "N": N, "H": round(rng.uniform(0.3, 0.8), 4), "gexp": 4.0 / 3.0, "db_over_sigma": 10.0,
                "sigma0": round(sigma, 6), "levels": 1, "tubes0": float(int(tubes)), "nodes0": nodes, "tubes_growth": 4}
    if kind == "spectral":
        precision = rng.choice([32, 32, 64])
        return {"kind": kind, "N": 2 * _log_int(rng, 12, 128 if precision == 64 else 256), "precision": precision,
                "bins": rng.choice([100, 201, 1000]), "order": rng.choice([4, 6, 10])}
    if kind == "generate":
        return {"kind": kind, "levels": rng.randint(1, 4), "tubes0": rng.randint(1, 16), "nodes0": rng.choice([64, 128, 200, 256, 300]),
                "H": round(rng.uniform(0.3, 0.8), 4), "sigma0": round(rng.uniform(0.2, 0.5), 4)}
    if kind == "train":
        return {"kind": kind, "batch": _log_int(rng, 16, 2048), "steps": rng.randint(2, 8), "width": rng.choice([64, 128, 256]),
                "depth": rng.randint(1, 4)}
    return {"kind": kind, "batch": _log_int(rng, 1, 4096), "width": rng.choice([64, 128, 256]), "depth": rng.randint(1, 4)}


# ------------------------------------------------------------------------------ inputs
def _bridges(gen, T, n, H, dB):
    """T closed fractional-Brownian-bridge loops of n nodes: (T, 3, n) FP64 in [-pi, pi)."""
    k = torch.arange(2 * n, dtype=torch.float64, device=DEV)
    k = torch.minimum(k, 2 * n - k)
    row = 0.5 * ((k + 1) ** (2 * H) - 2 * k ** (2 * H) + (k - 1).abs() ** (2 * H))
    lam = torch.fft.fft(row).real.clamp_min(0.0)
    z = torch.randn((T, 3, 2 * n, 2), generator=gen, dtype=torch.float64, device=DEV)
    z = torch.view_as_complex(z) * (lam / (2 * n)).sqrt()
    fbm = torch.fft.fft(z).real[..., :n].cumsum(-1)
    del z
    return _close(fbm, H, dB, (torch.rand((T, 3, 1), generator=gen, dtype=torch.float64, device=DEV) - 0.5) * PI2)


def _close(fbm, H, dB, shift):
    """Bridge, rms node step dB, shift and wrap of the paths fbm (T, 3, n)."""
    n = fbm.shape[-1]
    x = torch.arange(1, n + 1, dtype=torch.float64, device=DEV) / n
    f = 0.5 * (x ** (2 * H) + 1.0 - (1.0 - x) ** (2 * H))
    b = fbm - f * fbm[..., -1:]
    step = ((b[..., 1:] - b[..., :-1]) ** 2).sum((1, 2), keepdim=True) / (n - 1)
    v = b * (dB / step.sqrt()) + shift
    return v - torch.floor(v / PI2) * PI2 - math.pi


def _levels(c):
    out = []
    for l in range(int(c["levels"])):
        s = c["sigma0"] * 2.0 ** (-l)
        growth = c.get("tubes_growth", 8 if c.get("nodes_fixed") else 4)
        out.append((max(1, int(round(c["tubes0"] * growth ** l))), c["nodes0"] if c.get("nodes_fixed") else c["nodes0"] * 2 ** l, s,
                    (s / c["sigma0"]) ** c["gexp"]))
    return out


def _lines(c, seed):
    """Centerlines of a field or line case: per level the loops, and the per-line arrays."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    loops, npoint, sigma, Gamma, n_T = [], [], [], [], []
    for l, (T, n, s, G) in enumerate(_levels(c)):
        loops.append(_bridges(gen, T, n, c["H"], c["db_over_sigma"] * s))
        sign = 1 - 2 * torch.randint(0, 2, (T,), generator=gen, device=DEV)
        npoint += [n] * T
        sigma += [s] * T
        Gamma += (G * sign.double()).tolist()
        n_T += [2 ** l if c.get("core_ratio", 1.0) != 1.0 else 1] * T
    return loops, np.array(npoint, dtype=np.int64), np.array(sigma), np.array(Gamma), np.array(n_T, dtype=np.int32)


def _omega(N, precision, seed):
    """A random solenoidal field of the woven fields' kind (energy falling as k^-5/3 from the
    largest scales, vorticity as k^1/3), made in FP64 and given the field's precision."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    real = torch.float64 if precision == 64 else torch.float32
    kx = torch.arange(N // 2 + 1, device=DEV, dtype=real)
    ky = torch.fft.fftfreq(N, 1.0 / N, device=DEV).to(real)
    k = (ky[:, None, None], ky[None, :, None], kx[None, None, :])        # z, y, x
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    amp = torch.where(k2 > 0, k2.clamp_min(1.0) ** (-5.0 / 6.0), torch.zeros_like(k2)) * torch.exp(-(k2 / (N / 3.0) ** 2))
    out = torch.empty((3, N, N, N), dtype=real, device=DEV)
    pot = []
    for _ in range(3):
        pot.append(torch.fft.rfftn(torch.randn((N, N, N), generator=gen, dtype=real, device=DEV)) * amp)
    for d in range(3):
        a, b = (d + 1) % 3, (d + 2) % 3                                  # curl of the potential, x y z order
        out[d] = torch.fft.irfftn(1j * (k[2 - a] * pot[b] - k[2 - b] * pot[a]), s=(N, N, N))
    return out / out.square().mean().sqrt()


def _mlp_batch(c, seed):
    rng = np.random.default_rng(int(seed))
    steps = int(c.get("steps", 1))
    x = rng.uniform(-1.0, 1.0, (steps, c["batch"], N_IN)).astype(np.float32)
    # smooth targets of unit size, as the standardised statistics are
    A = rng.normal(0.0, 1.0, (N_IN, N_OUT))
    t = (np.sin(x @ A) + 0.3 * np.tanh(2.0 * x[..., :1])).astype(np.float32)
    w = np.zeros(N_OUT, dtype=np.float32)
    w[:40] = 1.0                                                         # spectrum and flatness
    return x, t, w


def _weights(c, seed):
    """The network's parameters, layer by layer: W (N x K) then b."""
    rng = np.random.default_rng(int(seed) + 7)
    widths = [N_IN] + [c["width"]] * c["depth"] + [N_OUT]
    out = []
    for K, N in zip(widths[:-1], widths[1:]):
        a = math.sqrt(6.0 / (K + N))
        out += [rng.uniform(-a, a, N * K).astype(np.float32), rng.uniform(-0.1, 0.1, N).astype(np.float32)]
    return np.concatenate(out), widths


# ------------------------------------------------------------------------------ passes
def prepare(c, seed):
    kind = c["kind"]
    if kind in ("field", "lines"):
        loops, npoint, sigma, Gamma, n_T = _lines(c, seed)
        xyz = torch.cat([p.permute(1, 0, 2).reshape(3, -1) for p in loops], 1).contiguous()
        # lines of one context as the ensemble makes it: 201 bins, order 6, no field output
        ctx = F.Context(F.Params(N=c["N"], N_downsample=c["N"], line_s=1, line_e=len(npoint), sigma_ratio=c.get("core_ratio", 1.0),
                                 precision=c.get("precision", 32), pdf_bins=201, Sp_order=6, vorticity_output=0))
        arrays = (npoint, xyz[0].data_ptr(), xyz[1].data_ptr(), xyz[2].data_ptr(), sigma, Gamma, n_T)
        torch.cuda.synchronize()
        ctx.set_centerlines_device(*arrays)
        return {"case": c, "ctx": ctx, "xyz": xyz, "arrays": arrays}
    if kind == "spectral":
        N = c["N"]
        omega = _omega(N, c["precision"], seed)
        ctx = F.Context(F.Params(N=N, N_downsample=N, line_s=1, line_e=1, sigma_ratio=1.0, precision=c["precision"],
                                 pdf_bins=c["bins"], Sp_order=c["order"], vorticity_output=0))
        # a context owns its omega: one line is deposited, then the field is written over it
        ang = np.linspace(0.0, PI2, 64, endpoint=False)
        ctx.set_centerlines([64], np.stack([np.cos(ang), np.sin(ang), 0 * ang], 1), [0.3], [1.0], [1])
        ctx.deposit()
        ctx.field_tensor(0).copy_(omega)
        del omega
        torch.cuda.synchronize()
        return {"case": c, "ctx": ctx}
    if kind == "generate":
        n = sum(T * p for T, p in _gen_levels(c))
        ctx = F.Context(F.Params(N=64, N_downsample=64))
        return {"case": c, "ctx": ctx, "seed": int(seed), "xyz": torch.empty((3, n), dtype=torch.float64, device=DEV)}
    x, t, w = _mlp_batch(c, seed)
    p, _ = _weights(c, seed)
    net = MLP(N_IN, c["width"], c["depth"], N_OUT, batch_max=4096)
    net.set_params(p)
    return {"case": c, "net": net, "x": x, "t": t, "w": w}


def _gen_levels(c):
    return [(c["tubes0"] * 4 ** l, c["nodes0"] * 2 ** l) for l in range(c["levels"])]


def _field(s, which):
    """The context's own field, as a tensor that keeps the context alive (field_tensor is a view
    of memory the context frees)."""
    view = s["ctx"].field_tensor(which)
    view.owner = s["ctx"]
    return view


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "field":
        ctx = s["ctx"]
        ctx.run()
        st = member_statistics(ctx, c["N"])
        real = np.float64 if c["precision"] == 64 else np.float32
        return {"omega": _field(s, 0), "u": _field(s, 1), "Ek": st["Ek"].astype(real), "Sp": st["Sp"].astype(real),
                "up": np.array(st["up"], dtype=real)}
    if kind == "lines":
        ctx = s["ctx"]
        ctx.set_centerlines_device(*s["arrays"])
        ctx.deposit()
        return {"omega": _field(s, 0)}
    if kind == "spectral":
        ctx = s["ctx"]
        ctx.biot_savart()
        up = ctx.cal_helicity()["up"]
        Ew, Eu = ctx.spectrum(0), ctx.spectrum(1)
        pu, pw = ctx.export_pdf(0, nbins=c["bins"]), ctx.export_pdf(1, nbins=c["bins"])
        Sp = ctx.Sp_calculate(pmax=c["order"])[1]
        real = np.float64 if c["precision"] == 64 else np.float32
        return {"u": _field(s, 1), "Ew": Ew.astype(real), "Eu": Eu.astype(real), "Sp": Sp.astype(real),
                "up": np.array(up, dtype=real), "pdf_u": pu[1], "pdf_w": pw[1], "bins_u": pu[0], "bins_w": pw[0],
                "counts_u": pu[2].astype(np.int64), "counts_w": pw[2].astype(np.int64)}
    if kind == "generate":
        lev = _gen_levels(c)
        x = s["xyz"]
        s["ctx"].fbb_generate(s["seed"], [T for T, _ in lev], [n for _, n in lev], [c["H"]] * len(lev),
                              [10.0 * c["sigma0"] * 2.0 ** (-l) for l in range(len(lev))], x[0].data_ptr(), x[1].data_ptr(),
                              x[2].data_ptr())
        return {"xyz": x}
    net = s["net"]
    if kind == "train":
        loss = [net.train_step(s["x"][k], s["t"][k], 1e-3) for k in range(c["steps"])]
        return {"loss": np.array(loss, dtype=np.float32), "params": net.params()}
    loss, _, gx = net.loss_grad(s["x"][0], s["t"][0], w_out=s["w"], params=False, inputs=True)
    return {"loss": np.array(loss, dtype=np.float32), "grad_x": gx}


# ------------------------------------------------------------------------------ work
def work(c):
    """Bytes: nodes in, fields and statistics out.  Operations: 145 per accepted (grid point,
    tube) pair (the tests and the Burgers profile), 5/2 n log2 n per real transform, and the
    matrix products of the network."""
    kind = c["kind"]
    if kind in ("field", "lines"):
        N, rb = c["N"], c.get("precision", 32) // 8
        nodes = pairs = 0
        r = c.get("core_ratio", 1.0)
        area = 1.0 + (r - 1.0) + 0.375 * (r - 1.0) ** 2                  # mean square core over its minimum's
        for T, n, s, _ in _levels(c):
            nodes += T * n
            pairs += T * n * c["db_over_sigma"] * s * 9.0 * math.pi * s * s * area / (PI2 / N) ** 3
        whole = kind == "field"
        fft = 6 * 2.5 * N ** 3 * math.log2(N ** 3) if whole else 0.0
        return {"bytes": 24.0 * nodes + (6 if whole else 3) * rb * float(N) ** 3, "flops": 145.0 * pairs + fft}
    if kind == "spectral":
        N, rb = c["N"], c["precision"] // 8
        nr = 2 * int(math.log2(N)) + 1
        return {"bytes": 6.0 * rb * N ** 3, "flops": 15.0 * N ** 3 * math.log2(N ** 3) + 3.0 * N ** 3 * nr * 2 * c["order"]}
    if kind == "generate":
        n = sum(T * p for T, p in _gen_levels(c))
        return {"bytes": 24.0 * n, "flops": sum(3 * T * 5 * 2 * p * math.log2(2 * p) for T, p in _gen_levels(c))}
    _, widths = _weights({"width": c["width"], "depth": c["depth"]}, 0)
    macs = sum(K * N for K, N in zip(widths[:-1], widths[1:]))
    nw = macs + sum(widths[1:])
    if kind == "train":
        return {"bytes": c["steps"] * (4.0 * c["batch"] * (N_IN + N_OUT) + 24.0 * nw), "flops": 6.0 * macs * c["batch"] * c["steps"]}
    return {"bytes": 4.0 * c["batch"] * (2 * N_IN + N_OUT) + 4.0 * nw, "flops": 4.0 * macs * c["batch"]}


# ------------------------------------------------------------------------------ 64 bits
def exact(c, seed):
    kind = c["kind"]
    if kind == "lines":
        if _box_points(c) > 3e9:
            return None
        return {"omega": _deposit64(c, *_lines(c, seed))}
    if kind == "field":
        if _box_points(c) > 3e9:
            return None
        omega = _deposit64(c, *_lines(c, seed))
        u, _, Eu = _biot_savart64(omega)
        up = math.sqrt(float(u.square().sum()) / c["N"] ** 3 / 3.0)
        return {"omega": omega, "u": u, "Ek": (Eu / up ** 2).cpu().numpy(), "Sp": _sp64(u / up, 6), "up": np.array(up)}
    if kind == "spectral":
        omega = _omega(c["N"], c["precision"], seed).double()
        u, Ew, Eu = _biot_savart64(omega)
        up = math.sqrt(float(u.square().sum()) / c["N"] ** 3 / 3.0)
        del omega
        # the histograms' edges are rounded in single precision by definition: no 64-bit value
        return {"u": u, "Ew": Ew.cpu().numpy(), "Eu": (Eu / up ** 2).cpu().numpy(), "Sp": _sp64(u / up, c["order"]), "up": np.array(up),
                "pdf_u": None, "pdf_w": None, "bins_u": None, "bins_w": None, "counts_u": None, "counts_w": None}
    if kind == "generate":
        return {"xyz": _generate64(c, seed)}
    return _mlp64(c, seed)


def _box_points(c):
    total, r = 0.0, c.get("core_ratio", 1.0)
    for T, n, s, _ in _levels(c):
        dx = PI2 / c["N"]
        side = 2.0 * 3.0 * s * r / dx + c["db_over_sigma"] * s / 14.0 / dx + 2.0
        total += T * n * 14.0 * side ** 3
    return total


def _wrap(v):
    v = torch.where(v > math.pi, v - PI2, v)
    return torch.where(v < -math.pi, v + PI2, v)


def _deposit64(c, loops, npoint, sigma, Gamma, n_T):
    """The reference's construction loop in FP64: periodic arc length, quintic splines, the
    1001-sample turning angle, sub-segments, and the box walk of every sub-segment."""
    N = c["N"]
    omega = torch.zeros((3, N * N * N), dtype=torch.float64, device=DEV)
    first = 0
    for loop in loops:
        T = loop.shape[0]
        sl = slice(first, first + T)
        group = max(1, int(4e5 // loop.shape[2]))
        for a in range(0, T, group):
            b = min(T, a + group)
            _deposit64_lines(c, loop[a:b].permute(0, 2, 1), sigma[sl][a:b], Gamma[sl][a:b], n_T[sl][a:b], omega)
        first += T
    return omega.reshape(3, N, N, N)


def _poly(a, z, der=0):
    """Quintic a[..., 3, 6] (or its derivatives) at z[...]: (..., 3)."""
    out = 0.0
    for m in range(5, der - 1, -1):
        k = float(math.perm(m, der))
        out = out * z[..., None] + k * a[..., m]
    return out


def _deposit64_lines(c, x, sigma, Gamma, n_T, omega):
    N = c["N"]
    t64 = dict(dtype=torch.float64, device=DEV)
    L_, n, _ = x.shape
    smin = torch.tensor(sigma, **t64)
    smax = smin * c.get("core_ratio", 1.0)
    G = torch.tensor(Gamma, **t64)
    step = torch.roll(x, -1, 1) - x
    step = step.abs()
    step = torch.where(step > math.pi, step - PI2, step).square().sum(-1).sqrt()
    total = step.sum(1)
    ze = torch.cat([torch.zeros_like(total)[:, None], step.cumsum(1)[:, :-1]], 1) * PI2 / total[:, None]
    Len = total / PI2
    z_ext = torch.cat([ze, torch.full_like(total, PI2)[:, None], PI2 + ze[:, 1:2]], 1)      # n + 2
    dz = (torch.roll(ze, -1, 1) - torch.roll(ze, 1, 1))
    dz = torch.where(dz < 0, dz + PI2, dz) * Len[:, None]
    v = _wrap(torch.roll(x, -1, 1) - torch.roll(x, 1, 1)) / dz[..., None]
    acc = (torch.roll(v, -1, 1) - torch.roll(v, 1, 1)) / dz[..., None]

    def nxt(q):
        return torch.roll(q, -1, 1)
    zr = ((z_ext[:, 1:n + 1] - z_ext[:, :n]) * Len[:, None])[..., None]
    xl, xr, vl, vr, al, ar = x, nxt(x), v, nxt(v), acc, nxt(acc)
    d = xr - xl
    d = torch.where(d > math.pi, d - PI2, torch.where(d < -math.pi, d + PI2, d))
    coe = torch.stack([xl, vl, al / 2,
                       (20 * d - (12 * vl + 8 * vr) * zr - (3 * al - ar) * zr ** 2) / (2 * zr ** 3),
                       (-30 * d + (16 * vl + 14 * vr) * zr + (3 * al - 2 * ar) * zr ** 2) / (2 * zr ** 4),
                       (12 * d - 6 * (vl + vr) * zr - (al - ar) * zr ** 2) / (2 * zr ** 5)], -1)   # line, section, 3, 6
    # turning angle over 1001 samples
    h = (z_ext[:, 1:n + 1] - z_ext[:, :n]) / 1000.0
    theta = torch.zeros_like(h)
    for j0 in range(0, 1001, 13):
        j = torch.arange(j0, j0 + 13, **t64)
        zz = h[..., None] * j * Len[:, None, None]
        c1, c2 = _poly(coe[:, :, None], zz, 1), _poly(coe[:, :, None], zz, 2)
        theta += (torch.linalg.cross(c1, c2).norm(dim=-1) / c1.square().sum(-1)).sum(-1)
    theta = theta * h * Len[:, None]
    ntf = (torch.ceil(50.0 * theta / PI2) + 1).long()
    dtf = (z_ext[:, 1:n + 1] - z_ext[:, :n]) / ntf
    # sub-segments
    cnt = ntf.reshape(-1)
    sec = torch.repeat_interleave(torch.arange(L_ * n, device=DEV), cnt)
    jj = torch.arange(len(sec), device=DEV) - torch.repeat_interleave(cnt.cumsum(0) - cnt, cnt)
    line, t = sec // n, sec % n
    cf, zl, dt, ns = coe.reshape(-1, 3, 6), z_ext[:, :n].reshape(-1), dtf.reshape(-1), cnt
    nextsec = line * n + (t + 1) % n

    def sample(k):
        p = _poly(cf[sec], dt[sec] * k * Len[line])
        p = torch.where(p >= math.pi, p - PI2, p)
        p = torch.where(p < -math.pi, p + PI2, p)
        q = _poly(cf[nextsec], dt[nextsec] * Len[line])
        q = torch.where(q >= math.pi, q - PI2, q)
        q = torch.where(q < -math.pi, q + PI2, q)
        node = x.reshape(-1, 3)[nextsec]
        kk = k[:, None]
        n_ = ns[sec][:, None]
        return torch.where(kk < n_, p, torch.where(kk == n_, node, q))
    s0, s1, s2 = sample(jj), sample(jj + 1), sample(jj + 2)
    ch0, ch1 = _wrap(s1 - s0), _wrap(s2 - s1)
    nd = ch0.norm(dim=-1)
    tc0, tc1 = ch0 / nd[:, None], ch1 / ch1.norm(dim=-1, keepdim=True)
    gap = s1 - s0
    ci0 = torch.where(gap > math.pi, s0 + PI2, s0)
    ci1 = torch.where(gap < -math.pi, s1 + PI2, s1)
    za, zb = zl[sec] + dt[sec] * jj, zl[sec] + dt[sec] * (jj + 1)
    wave = torch.floor(Len * PI2 / math.pi + 0.5) * torch.tensor(n_T, **t64)

    def core(zeta, ln):
        return smin[ln] + (smax - smin)[ln] * (torch.sin(wave[ln] * zeta) + 1) / 2
    Rt = 3.0 * torch.maximum(core(za, line), core(zb, line))
    dx = PI2 / N
    lo = torch.floor((torch.minimum(ci0, ci1) + math.pi - Rt[:, None]) / dx + 1).long()
    hi = torch.ceil((torch.maximum(ci0, ci1) + math.pi + Rt[:, None]) / dx + 1).long()
    ext = hi - lo + 1
    vol = ext.prod(-1)
    ends = vol.cumsum(0)
    a, at = 0, 0
    while a < len(vol):
        b = max(a + 1, int(torch.searchsorted(ends, at + 12_000_000, right=True)))
        q = torch.repeat_interleave(torch.arange(a, b, device=DEV), vol[a:b])
        o = torch.arange(len(q), device=DEV) - torch.repeat_interleave(ends[a:b] - vol[a:b] - at, vol[a:b])
        at, a = int(ends[b - 1]), b
        e = ext[q]
        idx = torch.stack([o % e[:, 0], (o // e[:, 0]) % e[:, 1], o // (e[:, 0] * e[:, 1])], -1) + lo[q]
        m = (idx.double() - 1) * dx - math.pi
        d0, d1 = m - ci0[q], m - ci1[q]
        t0, t1 = (d0 * tc0[q]).sum(-1), (d1 * tc1[q]).sum(-1)
        keep = (t0 >= 0) & (t1 < 0)
        keep &= (d0.square().sum(-1) - t0 * t0).clamp_min(0).sqrt() < Rt[q]
        q, idx, m, t0 = q[keep], idx[keep], m[keep], t0[keep]
        t1 = ((m - ci1[q]) * tc0[q]).sum(-1)
        zeta = (zb[q] * t0 - za[q] * t1) / nd[q]
        s_, ln = sec[q], line[q]
        zz = (zeta - zl[s_]) * Len[ln]
        p = _poly(cf[s_], zz)
        p = torch.where(p >= math.pi, p - PI2, p)
        p = torch.where(p < -math.pi, p + PI2, p)
        c1, c2 = _poly(cf[s_], zz, 1), _poly(cf[s_], zz, 2)
        n1 = c1.norm(dim=-1, keepdim=True)
        tan = c1 / n1
        X = torch.linalg.cross(c1, c2)
        nX = X.norm(dim=-1, keepdim=True)
        r = _wrap(m - p)
        rho = r.norm(dim=-1, keepdim=True)
        sg = core(zeta, ln)[:, None]
        prof = (torch.exp(-rho ** 2 / 2 / sg ** 2) - torch.exp(-Rt[q][:, None] ** 2 / 2 / sg ** 2)) / (PI2 * sg ** 2) * G[ln][:, None]
        val = prof * tan
        if c.get("core_ratio", 1.0) != 1.0:
            hz = dt[s_].clamp_max(1e-4)
            ds = ((core(zeta + hz, ln) - core(zeta - hz, ln)) / (2 * hz))[:, None] / n1 / Len[ln][:, None]
            B = X / nX.clamp_min(1e-300)
            Nv = torch.linalg.cross(B, tan)
            kap = nX / n1 ** 3
            ct = (r * Nv).sum(-1, keepdim=True) / (rho + 1e-15)
            st = (r * B).sum(-1, keepdim=True) / (rho + 1e-15)
            den = 1 - kap * rho * ct
            curved = ct * rho * ds / sg / den * Nv + st * rho * ds / sg / den * B
            straight = rho * ds / sg * r / (rho + 1e-15)
            val = val + prof * torch.where(nX < 1e-8, straight, curved)
        g = (idx - 1) % N
        cell = g[:, 0] + N * (g[:, 1] + N * g[:, 2])
        for k in range(3):
            omega[k].index_add_(0, cell, val[:, k])


def _biot_savart64(w):
    """u = curl^-1 of w (3, N, N, N) [z, y, x], and the shell spectra of w and u."""
    N = w.shape[-1]
    kx = torch.arange(N // 2 + 1, device=DEV, dtype=torch.float64)
    kf = torch.arange(N, device=DEV, dtype=torch.float64)
    kf = torch.where(kf >= N // 2, kf - N, kf)
    k = [kx[None, None, :], kf[None, :, None], kf[:, None, None]]
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    shell = (torch.sqrt(k2 + 1e-8) + 0.5).long().reshape(-1)
    wgt = torch.full((N // 2 + 1,), 2.0, device=DEV, dtype=torch.float64)
    wgt[0] = wgt[N // 2] = 1.0
    odd = [torch.where(q.abs() == N // 2, torch.zeros_like(q), q) for q in k]   # the Nyquist planes' derivative is zero
    inv = torch.where(k2 > 0, 1.0 / k2.clamp_min(1.0), torch.zeros_like(k2))
    W = [torch.fft.rfftn(w[d]) / N ** 3 for d in range(3)]
    u = torch.empty_like(w)
    e = [torch.zeros_like(k2), torch.zeros_like(k2)]
    for d in range(3):
        a, b = (d + 1) % 3, (d + 2) % 3
        U = 1j * (odd[a] * W[b] - odd[b] * W[a]) * inv
        e[0] += 0.5 * wgt * (W[d].real ** 2 + W[d].imag ** 2)
        e[1] += 0.5 * wgt * (U.real ** 2 + U.imag ** 2)
        u[d] = torch.fft.irfftn(U, s=(N, N, N)) * N ** 3
    spec = [torch.zeros(int(shell.max()) + 1, device=DEV, dtype=torch.float64).index_add_(0, shell, q.reshape(-1)) for q in e]
    return u, spec[0][1:N // 2 + 1], spec[1][1:N // 2 + 1]


def _sp64(u, order):
    N = u.shape[-1]
    out = np.zeros((order, len(F.sp_separations(N))))
    for m, r in enumerate(F.sp_separations(N)):
        for d in range(3):
            du = torch.roll(u[d], -int(r), 2 - d) - u[d]
            pw = du.clone()
            for p in range(order):
                out[p, m] += float(pw.sum())
                pw *= du
    return out / (3.0 * N ** 3)


def _philox(ctr, key):
    """Philox4x32-10 on int64 tensors holding 32-bit words."""
    mask = 0xFFFFFFFF
    c = [torch.as_tensor(v, dtype=torch.int64, device=DEV) for v in ctr]
    k0, k1 = key & mask, (key >> 32) & mask
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & mask) ^ c[1] ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _generate64(c, seed):
    out, t0 = [], 0
    for l, (T, n) in enumerate(_gen_levels(c)):
        M = max(n, 128)
        H, dB = c["H"], 10.0 * c["sigma0"] * 2.0 ** (-l)
        k = torch.arange(2 * M, dtype=torch.float64, device=DEV)
        k = torch.minimum(k, 2 * M - k)
        lam = torch.fft.fft(0.5 * ((k + 1) ** (2 * H) - 2 * k ** (2 * H) + (k - 1).abs() ** (2 * H))).real.clamp_min(0.0)
        tube = torch.arange(t0, t0 + T, device=DEV)
        w = _philox([torch.arange(2 * M, device=DEV)[None, None, :].expand(T, 3, -1), tube[:, None, None].expand(-1, 3, 2 * M),
                     torch.arange(3, device=DEV)[None, :, None].expand(T, -1, 2 * M), torch.zeros((T, 3, 2 * M), dtype=torch.int64, device=DEV)], seed)
        a, b = (((w[i] >> 5).double() * 67108864.0 + (w[i + 1] >> 6).double() + 0.5) / 9007199254740992.0 for i in (0, 2))
        r = torch.sqrt(-2.0 * torch.log(a)) * (lam / (2 * M)).sqrt()
        fbm = torch.fft.fft(torch.complex(r * torch.cos(PI2 * b), r * torch.sin(PI2 * b))).real[..., :M].cumsum(-1)
        if n < 128:
            fbm = fbm[..., torch.arange(1, n + 1, device=DEV) * (128 // n) - 1]
        s = _philox([torch.arange(3, device=DEV)[None, :].expand(T, -1), tube[:, None].expand(-1, 3),
                     torch.full((T, 3), 3, device=DEV), torch.zeros((T, 3), dtype=torch.int64, device=DEV)], seed)
        shift = (((s[0] >> 5).double() * 67108864.0 + (s[1] >> 6).double()) / 9007199254740992.0 - 0.5) * PI2
        out.append(_close(fbm, H, dB, shift[..., None]).permute(1, 0, 2).reshape(3, -1))
        t0 += T
    return torch.cat(out, 1)


def _mlp64(c, seed):
    x, t, w = _mlp_batch(c, seed)
    flat, widths = _weights(c, seed)
    p, o = [], 0
    for K, N in zip(widths[:-1], widths[1:]):
        p += [torch.tensor(flat[o:o + N * K].reshape(N, K).astype(np.float64)), torch.tensor(flat[o + N * K:o + N * K + N].astype(np.float64))]
        o += N * K + N
    p = [q.requires_grad_() for q in p]

    def loss_of(x, t, w):
        h = x
        for i in range(0, len(p), 2):
            h = h @ p[i].T + p[i + 1]
            h = torch.nn.functional.gelu(h) if i + 2 < len(p) else h
        return (w * (h - t) ** 2).sum() / t.numel()
    if c["kind"] == "gradient":
        X = torch.tensor(x[0].astype(np.float64), requires_grad=True)
        loss = loss_of(X, torch.tensor(t[0].astype(np.float64)), torch.tensor(w.astype(np.float64)))
        return {"loss": np.array(loss.item()), "grad_x": torch.autograd.grad(loss, X)[0].numpy()}
    opt = torch.optim.Adam(p, lr=1e-3, eps=1e-8)
    losses = []
    for k in range(c["steps"]):
        opt.zero_grad()
        loss = loss_of(torch.tensor(x[k].astype(np.float64)), torch.tensor(t[k].astype(np.float64)), 1.0)
        loss.backward()
        opt.step()
        losses.append(loss.item())
    return {"loss": np.array(losses), "params": np.concatenate([q.detach().numpy().ravel() for q in p])}
