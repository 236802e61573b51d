"""Timed cases of the framework's public entry points.

Each case is a dict of plain values; ``prepare`` builds what a user's program
holds before the call (engine, fields, packets, network), ``run`` makes one pass
through the public API, ``work`` counts the bytes and operations such a pass
cannot do without, and ``exact`` evaluates the same pass in 64 bits with plain
torch / numpy, without the package (None where that is not defined or takes too
long).

Kinds:

* ``iterate``  -- ``TransportEngine.run_iterations(1)``: one shoot + balance
  iteration of the plain photoionization method on fields resident on the GPU,
  the step that the driver repeats.  ``coupled``: the host sends n_H and x_H
  before it and reads x_H after it, as a code that owns the gas does every step.
* ``batch``    -- the same for many uneven instances in one engine.
* ``dust``     -- ``TransportEngine.dust_image``: the dust driver's photon loop.
* ``traverse`` -- ``TransportEngine.traverse_buffer``: one photon buffer through
  one subgrid, the drop-in for ``do_photon_traversal``.
* ``train``    -- ``UNet.gradients``: forward and backward pass of the warm-start
  network.
* ``predict``  -- ``warmstart.warm_start``: features, network and x_H into an
  engine, once per simulation start.
"""
import math
import os

import numpy as np
import torch

PC = 3.086e16
BOX = (-5.0 * PC, -5.0 * PC, -5.0 * PC, 10.0 * PC, 10.0 * PC, 10.0 * PC)
ALPHA, SIGMA = 4.0e-19, 6.3e-22
DEV = "cuda:0"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _iterate(ncell, nsub, packets, sources=4, sigma_ln=1.0, precision="mixed", reemission=0.0,
             coupled=False):
    nc = ncell if isinstance(ncell, tuple) else (ncell,) * 3
    ns = nsub if isinstance(nsub, tuple) else (nsub,) * 3
    return {"kind": "iterate", "nx": nc[0], "ny": nc[1], "nz": nc[2], "sx": ns[0], "sy": ns[1],
            "sz": ns[2], "packets": packets, "sources": sources, "sigma_ln": sigma_ln,
            "precision": precision, "reemission": reemission, "coupled": coupled}


def listed():
    cases = [
        # a first look at a set-up, a unit test, one small member of a parameter study:
        # launch latency is most of it
        ("small32", _iterate(32, 4, 20_000, sources=1)),
        # the reference's own Stromgren test: uniform gas, one central source
        ("stromgren64", _iterate(64, 8, 1_000_000, sources=1, sigma_ln=0.0)),
        # the benchmark workload: log-normal gas, 4 sources
        ("lognormal128", _iterate(128, 8, 10_000_000)),
        # a production-size run: 256^3 cells, strong contrast, 16 sources
        ("large256", _iterate(256, 16, 100_000_000, sources=16, sigma_ln=1.5)),
        # a parameter study in one engine: uneven sides, 1-4 sources, 5 packets per cell
        ("batch12", {"kind": "batch", "count": 12, "max_side": 96, "packets_per_cell": 5}),
        # the faster FP32 walk inside a hydro code: fields from and to the host each step,
        # sides that are no powers of two
        ("coupled_fp32", _iterate((96, 80, 112), 8, 4_000_000, precision="fp32", coupled=True)),
        # the reference's arithmetic throughout, for validation runs
        ("lognormal64_fp64", _iterate(64, 4, 1_000_000, precision="fp64")),
        # diffuse radiation: the reference's reemission probability
        ("reemission64", _iterate(64, 8, 1_000_000, sources=1, sigma_ln=0.0, reemission=0.364)),
        # the dust driver's scattering and peel-off image
        ("dust128", {"kind": "dust", "side": 128, "sub": 8, "packets": 4_000_000, "albedo": 0.5,
                     "npix": 101}),
        # a host code's own photon buffers (200 photons, the reference's buffer size)
        ("traverse200", {"kind": "traverse", "nx": 16, "ny": 16, "nz": 16, "photons": 200,
                         "entry": "INSIDE", "precision": "mixed"}),
        # training of the warm-start network at its training shape
        ("train64", {"kind": "train", "side": 64, "batch": 8}),
        # the warm start of one 64^3 run
        ("predict64", {"kind": "predict", "side": 64, "sources": 4}),
    ]
    return [dict(c, name=n) for n, c in cases]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: the transport iteration most often."""
    kind = rng.choice(["iterate"] * 6 + ["batch", "dust", "traverse", "train", "predict"])
    if kind == "iterate":
        precision = rng.choice(["mixed", "mixed", "mixed", "fp32", "fp64"])
        nsub = tuple(rng.randint(2, 12) for _ in range(3))
        side = tuple(rng.randint(6, 16) for _ in range(3))
        nc = tuple(a * b for a, b in zip(nsub, side))
        cells = nc[0] * nc[1] * nc[2]
        packets = min(_log_int(rng, 1e4, 2e7), 40 * cells) + rng.randint(0, 999)
        return _iterate(nc, nsub, packets, sources=rng.randint(1, 16),
                        sigma_ln=round(rng.uniform(0.0, 1.5), 3), precision=precision,
                        reemission=rng.choice([0.0, 0.0, 0.0, round(rng.uniform(0.1, 0.4), 3)]),
                        coupled=rng.random() < 0.25)
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(2, 24), "max_side": rng.choice([48, 64, 96]),
                "packets_per_cell": rng.randint(2, 8)}
    if kind == "dust":
        sub = rng.randint(2, 12)
        side = sub * rng.randint(5, 16)
        return {"kind": "dust", "side": side, "sub": sub, "packets": _log_int(rng, 1e4, 4e6),
                "albedo": round(rng.uniform(0.1, 0.9), 3), "npix": rng.randint(33, 257)}
    if kind == "traverse":
        return {"kind": "traverse", "nx": rng.randint(4, 16), "ny": rng.randint(4, 16),
                "nz": rng.randint(4, 16), "photons": _log_int(rng, 1, 20_000),
                "entry": rng.choice(["INSIDE", "FACE_X_N", "FACE_Z_P"]),
                "precision": rng.choice(["mixed", "fp64"])}
    if kind == "train":
        return {"kind": "train", "side": rng.choice([32, 64]), "batch": rng.randint(1, 8)}
    return {"kind": "predict", "side": rng.choice([32, 64, 96]), "sources": rng.randint(1, 8)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rng(seed, *more):
    return np.random.default_rng([int(seed), *more])


def _lognormal(ncell, sigma_ln, seed, mean=1.0e8, smoothing=4.0):
    """Cube of a log-normal density: Gaussian noise smoothed over 4 cells
    (periodic), unit variance, exp(mu + sigma g) with the given mean."""
    if sigma_ln == 0.0:
        return torch.full(tuple(ncell), mean, dtype=torch.float64, device=DEV)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    g = torch.randn(tuple(ncell), generator=gen, dtype=torch.float64, device=DEV)
    f = torch.fft.rfftn(g)
    k2 = 0
    for a, n in enumerate(ncell):
        k = (torch.fft.rfftfreq if a == 2 else torch.fft.fftfreq)(n, dtype=torch.float64,
                                                                  device=DEV)
        k2 = k2 + (k * k).reshape([-1 if b == a else 1 for b in range(3)])
    f *= torch.exp(-0.5 * (2 * math.pi * smoothing) ** 2 * k2)
    g = torch.fft.irfftn(f, s=tuple(ncell))
    g = (g - g.mean()) / g.std()
    return torch.exp(math.log(mean) - 0.5 * sigma_ln ** 2 + sigma_ln * g)


def _sources(count, rng):
    if count == 1:  # the reference's central source
        return [(0.0, 0.0, 0.0, 4.26e49)]
    box = np.asarray(BOX)
    pos = box[:3] + rng.uniform(size=(count, 3)) * box[3:]
    lum = 10.0 ** rng.uniform(48.0, 49.0, size=count)
    return [tuple(float(v) for v in p) + (float(l),) for p, l in zip(pos, lum)]


def _centres(ncell, box=BOX):
    return [(box[a] + (torch.arange(ncell[a], dtype=torch.float64, device=DEV) + 0.5)
             * (box[3 + a] / ncell[a])).reshape([-1 if b == a else 1 for b in range(3)])
            for a in range(3)]


def _near_balance(nH, sources, sigma_ln):
    """x_H as an iteration meets it some steps into a run: optically thin balance
    around each source out to its Stromgren radius (with the clumping of the
    log-normal gas), neutral beyond."""
    c = _centres(nH.shape)
    gamma = torch.zeros_like(nH)
    for s in sources:
        r2 = (c[0] - s[0]) ** 2 + (c[1] - s[1]) ** 2 + (c[2] - s[2]) ** 2
        rs = (3.0 * s[3] / (4.0 * math.pi * 1.0e16 * math.exp(sigma_ln ** 2) * ALPHA)) ** (1 / 3)
        r2 = r2.clamp_min((0.5 * BOX[3] / nH.shape[0]) ** 2)
        gamma += torch.where(r2 < rs * rs, s[3] * SIGMA / (4.0 * math.pi * r2), 0.0)
    return _balance(gamma, nH)


def _balance(gamma, nH):
    a = 0.5 * gamma / (nH * ALPHA)
    return torch.where(gamma > 0, 1.0 / (1.0 + a + torch.sqrt(a * (a + 2.0))), 1.0)


def _to_blocked(cube, nsub):
    n = cube.shape
    c = [n[a] // nsub[a] for a in range(3)]
    return (cube.reshape(nsub[0], c[0], nsub[1], c[1], nsub[2], c[2])
            .permute(0, 2, 4, 1, 3, 5).reshape(-1).contiguous())


class _DeviceArray:
    """A library field as a CUDA array (no copy).  It holds the engine, so that the
    memory lives as long as any tensor made from it."""

    def __init__(self, eng, address, count):
        self.eng = eng
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8",
                                         "data": (address, False), "version": 3}


def _field(eng, instance, which):
    """The library's own array of a field, subgrid after subgrid, without the
    padding at the end of each subgrid."""
    g = eng.grids[instance]
    address, count = eng.device_field(instance, which)
    nsub = int(np.prod(g.num_subgrid))
    t = torch.as_tensor(_DeviceArray(eng, address, count), device=DEV)
    return t.view(nsub, count // nsub)[:, : g.num_cells // nsub]


def _iterate_inputs(case, seed):
    ncell, nsub = (case["nx"], case["ny"], case["nz"]), (case["sx"], case["sy"], case["sz"])
    src = _sources(case["sources"], _rng(seed, 1))
    nH = _lognormal(ncell, case["sigma_ln"], seed)
    return ncell, nsub, src, nH, _near_balance(nH, src, case["sigma_ln"])


def _batch_inputs(case, seed):
    rng = _rng(seed, 2)
    sizes = _rng(1, case["count"])  # the work of a case does not depend on the seed
    sides = [s for s in (32, 48, 64, 96) if s <= case["max_side"]]
    out = []
    for i in range(case["count"]):
        side = int(sizes.choice(sides))
        s_ln = float(sizes.uniform(0.5, 1.5))
        nsrc = int(sizes.integers(2, 5))
        src = _sources(nsrc, rng)
        nH = _lognormal((side,) * 3, s_ln, seed * 1009 + i)
        out.append((side, src, nH, _near_balance(nH, src, s_ln)))
    return out


def _dust_inputs(case, seed):
    """The dust driver's unit sphere with clumps."""
    n = case["side"]
    c = _centres((n,) * 3, (-1.0, -1.0, -1.0, 2.0, 2.0, 2.0))
    r2 = c[0] ** 2 + c[1] ** 2 + c[2] ** 2
    return torch.where(r2 < 1.0, _lognormal((n,) * 3, 0.5, seed, mean=1.0), 0.0)


def _photons(case, seed):
    rng = _rng(seed, 3)
    n = case["photons"]
    cells = np.array([case["nx"], case["ny"], case["nz"]], dtype=np.float64)
    side = cells * (10.0 * PC / 128)
    pos = rng.uniform(size=(n, 3)) * side
    mu, phi = rng.uniform(-1, 1, n), rng.uniform(0, 2 * np.pi, n)
    d = np.stack([np.sqrt(1 - mu ** 2) * np.cos(phi), np.sqrt(1 - mu ** 2) * np.sin(phi), mu], 1)
    if case["entry"] == "FACE_X_N":
        pos[:, 0], d[:, 0] = 0.0, np.abs(d[:, 0])
    if case["entry"] == "FACE_Z_P":
        pos[:, 2], d[:, 2] = side[2], -np.abs(d[:, 2])
    nH = np.exp(rng.normal(math.log(1e8), 1.0, int(cells.prod())))
    xH = 10.0 ** rng.uniform(-5, -1, int(cells.prod()))
    return side, pos, d, rng.exponential(size=n), nH, xH


def _train_inputs(case, seed):
    n = case["side"]
    feats, target = [], []
    for b in range(case["batch"]):
        nH = _lognormal((n,) * 3, 1.0, seed * 17 + b)
        src = _sources(4, _rng(seed, 4, b))
        c = _centres(nH.shape)
        flux = sum(s[3] / (4 * math.pi * ((c[0] - s[0]) ** 2 + (c[1] - s[1]) ** 2
                                          + (c[2] - s[2]) ** 2)) for s in src)
        x = _near_balance(nH, src, 1.0)
        f = torch.stack([torch.log10(nH) - 8.0, (torch.log10(flux) - 13.0) / 1.5,
                         torch.log10(flux / nH) / 3.0 - 1.7], -1)
        feats.append(f.reshape(-1, 3).float())
        target.append(torch.log10(x).clamp_min(-8.0).reshape(-1).float())
    return torch.stack(feats).contiguous(), torch.stack(target).contiguous()


def _weights_file():
    return os.path.join("parallelcmacionize_b200", "weights", "warmstart_unet64.npz")


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    from parallelcmacionize_b200 import GridSpec, TransportEngine
    kind = case["kind"]
    if kind == "iterate":
        ncell, nsub, src, nH, x = _iterate_inputs(case, seed)
        eng = TransportEngine(
            GridSpec(box=BOX, ncell=ncell, num_subgrid=nsub, sources=src,
                     num_photon=case["packets"], reemission_probability=case["reemission"]),
            precision=case["precision"])
        n, x = _to_blocked(nH, nsub), _to_blocked(x, nsub)
        s = {"kind": kind, "eng": eng, "seed": seed, "coupled": case["coupled"]}
        if case["coupled"]:
            for k, v in (("n", n), ("x", x)):
                s["t" + k] = v.cpu().pin_memory()
                s[k] = s["t" + k].numpy()
        else:
            torch.cuda.synchronize()
            eng.set_fields_device(0, n.data_ptr(), x.data_ptr())
            s["x"] = _field(eng, 0, "x")
        return s
    if kind == "batch":
        specs, fields = [], []
        for side, src, nH, x in _batch_inputs(case, seed):
            ns = (side // 16,) * 3
            specs.append(GridSpec(box=BOX, ncell=(side,) * 3, num_subgrid=ns, sources=src,
                                  num_photon=case["packets_per_cell"] * side ** 3))
            fields.append((_to_blocked(nH, ns), _to_blocked(x, ns)))
        eng = TransportEngine(specs)
        torch.cuda.synchronize()
        for i, (n, x) in enumerate(fields):
            eng.set_fields_device(i, n.data_ptr(), x.data_ptr())
        return {"kind": kind, "eng": eng, "seed": seed,
                "x": [_field(eng, i, "x") for i in range(len(specs))]}
    if kind == "dust":
        nsub = (case["sub"],) * 3
        eng = TransportEngine(GridSpec(box=(-1.0, -1.0, -1.0, 2.0, 2.0, 2.0),
                                       ncell=(case["side"],) * 3, num_subgrid=nsub),
                              precision="fp64" if (case["side"] // case["sub"]) ** 3 <= 4096
                              else "mixed")
        n = _to_blocked(_dust_inputs(case, seed), nsub)
        x = torch.ones_like(n)
        torch.cuda.synchronize()
        eng.set_fields_device(0, n.data_ptr(), x.data_ptr())
        return {"kind": kind, "eng": eng, "seed": seed, "case": case}
    if kind == "traverse":
        from parallelcmacionize_b200 import PHOTON_DTYPE
        from parallelcmacionize_b200.engine import TravelDirection
        side, pos, d, tau, nH, xH = _photons(case, seed)
        eng = TransportEngine(GridSpec(box=(0.0, 0.0, 0.0) + tuple(float(v) for v in side),
                                       ncell=(case["nx"], case["ny"], case["nz"]),
                                       num_subgrid=(1, 1, 1)), precision=case["precision"])
        eng.set_fields(0, nH, xH)
        ph = np.zeros(case["photons"], PHOTON_DTYPE)
        ph["position"], ph["direction"], ph["tau"] = pos, d, tau
        ph["sigma"], ph["weight"] = SIGMA, 1.0
        return {"kind": kind, "eng": eng, "photons": ph, "entry": TravelDirection[case["entry"]],
                "J": _field(eng, 0, "J")}
    from parallelcmacionize_b200 import warmstart
    net = warmstart.UNet.load()
    if kind == "train":
        feats, target = _train_inputs(case, seed)
        return {"kind": kind, "net": net, "feats": feats, "target": target,
                "ncell": (case["side"],) * 3}
    n, src = (case["side"],) * 3, _sources(case["sources"], _rng(seed, 5))
    nH = _lognormal(n, 1.0, seed)
    eng = TransportEngine(GridSpec(box=BOX, ncell=n, num_subgrid=(case["side"] // 16,) * 3,
                                   sources=src))
    return {"kind": kind, "net": net, "eng": eng, "nH": nH.reshape(-1)}


def run(state):
    kind = state["kind"]
    if kind == "iterate":
        eng = state["eng"]
        if state["coupled"]:
            eng.set_fields(0, state["n"], state["x"])
            stats = eng.run_iterations(1, state["seed"])
            eng.get_fields(0, intensity=False, out_x=state["x"])
            return {"x": state["tx"], "stats": stats[0][0]}
        stats = eng.run_iterations(1, state["seed"])
        return {"x": state["x"], "stats": stats[0][0]}
    if kind == "batch":
        stats = state["eng"].run_iterations(1, state["seed"])[0]
        return {"x": state["x"],
                "stats": np.array([[s["packets_absorbed"], s["packets_escaped"],
                                    s["cell_crossings"], s["subgrid_transits"], s["rounds"]]
                                   for s in stats])}
    if kind == "dust":
        c = state["case"]
        image, stats = state["eng"].dust_image(0, c["packets"], c["albedo"],
                                               npix=(c["npix"], c["npix"]), seed=state["seed"])
        return {"image": image, "stats": stats}
    if kind == "traverse":
        out, counts, done = state["eng"].traverse_buffer(0, 0, state["entry"], state["photons"])
        return {"position": out["position"], "direction": out["direction"], "tau": out["tau"],
                "counts": counts, "done": done, "J": state["J"]}
    if kind == "train":
        loss, g = state["net"].gradients(state["feats"], state["target"], state["ncell"])
        return {"loss": loss, "gradients": g}
    from parallelcmacionize_b200 import warmstart
    return {"x": warmstart.warm_start(state["net"], state["eng"], 0, state["nH"])}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
# one crossing of a cell: 3 face distances, the smallest, 3 coordinates, the depth
CROSSING_FLOPS = 18.0


def _crossings(side, packets, sources, sigma_ln):
    """Cells crossed by the packets: the mean path inside a Stromgren sphere (3/4 of
    its radius, with the gas's clumping), 1.5 cells per cell side of path."""
    lum = 4.26e49 if sources == 1 else 5.0e48
    rs = (3.0 * lum / (4.0 * math.pi * 1.0e16 * math.exp(sigma_ln ** 2) * ALPHA)) ** (1 / 3)
    return packets * 1.125 * min(rs, 0.5 * BOX[3]) * side / BOX[3]


_LAYERS = [(3, 12, 1), (12, 12, 1), (12, 24, 8), (24, 24, 8), (24, 48, 64), (48, 48, 64),
           (72, 24, 8), (24, 24, 8), (36, 12, 1), (12, 12, 1)]  # c_in, c_out, 1 / voxel share


def work(case):
    kind = case["kind"]
    if kind == "iterate":
        cells = case["nx"] * case["ny"] * case["nz"]
        side = cells ** (1 / 3)
        k = _crossings(side, case["packets"], case["sources"], case["sigma_ln"])
        k /= 1.0 - case["reemission"]
        # n_H and x_H in, x_H out
        return {"bytes": 24.0 * cells, "flops": CROSSING_FLOPS * k}
    if kind == "batch":
        sizes = _rng(1, case["count"])
        sides = [s for s in (32, 48, 64, 96) if s <= case["max_side"]]
        cells = flops = 0.0
        for _ in range(case["count"]):
            side, s_ln, nsrc = int(sizes.choice(sides)), float(sizes.uniform(0.5, 1.5)), \
                int(sizes.integers(2, 5))
            cells += side ** 3
            flops += CROSSING_FLOPS * _crossings(side, case["packets_per_cell"] * side ** 3, nsrc,
                                                 s_ln)
        return {"bytes": 24.0 * cells, "flops": flops}
    if kind == "dust":
        # to the edge, to the scattering and per scattering a peel-off and the next walk
        walks = 1.6 + 1.0 * case["albedo"] / (1.0 - case["albedo"])
        return {"bytes": 16.0 * case["side"] ** 3 + 8.0 * case["npix"] ** 2,
                "flops": CROSSING_FLOPS * 0.7 * case["side"] * walks * case["packets"]}
    if kind == "traverse":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 160.0 * case["photons"] + 32.0 * cells,
                "flops": CROSSING_FLOPS * 8.0 * case["photons"]}
    voxels = float(case["side"] ** 3) * case.get("batch", 1)
    flops = sum(2.0 * 27 * ci * co * voxels / share for ci, co, share in _LAYERS)
    if kind == "train":
        return {"bytes": voxels * 16.0 + 8.0 * 199_513, "flops": 3.0 * flops}
    # and the midpoint sums along the rays, 2 samples per cell over half a side on average
    return {"bytes": voxels * 16.0, "flops": flops + voxels * case["sources"] * case["side"] * 10.0}


# ---------------------------------------------------------------------------
# exact: the same passes in 64 bits
# ---------------------------------------------------------------------------
_M32 = 0xFFFFFFFF


def _philox(c, k0, k1):
    """Philox4x32-10 (Salmon et al. 2011) of int64 tensors holding 32-bit words."""
    def mul(a, m):
        lo = (a & 0xFFFF) * m
        p = (a >> 16) * m + (lo >> 16)
        return p >> 16, ((p & 0xFFFF) << 16) | (lo & 0xFFFF)
    c0, c1, c2, c3 = c
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
        h0, l0 = mul(c0, 0xD2511F53)
        h1, l1 = mul(c2, 0xCD9E8D57)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
    return c0, c1, c2, c3


def _emitted(seed, instance, iteration, ids):
    """Direction and optical depth of the packets with these ids."""
    o = torch.zeros_like(ids)
    w = _philox((ids & _M32, ids >> 32, o + iteration, o + 0x434D4901), seed & _M32,
                ((seed >> 32) + instance) & _M32)
    u0, u1 = (w[0].double() + 0.5) / 2.0 ** 32, (w[1].double() + 0.5) / 2.0 ** 32
    u2 = ((w[2] * 2 ** 21 ^ (w[3] >> 11)).double() + 0.5) / 2.0 ** 53
    cost, phi = 2.0 * u0 - 1.0, 2.0 * math.pi * u1
    sint = torch.sqrt((1.0 - cost * cost).clamp_min(0.0))
    return torch.stack([sint * torch.cos(phi), sint * torch.sin(phi), cost]), -torch.log(u2)


def _split(seed, instance, iteration, lum, packets):
    """Packets per source: truncated shares, the rest to the smallest draws."""
    total = 0.0
    for l in lum:
        total += l
    n = [int(l / total * float(packets)) for l in lum]
    k = torch.arange(len(lum), dtype=torch.int64)
    z = torch.zeros_like(k)
    w = _philox((k, z, z + iteration, z + 0x434D4902), seed & _M32,
                ((seed >> 32) + instance) & _M32)[0].tolist()
    for i in sorted(range(len(lum)), key=lambda i: (w[i], i))[: packets - sum(n)]:
        n[i] += 1
    return n


def _walk(opacity, box, pos, d, target=None, tally=None, start=None):
    """Straight walks through a cube of cells until the target depth is used up or the
    packet leaves.  pos, d: [3, n]; returns (end positions, depth so far, absorbed,
    cell index at the end, [3, n]).  tally: flat array that receives the path lengths."""
    n3 = opacity.shape
    h = [box[3 + a] / n3[a] for a in range(3)]
    N = pos.shape[1]
    end, depth = pos.clone(), torch.zeros(N, dtype=torch.float64, device=pos.device)
    hit = torch.zeros(N, dtype=torch.bool, device=pos.device)
    if start is None:
        start = torch.stack([((pos[a] - box[a]) / h[a]).floor().long() for a in range(3)])
    last = start.clone()
    live = torch.arange(N, device=pos.device)
    p = torch.stack([pos[a] - box[a] for a in range(3)])
    v, idx, tau = d.clone(), start.clone(), depth.clone()
    goal = target
    flat = opacity.reshape(-1)
    hh = torch.tensor(h, dtype=torch.float64, device=pos.device).reshape(3, 1)
    for _ in range(2 * sum(n3) + 8):
        if live.numel() == 0:
            break
        cell = (idx[0] * n3[1] + idx[1]) * n3[2] + idx[2]
        face = (idx + (v > 0)).double() * hh
        l = torch.where(v != 0, (face - p) / v, math.inf)
        lm = l.min(0).values
        dt = lm * flat[cell]
        done = torch.zeros_like(lm, dtype=torch.bool)
        length = lm
        if goal is not None:
            done = tau + dt >= goal
            length = torch.where(done, lm * ((goal - tau) / dt).clamp(max=1.0), lm)
        if tally is not None:
            tally.index_add_(0, cell, length)
        tau = tau + dt
        cross = (l == lm) & ~done
        p = torch.where(cross, face, p + length * v)
        idx = idx + torch.where(cross, torch.sign(v).long(), 0)
        out = (idx[0] < 0) | (idx[0] >= n3[0]) | (idx[1] < 0) | (idx[1] >= n3[1]) | \
            (idx[2] < 0) | (idx[2] >= n3[2])
        stop = done | out
        if bool(stop.any()):
            w = live[stop]
            for a in range(3):
                end[a, w] = p[a, stop] + box[a]
            last[:, w], depth[w], hit[w] = idx[:, stop], tau[stop], done[stop]
            keep = ~stop
            live, p, v, idx, tau = live[keep], p[:, keep], v[:, keep], idx[:, keep], tau[keep]
            goal = goal[keep] if goal is not None else None
    return end, depth, hit, last


def _exact_x(nH, x, sources, packets, seed, instance=0):
    """x_H after one iteration of the packets of iteration 0."""
    lum = [s[3] for s in sources]
    opacity = SIGMA * nH * x
    J = torch.zeros(nH.numel(), dtype=torch.float64, device=nH.device)
    first = 0
    for s, n in zip(sources, _split(seed, instance, 0, lum, packets)):
        for at in range(0, n, 4_000_000):
            ids = torch.arange(first + at, first + min(n, at + 4_000_000), device=nH.device)
            d, tau = _emitted(seed, instance, 0, ids)
            pos = torch.tensor(s[:3], dtype=torch.float64, device=nH.device).reshape(3, 1)
            _walk(opacity, BOX, pos.expand(3, ids.numel()).contiguous(), d, tau, tally=J)
        first += n
    cells = [BOX[3 + a] / nH.shape[a] for a in range(3)]
    gamma = sum(lum) / packets * (J * SIGMA).reshape(nH.shape) / (cells[0] * cells[1] * cells[2])
    return _balance(gamma, nH)


def _by_subgrid(cube, nsub):
    return _to_blocked(cube, nsub).view(int(np.prod(nsub)), -1)


def _dust_draw(seed, ids, gen, purpose):
    """Isotropic direction (Marsaglia's rejection from the square), the first word's and the
    accepted attempt's last word's uniforms."""
    n = ids.numel()
    z = torch.zeros_like(ids)
    d = torch.zeros(3, n, dtype=torch.float64, device=ids.device)
    d[2] = 1.0
    u0 = u3 = None
    open_ = torch.ones(n, dtype=torch.bool, device=ids.device)
    for k in range(16):
        w = _philox((ids, gen, z, z + (0x44555354 + (purpose << 8) + k)), seed & _M32,
                    (seed >> 32) & _M32)
        u = [(q.double() + 0.5) / 2.0 ** 32 for q in w]
        if k == 0:
            u0, u3 = u[0], u[3].clone()
        x1, x2 = 2.0 * u[1] - 1.0, 2.0 * u[2] - 1.0
        s = x1 * x1 + x2 * x2
        ok = open_ & (s < 1.0)
        f = 2.0 * torch.sqrt((1.0 - s).clamp_min(0.0))
        d = torch.where(ok, torch.stack([x1 * f, x2 * f, 1.0 - 2.0 * s]), d)
        u3 = torch.where(ok, u[3], u3)
        open_ = open_ & ~ok
    return d, u0, u3


def _exact_dust(case, seed):
    box = (-1.0, -1.0, -1.0, 2.0, 2.0, 2.0)
    opacity = _dust_inputs(case, seed)
    npix, N = case["npix"], case["packets"]
    image = torch.zeros(npix * npix, dtype=torch.float64, device=DEV)
    ids = torch.arange(N, device=DEV)
    pos = torch.zeros(3, N, dtype=torch.float64, device=DEV)
    d, _, _ = _dust_draw(seed, ids, torch.zeros_like(ids), 0)
    _, tau0, _, _ = _walk(opacity, box, pos, d)
    weight = 1.0 - torch.exp(-tau0)
    z = torch.zeros_like(ids)
    w = _philox((ids, z, z, z + (0x44555354 + (1 << 8))), seed & _M32, (seed >> 32) & _M32)
    target = -torch.log(1.0 - (w[0].double() + 0.5) / 2.0 ** 32 * weight)
    gen = 0
    start = None
    while ids.numel():
        pos, _, hit, cell = _walk(opacity, box, pos, d, target, start=start)
        gen += 1
        ids, pos, weight, start = ids[hit], pos[:, hit], weight[hit], cell[:, hit]
        d, u0, u3 = _dust_draw(seed, ids, torch.zeros_like(ids) + gen, 2)
        sc = u0 < case["albedo"]
        ids, pos, d, weight, u3 = ids[sc], pos[:, sc], d[:, sc], weight[sc] / (4.0 * math.pi), \
            u3[sc]
        start, target = start[:, sc], -torch.log(u3)
        if not ids.numel():
            break
        up = torch.zeros_like(pos)
        up[2] = 1.0
        out, depth, _, _ = _walk(opacity, box, pos, up, start=start)
        px = [((out[a] + 1.0) / 2.0 * npix).floor().long().clamp(0, npix - 1) for a in range(2)]
        image.index_add_(0, px[0] * npix + px[1], weight * torch.exp(-depth))
    return {"image": (image / N).reshape(npix, npix), "stats": None}


# TravelDirection values by exit signs (x, y, z)
_DIRECTIONS = [(0, 0, 0)] + \
    [(a, b, c) for a in (1, -1) for b in (1, -1) for c in (1, -1)] + \
    [(0, b, c) for b in (1, -1) for c in (1, -1)] + \
    [(a, 0, c) for a in (1, -1) for c in (1, -1)] + \
    [(a, b, 0) for a in (1, -1) for b in (1, -1)] + \
    [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]


def _exact_traverse(case, seed):
    side, pos, d, tau, nH, xH = _photons(case, seed)
    n3 = (case["nx"], case["ny"], case["nz"])
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    opacity = to(nH * xH).reshape(n3) * SIGMA
    J = torch.zeros(nH.size, dtype=torch.float64, device=DEV)
    p, v, t = to(pos.T), to(d.T), to(tau)
    box = (0.0, 0.0, 0.0) + tuple(float(s) for s in side)
    start = torch.stack([(p[a] / (side[a] / n3[a])).floor().long().clamp(0, n3[a] - 1)
                         for a in range(3)])
    end, depth, hit, last = _walk(opacity, box, p, v, t, tally=J, start=start)
    sign = torch.stack([(last[a] >= n3[a]).long() - (last[a] < 0).long() for a in range(3)])
    table = torch.zeros(27, dtype=torch.long, device=DEV)
    for k, s in enumerate(_DIRECTIONS):
        table[(s[0] + 1) * 9 + (s[1] + 1) * 3 + s[2] + 1] = k
    out = table[(sign[0] + 1) * 9 + (sign[1] + 1) * 3 + sign[2] + 1]
    order = torch.argsort(out, stable=True)
    return {"position": end[:, order].T.contiguous(), "direction": v[:, order].T.contiguous(),
            "tau": (t - depth)[order], "counts": torch.bincount(out, minlength=27),
            "done": None, "J": (J * SIGMA).reshape(1, -1)}


def _network(params, feats, side, slope):
    """The U-Net in 64 bits: feats [B, cells, 3] -> prediction [B, cells]."""
    at = 0
    convs = []
    for ci, co, _ in _LAYERS:
        w = params[at: at + co * 27 * ci].reshape(co, 3, 3, 3, ci).permute(0, 4, 1, 2, 3)
        at += co * 27 * ci
        convs.append((w, params[at: at + co]))
        at += co
    hw, hb = params[at: at + 12], params[at + 12]
    F = torch.nn.functional

    def conv(x, i):
        # a matrix product per tap: no 64-bit convolution library is needed
        w, b = convs[i]
        xp = F.pad(x, (1, 1, 1, 1, 1, 1))
        Z, Y, X = x.shape[2:]
        y = b.reshape(1, -1, 1, 1, 1)
        for t in range(27):
            dz, dy, dx = t // 9, t // 3 % 3, t % 3
            y = y + torch.einsum("oc,bczyx->bozyx", w[:, :, dz, dy, dx],
                                 xp[:, :, dz:dz + Z, dy:dy + Y, dx:dx + X])
        return F.leaky_relu(y, slope)

    up = lambda x: F.interpolate(x, scale_factor=2, mode="nearest")  # noqa: E731
    B = feats.shape[0]
    x = feats.reshape(B, side, side, side, 3).permute(0, 4, 1, 2, 3)
    e1 = conv(conv(x, 0), 1)
    e2 = conv(conv(F.avg_pool3d(e1, 2), 2), 3)
    b = conv(conv(F.avg_pool3d(e2, 2), 4), 5)
    d2 = conv(conv(torch.cat([up(b), e2], 1), 6), 7)
    d1 = conv(conv(torch.cat([up(d2), e1], 1), 8), 9)
    return torch.einsum("c,bczyx->bzyx", hw, d1).reshape(B, -1) + hb


def _exact_train(case, seed):
    d = np.load(_weights_file())
    params = torch.from_numpy(d["params"]).to(DEV).double().requires_grad_()
    feats, target = _train_inputs(case, seed)
    loss, n = 0.0, feats.shape[0]
    for b in range(n):
        pred = _network(params, feats[b: b + 1].double(), case["side"], float(d["slope"]))
        part = ((pred - target[b: b + 1].double()) ** 2).mean() / n
        part.backward()
        loss += float(part)
    return {"loss": loss, "gradients": params.grad.float().double()}


def _exact_predict(case, seed):
    d = np.load(_weights_file())
    n, src = case["side"], _sources(case["sources"], _rng(seed, 5))
    if "ratio_factor" in d.files or n not in (32, 64, 96):
        return None
    nH = _lognormal((n,) * 3, 1.0, seed)
    h = BOX[3] / n
    c = _centres((n,) * 3)
    flux = ratio = 0.0
    for s in src:
        dm = torch.stack(torch.broadcast_tensors(*[c[a] - s[a] for a in range(3)]))
        r = torch.sqrt((dm ** 2).sum(0))
        flux = flux + s[3] / (4 * math.pi * r.clamp_min(0.5 * h) ** 2)
        steps = (r / h / 0.5).ceil().clamp_min(1.0)
        R = torch.zeros_like(r)
        for k in range(int(steps.max())):
            t = (k + 0.5) / steps
            i = [((s[a] - BOX[a] + t * dm[a]) / h).floor().long().clamp(0, n - 1)
                 for a in range(3)]
            R += torch.where(k < steps, nH[i[0], i[1], i[2]] ** 2 * (t * r) ** 2 * r / steps, 0.0)
        ratio = ratio + s[3] / (4 * math.pi * ALPHA * R.clamp_min(1e-300))
    f = torch.stack([torch.log10(nH), torch.log10(flux),
                     torch.log10(ratio.clamp(1e-30, 1e30))], -1).reshape(1, -1, 3)
    norm = torch.from_numpy(d["norm"].astype(np.float64)).to(DEV)
    params = torch.from_numpy(d["params"]).to(DEV).double()
    with torch.no_grad():
        pred = _network(params, (f - norm[0::2]) / norm[1::2], n, float(d["slope"]))
    return {"x": (10.0 ** pred.clamp(-8.0, 0.0)).reshape(-1)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "iterate":
        # reemission draws hang on the bits of the absorption points; above 2e7 packets the
        # plain walk takes too long
        if case["reemission"] or case["packets"] > 20_000_000:
            return None
        ncell, nsub, src, nH, x = _iterate_inputs(case, seed)
        x = _by_subgrid(_exact_x(nH, x, src, case["packets"], seed), nsub)
        return {"x": x.reshape(-1).cpu() if case["coupled"] else x, "stats": None}
    if kind == "batch":
        out = []
        for i, (side, src, nH, x) in enumerate(_batch_inputs(case, seed)):
            out.append(_by_subgrid(_exact_x(nH, x, src, case["packets_per_cell"] * side ** 3,
                                            seed, i), (side // 16,) * 3))
        return {"x": out, "stats": None}
    return {"dust": _exact_dust, "traverse": _exact_traverse, "train": _exact_train,
            "predict": _exact_predict}[kind](case, seed)
