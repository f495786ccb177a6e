"""The work that a user of the propagator has it do, as cases to be timed.

Each case is one call pattern of the public interface on inputs made from a
seed:

* ``steps``   -- ``Simulation.run`` on a box that is full of waves: the time
                 loop, with each medium storage (FP32, FP16, BF16, vpz/vsv),
                 equal or unequal spacing, with and without a sponge, with
                 the fast or the exact kernel.
* ``shot``    -- a whole short shot: fields cleared, steps with a source, a
                 sponge, receivers and the energy log, traces read back.
* ``abi``     -- the reference's own time loop: ``dc_device_add_source``,
                 seven ``dc_propagate`` boxes and ``dc_device_swap_arrays``
                 per step.
* ``batch``   -- uneven shots cropped out of one shared medium, advanced
                 together, with the 48-cell sponge or the learned layer.
* ``learned`` -- one box with the learned 8-cell absorbing layer.
* ``train``   -- Adam steps of the learned layer's network on samples.

Wavefields come back as views of the device buffers that
``dc_device_data`` points at.
"""
from __future__ import annotations

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
PKG = ROOT / "distributed-cube-average_gb300"

DX, DT = 12.5, 0.8e-3          # the benchmark's spacing and time step
KAPPA, LAYER = 0.35, 8         # its sponge strength and learned-layer width
FEATURES = (12, 6, 6)          # random Fourier features of the medium fields
NLAYERS = 12
HALO = 4
K2 = (-205.0 / 72.0, 8.0 / 5.0, -1.0 / 5.0, 8.0 / 315.0, -1.0 / 560.0)
L1 = (4.0 / 5.0, -1.0 / 5.0, 4.0 / 105.0, -1.0 / 280.0)
MEDIUM_BYTES = {"f32": 40, "f16": 20, "bf16": 20, "vv": 8}
FLOPS = 220                    # per updated point, both fields
PRE_STEPS = {0: 96, LAYER: 320}  # steps a batch has run before (waves in the layer)


def _dc():
    """The package (its folder's name is no Python identifier)."""
    if "dc_gb300" not in sys.modules:
        spec = importlib.util.spec_from_file_location("dc_gb300", PKG / "__init__.py",
                                                      submodule_search_locations=[str(PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["dc_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["dc_gb300"]


# ---------------------------------------------------------------------------
# cases

def listed():
    def steps(name, sizes, n, form="f32", absorb=0, kernel="fast", dy=DX, dz=DX):
        return {"name": name, "kind": "steps", "sx": sizes[0], "sy": sizes[1], "sz": sizes[2],
                "steps": n, "form": form, "absorb": absorb, "kernel": kernel, "dy": dy, "dz": dz}

    return [
        # the smallest workload: one short shot on 64^3 + a 16-cell sponge,
        # 64 receivers, the whole call from cleared fields to traces
        {"name": "shot_64", "kind": "shot", "sx": 104, "sy": 104, "sz": 104, "steps": 96,
         "absorb": 16, "receivers": 64, "energy": False, "dy": DX, "dz": DX},
        # a mid-size shot on an odd-sized box with unequal spacing and energy
        {"name": "shot_ragged", "kind": "shot", "sx": 201, "sy": 157, "sz": 183, "steps": 64,
         "absorb": 24, "receivers": 200, "energy": True, "dy": 10.0, "dz": 8.0},
        # the headline workload: 512^3 + a 48-cell sponge, FP32 medium
        steps("plain_616", (616, 616, 616), 20, absorb=48),
        # a box of ordinary size, odd extents
        steps("plain_300", (307, 291, 299), 48, absorb=48),
        # mixed precision at scale: FP16 medium, 768 x 768 x 512 + sponge
        steps("fp16_872", (872, 872, 616), 8, form="f16", absorb=48),
        # the other 16-bit medium, on an ordinary box without a sponge
        steps("bf16_240", (240, 222, 251), 48, form="bf16"),
        # the medium of the reference's GPU backend (vpz, vsv)
        steps("vv_408", (408, 408, 408), 32, form="vv"),
        # bit-exact runs: the parity kernel
        steps("exact_168", (168, 168, 152), 8, kernel="exact"),
        # the reference's own host loop linked against the library
        {"name": "abi_216", "kind": "abi", "sx": 216, "sy": 208, "sz": 200, "steps": 24},
        # shots over one shared medium, FP16 storage, 48-cell sponge
        {"name": "batch_fp16", "kind": "batch", "mx": 424, "my": 424, "mz": 268, "shots": 8,
         "lo": 96, "hi": 160, "depth": 128, "form": "f16", "layer": 0, "steps": 32,
         "receivers": 512, "fields": 0},
        # the same with the learned layer in the sponge's place
        {"name": "batch_learned", "kind": "batch", "mx": 424, "my": 424, "mz": 268, "shots": 12,
         "lo": 120, "hi": 200, "depth": 160, "form": "f16", "layer": LAYER, "steps": 32,
         "receivers": 512, "fields": 0},
        # the network's training
        {"name": "train", "kind": "train", "samples": 400000, "batch": 8192, "steps": 24},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sizes(rng, lo, hi):
    """Padded sizes with about log-uniform volume in [lo, hi]."""
    v = _log(rng, lo, hi)
    a, b = _log(rng, 0.7, 1.4), _log(rng, 0.7, 1.4)
    c = v ** (1.0 / 3.0)
    return [max(40, int(round(t))) for t in (c * a, c * b, c / (a * b))]


def draw(rng):
    kind = rng.choice(["steps"] * 8 + ["shot"] * 2 + ["abi", "batch", "batch", "learned", "train"])
    if kind == "train":
        return {"kind": kind, "samples": int(_log(rng, 2e4, 1e6)),
                "batch": int(_log(rng, 1000, 16384)), "steps": rng.randint(8, 48)}
    if kind == "batch":
        layer = rng.choice([0, LAYER])
        lo = rng.randint(56, 120)
        hi = rng.randint(lo + 1, 170)
        mx, my = rng.randint(hi + 120, 430), rng.randint(hi + 120, 430)
        return {"kind": kind, "mx": mx, "my": my, "mz": rng.randint(230, 270),
                "shots": rng.randint(2, 10), "lo": lo, "hi": hi, "depth": rng.randint(48, 120),
                "form": rng.choice(["f16", "f16", "f32", "bf16"]), "layer": layer,
                "steps": rng.randint(16, 48), "receivers": rng.randint(32, 512),
                "fields": rng.choice([0, 0, 1])}
    form = rng.choice(["f32", "f32", "f16", "f16", "bf16", "vv"])
    kernel = "exact" if kind == "steps" and form in ("f32", "vv") and rng.random() < 0.15 else "fast"
    top = {"abi": 4e7, "learned": 6e7, "shot": 3e7}.get(kind, 1e7 if kernel == "exact" else 2e8)
    sx, sy, sz = _sizes(rng, 8e4, top)
    n = max(4, min(96, int(2e9 / (sx * sy * sz))))
    n = max(2, n // 6) if kernel == "exact" else n
    case = {"kind": kind, "sx": sx, "sy": sy, "sz": sz, "steps": n}
    if kind in ("abi", "learned"):
        return case
    even = rng.random() < 0.7
    case["dy"], case["dz"] = (DX, DX) if even else (10.0, 8.0)
    most = (min(sx, sy, sz) - 2 * HALO - 8) // 2
    if kind == "shot":
        return dict(case, steps=min(n, 64), absorb=min(most, rng.randint(8, 48)),
                    receivers=rng.randint(1, 600), energy=rng.random() < 0.5)
    return dict(case, form=form, kernel=kernel,
                absorb=0 if rng.random() < 0.3 else min(most, rng.randint(8, 48)))


def _pts(sizes):
    return math.prod(s - 2 * HALO for s in sizes)


def work(case):
    if case["kind"] == "train":
        n = case["batch"] * case["steps"]
        return {"bytes": n * 35 * 4, "flops": n * 6 * (32 * 32 + 32 * 32 + 32 * 2)}
    if case["kind"] == "batch":
        pts = sum(_pts(s["sizes"]) for s in _shots(case, 1))
    else:
        pts = _pts((case["sx"], case["sy"], case["sz"]))
    # per update: (pc, qc) and (pp, qp) read, (pp, qp) written, the medium
    per = 24 + MEDIUM_BYTES[case.get("form", "f32")]
    return {"bytes": pts * case["steps"] * per, "flops": pts * case["steps"] * FLOPS}


# ---------------------------------------------------------------------------
# inputs

def _gen(seed):
    return np.random.Generator(np.random.PCG64(seed))


def _medium(seed, depth):
    """A layered medium's random parameters (12 layers, velocity increasing
    with depth, smooth angle fields), as drawn for the benchmark but with
    fewer Fourier features."""
    rng = _gen(seed)

    def rff(m, sigma):
        k = rng.normal(0.0, 1.0 / (sigma * math.sqrt(2.0)), size=(m, 3))
        return np.concatenate([k, rng.uniform(0.0, 2.0 * math.pi, size=(m, 1))], 1).astype(np.float32)

    eps = rng.uniform(0.0, 0.3, NLAYERS).astype(np.float32)
    return {"top": (np.arange(NLAYERS) * float(depth) / NLAYERS).astype(np.float32),
            "vp": np.sort(rng.uniform(1500.0, 4500.0, NLAYERS)).astype(np.float32),
            "eps": eps, "delta": (rng.uniform(0.0, 1.0, NLAYERS) * eps).astype(np.float32),
            "noise": rff(FEATURES[0], 2.0), "theta": rff(FEATURES[1], 20.0),
            "phi": rff(FEATURES[2], 20.0), "vp_noise": np.float32(0.02),
            "theta_range": np.float32([-math.pi / 3, math.pi / 3]),
            "phi_range": np.float32([0.0, 2.0 * math.pi])}


def _spec(m):
    """The library's struct of a medium's parameters."""
    s = _dc().LayeredSpec()
    s.nlayers = NLAYERS
    for l in range(NLAYERS):
        s.layer_top[l], s.vp[l] = m["top"][l], m["vp"][l]
        s.epsilon[l], s.delta[l] = m["eps"][l], m["delta"][l]
    s.vp_noise, s.sigma_ratio = m["vp_noise"], 0.75
    s.theta_lo, s.theta_hi = m["theta_range"]
    s.phi_lo, s.phi_hi = m["phi_range"]
    s.n_noise, s.n_theta, s.n_phi = FEATURES
    for name, dst in (("noise", s.k_noise), ("theta", s.k_theta), ("phi", s.k_phi)):
        for j, row in enumerate(m[name]):
            for c in range(4):
                dst[j][c] = row[c]
    return s


def _vv(seed, sizes):
    """(vpz, vsv): velocity growing with depth, rough at the rim, as the
    reference's medium with its random boundary is."""
    g = torch.Generator("cuda").manual_seed(seed)
    shape = (sizes[2], sizes[1], sizes[0])
    z = torch.linspace(0.0, 1.0, sizes[2], device="cuda")[:, None, None]
    r = torch.rand(shape, generator=g, device="cuda")
    vpz = (2000.0 + 1500.0 * z) * (1.0 - 0.05 * r)
    return vpz.float(), (vpz * 0.4).float()


def _waves(seed, sizes):
    """(pp, pc, qp, qc) of a box full of plane waves, about ten cells long,
    zero in the halo."""
    rng = _gen(seed + 7)
    sx, sy, sz = sizes
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) for n in (sz, sy, sx)]
    out = [torch.zeros((sz, sy, sx), device="cuda") for _ in range(4)]
    for _ in range(4):
        k = rng.normal(size=3)
        k *= 2.0 * math.pi / rng.uniform(8.0, 16.0) / np.linalg.norm(k)
        a, ph, w = rng.uniform(0.5, 1.0), rng.uniform(0.0, 6.28), np.linalg.norm(k) * 0.2
        arg = (k[0] * ax[0])[:, None, None] + (k[1] * ax[1])[None, :, None] + (k[2] * ax[2])[None, None, :]
        now, before = a * torch.sin(arg + ph), a * torch.sin(arg + (ph - w))
        for f, v, s in zip(out, (before, now, before, now), (1.0, 1.0, 0.9, 0.9)):
            f.add_(v, alpha=s)
        del arg, now, before
    for f in out:
        for d in range(3):
            f.narrow(d, 0, HALO).zero_()
            f.narrow(d, f.shape[d] - HALO, HALO).zero_()
    return out


def _sponge(n, absorb):
    return _dc().sponge_profile(n, absorb, KAPPA)


def _ricker(seed, count):
    """A band-limited source wavelet that starts at once."""
    rng = _gen(seed + 3)
    t = np.arange(count) * DT
    f = rng.uniform(15.0, 25.0, 3)
    return (10.0 * sum(np.sin(2 * math.pi * v * t + i) for i, v in enumerate(f))).astype(np.float32)


def _receivers(seed, sizes, count):
    """Receiver positions (x, y, z) all over the updated box."""
    rng = _gen(seed + 5)
    return np.stack([rng.integers(HALO, s - HALO, count) for s in sizes], 1).astype(np.int64)


def _index(sizes, xyz):
    x, y, z = (np.asarray(xyz)[..., c] for c in range(3))
    return x + y * sizes[0] + z * sizes[0] * sizes[1]


def _shots(case, seed):
    """Uneven crops around sources spread over the medium; the layout
    belongs to the case, the sources to the seed."""
    rng, jit = _gen(case["mx"] * 31 + case["my"]), _gen(seed + 11)
    pad = HALO + (case["layer"] or 48)
    out = []
    for _ in range(case["shots"]):
        inner = [int(v) for v in rng.integers(case["lo"], case["hi"] + 1, 2)] + [case["depth"]]
        sizes = [v + 2 * pad for v in inner]
        origin = [int(rng.integers(0, max(1, m - s + 1))) for m, s in
                  zip((case["mx"], case["my"], case["mz"]), sizes)]
        origin[0] = origin[0] // 4 * 4
        src = [pad + int(jit.integers(8, v - 8)) for v in inner]
        out.append({"sizes": sizes, "origin": origin, "src": src,
                    "fcut": float(jit.uniform(45.0, 75.0))})
    return out


class _Buffer:
    """Device memory of a state, which it keeps alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4",
                                         "version": 2}


def _view(dc, state, data, sizes, pitch):
    """The current and previous (p, q) fields on the device, shape
    (sz, sy, sx, 2)."""
    v = dc.device_view(data)
    shape = (sizes[2], sizes[1], pitch, 2)
    return [torch.as_tensor(_Buffer(dc.C.cast(p, dc.C.c_void_p).value, shape, state),
                            device="cuda")[:, :, :sizes[0]] for p in (v.pc, v.pp)]


FORMS = {"f32": "MEDIUM_PRECOMP", "f16": "MEDIUM_PRECOMP_F16", "bf16": "MEDIUM_PRECOMP_BF16",
         "vv": "MEDIUM_VPZ_VSV"}


def _coef(m, sizes, origin=(0, 0, 0)):
    """The ten coefficients (float64 holding what the medium generator
    rounds to float32) of a box, dc_precomp_vars order."""
    dev = {"device": "cuda", "dtype": torch.float64}
    sx, sy, sz = sizes
    gx, gy, gz = (torch.arange(n, **dev) + o for n, o in zip(sizes, origin))
    top = torch.tensor(m["top"], **dev)
    layer = (torch.searchsorted(top, gz, right=True) - 1).clamp(0, NLAYERS - 1)

    def field(feat):
        s = torch.zeros((sz, sy, sx), **dev)
        for k in feat.astype(np.float64):
            s += torch.cos((k[0] * gx + k[3])[None, None, :] + (k[1] * gy)[None, :, None] +
                           (k[2] * gz)[:, None, None])
        return s * math.sqrt(2.0 / feat.shape[0])

    def f32(v):
        return v.to(torch.float32).to(torch.float64)

    def per_layer(name):
        return torch.tensor(m[name], **dev)[layer][:, None, None]

    def angle(name):
        lo, hi = (float(v) for v in m[name + "_range"])
        u = 0.5 * torch.erfc(field(m[name]) * -math.sqrt(0.5))
        return f32(lo + (hi - lo) * u)

    vp = f32(per_layer("vp") * (1.0 + float(m["vp_noise"]) * field(m["noise"])))
    eps, delta = per_layer("eps"), per_layer("delta")
    vs = f32(vp * f32(torch.sqrt(f32(f32(eps - delta).abs() / 0.75))))
    th, ph = angle("theta"), angle("phi")
    return _precomp(th, ph, vp, vs, eps, delta)


def _precomp(th, ph, vp, vs, eps, delta):
    def f32(v):
        return v.to(torch.float32).to(torch.float64)

    st, ct, s2t = f32(torch.sin(th)), f32(torch.cos(th)), f32(torch.sin(2 * th))
    sp, cp, s2p = f32(torch.sin(ph)), f32(torch.cos(ph)), f32(torch.sin(2 * ph))
    v2pz = f32(vp * vp)
    return [f32(st * st * cp * cp), f32(st * st * sp * sp), f32(ct * ct), f32(st * st * s2p),
            f32(s2t * sp), f32(s2t * cp), f32(v2pz * (1 + 2 * eps)), v2pz, f32(vs * vs),
            f32(v2pz * (1 + 2 * delta))]


def _vv_coef(seed, sizes):
    vpz, vsv = (v.double() for v in _vv(seed, sizes))
    one = torch.ones((1, 1, 1), device="cuda", dtype=torch.float64)
    c = [0.1459632909, 0.3540367091, 0.5, 0.4546487134, 0.8414709848, 0.5403023059]
    return [one * v for v in c] + [vpz * vpz * 1.48, vpz * vpz, vsv * vsv, vpz * vpz * 1.2]


def prepare(case, seed):
    dc = _dc()
    kind = case["kind"]
    if kind == "train":
        g = torch.Generator("cuda").manual_seed(seed)
        n = case["samples"]
        w = torch.arange(8, device="cuda") * 0.6
        ph = 6.28 * torch.rand((n, 4, 1), generator=g, device="cuda")
        amp = torch.exp(torch.randn((n, 1, 1), generator=g, device="cuda"))
        x = (amp * torch.sin(ph + w)).reshape(n, 32)
        depth = torch.randint(4, 8, (n, 1), generator=g, device="cuda").float()
        xs = torch.cat([x, depth], 1).contiguous()
        ts = (0.2 * x[:, 0:16:8] - 0.1 * x[:, 1:17:8] * depth / 8.0).contiguous()
        mlp = dc.MLP(seed=seed % 10007)
        torch.cuda.synchronize()
        return {"case": case, "mlp": mlp, "xs": xs, "ts": ts, "seed": seed}
    if kind == "batch":
        box = (case["mx"], case["my"], case["mz"])
        b = dc.Batch(box, (DX,) * 3, DT, medium=getattr(dc, FORMS[case["form"]]), max_steps=100000)
        b.generate_layered(_spec(_medium(seed, box[2])))
        for k, sh in enumerate(_shots(case, seed)):
            b.add_shot(sh["sizes"], sh["origin"], sh["src"], sh["fcut"],
                       0 if case["layer"] else 48, 0.0 if case["layer"] else KAPPA)
            b.set_receivers(k, _receivers(seed + k, sh["sizes"], case["receivers"]))
        b.autotune(3)
        state = {"case": case, "batch": b}
        if case["layer"]:
            state["mlp"] = dc.MLP(params=np.load(PKG / "data" / "learned_layer8.npy"))
            b.set_learned_layer(state["mlp"], case["layer"])
        b.run(PRE_STEPS[case["layer"]])
        b.synchronize()
        return state
    sizes = (case["sx"], case["sy"], case["sz"])
    d = (DX, case.get("dy", DX), case.get("dz", DX))
    if kind == "abi":
        coef = [c.expand(sizes[::-1]).float().cpu().numpy() for c in
                _coef(_medium(seed, sizes[2]), sizes)]
        pp, pc, qp, qc = (f.cpu().numpy() for f in _waves(seed, sizes))
        proc = dc.Process(sizes, d, DT, pp=pp, pc=pc, qp=qp, qc=qc, precomp=coef)
        data = dc.device_data_init(proc)
        sx, sy, sz = sizes
        r = HALO
        boxes = [((r if s == 0 else sx - 2 * r, r, r), (2 * r if s == 0 else sx - r, sy - r, sz - r))
                 for s in range(2)]
        boxes += [((2 * r, r if s == 0 else sy - 2 * r, r),
                   (sx - 2 * r, 2 * r if s == 0 else sy - r, sz - r)) for s in range(2)]
        boxes += [((2 * r, 2 * r, r if s == 0 else sz - 2 * r),
                   (sx - 2 * r, sy - 2 * r, 2 * r if s == 0 else sz - r)) for s in range(2)]
        boxes.append(((2 * r,) * 3, (sx - 2 * r, sy - 2 * r, sz - 2 * r)))
        pitch = int(dc.lib().dc_gb300_device_pitch(dc.lib().dc_gb300_from_device_data(data)))
        return _Abi({"case": case, "proc": proc, "data": data, "boxes": boxes, "pitch": pitch,
                     "src": [float(v) for v in _ricker(seed, case["steps"])],
                     "at": int(_index(sizes, [s // 2 for s in sizes]))})
    form = case.get("form", "f32")
    exact_kernel = case.get("kernel") == "exact"
    sim = dc.Simulation(sizes, d, DT, kernel=dc.KERNEL_EXACT if exact_kernel else dc.KERNEL_FAST,
                        medium=getattr(dc, FORMS[form]))
    if form == "vv":
        sim.set_vpz_vsv(*(v.cpu().numpy() for v in _vv(seed, sizes)))
    else:
        sim.generate_layered(_spec(_medium(seed, sizes[2])))
    if case.get("absorb"):
        sim.set_sponge(*(_sponge(n, case["absorb"]) for n in sizes))
    state = {"case": case, "sim": sim}
    if kind == "shot":
        sim.set_source(int(_index(sizes, [s // 2 for s in sizes])), _ricker(seed, case["steps"] + 8))
        sim.set_receivers(_index(sizes, _receivers(seed, sizes, case["receivers"])), case["steps"])
        if case["energy"]:
            sim.enable_energy(case["steps"])
        return state
    sim.set_fields(*(f.cpu().numpy() for f in _waves(seed, sizes)))
    if kind == "learned":
        state["mlp"] = dc.MLP(params=np.load(PKG / "data" / "learned_layer8.npy"))
        dc.set_learned_layer(sim, state["mlp"], LAYER)
    else:
        sim.set_source(int(_index(sizes, [s // 2 for s in sizes])), _ricker(seed, 4000))
    return state


class _Abi(dict):
    """A state whose device data ends with it."""

    def __del__(self):
        _dc().device_data_free(self["data"])


# ---------------------------------------------------------------------------
# one pass

def run(state):
    dc = _dc()
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        loss = state["mlp"].train(state["xs"].data_ptr(), state["ts"].data_ptr(),
                                  case["samples"], case["steps"], case["batch"], 2e-3,
                                  state["seed"])
        return {"loss": loss, "params": state["mlp"].params()}
    if kind == "batch":
        b = state["batch"]
        b.run(case["steps"])
        done = b.steps_done
        out = {"traces": [b.traces(k, done) for k in range(case["shots"])]}
        if case["fields"]:
            out["fields"] = [b.get_fields(k) for k in range(case["fields"])]
        return out
    sizes = (case["sx"], case["sy"], case["sz"])
    if kind == "abi":
        data = state["data"]
        for s in state["src"]:
            dc.device_add_source(data, state["at"], s)
            for b0, b1 in state["boxes"]:
                dc.propagate(b0, b1, sizes, data, DX, DX, DX, DT)
            dc.device_swap_arrays(data)
        return _view(dc, state, data, sizes, state["pitch"])
    sim = state["sim"]
    if kind == "shot":
        sim.set_fields()
        sim.run(case["steps"])
        out = {"traces": sim.traces(case["steps"])}
        if case["energy"]:
            out["energy"] = sim.energy(case["steps"])
        return dict(out, fields=_view(dc, state, sim.device_data, sizes, sim.pitch))
    sim.run(case["steps"])
    return _view(dc, state, sim.device_data, sizes, sim.pitch)


# ---------------------------------------------------------------------------
# the same in 64 bits

def _taps(u, axis, weights, odd):
    """8th-order central difference along `axis`, over the points with four
    neighbours on both sides."""
    n = u.shape[axis] - 2 * HALO
    out = u.narrow(axis, HALO, n) * (0.0 if odd else K2[0])
    for j, w in enumerate(weights, 1):
        out.add_(u.narrow(axis, HALO + j, n), alpha=w)
        out.add_(u.narrow(axis, HALO - j, n), alpha=-w if odd else w)
    return out


def _inner(u, axes):
    for a in axes:
        u = u.narrow(a, HALO, u.shape[a] - 2 * HALO)
    return u


def _h(u, c, d):
    """(H1, Laplacian) of one field; c: the six angle terms, interior."""
    dx, dy, dz = d
    xx = _inner(_taps(u, 2, K2[1:], False), (0, 1)) / dx ** 2
    h1, lap = c[0] * xx, xx
    yy = _inner(_taps(u, 1, K2[1:], False), (0, 2)) / dy ** 2
    h1 += c[1] * yy
    lap += yy
    del xx, yy
    zz = _inner(_taps(u, 0, K2[1:], False), (1, 2)) / dz ** 2
    h1 += c[2] * zz
    lap += zz
    del zz
    uy = _taps(u, 1, L1, True)
    h1 += c[3] * (_inner(_taps(uy, 2, L1, True), (0,)) / (dx * dy))
    h1 += c[4] * (_inner(_taps(uy, 0, L1, True), (2,)) / (dy * dz))
    del uy
    h1 += c[5] * (_inner(_taps(_taps(u, 2, L1, True), 0, L1, True), (1,)) / (dx * dz))
    return h1, lap


def _loop64(cur, prev, coef, d, steps, sponge=None, at=None, src=None, late=True, rec=None,
            energy=None):
    """The time loop of the reference in float64.  `cur`, `prev`: [p, q].
    src[it] is added before step it, and src[steps] after the last one where
    `late` (the library adds the next amplitude with the store).  Returns
    the fields and the traces."""
    c = [_inner(v, (0, 1, 2)) if v.numel() > 1 else v for v in coef]
    dt2 = float(np.float32(DT)) ** 2
    traces = []
    for it in range(steps):
        if at is not None and it < len(src):
            for f in cur:
                f.view(-1)[at] += float(src[it])
        h1p, lp = _h(cur[0], c[:6], d)
        h1q, lq = _h(cur[1], c[:6], d)
        h2p, h2q = lp - h1p, lq - h1q
        del lp, lq
        rhs = [c[6] * h2p + c[7] * h1q + c[8] * (h1p - h1q),
               c[9] * h2p + c[7] * h1q - c[8] * (h2p - h2q)]
        del h1p, h1q, h2p, h2q
        for f, o, r in zip(cur, prev, rhs):
            inner = _inner(o, (0, 1, 2))
            if sponge is None:
                inner.neg_()
                inner.add_(_inner(f, (0, 1, 2)), alpha=2.0).add_(r, alpha=dt2)
            else:
                inner.mul_(sponge).neg_()
                inner.add_(_inner(f, (0, 1, 2)), alpha=2.0).add_(r, alpha=dt2).mul_(sponge)
        cur, prev = prev, cur
        if rec is not None:
            traces.append(cur[0].view(-1)[rec].clone())
        if energy is not None:
            energy.append(float(sum(_inner(f, (0, 1, 2)).square().sum() for f in cur)))
    if late and at is not None and steps < len(src):
        for f in cur:
            f.view(-1)[at] += float(src[steps])
    return cur, prev, traces


def _sponge64(sizes, absorb):
    """exp(-(kappa d / a)^2) for d cells into the shell, per axis (float32
    profiles), multiplied."""
    g = []
    for n in sizes:
        i = np.arange(n)
        dist = np.maximum(np.maximum(HALO + absorb - i, i - (n - 1 - HALO - absorb)), 0)
        dist = np.minimum(dist, absorb)
        v = np.exp(-(KAPPA * dist / absorb) ** 2).astype(np.float32)
        g.append(torch.tensor(v[HALO:n - HALO], device="cuda", dtype=torch.float64))
    return g[2][:, None, None] * g[1][None, :, None] * g[0][None, None, :]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "learned") or (kind == "batch" and case["layer"]):
        return None  # a BF16 network with the hardware's tanh has no 64-bit value
    if kind == "batch":
        return _exact_batch(case, seed)
    sizes = (case["sx"], case["sy"], case["sz"])
    d = (DX, case.get("dy", DX), case.get("dz", DX))
    if case.get("form") == "vv":
        coef = _vv_coef(seed, sizes)
    else:
        coef = _coef(_medium(seed, sizes[2]), sizes)
    absorb = case.get("absorb")
    sponge = _sponge64(sizes, absorb) if absorb else None
    at = int(_index(sizes, [s // 2 for s in sizes]))
    rec = None
    energy = [] if case.get("energy") else None
    if kind == "shot":
        shape = sizes[::-1]
        cur, prev = ([torch.zeros(shape, device="cuda", dtype=torch.float64) for _ in range(2)]
                     for _ in range(2))
        src = _ricker(seed, case["steps"] + 8)
        rec = torch.tensor(_index(sizes, _receivers(seed, sizes, case["receivers"])), device="cuda")
    else:
        pp, pc, qp, qc = (f.double() for f in _waves(seed, sizes))
        cur, prev = [pc, qc], [pp, qp]
        src = _ricker(seed, case["steps"] if kind == "abi" else 4000)
    cur, prev, traces = _loop64(cur, prev, coef, d, case["steps"], sponge, at, src, True, rec, energy)
    fields = [torch.stack(cur, -1), torch.stack(prev, -1)]
    if kind != "shot":
        return fields
    out = {"traces": torch.stack(traces)}
    if energy is not None:
        out["energy"] = np.array(energy)
    return dict(out, fields=fields)


def _exact_batch(case, seed):
    steps = PRE_STEPS[0] + case["steps"]
    shots = _shots(case, seed)
    if sum(math.prod(s["sizes"]) for s in shots) * steps > 6e9:
        return None
    m = _medium(seed, case["mz"])
    out = {"traces": []}
    if case["fields"]:
        out["fields"] = []
    for k, sh in enumerate(shots):
        sizes = sh["sizes"]
        cur, prev = ([torch.zeros(sizes[::-1], device="cuda", dtype=torch.float64)
                      for _ in range(2)] for _ in range(2))
        rec = torch.tensor(_index(sizes, _receivers(seed + k, sizes, case["receivers"])),
                           device="cuda")
        cur, prev, traces = _loop64(cur, prev, _coef(m, sizes, sh["origin"]), (DX,) * 3, steps,
                                    _sponge64(sizes, 48), int(_index(sizes, sh["src"])),
                                    _wavelet64(steps + 1, sh["fcut"]), False, rec)
        out["traces"].append(torch.stack(traces))
        if k < case["fields"]:
            out["fields"].append({"pp": prev[0], "pc": cur[0], "qp": prev[1], "qc": cur[1]})
    return out


def _wavelet64(count, fcut):
    """The reference's source wavelet, with its float32 rounding points."""
    f = np.float32
    tf, fc = f(2.0 * math.sqrt(math.pi) / fcut), f(fcut / (3.0 * math.sqrt(math.pi)))
    x = fc * (np.arange(count, dtype=f) * f(DT) - tf)
    x = (math.pi ** 3 * x.astype(np.float64) * x).astype(f).astype(np.float64)
    return ((1.0 - 2.0 * x) * np.exp(-x)).astype(f)
