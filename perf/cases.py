"""Timed workloads of the library: what a program that uses it has it do.

Each case is one pass of a program's loop through the public entry points
(the C API of include/sunlightlb.h as ``sunlightlb_gb300.library()`` exposes
it, and the network of ``sunlightlb_gb300.warmstart``).  Kinds:

``sphere``   a sphere in a periodic box under a body force, the smallest
             driver of the library (its default, FP64 precision): a check
             interval of ``lbsteps`` + ``measure``.  Latency and launches.
``bed``      a check interval of a packed bed (permeability or calibration
             run): ``lbsteps`` + ``measure``, then the velocity and density
             field (``lbstate``) where the storage has one.  FP32, FP64 or
             BF16 populations, Stokes or Navier-Stokes, cubic or ragged.
``batch``    an ensemble of small domains, one moving sphere each,
             advanced together by ``batchsteps``.
``tracer``   a passive scalar carried through a bed, with a source and an
             absorbing plane set again before every update: on a frozen flow
             (breakthrough run) or interleaved with the flow's own steps;
             FP32 or FP64; the field is read back at the end.
``conv``     one 3x3x3 convolution layer of the warm-start network, forward
             and input gradient.
``predict``  the warm start: a solid mask through the committed network to
             the predicted state.
``train``    one training iteration of the network.

Sizes follow the repository's benchmark and tests (512^3, 256^3 and 128^3
beds, domains of 24 to 64, 64^3 training packings in batches of 4, 128^3
prediction) and spread around them.  Inputs are made on the GPU from the
seed; geometries are random (overlapping) spheres.
"""

import math

import numpy as np
import torch

FP64, FP32, BF16 = 0, 1, 2
PRECISION = {"fp64": FP64, "fp32": FP32, "bf16": BF16}
# velocity set (i, j, k components of link q) and weights
CX = (0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1)
CY = (0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1)
CZ = (0, 0, 0, 0, 0, 1, -1, 1, 1, 1, 1, -1, -1, -1, -1)
OPP = (0, 2, 1, 4, 3, 6, 5, 14, 13, 12, 11, 10, 9, 8, 7)
RHO0 = 72.0
NET_WIDTHS = (32, 64, 128, 256)
# (name, level, cin, cout) of the network's convolutions
NET_LAYERS = ((0, 32, 32), (0, 32, 32), (1, 32, 64), (1, 64, 64), (2, 64, 128), (2, 128, 128), (3, 128, 256),
              (3, 256, 256), (2, 384, 128), (2, 128, 128), (1, 192, 64), (1, 64, 64), (0, 96, 32), (0, 32, 32),
              (0, 32, 32))


def listed():
    return [
        # the smallest driver: one sphere, default precision, 50-step checks
        {"name": "sphere_24_fp64", "kind": "sphere", "ni": 24, "nj": 24, "nk": 24, "precision": "fp64", "steps": 50,
         "rad": 4.5, "tau": 0.8},
        # permeability of a 128^3 packing, Stokes flow, 100-step checks
        {"name": "bed_128_fp32", "kind": "bed", "ni": 128, "nj": 128, "nk": 128, "precision": "fp32", "stokes": True,
         "steps": 100, "phi": 0.30, "rmin": 4.0, "rmax": 8.0, "tau": 1.0, "bf": 1e-6},
        # the largest single-lattice run: 512^3 bed with inertia
        {"name": "bed_512_fp32_ns", "kind": "bed", "ni": 512, "nj": 512, "nk": 512, "precision": "fp32",
         "stokes": False, "steps": 50, "phi": 0.35, "rmin": 6.0, "rmax": 12.0, "tau": 1.0, "bf": 1e-6},
        # the reference's own precision on a scanned sample, no side a round number
        {"name": "bed_ragged_fp64", "kind": "bed", "ni": 126, "nj": 110, "nk": 97, "precision": "fp64", "stokes": True,
         "steps": 50, "phi": 0.25, "rmin": 4.0, "rmax": 8.0, "tau": 0.85, "bf": 1e-6},
        # BF16 storage on a bed where memory traffic matters
        {"name": "bed_192_bf16", "kind": "bed", "ni": 192, "nj": 192, "nk": 192, "precision": "bf16", "stokes": True,
         "steps": 100, "phi": 0.30, "rmin": 4.0, "rmax": 8.0, "tau": 1.0, "bf": 1e-6},
        # an ensemble of moving spheres
        {"name": "batch_64_domains", "kind": "batch", "domains": 64, "side_lo": 24, "side_hi": 64, "precision": "fp32",
         "steps": 100, "rmin": 3.0, "rmax": 6.0, "tau": 1.0, "speed": 1e-3},
        # breakthrough run on a frozen flow
        {"name": "tracer_256_frozen", "kind": "tracer", "ni": 256, "nj": 256, "nk": 256, "precision": "fp32",
         "frozen": True, "steps": 250, "phi": 0.35, "rmin": 6.0, "rmax": 12.0, "tau": 1.0, "bf": 1e-6, "alpha": 0.5,
         "adprob": 0.01},
        # tracer carried by a developing flow
        {"name": "tracer_live_fp32", "kind": "tracer", "ni": 160, "nj": 120, "nk": 140, "precision": "fp32",
         "frozen": False, "steps": 100, "phi": 0.30, "rmin": 4.0, "rmax": 8.0, "tau": 1.0, "bf": 1e-6, "alpha": 0.5,
         "adprob": 0.01},
        # the same in the reference's precision, all-or-nothing adsorption
        {"name": "tracer_live_fp64", "kind": "tracer", "ni": 96, "nj": 96, "nk": 96, "precision": "fp64",
         "frozen": False, "steps": 40, "phi": 0.30, "rmin": 4.0, "rmax": 8.0, "tau": 0.8, "bf": 1e-6, "alpha": 0.3,
         "adprob": 1.0},
        # a layer of the network's second level
        {"name": "conv_64ch_64", "kind": "conv", "batch": 1, "d": 64, "h": 64, "w": 64, "cin": 64, "cout": 64},
        # the warm start of a 128^3 packing
        {"name": "predict_128", "kind": "predict", "d": 128, "h": 128, "w": 128, "phi": 0.3, "rmin": 3.0,
         "rmax": 8.0},
        # a training iteration as the network was trained
        {"name": "train_4x64", "kind": "train", "batch": 4, "d": 64, "h": 64, "w": 64, "phi": 0.3, "rmin": 3.0,
         "rmax": 8.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sphere", "bed", "bed", "bed", "batch", "tracer", "tracer", "conv", "predict", "train"])
    if kind == "sphere":
        n = [_log_int(rng, 12, 72) for _ in range(3)]
        return {"kind": kind, "ni": n[0], "nj": n[1], "nk": n[2], "precision": rng.choice(["fp64", "fp32"]),
                "steps": rng.randint(20, 120), "rad": round(rng.uniform(0.15, 0.33) * min(n), 3),
                "tau": round(rng.uniform(0.6, 1.2), 3)}
    if kind in ("bed", "tracer"):
        prec = rng.choice(["fp32", "fp32", "fp64", "bf16"] if kind == "bed" else ["fp32", "fp64"])
        hi = 200 if prec == "fp64" or kind == "tracer" else 400
        base = _log_int(rng, 40, hi)
        n = [max(24, int(base * rng.uniform(0.7, 1.25))) for _ in range(3)]
        case = {"kind": kind, "ni": n[0], "nj": n[1], "nk": n[2], "precision": prec, "phi": round(rng.uniform(0.1, 0.45), 3),
                "rmin": 3.0, "rmax": round(rng.uniform(5.0, 9.0), 2), "tau": round(rng.uniform(0.7, 1.1), 3), "bf": 1e-6}
        if kind == "bed":
            case.update(stokes=rng.random() < 0.5, steps=rng.randint(20, 100 if prec != "fp64" else 50))
        else:
            case.update(frozen=prec == "fp32" and rng.random() < 0.5, steps=rng.randint(20, 60),
                        alpha=round(rng.uniform(0.1, 0.8), 3), adprob=rng.choice([1.0, 0.01, 0.3]))
        return case
    if kind == "batch":
        lo = rng.randint(16, 40)
        return {"kind": kind, "domains": _log_int(rng, 4, 100), "side_lo": lo, "side_hi": lo + rng.randint(0, 30),
                "precision": rng.choice(["fp32", "fp32", "fp64"]), "steps": rng.randint(40, 100), "rmin": 3.0,
                "rmax": round(rng.uniform(4.0, 7.0), 2), "tau": round(rng.uniform(0.7, 1.1), 3), "speed": 1e-3}
    if kind == "conv":
        level, cin, cout = rng.choice(NET_LAYERS[:8] + NET_LAYERS[10:])
        batch = rng.choice([1, 2, 4])
        side = rng.choice([64, 128 if batch == 1 else 64]) >> level
        return {"kind": kind, "batch": batch, "d": side * rng.choice([1, 2] if side < 64 else [1]), "h": side,
                "w": side, "cin": cin, "cout": cout}
    phi = round(rng.uniform(0.1, 0.5), 4)
    if kind == "predict":
        d, h, w = rng.choice([(64, 64, 64), (128, 64, 64), (64, 128, 64), (64, 64, 128), (128, 128, 64), (64, 128, 128)])
        return {"kind": kind, "d": d, "h": h, "w": w, "phi": phi, "rmin": 3.0, "rmax": 8.0}
    d, h, w = rng.choice([(64, 64, 64), (32, 64, 64), (64, 64, 32), (64, 32, 64)])
    return {"kind": kind, "batch": rng.choice([1, 2, 3, 4]), "d": d, "h": h, "w": w, "phi": phi, "rmin": 3.0, "rmax": 8.0}


# ---- inputs --------------------------------------------------------------------

def _spheres(shape, phi, rmin, rmax, gen):
    """Solid mask (bool, GPU) of randomly placed spheres of radii U[rmin, rmax],
    periodic, overlaps allowed, expected solid fraction phi."""
    vol = float(np.prod(shape))
    mean_vol = 4.0 / 3.0 * math.pi * (rmax ** 4 - rmin ** 4) / (4.0 * (rmax - rmin))
    count = max(1, int(round(-math.log(1.0 - phi) * vol / mean_vol)))
    size = torch.tensor(shape, device="cuda", dtype=torch.float64)
    centre = torch.rand(count, 3, device="cuda", dtype=torch.float64, generator=gen) * size
    rad = rmin + (rmax - rmin) * torch.rand(count, device="cuda", dtype=torch.float64, generator=gen)
    reach = int(math.ceil(rmax)) + 1
    o = torch.arange(-reach, reach + 1, device="cuda")
    box = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).view(1, -1, 3)
    solid = torch.zeros(int(vol), device="cuda", dtype=torch.bool)
    per = max(1, 8_000_000 // box.shape[1])
    dims = torch.tensor(shape, device="cuda")
    for a in range(0, count, per):
        c, r = centre[a:a + per].unsqueeze(1), rad[a:a + per].unsqueeze(1)
        node = torch.floor(c).to(torch.int64) + box
        inside = (node - c).square().sum(-1) < r * r
        node = node[inside] % dims
        solid[(node[:, 0] * shape[1] + node[:, 1]) * shape[2] + node[:, 2]] = True
    return solid.view(*shape)


def _smooth_state(shape, solid, gen, speed):
    """Smooth random velocity (3, ...) and density deviation of a lattice, as
    a run that goes on from an earlier state has them; zero on solids."""
    grid = [torch.arange(n, device="cuda", dtype=torch.float32) * (2.0 * math.pi / n) for n in shape]
    phase = torch.rand(4, 4, 3, device="cuda", generator=gen) * 2.0 * math.pi
    amp = torch.randn(4, 4, device="cuda", generator=gen)
    fields = []
    for f in range(4):
        v = torch.zeros(shape, device="cuda", dtype=torch.float32)
        for m in range(4):
            s = [torch.sin((1 + (m + a) % 3) * grid[a] + phase[f, m, a]) for a in range(3)]
            v += amp[f, m] * (s[0][:, None, None] * s[1][None, :, None] * s[2][None, None, :])
        fields.append(v * (speed if f < 3 else 20.0 * speed))
    fields[0] += speed
    out = torch.stack(fields)
    out[:, solid] = 0.0
    return out[:3].contiguous(), out[3].contiguous()


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _shape(case):
    return (case["ni"], case["nj"], case["nk"])


def _sphere_mask(shape, rad, centre):
    """The nodes insertsph sets for a sphere that lies inside the box."""
    g = [torch.arange(n, device="cuda", dtype=torch.float64) for n in shape]
    rsq = ((g[0] - centre[0]).square()[:, None, None] + (g[1] - centre[1]).square()[None, :, None]
           + (g[2] - centre[2]).square()[None, None, :])
    return rsq < rad * rad


def _flow_inputs(case, seed):
    """(solid, u, drho, body force) of the sphere, bed and tracer kinds."""
    gen, shape = _gen(seed), _shape(case)
    if case["kind"] == "sphere":
        shift = torch.rand(3, device="cuda", generator=gen, dtype=torch.float64).tolist()
        centre = [0.5 * n - 0.5 + (s - 0.5) for n, s in zip(shape, shift)]
        solid, bf, speed = _sphere_mask(shape, case["rad"], centre), 1e-4, 1e-4
    else:
        solid, bf, speed = _spheres(shape, case["phi"], case["rmin"], case["rmax"], gen), case["bf"], 2e-5
        centre = None
    u, drho = _smooth_state(shape, solid, gen, speed)
    return solid, u, drho, bf, centre


class _State:
    """What a program holds between passes: its lattices, tracers and output
    buffers; the library's objects are freed with it."""

    def __init__(self, lib):
        self.lib, self.lbs, self.mp, self.batch = lib, [], None, None

    def __del__(self):
        if self.mp is not None:
            self.lib.freemp(self.mp)
        if self.batch is not None:
            self.lib.freebatch(self.batch)
        for lb in self.lbs:
            self.lib.freelb(lb)


def _domains(case, seed):
    """(side, radius, centre, velocity) of every domain of a batch; the sides
    are the ensemble's and do not depend on the seed."""
    rng = np.random.default_rng(seed)
    sides = np.random.default_rng(case["domains"]).integers(case["side_lo"], case["side_hi"] + 1, case["domains"])
    out = []
    for side in sides.tolist():
        rad = float(rng.uniform(case["rmin"], case["rmax"]))
        centre = rng.uniform(rad + 0.5, side - 1.5 - rad, 3).tolist()
        vel = rng.normal(size=3)
        out.append((side, rad, centre, (case["speed"] * vel / np.linalg.norm(vel)).tolist()))
    return out


def _net_inputs(case, seed):
    gen = _gen(seed)
    shape = (case["d"], case["h"], case["w"])
    n = case.get("batch", 1)
    solid = torch.stack([_spheres(shape, case["phi"], case["rmin"], case["rmax"], gen) for _ in range(n)])
    labels = None
    if case["kind"] == "train":
        labels = torch.empty(n, *shape, 4, device="cuda")
        for b in range(n):
            u, drho = _smooth_state(shape, solid[b], gen, 1.0)
            labels[b, ..., :3] = u.permute(1, 2, 3, 0)
            labels[b, ..., 3] = 0.05 * drho
    return solid.to(torch.uint8), labels


def _conv_inputs(case, seed):
    """Activations (post-ReLU), output gradient, FP32 master weights, bias."""
    gen, cin, cout = _gen(seed), case["cin"], case["cout"]
    shape = (case["batch"], case["d"], case["h"], case["w"])
    x = torch.randn(*shape, cin, device="cuda", generator=gen).relu_().to(torch.bfloat16)
    g = torch.randn(*shape, cout, device="cuda", generator=gen).to(torch.bfloat16)
    w = torch.randn(27, cout, cin, device="cuda", generator=gen) * math.sqrt(2.0 / (27 * cin))
    b = torch.randn(cout, device="cuda", generator=gen) * 0.1
    return x, g, w, b


def _lattice(st, shape, case):
    """A lattice with its device state in place before the geometry is built
    (a program orders its own GPU work against the lattice's stream)."""
    lb = st.lib.newlb(*shape, "null")
    st.lbs.append(lb)
    lb.precision = PRECISION[case["precision"]]
    lb.tau = case["tau"]
    st.lib.lbgetstream(lb)
    return lb


def prepare(case, seed):
    import sunlightlb_gb300
    from sunlightlb_gb300 import warmstart
    from sunlightlb_gb300 import workloads
    L = sunlightlb_gb300.library()
    st = _State(L)
    st.case = case
    kind = case["kind"]
    if kind in ("sphere", "bed", "tracer"):
        solid, u, drho, bf, centre = _flow_inputs(case, seed)
        lb = _lattice(st, _shape(case), case)
        lb.stokes_flow = 1 if case.get("stokes", True) else 0
        torch.cuda.synchronize()
        if kind == "sphere":
            st.obj = L.insertsph(lb, case["rad"], *centre)
        else:
            st.obj = workloads.insert_solid(L, lb, solid.cpu().numpy())
        L.syncobjs(lb)
        L.addbf(lb, bf, 0.0, 0.0)
        L.lbsetstatedev(lb, u.data_ptr(), drho.data_ptr())
        n = lb.nnodes
        if lb.precision != BF16:
            st.field = torch.empty(4, n, device="cuda", dtype=torch.float32)
        st.real = np.float64 if lb.precision == FP64 else np.float32
        if kind == "tracer":
            L.lbsteps(lb, 20)
            mp = st.mp = L.newmp(lb, "null")
            mp.alpha, mp.adprob = case["alpha"], case["adprob"]
            L.mpinit(mp)
            L.adall(mp)
            L.mpslab(mp, 0.5, 0.4 * case["ni"], -1.0, case["nj"], -1.0, case["nk"], 0.5)
    elif kind == "batch":
        st.batch = L.newbatch()
        total = 0
        for side, rad, centre, vel in _domains(case, seed):
            lb = _lattice(st, (side,) * 3, case)
            lb.stokes_flow, lb.objects_moving = 1, 1
            torch.cuda.synchronize()
            obj = L.insertsph(lb, rad, *centre)
            obj.velx, obj.vely, obj.velz = vel
            L.syncobjs(lb)
            L.vspread(lb)
            L.lbgetstream(lb)  # the geometry goes to the GPU here
            L.batchadd(st.batch, lb)
            total += lb.nnodes
        st.field = torch.empty(4 * total, device="cuda", dtype=torch.float32)
    elif kind == "conv":
        x, g, w, b = _conv_inputs(case, seed)
        k = st.k = warmstart.Kernels(L.dll)
        B, D, H, W = x.shape[:4]
        st.dims, st.stream = (B, D, H, W), torch.cuda.current_stream().cuda_stream

        def padded(c):
            return torch.zeros(B, D + 2, H + 2, W + 2, c, device="cuda", dtype=torch.bfloat16)

        st.x, st.g, st.y, st.gx = padded(x.shape[-1]), padded(g.shape[-1]), padded(g.shape[-1]), padded(x.shape[-1])
        for buf, v in ((st.x, x), (st.g, g)):
            buf[:, 1:-1, 1:-1, 1:-1] = v
            k.tc_halo(buf.data_ptr(), B, D, H, W, v.shape[-1], 0, v.shape[-1], st.stream)
        st.bias = b
        st.wf = torch.empty(w.numel(), device="cuda", dtype=torch.bfloat16)
        st.wd = torch.empty(w.numel(), device="cuda", dtype=torch.bfloat16)
        k.nn_wfwd(w.data_ptr(), case["cout"], case["cin"], st.wf.data_ptr(), st.stream)
        k.nn_wdgrad(w.data_ptr(), case["cout"], case["cin"], 0, case["cin"], st.wd.data_ptr(), st.stream)
    else:
        st.solid, st.labels = _net_inputs(case, seed)
        dims = (case["d"], case["h"], case["w"])
        if kind == "predict":
            params, widths, features, _ = warmstart.load_weights()
            st.net = warmstart.UNet(L, *dims, batch=1, widths=widths, params=params, features=features)
            st.predict_state = warmstart.predict_state
            st.eta = warmstart.ETA_TAU1
        else:
            st.net = warmstart.UNet(L, *dims, batch=case["batch"], widths=NET_WIDTHS, seed=seed % 1000, features=2)
            lab = st.labels[..., :3].square().mean(dim=(1, 2, 3, 4))
            st.sample_w = (1.0 / lab).float().contiguous()
    torch.cuda.synchronize()
    return st


def run(st):
    L, kind = st.lib, st.case["kind"]
    if kind in ("sphere", "bed"):
        lb = st.lbs[0]
        L.lbsteps(lb, st.case["steps"] - 2)
        L.measure(lb)
        out = {"flow": np.array([lb.vmeanx, lb.vmeany, lb.vmeanz], dtype=st.real),
               "force": np.array([st.obj.frcx, st.obj.frcy, st.obj.frcz], dtype=st.real)}
        if lb.precision != BF16:
            L.lbstate(lb, st.field.data_ptr(), st.field[3].data_ptr())
            out["field"] = st.field
        return out
    if kind == "batch":
        L.batchsteps(st.batch, st.case["steps"])
        at = 0
        for lb in st.lbs:
            n = lb.nnodes
            L.lbstate(lb, st.field[at:].data_ptr(), st.field[at + 3 * n:].data_ptr())
            at += 4 * n
        return {"field": st.field}
    if kind == "tracer":
        lb, mp = st.lbs[0], st.mp
        frozen, sink = st.case["frozen"], lb.esi - 1
        if not frozen:  # the density snapshot follows a changing flow, once per pass
            L.mprhoinit(mp)
        for _ in range(st.case["steps"]):
            if not frozen:
                L.lbstep(lb)
            L.mpwall(mp, "x", 0, 1.0)
            L.mpwall(mp, "x", sink, 0.0)
            L.mpstep(mp)
        L.mppull(mp)
        p = mp.field()
        out = {"p": p.astype(st.real),  # a copy: the mirror is the tracer's
               "held": float(L.mptotal(mp, "all")), "breakthrough": float(L.mpplane(mp, "x", lb.esi - 2))}
        if not frozen:
            L.lbstate(lb, st.field.data_ptr(), st.field[3].data_ptr())
            out["field"] = st.field
        return out
    if kind == "conv":
        k, (B, D, H, W), cin, cout = st.k, st.dims, st.case["cin"], st.case["cout"]
        k.tc_conv3d(st.x.data_ptr(), B, D, H, W, cin, 0, cin, st.wf.data_ptr(), st.bias.data_ptr(), cout,
                    st.y.data_ptr(), cout, 0, 1, None, st.stream)
        k.tc_halo(st.y.data_ptr(), B, D, H, W, cout, 0, cout, st.stream)
        k.tc_conv3d(st.g.data_ptr(), B, D, H, W, cout, 0, cout, st.wd.data_ptr(), None, cin, st.gx.data_ptr(), cin, 0, 0,
                    st.x.data_ptr(), st.stream)
        k.tc_halo(st.gx.data_ptr(), B, D, H, W, cin, 0, cin, st.stream)
        return {"y": st.y, "gx": st.gx}
    net = st.net
    if kind == "predict":
        u, drho = st.predict_state(net, st.solid[0], 1e-6, st.eta)
        return {"u": u, "drho": drho, "logits": net.buf["OUT"]}
    net.encode(st.solid)
    logits = net.forward()
    loss = net.loss_and_backward(st.labels, st.sample_w)
    net.clip_grads(3.0)
    net.adam(1e-4)
    out = {"loss": loss, "logits": logits}
    for name, p in net.params.items():
        out[name] = {"gw": p["gw"], "gb": p["gb"], "w": p["w"]}
    return out


# ---- the work of a pass ----------------------------------------------------------

def work(case):
    """Bytes and operations of a pass: the state (populations, tracer,
    activations) read once and written once, outputs written once; about 190
    operations per lattice update (150 in Stokes flow) and 75 per tracer
    update; 2 per multiply-add of a convolution."""
    kind = case["kind"]
    size = {"fp64": 8, "fp32": 4, "bf16": 4}
    if kind in ("sphere", "bed", "tracer"):
        n, s = float(np.prod(_shape(case))), size[case["precision"]]
        state = 32.0 if case["precision"] == "bf16" else 15.0 * s
        if kind == "tracer":
            flow = 0.0 if case["frozen"] else 15.0 * s + 16.0
            return {"bytes": n * (15.0 * s + 2.0 * s + 2.0 + flow),
                    "flops": n * case["steps"] * (75.0 + (0.0 if case["frozen"] else 150.0))}
        out = 0.0 if case["precision"] == "bf16" else 16.0
        return {"bytes": n * (2.0 * state + 2.0 + out),
                "flops": n * case["steps"] * (150.0 if case.get("stokes", True) else 190.0)}
    if kind == "batch":
        n = case["domains"] * (0.5 * (case["side_lo"] + case["side_hi"])) ** 3
        return {"bytes": n * (30.0 * size[case["precision"]] + 18.0), "flops": n * case["steps"] * 150.0}
    vox = float(case["d"] * case["h"] * case["w"] * case.get("batch", 1))
    if kind == "conv":
        cin, cout = case["cin"], case["cout"]
        return {"bytes": vox * 2 * (3 * cin + 2 * cout) + 4.0 * 27 * cin * cout, "flops": 4.0 * 27 * cin * cout * vox}
    weights = sum(27.0 * ci * co for _, ci, co in NET_LAYERS)
    macs = sum(27.0 * ci * co * vox / 8 ** lv for lv, ci, co in NET_LAYERS)
    if kind == "predict":
        return {"bytes": 2.0 * weights + vox * (1.0 + 128.0 + 16.0), "flops": 2.0 * macs}
    first = 27.0 * 32 * 32 * vox  # no input gradient of the first layer
    return {"bytes": weights * 4.0 * 8 + vox * (1.0 + 16.0 + 128.0), "flops": 2.0 * (3 * macs - first)}


# ---- the same in 64 bits -----------------------------------------------------------

class _Flow64:
    """The lattice Boltzmann update (link bounce-back, streaming, collision)
    of a list of 15 FP64 arrays, by plain array operations."""

    def __init__(self, solid, tau, stokes, bf, wall=None):
        self.solid, self.omega, self.stokes, self.bf = solid, 1.0 / tau, stokes, bf
        self.wall = wall  # wall velocity times rho0 / 12, uniform over the solids
        self.fluid = (~solid).double()
        self.link = [None] + [self.shift(solid, q) != solid for q in range(1, 15)]

    @staticmethod
    def shift(v, q):
        moves = [(c, d) for d, c in enumerate((CX[q], CY[q], CZ[q])) if c]
        return torch.roll(v, [m[0] for m in moves], [m[1] for m in moves])

    def start(self, u, drho):
        u, drho = u.double(), drho.double()
        ru = [(RHO0 + drho) * u[a] for a in range(3)]
        s = None if self.stokes else [ru[a] * u[b] for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
        self.f = self.rebuild(drho, ru, s)
        self.collide()

    @staticmethod
    def rebuild(drho, ru, s):
        t = [16.0 / 72.0 * drho]
        tr = None
        if s is not None:
            tr = (s[0] + s[1] + s[2]) / 3.0
            t[0] = t[0] - tr
        for q in range(1, 15):
            w = 8.0 if q <= 6 else 1.0
            v = drho * (w / 72.0)
            for c, r in zip((CX[q], CY[q], CZ[q]), ru):
                if c:
                    v.add_(r, alpha=c * w / 24.0)
            if s is not None:
                if q <= 6:
                    v.add_(s[(q - 1) // 2], alpha=0.5).sub_(tr, alpha=0.5)
                else:
                    v.add_(tr, alpha=0.125).add_(s[3], alpha=0.125 * CX[q] * CY[q])
                    v.add_(s[4], alpha=0.125 * CX[q] * CZ[q]).add_(s[5], alpha=0.125 * CY[q] * CZ[q])
            t.append(v)
        return t

    def moments(self):
        drho = self.f[0].clone()
        ru = [torch.zeros_like(drho) for _ in range(3)]
        for q in range(1, 15):
            drho.add_(self.f[q])
            for c, r in zip((CX[q], CY[q], CZ[q]), ru):
                if c:
                    r.add_(self.f[q], alpha=c)
        return drho, ru

    def collide(self):
        drho, ru = self.moments()
        ru[0].add_(self.fluid, alpha=self.bf)
        s = []
        for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)):
            v = drho * (-1.0 / 3.0) if a == b else torch.zeros_like(drho)
            for q in range(1, 15):
                c = (CX[q], CY[q], CZ[q])
                if c[a] * c[b]:
                    v.add_(self.f[q], alpha=c[a] * c[b])
            v.mul_(1.0 - self.omega)
            if not self.stokes:
                v.addcdiv_(ru[a] * ru[b], RHO0 + drho, value=self.omega)
            s.append(v)
        self.f = None
        self.f = self.rebuild(drho, ru, s)

    def wall_term(self, q):
        w = 8.0 if q <= 6 else 1.0
        return w * (CX[q] * self.wall[0] + CY[q] * self.wall[1] + CZ[q] * self.wall[2])

    def step(self):
        new = [self.f[0]]
        for q in range(1, 15):
            back = self.f[OPP[q]]
            if self.wall is not None:  # + the term of q at fluid nodes, - that of opp(q) at solid ones: the same number
                back = back + self.wall_term(q)
            new.append(torch.where(self.link[q], back, self.shift(self.f[q], q)))
        self.f = new
        self.collide()

    def field(self):
        drho, ru = self.moments()
        ru[0].sub_(self.fluid, alpha=0.5 * self.bf)
        rho = RHO0 + drho
        return torch.stack([r / rho * self.fluid for r in ru] + [drho * self.fluid])

    def mean_flow(self):
        return (self.field()[:3].sum(dim=(1, 2, 3)) / self.solid.numel()).cpu().numpy()

    def force(self):
        total = np.zeros(3)
        for q in range(1, 15):
            # links solid s -> fluid s + c_q, seen from the fluid node
            a, b = self.shift(self.f[q], q), self.f[OPP[q]]
            d = torch.where(self.link[q] & ~self.solid, a - b, 0.0).sum().item()
            total += 2.0 * d * np.array([CX[q], CY[q], CZ[q]])
        return total


def _exact_tracer(case, flow):
    """The tracer run of `run` on the flow's 64-bit populations."""
    shape, solid, alpha, P = _shape(case), flow.solid, case["alpha"], case["adprob"]
    fluid = ~solid
    p = torch.zeros(shape, device="cuda", dtype=torch.float64)
    i = torch.arange(shape[0], device="cuda")
    j = torch.arange(shape[1], device="cuda")
    k = torch.arange(shape[2], device="cuda")
    slab = ((i > 0.5) & (i < 0.4 * shape[0]))[:, None, None] & (j >= 0)[None, :, None] & (k >= 0)[None, None, :]
    p[slab & fluid] = 0.5
    rho = torch.where(fluid, RHO0 + flow.moments()[0], torch.full_like(p, RHO0))
    scale = (RHO0 / rho - alpha) / 72.0
    kept = [None] + [torch.where(flow.link[q], torch.where(fluid, 1.0 - P, P), torch.where(fluid, 1.0, 0.0)).double()
                     for q in range(1, 15)]
    for _ in range(case["steps"]):
        if not case["frozen"]:
            flow.step()
        p[0][fluid[0]] = 1.0
        p[-1][fluid[-1]] = 0.0
        fac, piece = p / rho, p * scale
        new = torch.where(fluid, fac * flow.f[0] + 16.0 * piece + alpha * p, p)
        for q in range(1, 15):
            w = 8.0 if q <= 6 else 1.0
            sent = fac * flow.f[q] + w * piece
            here = flow.link[q] & fluid  # what x sent along opp(q) comes back
            back = fac * flow.f[OPP[q]] + w * piece
            new.add_(torch.where(here, back, flow.shift(sent, q)) * kept[q])
        p = new
    plane = p[-2][fluid[-2]]
    out = {"p": p.reshape(-1), "held": float(p.sum()),
           "breakthrough": float(plane.mean()) if plane.numel() else 0.0}
    if not case["frozen"]:
        out["field"] = flow.field().reshape(4, -1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sphere", "bed", "tracer"):
        solid, u, drho, bf, _ = _flow_inputs(case, seed)
        flow = _Flow64(solid, case["tau"], case.get("stokes", True), bf)
        flow.start(u, drho)
        del u, drho
        if kind == "tracer":
            for _ in range(20):
                flow.step()
            return _exact_tracer(case, flow)
        for _ in range(case["steps"] - 2):
            flow.step()
        mean, force = 0.25 * flow.mean_flow(), 0.0
        for weight in (0.5, 0.25):
            force = force + 0.5 * flow.force()
            flow.step()
            mean = mean + weight * flow.mean_flow()
        out = {"flow": mean, "force": force}
        if case["precision"] != "bf16":
            out["field"] = flow.field().reshape(4, -1)
        return out
    if kind == "batch":
        fields = []
        for side, rad, centre, vel in _domains(case, seed):
            solid = _sphere_mask((side,) * 3, rad, centre)
            flow = _Flow64(solid, case["tau"], True, 0.0, wall=[RHO0 * v / 12.0 for v in vel])
            flow.f = [torch.zeros(side, side, side, device="cuda", dtype=torch.float64) for _ in range(15)]
            for _ in range(case["steps"]):
                flow.step()
            fields.append(flow.field().reshape(-1))
        return {"field": torch.cat(fields)}
    if kind == "conv":
        x, g, w, b = _conv_inputs(case, seed)
        wd = w.to(torch.bfloat16).double()
        x, g = x.double(), g.double()
        y = b.double().expand(*x.shape[:4], -1).clone()
        gx = torch.zeros_like(x)
        for t in range(27):
            off = (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3)
            y += torch.roll(x, off, (1, 2, 3)) @ wd[t].T
            gx += torch.roll(g, [-o for o in off], (1, 2, 3)) @ wd[t]

        def padded(v):
            for dim in (1, 2, 3):
                n = v.shape[dim]
                v = torch.cat([v.narrow(dim, n - 1, 1), v, v.narrow(dim, 0, 1)], dim)
            return v

        return {"y": padded(y.relu()), "gx": padded(gx * (x > 0))}
    return None  # the whole network in 64 bits: its 16-bit activations are not comparable with it
