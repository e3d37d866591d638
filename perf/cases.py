"""What a user of this framework has it do, at the sizes that occur: the cases its speed is measured on.

Each case is one pass through the public entry points: an engine stepping a
batch and handing back its fields, probe traces and energies (the path every
simulation takes), several grids stepped as one pack, the cylindrical engine,
and a forward and backward pass of the early-stop network.

`prepare` builds what a program keeps (operator, engine, probes, sources),
`run` is one pass, `exact` the same numbers in 64 bits from plain torch.
"""
import math

import numpy as np
import torch

import openems_b200 as oe

C0, EPS0, MU0, Z0 = 299792458.0, 8.854187817e-12, 1.256637062e-6, 376.730313668


def listed():
    return [
        # the smallest call: a unit-test sized grid, every step's cost is launches
        dict(name="tiny_cpml", kind="grid", nx=20, ny=24, nz=28, faces="5,5,4,0,6,6", steps=120, every=10, boxes=2,
             hard=1, probes=2),
        # plain cavity with point probes (the first benchmark configuration)
        dict(name="cavity_64", kind="grid", nx=64, ny=64, nz=64, faces="", steps=1000, every=100, boxes=0, probes=8),
        # one antenna of a parameter sweep: lumped port, port DFTs at 801 points, decay checks
        dict(name="patch_port", kind="patch", nx=121, ny=98, nz=75, steps=2000, every=100, freqs=801),
        # many uneven antennas stepped together
        dict(name="patch_pack", kind="pack", count=12, family=4, steps=300, every=100),
        # the headline configuration: 256^3, CPML on every face, 40 dielectric boxes
        dict(name="boxes_256", kind="grid", nx=256, ny=256, nz=256, faces="8,8,8,8,8,8", steps=1000, every=100,
             boxes=40, probes=2),
        # the same scene with second-order Mur faces
        dict(name="boxes_mur", kind="grid", nx=256, ny=256, nz=256, faces="mur2", steps=300, every=100, boxes=40,
             probes=2),
        # compressed coefficients on a grid with no round size, CPML on some faces, a voltage and a current probe
        dict(name="ragged_compressed", kind="grid", nx=151, ny=203, nz=187, faces="8,10,0,8,6,9", steps=500, every=50,
             boxes=25, probes=2, integrals=1, compressed=1),
        # the largest: 31 million cells, odd sizes
        dict(name="large_ragged", kind="grid", nx=353, ny=310, nz=287, faces="8,8,8,8,8,8", steps=400, every=100,
             boxes=40, probes=2),
        # dispersive sphere and shell, lumped port, CPML, near-field box with running DFTs
        dict(name="scatter_144", kind="scatter", n=144, steps=400, interval=10),
        # 2-byte field storage
        dict(name="boxes_f16", kind="grid", nx=200, ny=200, nz=200, faces="8,8,8,8,8,8", steps=400, every=100,
             boxes=40, probes=2, storage="f16"),
        # cylindrical mesh
        dict(name="cylinder", kind="cyl", nr=120, na=144, nz=160, r0=0, steps=200),
        # one training pass of the early-stop network
        dict(name="stage_net", kind="net", batch=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid", "grid", "grid", "grid", "grid", "patch", "pack", "scatter", "cyl", "net"])
    if kind == "grid":
        n = [_log(rng, 20, 320) for _ in range(3)]
        cells = n[0] * n[1] * n[2]
        steps = max(60, min(_log(rng, 100, 2000), int(8e9 / cells)))
        faces = rng.choice(["", "cpml", "cpml", "cpml", "mur1", "mur2"])
        if faces == "cpml":
            lim = [min(12, d // 3) for d in n for _ in (0, 1)]
            lay = [rng.choice([0, 4, 6, 8, 8, 8, 10, 12]) for _ in range(6)]
            lay = [min(a, b) for a, b in zip(lay, lim)]
            faces = ",".join(map(str, lay)) if any(lay) else "6,6,6,6,6,6"
        c = dict(kind="grid", nx=n[0], ny=n[1], nz=n[2], faces=faces, steps=steps, every=rng.choice([10, 50, 100, 100]),
                 boxes=rng.choice([0, 5, 20, 40]), probes=rng.choice([0, 1, 2, 8]), hard=rng.choice([0, 0, 1]),
                 integrals=rng.choice([0, 0, 1]), compressed=rng.choice([0, 0, 1]))
        if not faces.startswith("mur") and rng.random() < 0.2:
            c["storage"] = rng.choice(["f16", "bf16"])
        return c
    if kind == "patch":
        n = [rng.randint(48, 160) for _ in range(3)]
        return dict(kind="patch", nx=n[0], ny=n[1], nz=n[2], steps=_log(rng, 300, 2500), every=100,
                    freqs=rng.choice([101, 401, 801]))
    if kind == "pack":
        return dict(kind="pack", count=rng.randint(3, 12), family=rng.randint(1, 10**6), steps=_log(rng, 100, 400),
                    every=100)
    if kind == "scatter":
        return dict(kind="scatter", n=rng.randint(64, 176), steps=_log(rng, 100, 500), interval=rng.choice([1, 5, 10, 20]))
    if kind == "cyl":
        return dict(kind="cyl", nr=_log(rng, 24, 200), na=_log(rng, 24, 200), nz=_log(rng, 24, 300), r0=rng.choice([0, 1]),
                    steps=_log(rng, 50, 300))
    return dict(kind="net", batch=_log(rng, 32, 512))


# --------------------------------------------------------------------------- scenes, as plain numbers


def _grid_dt(delta):
    return 0.99 * (1.0 / (C0 * math.sqrt(3.0 / (delta * delta))))


def _gauss(fmax):
    tau = 1.0 / (math.pi * fmax)
    return 4.0 * tau, tau


def _grid_scene(c, seed):
    """Boxes, sources and probes of a grid case."""
    rng = np.random.default_rng([seed, 11])
    n = (c["nx"], c["ny"], c["nz"])
    lay = _layers(c)
    s = dict(n=n, delta=1e-3, steps=c["steps"], every=c["every"], layers=lay, mur=_mur(c), boxes=[], pec=[], port=None,
             storage=c.get("storage", "f32"))
    lo = [lay[2 * a] for a in range(3)]
    hi = [n[a] - lay[2 * a + 1] for a in range(3)]
    for _ in range(c["boxes"]):
        size = [int(rng.integers(min(4, hi[a] - lo[a]), min(41, hi[a] - lo[a] + 1))) for a in range(3)]
        at = [int(rng.integers(lo[a], hi[a] - size[a] + 1)) for a in range(3)]
        s["boxes"].append((float(rng.uniform(1, 10)), float(rng.uniform(0, 0.1)),
                           tuple(v for a in range(3) for v in (at[a], at[a] + size[a]))))

    def cell():
        return tuple(int(rng.integers(max(1, lo[a] + 1), max(max(1, lo[a] + 1) + 1, hi[a] - 1))) for a in range(3))

    # a modulated pulse that fills the batch: waves are in the grid at its end, and no static charge is left behind
    T = c["steps"] * _grid_dt(s["delta"])
    f0 = float(rng.uniform(8e9, 16e9))
    mid = tuple(v // 2 for v in n)
    s["src"] = [(mid, 2, True, 0.55 * T, 0.2 * T, 1.0, f0)]
    if c.get("hard"):
        s["src"].append((cell(), 0, False, 0.55 * T, 0.2 * T, float(rng.uniform(0.5, 1)), f0))
    comps = (2, 4, 0, 1, 3, 5, 2, 4)
    s["points"] = [(comps[p % 8], cell()) for p in range(c.get("probes", 0))]
    s["integrals"] = bool(c.get("integrals"))
    return s


def _layers(c):
    f = c.get("faces", "")
    return [int(v) for v in f.split(",")] if f and not f.startswith("mur") else [0] * 6


def _mur(c):
    f = c.get("faces", "")
    return int(f[3]) if f.startswith("mur") else 0


def _patch_scene(n, rng, steps, every, freqs):
    """A rectangular PEC patch on a substrate over a ground plane with a lumped 50 ohm feed, CPML 8 all round."""
    lay, kg = 8, 10
    h = int(rng.integers(2, 7))
    kp = kg + 1 + h
    W = max(4, min(int(rng.integers(16, 81)), n[0] - 24))
    L = max(4, min(int(rng.integers(16, 81)), n[1] - 24))
    x0, y0 = (n[0] - W) // 2, (n[1] - L) // 2
    fx, fy = x0 + W // 2, y0 + L // 2 - int(round(float(rng.uniform(0.2, 0.7)) * (L // 2)))
    eps = float(rng.uniform(2.2, 10.2))
    t0, tau = _gauss(8e9)
    s = dict(n=tuple(n), delta=0.5e-3, steps=steps, every=every, layers=[lay] * 6, mur=0, storage="f32",
             boxes=[(eps, 0.0, (0, n[0], 0, n[1], kg + 1, kp))],
             pec=[(0, n[0], 0, n[1], kg, kg + 1), (x0, x0 + W, y0, y0 + L, kp, kp + 1)], points=[], integrals=False)
    if kp > kg + 2:
        s["pec"].append((fx, fx + 1, fy, fy + 1, kg + 2, kp))
    s["port"] = dict(at=(fx, fy, kg + 1), eps=eps, freqs=np.linspace(0.0, 8e9, freqs) if freqs else None)
    s["src"] = [((fx, fy, kg + 1), 2, True, t0, tau, 1.0)]
    return s


def _pack_dims(c):
    rng = np.random.default_rng(c["family"])
    return [tuple(int(v) for v in rng.integers(48, 161, size=3)) for _ in range(c["count"])]


def _pack_scenes(c, seed):
    rng = np.random.default_rng([seed, 12])
    return [_patch_scene(n, rng, c["steps"], c["every"], 0) for n in _pack_dims(c)]


def _scatter(c, seed):
    """A Drude sphere in a Lorentz shell beside a wire dipole with a lumped port, lengths in proportion to n."""
    n = c["n"]
    rng = np.random.default_rng([seed, 13])
    sc = lambda v: max(1, int(round(v * n / 384)))  # noqa: E731
    ctr, r, t = n // 2, sc(96), sc(8)
    g = np.arange(ctr - r - t - 1, ctr + r + t + 2)
    I, J, K = np.meshgrid(g, g, g, indexing="ij")
    d = np.sqrt((I + 0.5 - ctr) ** 2 + (J + 0.5 - ctr) ** 2 + (K + 0.5 - ctr) ** 2)
    pts = np.stack([I, J, K], -1)
    px, arm, lo = ctr - r - t - sc(24), sc(20), 8 + sc(10)
    wp, f0 = 2 * math.pi * float(rng.uniform(4e9, 6e9)), float(rng.uniform(3e9, 5e9))
    tau = 1.0 / (math.pi * 2.5e9)
    return dict(n=(n, n, n), delta=1e-3, steps=c["steps"], every=0, layers=[8] * 6, mur=0, storage="f32", boxes=[],
                pec=[(px, px + 1, ctr, ctr + 1, ctr - arm, ctr), (px, px + 1, ctr, ctr + 1, ctr + 1, ctr + 1 + arm)],
                points=[], integrals=False, port=dict(at=(px, ctr, ctr), eps=1.0, freqs=np.array([2e9, 3.5e9, 5e9])),
                src=[((px, ctr, ctr), 2, True, 4 * tau, tau, 1.0, 3.5e9)], sphere=pts[d <= r], shell=pts[(d > r) & (d <= r + t)],
                drude=(wp, 1e9), lorentz=(2 * math.pi * f0, 1e8, 3.0, 2.0), box=((lo,) * 3, (n - 1 - lo,) * 3),
                interval=c["interval"])


# --------------------------------------------------------------------------- this framework


def _engine(s, compressed=False):
    op = oe.Operator(oe.Grid.uniform(*s["n"], s["delta"]), oe.BoundaryConditions.all_pec())
    if "shell" in s:
        op.set_material_cells(s["lorentz"][3], 1.0, 0.0, 0.0, s["shell"].astype(np.uint64))
    for eps, sig, reg in s["boxes"]:
        op.set_material(eps, 1.0, sig, 0.0, reg)
    for reg in s["pec"]:
        op.set_pec(reg)
    port = None
    if s["port"]:
        port = oe.fdtd.LumpedPort(1, 50.0, s["port"]["at"], 2, excite=1.0, eps_r=s["port"]["eps"]).apply(op)
    eng = oe.Engine(op, compressed=compressed, storage=s["storage"])
    if any(s["layers"]):
        eng.add_cpml(oe.CpmlBoundaries(layers=tuple(s["layers"])))
    if s["mur"]:
        eng.add_mur(oe.MurAbcConfig.all(s["mur"]))
    if "sphere" in s:
        w0, g, de, ei = s["lorentz"]
        eng.add_dispersive(oe.DrudeMaterial(*s["drude"], second_order=True), s["sphere"].astype(np.uint64))
        eng.add_dispersive(oe.LorentzMaterial(w0, g, de, eps_inf=ei, second_order=True), s["shell"].astype(np.uint64))
    for comp, at in s["points"]:
        eng.add_point_probe(comp, at)
    if s["integrals"]:
        a, b = _loop(s["n"])
        eng.add_probe(oe.fdtd.voltage_probe(a, (a[0], a[1], b[2]), 2))
        eng.add_probe(oe.fdtd.current_probe(a, (b[0], b[1], a[2]), 2))
    st = dict(eng=eng, port=port)
    if port is not None and s["port"]["freqs"] is not None:
        port.add_probes(eng, s["port"]["freqs"])
    elif port is not None:
        for kind in (0, 1):
            eng.add_probe(oe.fdtd.port_probe(op, s["port"]["at"], 2, kind))
    if "box" in s:
        st["box"] = oe.fdtd.Nf2ffBox(eng, *s["box"], list(s["port"]["freqs"]), interval=s["interval"])
    exc = []
    for at, d, soft, t0, tau, amp, *f0 in s["src"]:
        kind, par = (oe.fdtd.ExcitationType.GaussianModulated, (f0[0], t0, tau)) if f0 else (oe.fdtd.ExcitationType.Gaussian, (t0, tau))
        x = oe.Excitation(kind, par, d, at, amp, soft)
        if port is not None:
            x = port.excitation(x)
        exc.append(oe.ScheduledExcitation.from_excitation(x, 0, s["steps"], op.timestep()))
    decay = 50.0 if s["port"] and s["every"] else None
    st["batch"] = oe.EngineBatch(num_steps=s["steps"], excitations=exc,
                                 termination=oe.TerminationConfig(max_timesteps=s["steps"], energy_decay_db=decay, check_interval=100),
                                 energy_monitoring=oe.EnergyMonitorConfig(sample_interval=s["every"], track_peak=True))
    return st


def _loop(n):
    """Corners of the voltage line and the current face: the middle quarter of the grid."""
    return tuple(3 * v // 8 for v in n), tuple(min(5 * v // 8, 3 * v // 8 + 24) for v in n)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grid":
        return dict(kind=kind, **_engine(_grid_scene(case, seed), bool(case.get("compressed"))))
    if kind == "patch":
        n = (case["nx"], case["ny"], case["nz"])
        s = _patch_scene(n, np.random.default_rng([seed, 14]), case["steps"], case["every"], case["freqs"])
        return dict(kind="grid", **_engine(s))
    if kind == "scatter":
        return dict(kind="grid", **_engine(_scatter(case, seed)))
    if kind == "pack":
        parts = [_engine(s) for s in _pack_scenes(case, seed)]
        return dict(kind=kind, parts=parts, pack=oe.Pack([p["eng"] for p in parts]))
    if kind == "cyl":
        from openems_b200.cylindrical import CylindricalEngine, CylindricalGrid, CylindricalOperator
        r, dt, e, _ = _cyl_scene(case, seed)
        g = CylindricalGrid.uniform(r, 0.05, case["nr"], case["na"], 0.0, 0.05, case["nz"])
        eng = CylindricalEngine(CylindricalOperator(g, dt))
        eng.write_fields(e, [np.zeros_like(v) for v in e])
        return dict(kind=kind, eng=eng, steps=case["steps"])
    from openems_b200.stage_net import StageNet, StageNetConfig
    w, x, s, y = _net_scene(case, seed)
    net = StageNet(StageNetConfig()).load(dict(w, threshold=np.array([np.nan])))
    return dict(kind="net", net=net, x=x.cuda(), s=s.cuda(), y=y.cuda())


def _result(st, res):
    eng = st["eng"]
    e, h = eng.read_fields()
    out = {"e": e, "h": h}
    if eng.num_probes:
        out["traces"] = eng.probe_traces()
    if res.energy_samples:
        out["energy"] = np.array([(s.e_energy, s.h_energy) for s in res.energy_samples])
    if st.get("port") is not None and st["port"].freqs is not None:
        out["uf"], out["if"] = eng.probe_dft(st["port"].u_dft), eng.probe_dft(st["port"].i_dft)
    if "box" in st:
        for f in range(6):
            out["face%d" % f] = np.stack([st["box"].face(f, k) for k in range(3)])
    return out


def run(state):
    if state["kind"] == "grid":
        state["eng"].reset()
        return _result(state, state["eng"].run_batch(state["batch"]))
    if state["kind"] == "pack":
        for p in state["parts"]:
            p["eng"].reset()
        res = state["pack"].run_batch([p["batch"] for p in state["parts"]])
        return [_result(p, r) for p, r in zip(state["parts"], res)]
    if state["kind"] == "cyl":
        state["eng"].step(state["steps"])
        e, h = state["eng"].read_fields()
        return {"e": list(e), "h": list(h)}
    net, x, s, y = state["net"], state["x"], state["s"], state["y"]
    out = net.forward(x, s)
    g = torch.zeros_like(out)
    g[:, 0] = (2.0 / len(y)) * (out[:, 0] - y)
    net.backward(g)
    return {"out": out, "gw": [d.gw for d in net.dense_layers()], "gb": [d.gb for d in net.dense_layers()]}


# --------------------------------------------------------------------------- what a pass cannot do without


def _cells(case):
    if case["kind"] == "scatter":
        return case["n"] ** 3
    if case["kind"] == "pack":
        return sum(a * b * c for a, b, c in _pack_dims(case))
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Coefficients (or ids) read once, fields written once; 36 operations a cell and step for the two curls."""
    if case["kind"] == "cyl":
        n = case["nr"] * case["na"] * case["nz"]
        return {"bytes": n * (24 + 24 + 24), "flops": 30 * n * case["steps"]}
    if case["kind"] == "net":
        w = 128 * 40 + 3 * 128 * 640
        f = 2 * 256 * case["batch"] * w * 3
        return {"bytes": case["batch"] * 256 * 8 * 4 + 4 * w * 2, "flops": f}
    n = _cells(case)
    co = 1 if case.get("compressed") else 48
    return {"bytes": n * (co + 24), "flops": 36 * n * case["steps"]}


def tolerance(case):
    """About four times what a run differs from the same numbers in 64 bits: 1e-6 to 1.5e-5 for 32-bit fields after these
    step counts, up to 4e-5 with dispersive media; 2-byte storage rounds every value it keeps (2^-11 and 2^-8: 3e-2 and
    eight times that). The network's products take bf16 operands: sums in another order flip a few of their roundings."""
    if case["kind"] == "net":
        return {"rel": 2e-2}
    if case["kind"] == "scatter":
        return {"rel": 1.5e-4}
    return {"rel": {"f32": 5e-5, "f16": 1e-1, "bf16": 4e-1}[case.get("storage", "f32")]}


# --------------------------------------------------------------------------- the same in 64 bits, plain torch


class _Yee:
    """The update in float64 on the GPU, written from the equations."""

    def __init__(self, s):
        self.s, n, d = s, s["n"], s["delta"]
        self.dt = dt = _grid_dt(d)
        new = lambda v: torch.full(n, v, dtype=torch.float64, device="cuda")  # noqa: E731
        self.E, self.H = [new(0.0) for _ in range(3)], [new(0.0) for _ in range(3)]
        ca, cb, self.db = new(1.0), new(dt / (EPS0 * d)), -dt / (MU0 * d)
        if "shell" in s:
            q = tuple(torch.from_numpy(s["shell"][:, a]).cuda() for a in range(3))
            cb[q] = dt / (EPS0 * s["lorentz"][3] * d)
        for eps, sig, r in s["boxes"]:
            loss = sig * dt / (2 * eps * EPS0)
            at = (slice(r[0], r[1]), slice(r[2], r[3]), slice(r[4], r[5]))
            ca[at] = (1 - loss) / (1 + loss)
            cb[at] = dt / (eps * EPS0) / (1 + loss) / d
        for r in s["pec"]:
            at = (slice(r[0], r[1]), slice(r[2], r[3]), slice(r[4], r[5]))
            ca[at] = 0.0
            cb[at] = 0.0
        self.ca, self.cb = [ca, ca, ca], [cb, cb, cb]
        self.scale = 1.0
        if s["port"]:
            p, eps = s["port"]["at"], s["port"]["eps"] * EPS0
            loss = d / (50.0 * d * d) * dt / (2 * eps)
            self.ca[2], self.cb[2] = ca.clone(), cb.clone()
            self.ca[2][p] = (1 - loss) / (1 + loss)
            self.cb[2][p] = dt / eps / (1 + loss) / d
            self.scale = dt / eps / (1 + loss) / (50.0 * d * d)
        self.slabs = {True: [[], [], []], False: [[], [], []]}
        if any(s["layers"]):
            self._cpml()
        self.mur = self._mur() if s["mur"] else []

    def _cpml(self):
        s, d, dt = self.s, self.s["delta"], self.dt
        lay = [L if 0 < L < s["n"][f // 2] else 0 for f, L in enumerate(s["layers"])]
        smax = -4.0 * math.log(1e-6) / (2 * Z0 * max(s["layers"]) * d)
        for f, L in enumerate(lay):
            if not L:
                continue
            a = f // 2
            i = torch.arange(L, dtype=torch.float64, device="cuda")
            for is_h in (True, False):
                depth = (L - i if f % 2 == 0 else i) + (0 if not is_h else -0.5 if f % 2 == 0 else 0.5)
                sig = smax * (depth / L).clamp(0, 1) ** 3
                b = torch.exp(-sig / EPS0 * dt)
                c = torch.where(sig > 0, b - 1.0, torch.zeros_like(b))
                shape = [1, 1, 1]
                shape[a] = L
                size = list(s["n"])
                size[a] = L
                psi = [torch.zeros(size, dtype=torch.float64, device="cuda") for _ in (0, 1)]
                self.slabs[is_h][a].append((0 if f % 2 == 0 else s["n"][a] - L, L, b.view(shape), c.view(shape), psi))

    def _stretch(self, d, axis, slot, is_h):
        for at, L, b, c, psi in self.slabs[is_h][axis]:
            v = d.narrow(axis, at, L)
            psi[slot].mul_(b).add_(c * v)
            v.add_(psi[slot])
        return d

    def _diff(self, f, axis, is_h, slot):
        n = f.shape[axis]
        d = torch.zeros_like(f)
        torch.sub(f.narrow(axis, 1, n - 1), f.narrow(axis, 0, n - 1), out=d.narrow(axis, 0 if is_h else 1, n - 1))
        return self._stretch(d, axis, slot, is_h)

    def _curl(self, f, is_h, a):
        b, c = (a + 1) % 3, (a + 2) % 3
        # the difference along an axis feeds two components: the first of them in x, y, z order has slot 0
        slot = lambda axis: 0 if a == min(x for x in range(3) if x != axis) else 1  # noqa: E731
        return self._diff(f[c], b, is_h, slot(b)) - self._diff(f[b], c, is_h, slot(c))

    def _mur(self):
        s, d = self.s, self.s["delta"]
        out = []
        for f in range(6):
            ax, is_max = f // 2, f % 2 == 1
            p, q = (ax + 1) % 3, (ax + 2) % 3
            o = 1 if s["mur"] == 2 and not is_max else 0
            n, lo = s["n"], 1 if s["mur"] == 2 else 0
            out.append(dict(ax=ax, line=n[ax] - 1 if is_max else o, shift=n[ax] - 2 if is_max else o + 1, comp=(p, q), lo=lo,
                            v=[None, None], ob=[0.0, 0.0], os=[0.0, 0.0], n0=n[p], n1=n[q]))
        cdt = C0 * self.dt
        self.mc = ((cdt - d) / (cdt + d), 2 * d / (cdt + d), cdt * cdt * d / (2 * d * d * (cdt + d)))
        return out

    def _plane(self, m, c, line):
        t = self.E[c].select(m["ax"], line)
        return t.t() if m["ax"] == 1 else t

    def _mur_pre(self):
        c1, c2, c3 = self.mc
        for m in self.mur:
            for k, c in enumerate(m["comp"]):
                wb, ws = self._plane(m, c, m["line"]).clone(), self._plane(m, c, m["shift"]).clone()
                v = ws - c1 * wb
                a = m["lo"] + 2
                if self.s["mur"] == 2 and m["n0"] - 2 > a and m["n1"] - 2 > a:
                    P, Q = slice(a, m["n0"] - 2), slice(a, m["n1"] - 2)
                    tot = wb + ws
                    lap = (tot[a + 1:m["n0"] - 1, Q] + tot[a - 1:m["n0"] - 3, Q] + tot[P, a + 1:m["n1"] - 1]
                           + tot[P, a - 1:m["n1"] - 3] - 4 * tot[P, Q])
                    if isinstance(m["ob"][k], float):
                        m["ob"][k], m["os"][k] = torch.zeros_like(wb), torch.zeros_like(ws)
                    v[P, Q] = c1 * m["ob"][k][P, Q] - m["os"][k][P, Q] + c2 * tot[P, Q] + c3 * lap
                    m["ob"][k], m["os"][k] = wb, ws
                m["v"][k] = v

    def _mur_post(self):
        for m in self.mur:
            for k, c in enumerate(m["comp"]):
                m["v"][k] += self.mc[0] * self._plane(m, c, m["shift"])
        for m in self.mur:
            for k, c in enumerate(m["comp"]):
                self._plane(m, c, m["line"])[m["lo"]:, m["lo"]:] = m["v"][k][m["lo"]:, m["lo"]:]

    def _source(self, t, t0, tau, amp, f0=None):
        v = math.exp(-((t - t0) / tau) ** 2)
        return amp * self.scale * (v if f0 is None else v * math.sin(2 * math.pi * f0 * t))

    def run(self):
        s, E, H, d, dt = self.s, self.E, self.H, self.s["delta"], self.dt
        inner = (slice(1, None),) * 3
        disp = []
        if "sphere" in s:
            for kind, cells in (("d", s["sphere"]), ("l", s["shell"])):
                q = tuple(torch.from_numpy(cells[:, a]).cuda() for a in range(3))
                w, g = s["drude"] if kind == "d" else s["lorentz"][:2]
                de, ei = (1.0, 1.0) if kind == "d" else s["lorentz"][2:]
                den = 1 + g * dt / 2
                a = (2 - (0 if kind == "d" else w * w * dt * dt)) / den
                P = [torch.zeros(len(cells), dtype=torch.float64, device="cuda") for _ in range(6)]
                disp.append((q, a, (g * dt / 2 - 1) / den, EPS0 * de * w * w * dt * dt / den, 1 / (EPS0 * ei), P))
        terms = [[(c, at, 1.0)] for c, at in s["points"]]
        if s["integrals"]:
            a, b = _loop(s["n"])
            terms.append([(2, (a[0], a[1], slice(a[2], b[2] + 1)), 1.0)])
            face = (slice(a[0], b[0] + 1), slice(a[1], b[1] + 1), a[2])
            terms.append([(3, face, 1.0), (4, face, -1.0)])
        if s["port"]:
            x, y, z = s["port"]["at"]
            sg = 1.0 if s["port"]["freqs"] is not None else -1.0
            terms.append([(2, (x, y, z), sg * d)])
            terms.append([(4, (x, y, z), -sg * d), (4, (x - 1, y, z), sg * d), (3, (x, y, z), sg * d), (3, (x, y - 1, z), -sg * d)])
        traces, energy, peak, faces = [], [], 0.0, None
        if "box" in s:
            faces = [None] * 6
        for step in range(s["steps"]):
            for a in range(3):
                H[a].add_(self._curl(E, True, a), alpha=self.db)
            old = [[E[a][q].clone() for a in range(3)] for q, *_ in disp]
            if self.mur:
                self._mur_pre()
            new = [self.ca[a] * E[a] + self.cb[a] * self._curl(H, False, a) for a in range(3)]
            for a in range(3):
                E[a][inner] = new[a][inner]
            if self.mur:
                self._mur_post()
            for (q, pa, pb, pc, c2, P), en in zip(disp, old):
                for a in range(3):
                    pn = pa * P[a] + pb * P[3 + a] + pc * en[a]
                    E[a][q] -= c2 * (pn - P[a])
                    P[3 + a], P[a] = P[a], pn
            for at, dr, soft, *w in s["src"]:
                v = self._source(step * dt, *w)
                E[dr][at] = E[dr][at] + v if soft else v
            F = E + H
            if terms:
                traces.append(torch.stack([sum(w * F[c][at].sum() for c, at, w in tl) for tl in terms]))
            t = step + 1
            if faces is not None and t % s["interval"] == 0:
                self._faces(faces, t)
            if s["every"] and step % s["every"] == 0:
                e2 = [float(sum((v * v).sum() for v in f)) for f in (E, H)]
                energy.append(e2)
                peak = max(peak, sum(e2))
            if s["port"] and s["every"] and step > 0 and step % 100 == 0:
                tot = float(sum((v * v).sum() for v in F))
                if peak > 0 and tot > 0 and 10 * math.log10(tot / peak) < -50.0:
                    break
        out = {"e": torch.stack(E), "h": torch.stack(H)}
        if terms:
            out["traces"] = tr = torch.stack(traces).cpu().numpy()
        if energy:
            out["energy"] = np.array(energy)
        if s["port"] and s["port"]["freqs"] is not None:
            t = np.arange(1, len(tr) + 1)
            for name, k, half in (("uf", 0, 0.0), ("if", 1, 0.5)):
                out[name] = np.exp(-2j * np.pi * np.outer(s["port"]["freqs"], (t - half) * dt)) @ tr[:, k] * (2 * dt)
        if faces is not None:
            for f in range(6):
                out["face%d" % f] = faces[f].cpu().numpy()
        return out

    def _faces(self, faces, t):
        (lo, hi), dt = self.s["box"], self.dt
        fr = torch.tensor(self.s["port"]["freqs"], dtype=torch.float64, device="cuda")
        w = [torch.exp(torch.complex(torch.zeros_like(fr), -2 * math.pi * fr * (tt * dt))) * (2 * dt * self.s["interval"])
             for tt in (t, t - 0.5)]
        for f in range(6):
            a = f // 2
            b, c = (a + 1) % 3, (a + 2) % 3
            p = hi[a] if f % 2 else lo[a]

            def cut(v, at):
                x = v.select(a, at)
                rest = [k for k in range(3) if k != a]
                x = x[lo[rest[0]]:hi[rest[0]] + 1, lo[rest[1]]:hi[rest[1]] + 1]
                return x if rest == [b, c] else x.t()

            v = torch.stack([cut(self.E[b], p), cut(self.E[c], p), 0.5 * (cut(self.H[b], p - 1) + cut(self.H[b], p)),
                             0.5 * (cut(self.H[c], p - 1) + cut(self.H[c], p))])
            ww = torch.stack([w[0], w[0], w[1], w[1]], 1)[:, :, None, None]
            add = ww * v[None]
            faces[f] = add if faces[f] is None else faces[f] + add


def _cyl_scene(case, seed):
    """First radius, a timestep at which the fields stay finite, and the fields a run starts from."""
    r = 0.0 if case["r0"] else 0.005
    nr, na, nz = case["nr"], case["na"], case["nz"]
    dr, da, dz = (0.05 - r) / nr, 2 * math.pi / na, 0.05 / nz
    rr = max(r, dr * 0.5)
    dt = 0.002 * 0.95 / (C0 * math.sqrt(1 / dr ** 2 + 1 / (rr * da) ** 2 + 1 / dz ** 2))
    rng = np.random.default_rng([seed, 15])
    return r, dt, [rng.standard_normal((nr, na, nz), dtype=np.float32) for _ in range(3)], (dr, da, dz)


def _cyl_exact(case, seed):
    r0, dt, e, (dr, da, dz) = _cyl_scene(case, seed)
    nr = case["nr"]
    E = [torch.from_numpy(v).cuda().double() for v in e]
    H = [torch.zeros_like(v) for v in E]
    R = (r0 + torch.arange(nr, dtype=torch.float64, device="cuda") * dr).view(-1, 1, 1)
    zero = torch.zeros_like(R)
    safe = lambda num, den: torch.where(den > 0, num / torch.where(den > 0, den, torch.ones_like(den)), zero)  # noqa: E731
    vi = [safe(dt / EPS0, R * da * dz), zero + dt / EPS0 / (dr * dz), safe(dt / EPS0, 0.5 * ((R + dr) ** 2 - R ** 2) * da)]
    iv = [zero + dt / (MU0 * dr), safe(dt / MU0, R * da), zero + dt / (MU0 * dz)]

    def near(f, axis, step):
        g = torch.roll(f, -step, axis)
        if axis != 1:
            k = 0 if step < 0 else f.shape[axis] - 1
            g.select(axis, k).copy_(f.select(axis, k))
        return g

    for _ in range(case["steps"]):
        pr = lambda f, a: f - near(f, a, -1)  # noqa: E731
        c = [pr(H[2], 1) - pr(H[1], 2), pr(H[0], 2) - pr(H[2], 0), pr(H[1], 0) - pr(H[0], 1)]
        if case["r0"]:
            c[0][0] = 0.0
            c[2][0] = 0.0
        for a in range(3):
            E[a] += vi[a] * c[a]
        if case["r0"]:
            E[1][0] = 0.0
            E[2][0] = 0.5 * E[2][1]
        nx = lambda f, a: near(f, a, 1) - f  # noqa: E731
        c = [nx(E[1], 2) - nx(E[2], 1), nx(E[2], 0) - nx(E[0], 2), nx(E[0], 1) - nx(E[1], 0)]
        for a in range(3):
            H[a] += iv[a] * c[a]
    return {"e": E, "h": H}


def _net_scene(case, seed):
    """Weights, decaying port traces, diagnostics and targets of a training batch."""
    rng = np.random.default_rng([seed, 16])
    dims = [(40, 128)] + [(640, 128)] * 3 + [(136, 256), (256, 8)]
    w = {}
    for k, (i, o) in enumerate(dims):
        w["w%d" % k] = rng.normal(0.0, math.sqrt(2.0 / i), (o, i)).astype(np.float32)
        w["b%d" % k] = rng.normal(0.0, 0.01, o).astype(np.float32)
    B, t = case["batch"], np.arange(256)
    x = np.zeros((B, 256, 8), dtype=np.float32)
    for c in (0, 1):
        f, q, ph = rng.uniform(0.01, 0.2, (B, 1)), rng.uniform(20, 400, (B, 1)), rng.uniform(0, 6.3, (B, 1))
        x[:, :, c] = np.exp(-t / q) * np.cos(2 * np.pi * f * t + ph)
    s = rng.normal(0.0, 1.0, (B, 8)).astype(np.float32)
    y = rng.uniform(-2, 1, B).astype(np.float32)
    return w, torch.from_numpy(x), torch.from_numpy(s), torch.from_numpy(y)


def _net_exact(case, seed):
    w, x, s, y = _net_scene(case, seed)
    W = [torch.from_numpy(w["w%d" % k]).cuda().double().requires_grad_() for k in range(6)]
    b = [torch.from_numpy(w["b%d" % k]).cuda().double().requires_grad_() for k in range(6)]
    h = x.cuda().double()
    for k in range(4):
        dil, C = 4 ** k, h.shape[2]
        cols = torch.cat([torch.nn.functional.pad(h, (0, 0, (4 - j) * dil, 0))[:, :256] for j in range(5)], 2)
        h = torch.relu(cols @ W[k].t() + b[k])
    z = torch.relu(torch.cat([h[:, -1], s.cuda().double()], 1) @ W[4].t() + b[4])
    out = z @ W[5].t() + b[5]
    loss = ((out[:, 0] - y.cuda().double()) ** 2).mean()
    loss.backward()
    return {"out": out.detach(), "gw": [v.grad for v in W], "gb": [v.grad for v in b]}


def exact(case, seed):
    if case["kind"] == "net":
        return _net_exact(case, seed)
    if case["kind"] == "cyl":
        return _cyl_exact(case, seed)
    if case["kind"] == "pack":
        return [_Yee(s).run() for s in _pack_scenes(case, seed)]
    if case["kind"] == "patch":
        n = (case["nx"], case["ny"], case["nz"])
        return _Yee(_patch_scene(n, np.random.default_rng([seed, 14]), case["steps"], case["every"], case["freqs"])).run()
    if case["kind"] == "scatter":
        return _Yee(_scatter(case, seed)).run()
    return _Yee(_grid_scene(case, seed)).run()
