"""The work this framework is used for, as measured cases.

A case is one of
* ``rtm``: a shot through ``Simulator`` (forward with receivers and
  snapshots, adjoint of the residual against observed traces, both images),
  on the fused kernels or (``fused`` false) on the reference's launcher
  sequence, for either operator, any snapshot precision, with or without
  graphs and checkpoints;
* ``forward``: modelling only (traces, no snapshots);
* ``shot``: the run-level call ``serve.rtm_shot`` on host arrays, everything
  from the simulator's creation to the images in host memory;
* ``stress``, ``velocity``: the elastic proxy's step launchers.

Shots are short (a few time steps of the lengths that real shots repeat
500 to 3000 times).  Models: smooth random tilted fields, or flat layers.
"""
import math

import numpy as np
import torch

from miniappsforhpe_b200 import Config, Simulator, elastic, serve

R = 4  # halo
DX = 10.0


# ---------------------------------------------------------------------------
# The cases.
def _case(name, kind, nx, ny, nz, nt=0, **more):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, nt=nt, model="tti", scheme=0, snap="fp32", surface=True, sponge=24,
             fused=True, graphs=False, checkpoint=0, xcorr=4, rec_every=1)
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the headline shot: 256^3 TTI, 24-cell sponge, receivers on every cell of a plane, imaging every 4 steps
        _case("rtm_tti_256", "rtm", 256, 256, 256, 64),
        # the largest shot: layered 512x512x400, FP16 snapshots, checkpointed recomputation
        _case("rtm_vti_512_checkpoint", "rtm", 512, 512, 400, 8, model="vti", snap="fp16", checkpoint=4),
        # the served form's ordinary shot: layered, FP16 snapshots, receivers on every 4th cell
        _case("rtm_vti_224_fp16", "rtm", 224, 224, 160, 48, model="vti", snap="fp16", sponge=16, rec_every=4),
        # a ragged grid in plain FP32 whose rows no 16-byte copy fits
        _case("rtm_tti_odd", "rtm", 101, 93, 77, 60, sponge=10),
        # the smallest shots (tests, quick looks): launches and latency, replayed from a graph
        _case("rtm_tti_small_graph", "rtm", 48, 40, 40, 96, sponge=8, graphs=True),
        # modelling alone at 128^3, VTI
        _case("forward_vti_128", "forward", 128, 128, 128, 100, model="vti", sponge=0),
        # the centred constant-density operator on the headline grid
        _case("rtm_centred_256", "rtm", 256, 256, 256, 48, scheme=1),
        # a user's own schedule on the reference's launchers, both operators
        _case("launchers_tti_160", "rtm", 160, 160, 160, 16, fused=False, sponge=16),
        _case("launchers_centred_odd", "rtm", 150, 141, 133, 16, fused=False, scheme=1, sponge=16),
        # one whole small shot from host arrays to host images
        _case("shot_vti_96", "shot", 96, 96, 96, 160, model="vti", snap="fp16", sponge=12, rec_every=4),
        # the elastic proxy: stress update at the reference's size, velocity and strain updates on a ragged grid
        _case("elastic_stress_256", "stress", 256, 256, 256),
        _case("elastic_velocity_odd", "velocity", 211, 187, 150),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rtm", "rtm", "rtm", "rtm", "rtm", "forward", "shot", "launchers", "stress", "velocity"])
    top = {"launchers": 180, "shot": 160, "stress": 260, "velocity": 280}.get(kind, 330)
    nx, ny, nz = (_log_int(rng, 40, top) for _ in range(3))
    snap = rng.choice(["fp32", "fp32", "fp16", "bf16"])
    fused = kind != "launchers"
    if not fused:
        kind, snap = "rtm", "fp32"
    if kind in ("rtm", "shot") and snap != "fp32":
        nx = max(40, nx // 8 * 8)  # what reduced-precision stores take
    if kind in ("stress", "velocity"):
        return _case("", kind, nx, ny, nz)
    most = (40e6 if not fused else 256 ** 3 * 48.0) / (nx * ny * nz)  # step points of one pass
    nt = max(8, min(_log_int(rng, 8, 120), int(most)))
    xcorr = rng.choice([2, 4, 5])
    checkpoint = xcorr * max(1, nt // (3 * xcorr)) if fused and kind != "forward" and rng.random() < 0.25 else 0
    return _case("", kind, nx, ny, nz, nt, model=rng.choice(["tti", "tti", "vti"]),
                 scheme=rng.choice([0, 0, 0, 1]), snap="fp32" if kind == "forward" else snap,
                 surface=rng.random() < 0.75, sponge=rng.choice([0, 8, 16, 24]), fused=fused,
                 graphs=fused and rng.random() < 0.3, checkpoint=checkpoint, xcorr=xcorr,
                 rec_every=rng.choice([1, 2, 4]))


# ---------------------------------------------------------------------------
# Inputs.
def _smooth(shape, cells, gen):
    """A random field in [0, 1] that varies over `cells` cells."""
    coarse = [max(2, int(math.ceil(n / cells)) + 1) for n in shape]
    f = torch.rand([1, 1] + coarse, generator=gen, device="cuda")
    return torch.nn.functional.interpolate(f, size=list(shape), mode="trilinear", align_corners=True)[0, 0]


def _model(case, seed):
    """{name: float32 (nz, ny, nx) tensor on the GPU}, in the ranges of the synthetic earth models."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)
    shape = (case["nz"], case["ny"], case["nx"])
    if case["model"] == "tti":
        m = {"vp": 1500.0 + 3500.0 * _smooth(shape, 30, gen), "eps": 0.25 * _smooth(shape, 30, gen)}
        m["delta"] = torch.minimum(0.1 * _smooth(shape, 30, gen), m["eps"])
        m["theta"] = math.radians(45.0) * _smooth(shape, 30, gen)
        m["phi"] = math.radians(180.0) * _smooth(shape, 30, gen)
        m["rho"] = 1.0 + 1.2 * _smooth(shape, 30, gen)
        return m
    layer = torch.randint(0, 6, (case["nz"],), generator=gen, device="cuda").sort().values
    vp = 1500.0 + 3000.0 * torch.rand(6, generator=gen, device="cuda")
    eps = 0.3 * torch.rand(6, generator=gen, device="cuda")
    delta = torch.minimum(0.15 * torch.rand(6, generator=gen, device="cuda"), eps)
    return {k: v[layer][:, None, None].expand(shape).contiguous() for k, v in
            (("vp", vp), ("eps", eps), ("delta", delta))}


def _dt(m):
    return float(np.float32(0.4 * DX / float((m["vp"] * torch.sqrt(1.0 + 2.0 * m["eps"])).max())))


def _source(case):
    return case["nx"] // 2, case["ny"] // 3, min(6, case["nz"] - 1)


def _receivers(case):
    iy, ix = np.meshgrid(np.arange(0, case["ny"], case["rec_every"]), np.arange(0, case["nx"], case["rec_every"]),
                         indexing="ij")
    return np.stack([ix.ravel(), iy.ravel(), np.full(ix.size, 3)], axis=1).astype(np.int32)


def _wavelet(case, dt):
    """The first steps of a 15 Hz Ricker pulse that peaks at 53 ms."""
    a = (math.pi * 15.0 * (np.arange(case["nt"]) * dt - 0.8 / 15.0)) ** 2
    return (1e5 * (1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _observed(case, dt, seed):
    """Traces of a pulse that moves out from a random place, of the size that the modelled ones have."""
    rng = np.random.default_rng([int(seed), 5])
    rec = _receivers(case)
    at = rng.uniform(0.2, 0.8, 2) * (case["nx"], case["ny"])
    dist = np.hypot(rec[:, 0] - at[0], rec[:, 1] - at[1]) / (case["nx"] + case["ny"])
    n = np.arange(case["nt"], dtype=np.float32)[:, None]
    mid = ((0.3 + 0.8 * dist) * case["nt"]).astype(np.float32)[None, :]
    a = ((n - mid) / (0.15 * case["nt"])) ** 2
    return (0.1 * rng.uniform(0.5, 2.0) * (1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _config(case, dt):
    return Config(case["nx"], case["ny"], case["nz"], DX, DX, DX, dt, case["nt"], xcorr_step=case["xcorr"],
                  sponge_width=case["sponge"], free_surface=case["surface"], fused=case["fused"],
                  save_snapshots=case["kind"] != "forward", snap_precision=case["snap"],
                  checkpoint_every=case["checkpoint"], use_graphs=case["graphs"], scheme=case["scheme"])


def _elastic(case, seed):
    e = elastic.ElasticProxy(case["nx"], case["ny"], case["nz"])
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 104729 + 3)
    inside = (slice(R, R + case["nz"]), slice(R, R + case["ny"]), slice(R, R + case["nx"]))
    for f in e.v + e.s + e.d:
        f.zero_()
        f[inside] = torch.randn((case["nz"], case["ny"], case["nx"]), generator=gen, device="cuda")
    return e


def prepare(case, seed):
    if case["kind"] in ("stress", "velocity"):
        return {"case": case, "e": _elastic(case, seed)}
    m = _model(case, seed)
    dt = _dt(m)
    host = {k: v.cpu().numpy() for k, v in m.items()}
    observed = _observed(case, dt, seed)
    if case["kind"] == "shot":
        shot = serve.Shot(case["nx"], case["ny"], case["nz"], dt, case["nt"], host["vp"], _wavelet(case, dt),
                          _source(case), _receivers(case), **{k: v for k, v in host.items() if k != "vp"},
                          observed=observed, dx=DX, dy=DX, dz=DX, xcorr_step=case["xcorr"],
                          sponge_width=case["sponge"], free_surface=case["surface"])
        return {"case": case, "shot": shot, "opts": _config(case, dt)}
    sim = Simulator(_config(case, dt))
    sim.set_model(**host)
    sim.set_source(*_source(case), _wavelet(case, dt))
    sim.set_receivers(_receivers(case))
    s = {"case": case, "sim": sim, "traces": torch.zeros(observed.shape, device="cuda")}
    if case["kind"] == "rtm":
        s["observed"] = torch.from_numpy(observed).cuda()
        for k in ("vp", "rho"):
            s[k] = torch.zeros((case["nz"], case["ny"], case["nx"]), device="cuda")
    return s


# ---------------------------------------------------------------------------
# One pass.
def run(s):
    case = s["case"]
    if case["kind"] == "stress":
        e = s["e"]
        elastic.launch_splain(*e.s, e.M[:21], *e.d, e.pre, e.nx, e.ny, e.nz, e.ldimx, e.ldimy)
        return e.s + e.pre
    if case["kind"] == "velocity":
        e = s["e"]
        grid = (e.nx, e.ny, e.nz, e.ldimx, e.ldimy)
        elastic.launch_vplain(*e.v, *e.s, e.M[21], e.zprime, *grid)
        elastic.launch_mirror(e.v, e.ldimx, e.ldimy, R, e.ldimz)
        elastic.launch_vgplain(*e.v, *e.d, e.zprime, *grid)
        elastic.launch_compute_p(e.p, *e.s, e.p.numel())
        return e.v + e.d + [e.p]
    if case["kind"] == "shot":
        r = serve.rtm_shot(s["shot"], s["opts"])
        return [r.traces, r.image_vp] + ([r.image_rho] if case["scheme"] == 0 else [])
    sim = s["sim"]
    sim.forward(s["traces"])
    if case["kind"] == "forward":
        return [s["traces"]]
    sim.adjoint_observed(s["observed"])
    sim.image(s["vp"], s["rho"])
    return [s["traces"], s["vp"]] + ([s["rho"]] if case["scheme"] == 0 else [])


# ---------------------------------------------------------------------------
# What one pass cannot do without.
def work(case):
    n = float(case["nx"] * case["ny"] * case["nz"])
    if case["kind"] == "stress":  # 21 moduli, 6 strains, 12 mixed volumes written, 6 stresses updated
        return {"bytes": n * 4 * (21 + 6 + 12 + 12), "flops": n * 470}
    if case["kind"] == "velocity":  # 6 stresses, buoyancy, 3 velocities updated; strains from them; pressure
        return {"bytes": n * 4 * (6 + 1 + 6) + n * 4 * (3 + 6) + n * 4 * 7, "flops": n * 210}
    tilt = case["model"] == "tti"
    forward = case["nt"]
    if case["checkpoint"]:  # every step but the last segment's is modelled twice
        forward += (case["nt"] - 1) // case["checkpoint"] * case["checkpoint"]
    adjoint = case["nt"] if case["kind"] != "forward" else 0
    images = (case["nt"] - 1) // case["xcorr"] + 1 if adjoint else 0
    fields = 4 if case["scheme"] == 0 else 2
    elt = 4 if case["snap"] == "fp32" else 2
    if case["fused"]:  # p, q, pdot, qdot read and written, the model read
        model = 4 + (1 if case["scheme"] == 0 else 0) + (3 if tilt else 0)
        step, image = 4 * (8 + model), fields * elt + (8 + 8 if case["scheme"] == 0 else 8)
        byts = n * (step * (forward + adjoint) + image * images + fields * elt * images)
    elif case["scheme"] == 0:  # each launcher's volumes once per launch
        byts = n * 4 * ((6 + 9 + 20) * forward + (18 + 12 + 6) * adjoint + (6 + 4 + 9 + 18 + 8) * images)
    else:
        byts = n * 4 * ((6 + 13) * forward + (13 + 6) * adjoint + (6 + 4) * images)
    per_step = (360 if tilt else 220) if case["scheme"] == 0 else (300 if tilt else 150)
    return {"bytes": byts, "flops": n * (per_step * (forward + adjoint) + (280 if fields == 4 else 4) * images)}


def tolerance(case):
    # measured between the fused kernels and the launcher sequence, which sum in another order: at most 1e-6, and
    # 2e-4 of the largest; a stored 16-bit value that rounds the other way is off by its whole unit at that cell
    if case["kind"] in ("stress", "velocity"):
        return {"rel": 2e-6, "max": 1e-4}
    if case["kind"] != "forward" and case["snap"] != "fp32":
        return {"rel": 2e-4, "max": 0.5 if case["snap"] == "fp16" else 0.9}
    return {"rel": 1e-5, "max": 1e-3}


# ---------------------------------------------------------------------------
# The same in 64 bits.
C1 = [0.0] + [float(np.float32(v)) for v in (1.19628906250000e+00, -7.97526041666667e-02, 9.57031250000000e-03,
                                             -6.97544642857143e-04)]
C2 = [float(np.float32(v)) for v in (-2.903117, 1.645351, -0.2236606, 0.03265851, -0.002790073)]
CS = [float(np.float32(v)) for v in (1.1962891, -7.9752604e-2, 9.5703125e-3, -6.9754464e-4)]
E3 = [float(np.float32(v)) for v in (1.01, 2.01, 3.01, 4.01)]


class _Grid:
    def __init__(self, case):
        self.n = (case["nz"], case["ny"], case["nx"])
        self.inside = tuple(slice(R, R + k) for k in self.n)

    def zeros(self):
        return torch.zeros([k + 2 * R for k in self.n], dtype=torch.float64, device="cuda")

    def put(self, inner):
        v = self.zeros()
        v[self.inside] = inner
        return v

    def at(self, v, z=0, y=0, x=0):
        return v[tuple(slice(R + o, R + o + k) for o, k in zip((z, y, x), self.n))]

    def along(self, v, axis, o):
        return self.at(v, **{"zyx"[axis]: o})

    def minus(self, v, axis, c=C1[1:]):
        """Staggered derivative half a cell back, over the interior."""
        return sum(c[k - 1] * (self.along(v, axis, k - 1) - self.along(v, axis, -k)) for k in range(1, 5)) / DX

    def plus(self, v, axis, c=C1[1:]):
        return sum(c[k - 1] * (self.along(v, axis, k) - self.along(v, axis, 1 - k)) for k in range(1, 5)) / DX

    def second(self, v, axis):
        return (C2[0] * self.at(v) + sum(C2[k] * (self.along(v, axis, k) + self.along(v, axis, -k))
                                         for k in range(1, 5))) / (DX * DX)

    def cross(self, v, a, b):
        a, b = "zyx"[a], "zyx"[b]
        return sum(C2[k] * (self.at(v, **{a: k, b: k}) - self.at(v, **{a: k, b: -k}) +
                            self.at(v, **{a: -k, b: -k}) - self.at(v, **{a: -k, b: k}))
                   for k in range(1, 5)) / (4 * DX * DX)


def _mirror(v):
    """Free surface at plane R: zero there, odd above."""
    v[R] = 0.0
    for k in range(1, R + 1):
        v[R - k] = -v[R + k]


def _mirror_dz(v):
    for iz in range(R + 1):
        v[iz] = v[2 * R + 1 - iz]


def _edge(v):
    return torch.nn.functional.pad(v.double()[None, None], [R] * 6, mode="replicate")[0, 0]


class _Exact:
    def __init__(self, case, seed):
        m = _model(case, seed)
        self.case, self.g, self.dt = case, _Grid(case), _dt(m)
        self.vp = m["vp"].double()
        p = {k: _edge(v) for k, v in m.items()}
        vp2 = p["vp"] * p["vp"]
        zero = torch.zeros_like(vp2)
        self.m1, self.m3, self.m4 = vp2 * (1 + 2 * p["eps"]), vp2, zero
        self.m2 = torch.sqrt(vp2 * vp2 * (1 + 2 * p["delta"]))
        theta, phi = p.get("theta", zero), p.get("phi", zero)
        self.rx, self.ry, self.rz = torch.sin(theta) * torch.cos(phi), torch.sin(theta) * torch.sin(phi), torch.cos(theta)
        self.irho = 1.0 / p["rho"] if "rho" in p else torch.ones_like(vp2)
        axes = [self._sponge(k, low) for k, low in zip(self.g.n, (not case["surface"], True, True))]
        self.damp = torch.minimum(torch.minimum(axes[0][:, None, None], axes[1][None, :, None]), axes[2][None, None, :])
        self.rec = torch.from_numpy(_receivers(case).astype(np.int64)).cuda()
        self.src = tuple(R + k for k in reversed(_source(case)))
        self.state = [self.g.zeros() for _ in range(4)]

    def _sponge(self, n, low):
        w = self.case["sponge"]
        a = np.ones(n)
        for k in range(min(w, n)):
            f = float(np.float32(math.exp(-(0.3 * (w - k) / w) ** 2)))
            if low:
                a[k] = f
            a[n - 1 - k] = min(a[n - 1 - k], f)
        return torch.from_numpy(a).cuda()

    def _update_pq(self):
        p, q, pd, qd = self.state
        for f, fd in ((p, pd), (q, qd)):
            f[self.g.inside] = self.damp * self.g.at(f) + self.damp * self.g.at(fd) * self.dt
            if self.case["surface"]:
                _mirror(f)

    def _add(self, f, rhs, sponge):
        old = self.g.at(f)
        f[self.g.inside] = self.damp * old + self.damp * rhs * self.dt if sponge else old + rhs * self.dt

    def first(self, f):
        """Buoyancy-scaled first derivatives of one field, halos as the free surface makes them."""
        d = [self.g.put(self.g.minus(f, axis) * self.g.at(self.irho)) for axis in range(3)]
        if self.case["surface"]:
            _mirror_dz(d[0])
        return d

    def forward_rates(self):
        g, at = self.g, self.g.at
        V, H = [], []
        for f in self.state[:2]:
            if self.case["scheme"] == 0:
                d = self.first(f)
                zz, yy, xx = (g.plus(d[axis], axis) / at(self.irho) for axis in range(3))
            else:
                zz, yy, xx = (g.second(f, axis) for axis in range(3))
            rx, ry, rz = at(self.rx), at(self.ry), at(self.rz)
            V.append(rx * rx * xx + ry * ry * yy + rz * rz * zz + 2 * rx * ry * g.cross(f, 1, 2) +
                     2 * rz * rx * g.cross(f, 0, 2) + 2 * ry * rz * g.cross(f, 0, 1))
            H.append(xx + yy + zz - V[-1])
        return (at(self.m1) * H[0] + at(self.m4) * V[0] + at(self.m2) * V[1],
                at(self.m2) * H[0] + at(self.m3) * V[1] + at(self.m4) * H[1])

    def temporaries(self):
        """(S, H) of both fields, the model transposed onto the adjoint p, q."""
        p, q = self.state[:2]
        return ((self.m1 * p + self.m2 * q, (self.m4 - self.m1) * p - self.m2 * q),
                (self.m4 * q, self.m2 * p + (self.m3 - self.m4) * q))

    def adjoint_rates(self):
        g = self.g
        out = []
        for S, H in self.temporaries():
            r = (g.cross(2 * self.rx * self.ry * H, 1, 2) + g.cross(2 * self.ry * self.rz * H, 0, 1) +
                 g.cross(2 * self.rz * self.rx * H, 0, 2))
            for axis, ra in ((0, self.rz), (1, self.ry), (2, self.rx)):
                t = S + ra * ra * H
                if self.case["scheme"] == 1:
                    r = r + g.second(t, axis)
                    continue
                d = g.put(g.minus(t / self.irho, axis) * g.at(self.irho))
                if self.case["surface"] and axis == 0:
                    _mirror_dz(d)
                r = r + g.plus(d, axis)
            out.append(r)
        return out

    def image(self, gvp, grho, snap):
        g, at = self.g, self.g.at
        gvp += at(self.state[2]) * snap[0] + at(self.state[3]) * snap[1]
        if self.case["scheme"] == 1:
            return
        rhs = 0.0
        for (S, H), stored in zip(self.temporaries(), snap[2:]):
            f = g.put(stored)
            if self.case["surface"]:
                _mirror(f)
            d = self.first(f)
            for axis, ra in ((0, self.rz), (1, self.ry), (2, self.rx)):
                t = (S + ra * ra * H) / self.irho
                rhs = rhs + at(t) * g.plus(d[axis], axis, CS) + g.minus(t, axis, CS) * at(d[axis])
        grho -= at(self.irho) * rhs

    def shot(self, seed):
        case, n = self.case, self.case["nt"]
        p, q, pd, qd = self.state
        wavelet, ix, iy, iz = _wavelet(case, self.dt), *(self.rec[:, k] + R for k in range(3))
        traces, snaps = [], {}
        adjoint = case["kind"] != "forward"
        for it in range(n):
            traces.append(-(2 * p[iz, iy, ix] + q[iz, iy, ix]) / 3)
            r3, r4 = self.forward_rates()
            for f, r in ((pd, r3), (qd, r4)):
                self._add(f, r, case["scheme"] == 1 and case["sponge"] > 0)
                f[self.src] += float(wavelet[it]) * self.dt
            if adjoint and it % case["xcorr"] == 0:
                keep = (pd, qd, p, q)[:4 if case["scheme"] == 0 else 2]
                snaps[it] = [self.g.at(f).clone() for f in keep]
            self._update_pq()
        traces = torch.stack(traces)
        if not adjoint:
            return [traces]
        for f in self.state:
            f.zero_()
        gvp, grho = torch.zeros_like(self.vp), torch.zeros_like(self.vp)
        residual = traces - torch.from_numpy(_observed(case, self.dt, seed)).cuda().double()
        for it in range(n - 1, -1, -1):
            pd[iz, iy, ix] += -2.0 / 3.0 * residual[it]
            qd[iz, iy, ix] += -1.0 / 3.0 * residual[it]
            r3, r4 = self.adjoint_rates()
            self._add(pd, r3, case["sponge"] > 0)
            self._add(qd, r4, case["sponge"] > 0)
            self._update_pq()
            if it % case["xcorr"] == 0:
                self.image(gvp, grho, snaps.pop(it))
        gvp *= -self.dt * case["xcorr"] * 2.0 / self.vp
        return [traces, gvp] + ([grho] if case["scheme"] == 0 else [])


def _exact_elastic(case, seed):
    e = _elastic(case, seed)
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    v, s, d = ([f.double() for f in fs] for fs in (e.v, e.s, e.d))

    def at(f, z=0, y=0, x=0):
        return f[R + z:R + z + nz, R + y:R + y + ny, R + x:R + x + nx]

    def drv(f, axis, back):
        o = -1 if back else 0
        return sum(E3[i] * (at(f, **{axis: o + i + 1}) - at(f, **{axis: o - i})) for i in range(4))

    inside = (slice(R, R + nz), slice(R, R + ny), slice(R, R + nx))
    if case["kind"] == "velocity":
        M, zp = e.M[21].double(), e.zprime.double()[R:R + nz, None, None]
        one, two, up = (float(np.float32(k)) for k in (1.01, 2.01, 2.02))
        f4, f5, f6, f7, f8, f9 = s
        new = [at(v[0]) + 2 * at(M, x=-1) * (drv(f4, "x", 1) * one + drv(f7, "y", 0) * two + drv(f8, "z", 0) * zp),
               at(v[1]) + 2 * at(M, y=-1) * (drv(f7, "x", 0) * one + drv(f5, "y", 1) * two + drv(f9, "z", 0) * zp),
               at(v[2]) + 2 * at(M, z=-1) * (drv(f8, "x", 0) * one + drv(f9, "y", 0) * two + drv(f6, "z", 1) * zp)]
        for f, k in zip(v, new):
            f[inside] = k
            _mirror(f)
        a, b, c = v
        new = [one * drv(a, "x", 0), up * drv(a, "y", 1) + one * drv(b, "x", 1), zp * drv(a, "z", 1) + one * drv(c, "x", 1),
               up * drv(b, "y", 0), zp * drv(b, "z", 1) + up * drv(c, "y", 1), zp * drv(c, "z", 0)]
        for f, k in zip(d, new):
            f[inside] = k
        return v + d + [-sum((k + 2) * f for k, f in enumerate(s)) / 27.0]

    M = [f.double() for f in e.M[:21]]
    # weights of the z-mixed averages: the first seven planes of each 64-plane block take the arriving plane's
    weight = np.empty((nz, 8))
    for o in range(nz):
        m = o % 64
        for k in range(8):
            weight[o, k] = E3[max(3 - (m + k), m + k - 4) if m + k <= 6 else max(k - 4, 3 - k)]
    weight = torch.from_numpy(weight).cuda()

    def mixed_z(f, xs, ys, zs):
        xz = yz = 0.0
        for k in range(8):
            i, z, w = 7 - k, k - 3 - zs, weight[:, k, None, None]
            xz = xz + w * (at(f, z=z, x=-3 - xs + i) + at(f, z=z, x=4 - xs - i))
            yz = yz + w * (at(f, z=z, y=-3 - ys + i) + at(f, z=z, y=4 - ys - i))
        return 0.5 * xz, 0.5 * yz

    def mixed_xy(f, xs, ys):
        return 0.5 * sum(E3[i] * (at(f, y=-ys + i + 1, x=-xs + i + 1) + at(f, y=-ys + i + 1, x=-xs - i) +
                                  at(f, y=-ys - i, x=-xs + i + 1) + at(f, y=-ys - i, x=-xs - i)) for i in range(4))

    e11, e12, e13, e22, e23, e33 = d
    pre = {}
    for (a, b), f, shift in (((10, 11), e11, (1, 1, 1)), ((16, 17), e22, (1, 1, 1)), ((20, 21), e33, (1, 1, 1)),
                             ((12, 13), e12, (0, 0, 1)), ((14, 15), e13, (0, 1, 0)), ((18, 19), e23, (1, 0, 0))):
        pre[a], pre[b] = mixed_z(f, *shift)

    def m(k):
        return at(M[k - 1])

    x12, a11, a22, a33 = mixed_xy(e12, 0, 0), mixed_xy(e11, 1, 1), mixed_xy(e22, 1, 1), mixed_xy(e33, 1, 1)
    x23, y13 = mixed_xy(e23, 1, 0), mixed_xy(e13, 0, 1)
    i11, i12, i13, i22, i23, i33 = (at(f) for f in d)
    rates = [m(1) * i11 + m(2) * i22 + m(3) * i33 + m(6) * x12 + m(5) * pre[14] + m(4) * pre[19],
             m(2) * i11 + m(7) * i22 + m(8) * i33 + m(11) * x12 + m(10) * pre[14] + m(9) * pre[19],
             m(3) * i11 + m(8) * i22 + m(12) * i33 + m(15) * x12 + m(14) * pre[14] + m(13) * pre[19],
             m(6) * a11 + m(11) * a22 + m(15) * a33 + m(20) * pre[15] + m(18) * pre[18] + m(21) * i12,
             m(5) * pre[10] + m(10) * pre[16] + m(14) * pre[20] + m(20) * pre[13] + m(17) * x23 + m(19) * i13,
             m(4) * pre[11] + m(9) * pre[17] + m(13) * pre[21] + m(18) * pre[12] + m(17) * y13 + m(16) * i23]
    for f, k in zip(s, rates):
        f[inside] += k
    full = []
    for k in range(10, 22):
        f = torch.zeros_like(s[0])
        f[inside] = pre[k]
        full.append(f)
    return s + full


def exact(case, seed):
    if case["kind"] in ("stress", "velocity"):
        return _exact_elastic(case, seed)
    out = _Exact(case, seed).shot(seed)
    return [v.cpu().numpy() for v in out] if case["kind"] == "shot" else out
