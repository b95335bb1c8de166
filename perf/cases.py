"""What is measured: the calls a user of this framework makes, from a right-hand
side of a few hundred elements to a run of 400,000, through the public entry
points (``dgcom_gb300.device``, ``.ensemble``, ``.adjoint``).

A case is a dict of plain values with a ``kind``:

- ``rhs``      the right-hand side of a device state, read back to the host
               (a host that keeps its own time integrator);
- ``step``     one CFL step of a state held on the host (upload, step, read back);
- ``run``      a case run: upload, steps over a time span with the state read
               back at every output interval, the final state; ``levels`` > 0
               is local time stepping, ``weather`` a storm's forcing;
- ``ensemble`` independent members of mixed size and order, advanced together;
- ``adjoint``  a station misfit's forward and reverse sweeps: its gradients.

Meshes are the repository's own generators: ``channel``, the tidal channel
(nx × ny affine quads, its head a drying flat), and ``coast``, the coastal box
(an unstructured, depth-graded quad paving, none of it affine; with
``islands`` > 0 part of it is dry or drying). The mesh and its bed belong to the
case; the state and the tide's phases come from the seed."""

from __future__ import annotations

import math

import numpy as np
import torch

from dgcom_gb300 import abi, cases, tides
from dgcom_gb300.adjoint import Adjoint
from dgcom_gb300.device import DeviceRun, SWEPhysics2D
from dgcom_gb300.ensemble import Ensemble
from dgcom_gb300.mesh import TAG_OPEN

MESH_SEED = 2026
START = 7200.0  # simulation time of every state, after the tide's one-hour ramp
CHANNEL = (50_000.0, 5_000.0)


def listed():
    return [
        # the smallest call: a few hundred elements, launches and latency
        dict(name="rhs channel 320 N2", kind="rhs", mesh="channel", nx=40, ny=8, order=2),
        # a host's own integrator on an ordinary unstructured mesh, all wet
        dict(name="rhs coast 30k N3", kind="rhs", mesh="coast", elements=30_011, order=3,
             islands=0),
        # the highest order
        dict(name="rhs coast 7k N4", kind="rhs", mesh="coast", elements=7_003, order=4,
             islands=0),
        # a host-held state stepped through the device, all wet
        dict(name="step coast 60k N3", kind="step", mesh="coast", elements=60_013, order=3,
             islands=0),
        # the tidal channel of the case files with its drying flat: small
        # steps, many of them, output every ten minutes
        dict(name="run channel 4k N2", kind="run", mesh="channel", nx=200, ny=20, order=2,
             span=1200.0, interval=600.0, scheme=3, levels=0, weather=False),
        # an ordinary coastal run with islands
        dict(name="run coast 50k N3", kind="run", mesh="coast", elements=50_021, order=3,
             islands=2, span=20.0, interval=10.0, scheme=3, levels=0, weather=False),
        # the largest: the headline's mesh family at 400,000 quads
        dict(name="run coast 400k N3", kind="run", mesh="coast", elements=400_009, order=3,
             islands=12, span=12.0, interval=12.0, scheme=3, levels=0, weather=False),
        # linear elements under a storm, the four-stage scheme
        dict(name="run coast 90k N1 storm", kind="run", mesh="coast", elements=90_001, order=1,
             islands=3, span=60.0, interval=30.0, scheme=43, levels=0, weather=True),
        # local time stepping
        dict(name="run coast 120k N3 levels", kind="run", mesh="coast", elements=120_011, order=3,
             islands=4, span=24.0, interval=24.0, scheme=3, levels=3, weather=False),
        # a batch of small members, orders 2 and 3
        dict(name="ensemble 24", kind="ensemble", members=24, smallest=400, largest=8000,
             steps=40),
        # the adjoint of a drying channel, every state stored
        dict(name="adjoint channel 6k N3", kind="adjoint", mesh="channel", nx=240, ny=24, order=3,
             steps=40, stations=20, every=0),
        # the adjoint of a coastal box, checkpointed
        dict(name="adjoint coast 40k N3", kind="adjoint", mesh="coast", elements=40_009, order=3,
             islands=2, steps=24, stations=30, every=6),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["rhs", "step", "run", "run", "run", "ensemble", "adjoint"])
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(3, 40), smallest=log(200, 1000),
                    largest=log(2000, 12_000), steps=rng.randint(10, 40))
    mesh = rng.choice(["channel", "coast", "coast"])
    order = rng.choice([1, 2, 2, 3, 3, 3, 4])
    # nodes rather than elements span the range, so that the orders share it
    top = {"rhs": 600_000, "step": 2_000_000, "run": 4_000_000, "adjoint": 500_000}[kind]
    elements = max(160, log(3_000, top) // (order + 1) ** 2)
    case = dict(kind=kind, mesh=mesh, order=order)
    if mesh == "channel":
        ny = max(4, int(round(math.sqrt(elements / 10.0))) + rng.randint(-1, 1))
        case |= dict(nx=max(40, elements // ny + rng.randint(0, 7)), ny=ny)
    else:
        case |= dict(elements=max(500, elements),
                     islands=0 if kind in ("rhs", "step") else rng.randint(0, 4))
    if kind == "run":
        levels = rng.choice([0, 0, 0, 2, 3])
        scheme = 3 if levels else rng.choice([3, 3, 43])
        steps = rng.randint(10, 60)
        span = round(steps * _dt(case), 2)
        case |= dict(span=span, interval=round(span / rng.choice([1, 2, 3]), 3), scheme=scheme,
                     levels=levels,
                     weather=_elements(case) * (order + 1) ** 2 < 800_000 and rng.random() < 0.4)
    if kind == "adjoint":
        case["order"] = rng.choice([2, 3])
        case |= dict(steps=rng.randint(6, 30), stations=rng.randint(2, 40),
                     every=rng.choice([0, 0, 5]))
    return case


# ---------------------------------------------------------------------------
# sizes

def _elements(case):
    return case["nx"] * case["ny"] if case["mesh"] == "channel" else case["elements"]


def _dt(case):
    """About the CFL step (CFL ½): the element size over the gravity wave's
    speed in the deepest water."""
    if case["mesh"] == "channel":
        size = min(CHANNEL[0] / case["nx"], CHANNEL[1] / case["ny"])
        return 0.5 * size / ((2 * case["order"] + 1) * math.sqrt(9.81 * 20.0))
    return 0.5 * 90.0 / ((2 * case["order"] + 1) * math.sqrt(9.81 * 250.0))


def work(case):
    """A pass reads each state, bed and element table entry of a stage once and
    writes each result once: per node-stage at N = 3 77.5 B (read the state's
    three fields, the step's start from the second stage on, write three
    fields, the bed, the corners, the face links and Manning's n), and ≈ 180
    FP64 operations (fluxes, sources, update)."""
    stages = 3
    if case["kind"] == "ensemble":
        mean = (case["largest"] - case["smallest"]) / math.log(case["largest"] / case["smallest"])
        nodes, count = case["members"] * mean * 12.5, case["steps"]
        io = 48.0
    else:
        nodes = _elements(case) * (case["order"] + 1) ** 2
        io = 24.0
        if case["kind"] == "rhs":
            return {"bytes": nodes * 80.0, "flops": nodes * 150.0}
        if case["kind"] == "step":
            count, io = 1, 48.0
        elif case["kind"] == "adjoint":
            # the forward, and its reverse at about twice its work
            count = 3 * case["steps"]
            io = 24.0 + 40.0
        else:
            count = max(1.0, case["span"] / _dt(case))
            io = 24.0 * (2 + case["span"] / case["interval"])
            stages = 4 if case["scheme"] == 43 else 3
            if case["levels"]:
                count *= 0.6  # most elements step at a multiple of the smallest step
    return {"bytes": nodes * (count * stages * 77.5 + io), "flops": nodes * count * stages * 180.0}


# ---------------------------------------------------------------------------
# inputs

_MESHES = {}  # the last cases' meshes and beds, as a program keeps its domain


def _domain(case):
    key = tuple(sorted((k, case.get(k)) for k in ("mesh", "nx", "ny", "elements", "order",
                                                  "islands")
                       if case.get(k) is not None))
    if key not in _MESHES:
        if len(_MESHES) >= 2:
            _MESHES.pop(next(iter(_MESHES)))
        if case["mesh"] == "channel":
            made = cases.tidal_channel(case["nx"], case["ny"], case["order"])
        else:
            scale = math.sqrt(case["elements"] / 1e6)
            made = cases.coastal_box(case["elements"], case["order"], MESH_SEED,
                                     lx=200_000.0 * scale, ly=150_000.0 * scale,
                                     n_islands=case["islands"],
                                     island_radius=(min(1000.0, 15_000.0 * scale),
                                                    min(5000.0, 30_000.0 * scale)))
        _MESHES[key] = made
    return _MESHES[key]


def _form(case, seed):
    """The case's physics with the seed's tide, and its flowing state."""
    made = _domain(case)
    form = made.form
    rng = np.random.default_rng(seed)
    bc = form.boundaries[TAG_OPEN]
    names = ["M2"] if case["mesh"] == "channel" else [n for n, _ in cases.COASTAL_TIDE]
    amps = [1.0] if case["mesh"] == "channel" else [a for _, a in cases.COASTAL_TIDE]
    bc.constituents = [tides.constituent(n, a, p)
                       for n, a, p in zip(names, amps, rng.uniform(0.0, 360.0, len(names)))]
    form.atmosphere = None
    if case.get("weather"):
        form.atmosphere = cases.synthetic_atmosphere(form, t0=0.0, t1=4 * 3600.0, dt_snap=7200.0,
                                                     seed=int(seed) % (1 << 31))
    return form, _state(form, rng)


def _state(form, rng):
    """Waves of decimetres over the bed with currents of decimetres a second,
    no water on land."""
    x, y = (p.reshape(-1) for p in form.positions())
    lx, ly = max(np.ptp(x), 1.0), max(np.ptp(y), 1.0)
    bed = form.bathymetry.reshape(-1)

    def wave(scale):
        out = np.zeros_like(x)
        for _ in range(3):
            kx, ky = rng.uniform(0.5, 4.0, 2) * (2.0 * math.pi)
            out += rng.uniform(0.2, 1.0) * np.cos(kx * x / lx + ky * y / ly
                                                  + rng.uniform(0.0, 2.0 * math.pi))
        return scale * out

    h = np.maximum(wave(0.15) - bed, 0.0)
    wet = h > 0.05
    u, v = wave(0.12), wave(0.08)
    return h, np.where(wet, h * u, 0.0), np.where(wet, h * v, 0.0)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        rng = np.random.default_rng(seed)
        made = cases.ensemble_members(case["members"], MESH_SEED,
                                      (case["smallest"], case["largest"]))
        for m in made:
            bc = m.form.boundaries[TAG_OPEN]
            bc.constituents = [tides.constituent("M2", 1.0, rng.uniform(0.0, 360.0))]
        return dict(case=case, handle=Ensemble([m.form for m in made]),
                    state=[_state(m.form, rng) for m in made])
    form, q = _form(case, seed)
    if kind == "adjoint":
        rng = np.random.default_rng(seed + 1)
        lo, hi = form.mesh.vertices.min(axis=0), form.mesh.vertices.max(axis=0)
        at = lo + (hi - lo) * rng.uniform(0.03, 0.6, (case["stations"], 2))
        handle = Adjoint(form, case["steps"], at, t_start=START, checkpoint_every=case["every"])
        seen = 0.2 * rng.standard_normal((case["steps"], case["stations"]))
        return dict(case=case, handle=handle, state=q, seen=seen)
    handle = SWEPhysics2D(form)
    if kind == "rhs":
        handle.upload(*q)
    return dict(case=case, handle=handle, state=tuple(q))


def run(state):
    case, handle, q = state["case"], state["handle"], state["state"]
    kind = case["kind"]
    if kind == "rhs":
        return handle.compute_rhs_into(START)
    if kind == "step":
        # the host keeps its state: a step of a copy leaves it as it was
        out = [x.copy() for x in q]
        dt = handle.step_host(START, 0.5, *out)
        return {"dt": np.array([dt]), "q": out}
    if kind == "run":
        handle.upload(*q)
        report = handle.run_with_callback(
            DeviceRun(span=(START, START + case["span"]), interval=case["interval"],
                      scheme=abi.SSP_RK43 if case["scheme"] == 43 else abi.SSP_RK3,
                      levels=case["levels"]))
        return {"q": handle.download(), "dt": np.array([report.dt_min, report.dt_max]),
                "steps": report.n_steps}
    if kind == "ensemble":
        for m, qm in enumerate(q):
            handle.upload(m, *qm)
        reports, _ = handle.run(case["steps"], 0.5, t_start=START)
        fields = [handle.download(m) for m in range(handle.n_members)]
        return {"h": np.concatenate([f[0] for f in fields]),
                "hu": np.concatenate([f[1] for f in fields]),
                "hv": np.concatenate([f[2] for f in fields]),
                "t": np.array([r.final_time for r in reports])}
    misfit, eta, dts = handle.forward(q, eta_obs=state["seen"])
    g = handle.reverse()
    return {"J": np.array([misfit]), "eta": eta, "dt": dts, "h0": g.h0, "hu0": g.hu0,
            "hv0": g.hv0, "bed": g.bed, "manning": g.manning, "tide": g.tide}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits: states that are wet everywhere (the coastal
# box without islands), under the uniform tide

def exact(case, seed):
    wet = case["kind"] in ("rhs", "step", "run") and case["mesh"] == "coast" \
        and case["islands"] == 0 and not case.get("weather") and not case.get("levels")
    if not wet:
        return None
    steps = case.get("span", 0.0) / _dt(case)
    if _elements(case) * (case["order"] + 1) ** 2 * max(1.0, steps) > 4e7:
        return None
    form, q = _form(case, seed)
    model = _Wet(form)
    q = torch.stack([torch.as_tensor(x) for x in q]).reshape(3, -1, model.n1, model.n1)
    q = q.to(model.device)
    if case["kind"] == "rhs":
        return tuple(x.reshape(-1).cpu().numpy() for x in model.rhs(q, START))
    scheme = case.get("scheme", 3)
    t, end, small, large, count = START, math.inf, math.inf, 0.0, 0
    if case["kind"] == "run":
        end = START + case["span"]
    while t < end:
        dt = model.step_size(q, 0.5, scheme)
        small, large = min(small, dt), max(large, dt)
        # the run lands on every output time
        k = math.floor((t - START) / case["interval"] + 1e-9) + 1 if end < math.inf else 0
        target = min(START + k * case["interval"], end) if k else math.inf
        landed = t + dt * (1.0 + 1e-9) >= target
        q = model.step(q, t, target - t if landed else dt, scheme)
        t = target if landed else t + dt
        count += 1
        if case["kind"] == "step":
            break
    fields = tuple(x.reshape(-1).cpu().numpy() for x in q)
    if case["kind"] == "step":
        return {"dt": np.array([small]), "q": list(fields)}
    return {"q": fields, "dt": np.array([small, large]), "steps": count}


class _Wet:
    """The split-form shallow-water equations on wet quads: flux differencing
    in the element, hydrostatic reconstruction with HLL between elements,
    walls, a tide on the open side, Coriolis and point-implicit Manning
    friction. A node is [element][s][r]."""

    def __init__(self, form):
        self.device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.form, self.g, self.n1 = form, form.g, form.order + 1
        n1 = self.n1

        def put(a):
            return torch.as_tensor(np.ascontiguousarray(a), device=self.device)

        # Gauss–Lobatto–Legendre points, weights and derivative matrix
        p = np.polynomial.legendre.Legendre.basis(form.order)
        x = np.concatenate([[-1.0], np.sort(p.deriv().roots().real), [1.0]])
        w = 2.0 / (form.order * (form.order + 1) * p(x) ** 2)
        bary = 1.0 / np.array([np.prod(x[j] - np.delete(x, j)) for j in range(n1)])
        d = np.zeros((n1, n1))
        for i in range(n1):
            for j in range(n1):
                if i != j:
                    d[i, j] = bary[j] / bary[i] / (x[i] - x[j])
            d[i, i] = -d[i].sum()
        self.w, self.d = put(w), put(d)
        # the bilinear map
        c = form.mesh.corners()
        r, s = np.meshgrid(x, x)
        r, s = r[None], s[None]
        cx, cy = (c[:, :, k, None, None] for k in (0, 1))
        x_r = 0.25 * ((1 - s) * (cx[:, 1] - cx[:, 0]) + (1 + s) * (cx[:, 2] - cx[:, 3]))
        y_r = 0.25 * ((1 - s) * (cy[:, 1] - cy[:, 0]) + (1 + s) * (cy[:, 2] - cy[:, 3]))
        x_s = 0.25 * ((1 - r) * (cx[:, 3] - cx[:, 0]) + (1 + r) * (cx[:, 2] - cx[:, 1]))
        y_s = 0.25 * ((1 - r) * (cy[:, 3] - cy[:, 0]) + (1 + r) * (cy[:, 2] - cy[:, 1]))
        det = x_r * y_s - x_s * y_r
        self.det = put(det)
        self.m = [[put(y_s), put(-x_s)], [put(-y_r), put(x_r)]]  # J∇r, J∇s
        self.mass = put(w[None, :, None] * w[None, None, :] * det)
        edge = np.zeros((n1, n1), bool)
        edge[[0, -1], :] = edge[:, [0, -1]] = True
        self.edge = put(edge)
        self.b = put(form.bathymetry.reshape(-1, n1, n1))
        # faces in their own direction round the element: south, east, north, west
        self.at = [(np.zeros(n1, int), np.arange(n1)), (np.arange(n1), np.full(n1, n1 - 1)),
                   (np.full(n1, n1 - 1), np.arange(n1)[::-1].copy()),
                   (np.arange(n1)[::-1].copy(), np.zeros(n1, int))]
        nrm = []
        for f, (jj, aa) in enumerate(self.at):
            e0, e1 = c[:, f], c[:, (f + 1) % 4]
            t = 0.5 * (e1 - e0)
            nrm.append(np.stack([t[:, 1], -t[:, 0]], axis=1))
        nrm = np.stack(nrm, axis=1)
        sj = np.hypot(nrm[..., 0], nrm[..., 1])
        self.sj, self.nx, self.ny = put(sj), put(nrm[..., 0] / sj), put(nrm[..., 1] / sj)
        # each face's neighbour (element · 4 + face), −1 at the boundary
        quads = form.mesh.elements
        a, e = quads, np.roll(quads, -1, axis=1)
        key = (np.minimum(a, e) * (quads.max() + 1) + np.maximum(a, e)).reshape(-1)
        order = np.argsort(key, kind="stable")
        same = np.flatnonzero(key[order][1:] == key[order][:-1])
        other = np.full(key.size, -1)
        other[order[same]], other[order[same + 1]] = order[same + 1], order[same]
        self.other = put(other)
        self.open = put((form.mesh.face_tags.reshape(-1) == TAG_OPEN) & (other < 0))

    def faces(self, f):
        """A field's values on the four faces: [element · 4 + face][node]."""
        return torch.stack([f[:, j, a] for j, a in self.at], dim=1).reshape(-1, self.n1)

    def across(self, own):
        """The neighbour's values at the same points (its face runs the other
        way); the face's own at the boundary."""
        got = own[self.other.clamp(min=0)].flip(1)
        return torch.where((self.other < 0)[:, None], own, got)

    def rhs(self, q, t):
        g, n1 = self.g, self.n1
        h, hu, hv = q
        u, v, b = hu / h, hv / h, self.b
        out = [torch.zeros_like(h) for _ in range(3)]
        # the two-point fluxes along each line, but for the diagonal: it and
        # the face's own flux cancel (summation by parts)
        for axis, (mx, my) in ((2, self.m[0]), (1, self.m[1])):
            def ends(f):
                return (f.unsqueeze(3), f.unsqueeze(2)) if axis == 2 else \
                    (f.unsqueeze(2), f.unsqueeze(1))

            def mean(f):
                l, r = ends(f)
                return 0.5 * (l + r)

            jx, jy = mean(mx), mean(my)
            mass = mean(hu) * jx + mean(hv) * jy
            hl, hr = ends(h)
            pressure = 0.5 * g * hl * hr
            off = 2.0 * (self.d - torch.diag(torch.diag(self.d)))
            dd = off if axis == 2 else off[:, :, None]
            for k, f in enumerate((mass, mass * mean(u) + pressure * jx,
                                   mass * mean(v) + pressure * jy)):
                out[k] -= (dd * f).sum(dim=3 if axis == 2 else 2)

            def slope(f):
                return torch.einsum("ac,ksc->ksa" if axis == 2 else "ac,kcr->kar", self.d, f)

            out[1] -= 0.5 * g * h * (mx * slope(b) + slope(b * mx))
            out[2] -= 0.5 * g * h * (my * slope(b) + slope(b * my))
        # numerical fluxes
        hi, ui, vi, bi = (self.faces(f) for f in (h, u, v, b))
        nx, ny = self.nx.reshape(-1, 1), self.ny.reshape(-1, 1)
        he, ue, ve, be = (self.across(f) for f in (hi, ui, vi, bi))
        wall = ((self.other < 0) & ~self.open)[:, None]
        un = ui * nx + vi * ny
        ue = torch.where(wall, ui - 2.0 * un * nx, ue)
        ve = torch.where(wall, vi - 2.0 * un * ny, ve)
        f = self.hydrostatic(hi, ui, vi, bi, he, ue, ve, be, nx, ny)
        o = self.open
        if bool(o.any()):
            made = self.tide(hi[o], ui[o], vi[o], bi[o], nx[o], ny[o], t)
            for k in range(3):
                f[k][o] = made[k]
        for k in range(3):
            flux = f[k].reshape(-1, 4, n1)
            for face, (j, a) in enumerate(self.at):
                out[k][:, j, a] -= self.sj[:, face, None] / self.w[0] * flux[:, face]
        r = [x / self.det for x in out]
        f0 = self.form.coriolis_f0
        r[1] = r[1] + f0 * hv
        r[2] = r[2] - f0 * hu
        return torch.stack(r)

    def hydrostatic(self, ha, ua, va, ba, hb, ub, vb, bb, nx, ny):
        g = self.g
        face = torch.maximum(ba, bb)
        sa, sb = (ha + ba - face).clamp(min=0.0), (hb + bb - face).clamp(min=0.0)
        na, ta = ua * nx + va * ny, -ua * ny + va * nx
        nb, tb = ub * nx + vb * ny, -ub * ny + vb * nx
        ra, rb = sa.sqrt(), sb.sqrt()
        ca, cb = math.sqrt(g) * ra, math.sqrt(g) * rb
        roe = (ra * na + rb * nb) / (ra + rb)
        c = (g * 0.5 * (sa + sb)).sqrt()
        sl, sr = torch.minimum(na - ca, roe - c), torch.maximum(nb + cb, roe + c)
        fa = (sa * na, sa * na * na + 0.5 * g * sa * sa, sa * na * ta)
        fb = (sb * nb, sb * nb * nb + 0.5 * g * sb * sb, sb * nb * tb)
        jump = (sb - sa, sb * nb - sa * na, sb * tb - sa * ta)
        f = []
        for x, y, z in zip(fa, fb, jump):
            star = (sr * x - sl * y + sl * sr * z) / (sr - sl)
            f.append(torch.where(sl >= 0.0, x, torch.where(sr <= 0.0, y, star)))
        p = 0.5 * g * (ha * ha - sa * sa)
        return [f[0], f[1] * nx - f[2] * ny + p * nx, f[1] * ny + f[2] * nx + p * ny]

    def tide(self, h, u, v, b, nx, ny, t):
        """The characteristic boundary state of the tide's elevation, sub-critical."""
        g = self.g
        bc = self.form.boundaries[TAG_OPEN]
        he = (tides.elevation(bc.constituents, t, bc.mean_elevation, bc.ramp_duration)
              - b).clamp(min=0.0)
        un, ut = u * nx + v * ny, -u * ny + v * nx
        out, into = un + 2.0 * (g * h).sqrt(), -2.0 * (g * he).sqrt()
        c = 0.25 * (out - into)
        hb, nb = c * c / g, 0.5 * (out + into)
        ub, vb = nb * nx - ut * ny, nb * ny + ut * nx
        mass, p = hb * ub * nx + hb * vb * ny, 0.5 * g * hb * hb
        return [mass, mass * ub + p * nx, mass * vb + p * ny]

    def stage(self, base, q, t, a, b, c):
        new = a * base + b * q + c * self.rhs(q, t)
        h, n = q[0], self.form.manning_n
        speed = ((q[1] / h) ** 2 + (q[2] / h) ** 2).sqrt()
        factor = 1.0 / (1.0 + c * self.g * n * n * speed / new[0] ** (4.0 / 3.0))
        new[1] *= factor
        new[2] *= factor
        return new

    def step(self, q, t, dt, scheme):
        table = [(1.0, 0.0, 1.0, 0.0), (0.75, 0.25, 0.25, 1.0), (1 / 3, 2 / 3, 2 / 3, 0.5)]
        if scheme == 43:
            table = [(1.0, 0.0, 0.5, 0.0), (0.0, 1.0, 0.5, 0.5), (2 / 3, 1 / 3, 1 / 6, 1.0),
                     (0.0, 1.0, 0.5, 0.5)]
        x = q
        for a, b, c, at in table:
            x = self.stage(q, x, t + at * dt, a, b, c * dt)
        return x

    def step_size(self, q, cfl, scheme):
        """The smallest element step: CFL over the largest wave rate of the
        element's nodes and its neighbours' face nodes, kept to the bound
        that keeps cell means positive."""
        n, g = self.form.order, self.g
        h, u, v = q[0], q[1] / q[0], q[2] / q[0]
        c = (g * h).sqrt()
        grad = [[m / self.det for m in row] for row in self.m]

        def rate(c, u, v, gr):
            return sum(0.25 * ((u * x + v * y).abs() + c * (x * x + y * y).sqrt()) for x, y in gr)

        most = rate(c, u, v, grad).amax(dim=(1, 2))
        cf, uf, vf = (self.across(self.faces(f)) for f in (c, u, v))
        gf = [[self.faces(x) for x in row] for row in grad]
        beyond = torch.where((self.other < 0)[:, None], 0.0, rate(cf, uf, vf, gf))
        most = torch.maximum(most, beyond.reshape(h.shape[0], -1).amax(dim=1))
        rk43 = scheme == 43
        bound = (2.0 if rk43 else 1.0) * (2 * n + 1) / (2.0 * n * (n + 1))
        linear = ((2.2, 1.51, 1.15, 0.93) if rk43 else (1.6, 1.04, 0.73, 0.56))[n - 1]
        water, weight = (self.mass * h), self.mass

        def ratio(m):
            return m.sum(dim=(1, 2)) / (m * self.edge).sum(dim=(1, 2))

        rho = (0.9 * torch.minimum(ratio(water), ratio(weight))).clamp(min=1.0)
        own = torch.minimum((bound * rho).clamp(max=max(bound, 0.9 * linear)),
                            torch.full_like(rho, cfl))
        return float((own / ((2 * n + 1) * most)).min())
