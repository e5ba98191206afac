"""The work that users of this package have it do, as cases for timing: fields at points, RK4
tracks, one optimiser generation and adjoint gradients, through the public entry points.

Sizes are those of the package's own workloads (cctpy_gb300/workloads.py), of cctpy's speed
test and of the tests, from one point or a handful of protons to the full field map and the
4096-proton gantry section.  `draw` gives further cases of the same ranges.
"""
import math

import numpy as np
import torch

from cctpy_gb300 import GPU_ACCELERATOR, HUST_SC_GANTRY, P3, adjoint, engine, optim, workloads as W
from cctpy_gb300.particles import ParticleFactory, PhaseSpaceParticle, RunningParticle, particles_to_array

PAIR_FLOPS = 26                 # of one (point, segment) term, |r|^-1 as one operation
SECTION_START = 1.9             # m: end of the second section's entrance drift
MAX_PAIRS = {"f64": 2.0e9, "f32c": 9.0e10}     # of one drawn case


def listed():
    return [
        # one field value asked of a magnet object, as cctpy's magnetic_field_at is used: the smallest call
        dict(name="field_point_f64", kind="field", magnet="dipole", part=360, n=1, precision="f64", io="host"),
        # the field along a design orbit, 1 cm apart over the second bending section (the default precision)
        dict(name="field_axis_f64", kind="field", magnet="section", part=120, n=351, precision="f64", io="host"),
        # an FP64 field map of moderate size, an odd number of points
        dict(name="field_map_f64", kind="field", magnet="dipole", part=360, n=30031, precision="f64", io="host"),
        # some hundred points in the finely divided gantry section, resident on the device
        dict(name="field_line_f32c", kind="field", magnet="section", part=600, n=517, precision="f32c", io="device"),
        # the field-map workload: 2^20 points x 46 080 segments
        dict(name="field_map_f32c", kind="field", magnet="dipole", part=360, n=1 << 20, precision="f32c",
             io="device"),
        # a few protons through the section as ParticleRunner.run_only tracks them (FP64), 1 m at 10 mm
        dict(name="track_few_f64", kind="track", magnet="section", part=120, n=5, steps=100, step_mm=10.0,
             precision="f64"),
        # the single-dipole workload: 32 protons over the whole arc at 1 mm
        dict(name="track_arc_f32c", kind="track", magnet="dipole", part=360, n=32, steps=374, step_mm=1.0,
             precision="f32c"),
        # the gantry-section workload, a slice of its steps: 4096 protons x 597 600 segments
        dict(name="track_gantry_f32c", kind="track", magnet="section", part=600, n=4096, steps=10, step_mm=1.0,
             precision="f32c"),
        # cctpy's own GPU speed test through the drop-in accelerator: 100 beamlines x 16 protons, 20 mm steps
        dict(name="speed_test_f32c", kind="speed", designs=100, n=16, step_mm=20.0, steps=544),
        # one optimiser generation: beamlines built, segments, tracking of 96 protons at 50 mm, eleven objectives
        dict(name="generation_f32c", kind="generation", designs=12, part=120, n=96, step_mm=50.0, steps=142),
        # gradient of the spot size, a few protons, in the default precision
        dict(name="adjoint_f64", kind="adjoint", designs=1, part=120, n=16, steps=10, step_mm=5.0, checkpoint=0,
             precision="f64"),
        # the design-gradient workload, a slice: some designs, checkpoints with recompute
        dict(name="adjoint_f32c", kind="adjoint", designs=6, part=120, n=512, steps=8, step_mm=1.0, checkpoint=4,
             precision="f32c"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["field", "field", "track", "track", "track", "speed", "generation", "adjoint"])
    precision = rng.choice(["f64", "f32c"])
    most = MAX_PAIRS[precision]
    if kind == "field":
        magnet = rng.choice(["dipole", "section"])
        part = rng.choice([360]) if magnet == "dipole" else rng.choice([60, 120, 360, 600])
        segs = _segments(magnet, part)
        n = _log(rng, 1, min(1 << 20, most / segs))
        return dict(kind=kind, magnet=magnet, part=part, n=n, precision=precision, io=rng.choice(["host", "device"]))
    if kind == "track":
        magnet = rng.choice(["dipole", "section"])
        part = 360 if magnet == "dipole" else rng.choice([60, 120, 360, 600])
        segs = _segments(magnet, part)
        n = _log(rng, 1, 512 if precision == "f64" else 4096)
        most = min(max(most / (4.0 * segs * max(n, 32)), 4), 374)
        return dict(kind=kind, magnet=magnet, part=part, n=n, steps=_log(rng, 3, most),
                    step_mm=1.0 if magnet == "dipole" else rng.choice([1.0, 2.0]), precision=precision)
    if kind == "speed":
        return dict(kind=kind, designs=_log(rng, 1, 100), n=_log(rng, 1, 16), step_mm=rng.choice([20.0, 50.0]),
                    steps=rng.randint(110, 217))
    if kind == "generation":
        return dict(kind=kind, designs=_log(rng, 2, 12), part=rng.choice([60, 120]), n=8 * _log(rng, 2, 12),
                    step_mm=50.0, steps=rng.randint(40, 142))
    n, designs = (_log(rng, 2, 40), 1) if precision == "f64" else (_log(rng, 8, 512), _log(rng, 1, 6))
    return dict(kind=kind, designs=designs, part=rng.choice([60, 120]), n=n, steps=rng.randint(2, 8),
                step_mm=rng.choice([1.0, 5.0]), checkpoint=rng.choice([0, 3, 4]), precision=precision)


# ---------------------------------------------------------------- inputs
def _segments(magnet, part):
    return 128 * part if magnet == "dipole" else 996 * part


def _length(case):
    # half a step short of the last step's end, so that the step count is no matter of rounding
    return (case["steps"] - 0.5) * case["step_mm"] * 1e-3


def _magnet(magnet, part):
    if magnet == "dipole":
        return W.build_single_dipole()
    bl = W.build_gantry_section(part_per_winding=part)
    return bl, bl


def _beam(trajectory, s, n, seed, kinetic_MeV, gaussian=True):
    """(n, 10) proton records around the ideal particle at arc length s."""
    ideal = ParticleFactory.create_proton_along(trajectory, s, kinetic_MeV)
    rows = W.gaussian_phase_space(n, seed) if gaussian else W.uniform_ellipse_phase_space(n, seed)
    return particles_to_array(ParticleFactory.create_from_phase_space_particles(
        ideal, ideal.get_natural_coordinate_system(), [PhaseSpaceParticle(*map(float, r)) for r in rows]))


def _points(case, trajectory, seed):
    if case["magnet"] == "dipole":
        return W.field_map_points(case["n"], seed)
    rng = np.random.default_rng(seed)
    s = np.sort(rng.uniform(0.0, 0.99 * trajectory.get_length(), case["n"]))
    pts = np.array([(p.x, p.y, 0.0) for p in (trajectory.point_at(float(x)) for x in s)])
    return pts + rng.uniform(-0.01, 0.01, pts.shape)


def _population(case, seed):
    return W.design_population(case["designs"], seed=seed, part_per_winding=case["part"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "field":
        traj, magnet = _magnet(case["magnet"], case["part"])
        pts = _points(case, traj, seed)
        ds = engine.design_of(magnet)
        if case["precision"] == "f32c":
            ds.packed()
        if case["io"] == "device":
            pts = torch.from_numpy(pts).cuda()
        return dict(case=case, magnet=magnet, ds=ds, points=pts)
    if kind == "track":
        traj, magnet = _magnet(case["magnet"], case["part"])
        if case["magnet"] == "dipole":
            c = W.SINGLE_DIPOLE
            ps = _beam(traj, c["drift"], case["n"], seed, c["kinetic_MeV"], gaussian=False)
        else:
            ps = _beam(traj, SECTION_START, case["n"], seed, W.GANTRY_SECTION["kinetic_MeV"])
        ds = engine.design_of(magnet)
        if case["precision"] == "f32c":
            ds.packed()
        return dict(case=case, ds=ds, particles=ps, length=_length(case))
    if kind == "speed":
        bl = W.build_speed_test_beamline()
        ps = _beam(bl, 0.0, case["n"], seed, 250.0)
        return dict(case=case, beamline=bl, accelerator=GPU_ACCELERATOR(GPU_ACCELERATOR.FLOAT32),
                    particles=[RunningParticle.from_numpy_array_data(r) for r in ps])
    if kind == "generation":
        rows = _population(case, seed)
        bl = HUST_SC_GANTRY(**rows[0]).create_second_bending_part_beamline()
        ps = _beam(bl, 0.0, case["n"], seed, 215.0)
        end = ParticleFactory.create_proton_along(bl, _length(case), 215.0)
        evaluate = optim.GenerationEvaluator(
            lambda row: HUST_SC_GANTRY(**rows[int(row[0])]).create_second_bending_part_beamline(), ps,
            _length(case), case["step_mm"] * 1e-3, end)
        return dict(case=case, rows=rows, evaluate=evaluate, particles=ps, end=end,
                    params=np.arange(case["designs"], dtype=np.float64)[:, None])
    bls = [HUST_SC_GANTRY(**r).create_second_bending_part_beamline() for r in _population(case, 3)]
    ps = _beam(bls[0], SECTION_START, case["n"], seed, 215.0)
    length = _length(case)
    frame = adjoint.exit_frame(bls[0].trajectory, SECTION_START + length, 215.0)
    ds = engine.design_set_of(bls, segments="device")
    if case["precision"] == "f32c":
        ds.packed()
    return dict(case=case, ds=ds, particles=ps, length=length, frames=np.tile(frame, (case["designs"], 1)))


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "field":
        if case["io"] == "device":
            return engine.field_at_points(state["ds"], state["points"], case["precision"])
        if case["n"] == 1 and case["precision"] == "f64":
            return np.array([state["magnet"].magnetic_field_at(P3(*state["points"][0])).to_list()])
        return state["magnet"].magnetic_field_at_points(state["points"], case["precision"])
    if kind == "track":
        return engine.track(state["ds"], state["particles"], state["length"], case["step_mm"] * 1e-3,
                            case["precision"])
    if kind == "speed":
        rows = state["accelerator"].track_multi_particle_beamline_for_magnet_with_multi_qs(
            [state["beamline"]] * case["designs"], state["particles"], _length(case), case["step_mm"] * 1e-3)
        return np.stack([particles_to_array(r) for r in rows])
    if kind == "generation":
        return state["evaluate"](state["params"])
    return adjoint.segment_gradient(state["ds"], state["particles"], state["length"], case["step_mm"] * 1e-3,
                                    state["frames"], case["checkpoint"] or None, case["precision"], on_device=True)


def work(case):
    kind = case["kind"]
    if kind == "field":
        segs = _segments(case["magnet"], case["part"])
        return dict(bytes=48 * segs + 48 * case["n"], flops=PAIR_FLOPS * segs * case["n"])
    if kind == "track":
        segs = _segments(case["magnet"], case["part"])
        return dict(bytes=48 * segs + 160 * case["n"], flops=PAIR_FLOPS * 4 * case["steps"] * segs * case["n"])
    if kind == "speed":
        pairs = 4 * case["steps"] * 24000 * case["n"] * case["designs"]
        return dict(bytes=48 * 24000 + 160 * case["n"] * case["designs"], flops=PAIR_FLOPS * pairs)
    # design_population: on average 1116 windings over its 16 layers
    segs = 1116 * case["part"] * case["designs"]
    pairs = 4 * case["steps"] * segs * case["n"]
    if kind == "generation":
        return dict(bytes=48 * segs + 160 * case["n"] * case["designs"], flops=PAIR_FLOPS * pairs)
    # forward, reverse sweep and segment gradient
    return dict(bytes=96 * segs + 160 * case["n"] * case["designs"], flops=3 * PAIR_FLOPS * pairs)


# ---------------------------------------------------------------- the same in plain torch, 64 bits
class _Field(torch.autograd.Function):
    """B(p) = sum_i kl_i x (p - p0_i) / |p - p0_i|^3, and its derivatives, in chunks."""

    @staticmethod
    def _chunks(p, kl):
        per = max(1, (1 << 22) // max(p.shape[0], 1))
        return [(i, min(i + per, kl.shape[0])) for i in range(0, kl.shape[0], per)]

    @staticmethod
    def forward(ctx, p, kl, p0):
        ctx.save_for_backward(p, kl, p0)
        out = torch.zeros_like(p)
        for a, b in _Field._chunks(p, kl):
            r = [p[:, c, None] - p0[None, a:b, c] for c in range(3)]
            w = (r[0] * r[0] + r[1] * r[1] + r[2] * r[2]).pow_(-1.5)
            k = kl[a:b].T
            for c in range(3):
                d, e = (c + 1) % 3, (c + 2) % 3
                out[:, c] += ((k[d] * r[e] - k[e] * r[d]) * w).sum(1)
        return out

    @staticmethod
    def backward(ctx, g):
        p, kl, p0 = ctx.saved_tensors
        gp, gk, gq = torch.zeros_like(p), torch.zeros_like(kl), torch.zeros_like(p0)
        for a, b in _Field._chunks(p, kl):
            r = [p[:, c, None] - p0[None, a:b, c] for c in range(3)]
            r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2]
            w = r2.pow(-1.5)
            k, v = kl[a:b].T, g.T[:, :, None]
            c3 = [v[(c + 1) % 3] * k[(c + 2) % 3] - v[(c + 2) % 3] * k[(c + 1) % 3] for c in range(3)]   # g x kl
            q = 3.0 * (c3[0] * r[0] + c3[1] * r[1] + c3[2] * r[2]) * w / r2
            for c in range(3):
                d, e = (c + 1) % 3, (c + 2) % 3
                t = c3[c] * w - q * r[c]
                gp[:, c] += t.sum(1)
                gq[a:b, c] -= t.sum(0)
                gk[a:b, c] += ((r[d] * v[e] - r[e] * v[d]) * w).sum(0)
        return gp, gk, gq


def _qs_field(rec, p):
    o, xi, yi, zi = rec[0:3], rec[3:6], rec[6:9], rec[9:12]
    length, g, s, ap = (float(v) for v in rec[12:16])
    x, y, z = ((p - o) @ xi, (p - o) @ yi, (p - o) @ zi)
    inside = (z >= 0) & (z <= length) & (x * x + y * y <= ap * ap)
    bx = torch.where(inside, g * y + s * x * y, 0.0)
    by = torch.where(inside, g * x + 0.5 * s * (x * x - y * y), 0.0)
    return bx[:, None] * xi + by[:, None] * yi


def _field64(p, kl, p0, qs):
    b = _Field.apply(p, kl, p0)
    for rec in qs:
        b = b + _qs_field(rec, p)
    return b


def _track64(rec, length, footstep, kl, p0, qs):
    """RK4 as the reference steps it: dt = length / speed / ceil(length / footstep)."""
    rec = torch.as_tensor(rec, device=kl.device)
    p, v, kq, speed = rec[:, 0:3], rec[:, 3:6], (rec[:, 7] / rec[:, 6])[:, None], rec[:, 8:9]
    steps = int(torch.ceil((length / speed) / (footstep / speed)).max())
    dt = length / speed / steps

    def f(p, v):
        return v, kq * torch.linalg.cross(v, _field64(p, kl, p0, qs))

    for _ in range(steps):
        p1, v1 = f(p, v)
        p2, v2 = f(p + dt / 2 * p1, v + dt / 2 * v1)
        p3, v3 = f(p + dt / 2 * p2, v + dt / 2 * v2)
        p4, v4 = f(p + dt * p3, v + dt * v3)
        p, v = p + dt / 6 * (p1 + 2 * p2 + 2 * p3 + p4), v + dt / 6 * (v1 + 2 * v2 + 2 * v3 + v4)
    return torch.cat([p, v, rec[:, 6:9], rec[:, 9:10] + length], 1)


def _winding64(m):
    """(kl, p0) of a CCT layer: points on its torus at equally spaced xi, in the global frame."""
    f = m.local_coordinate_system
    axes = torch.tensor([[a.x, a.y, a.z] for a in (f.XI, f.YI, f.ZI)], dtype=torch.float64, device="cuda")
    origin = torch.tensor([f.location.x, f.location.y, f.location.z], dtype=torch.float64, device="cuda")
    s, e = m.starting_point_in_ksi_phi_coordinate, m.end_point_in_ksi_phi_coordinate
    n = m.winding_number * m.disperse_number_per_winding
    xi = s.x + (e.x - s.x) * torch.arange(n + 1, dtype=torch.float64, device="cuda") / n
    a = math.sqrt(m.big_r ** 2 - m.small_r ** 2)
    eta = 0.5 * math.log((m.big_r + a) / (m.big_r - a))
    phi = s.y + (e.y - s.y) / (e.x - s.x) * (xi - s.x)
    for i, t in enumerate(m.tilt_angles):
        if abs(t - 90.0) > 1e-9:
            phi = phi + torch.sin((i + 1) * xi) / (math.tan(math.radians(t)) * (i + 1) * math.sinh(eta))
    d = a / (math.cosh(eta) - torch.cos(xi))
    w = origin + torch.stack([d * math.sinh(eta) * torch.cos(phi), d * math.sinh(eta) * torch.sin(phi),
                              d * torch.sin(xi)], 1) @ axes
    return 1e-7 * m.current * (w[1:] - w[:-1]), 0.5 * (w[1:] + w[:-1])


def _design64(magnets):
    parts = [_winding64(m) for m in magnets if hasattr(m, "winding_number")]
    qs = [torch.as_tensor(m.to_numpy_array(np.float64), device="cuda") for m in magnets
          if not hasattr(m, "winding_number")]
    return torch.cat([x[0] for x in parts]), torch.cat([x[1] for x in parts]), qs


def _objectives64(final, end, group):
    """The eleven objectives of a generation from one design's tracked records."""
    f = end.get_natural_coordinate_system()
    xi, yi = (np.array([a.x, a.y, a.z]) for a in (f.XI, f.YI))
    ideal = end.to_numpy_array_data(np.float64)
    dp, dv = final[:, 0:3] - ideal[0:3], final[:, 3:6] - ideal[3:6]
    v2 = (final[:, 3:6] ** 2).sum(1)
    cols = [dp @ xi, dv @ xi / np.sqrt(v2 - (dv @ xi) ** 2), dp @ yi, dv @ yi / np.sqrt(v2 - (dv @ yi) ** 2)]
    cols = [c / 0.001 for c in cols]
    wide = [np.abs(c).max() for c in cols]
    mean = [abs(math.fsum(c) / len(c)) for c in cols]
    half = [[np.ptp(c[i:i + group]) / 2 for i in range(0, len(c), group)] for c in (cols[0], cols[2])]
    return wide + mean + [abs(wide[0] - wide[2])] + [max(h) - min(h) for h in half]


def exact(case, seed):
    kind, st = case["kind"], prepare(case, seed)
    if kind in ("speed", "generation"):
        sets = [st["beamline"]] if kind == "speed" else [
            HUST_SC_GANTRY(**r).create_second_bending_part_beamline() for r in st["rows"]]
        ps = particles_to_array(st["particles"]) if kind == "speed" else st["particles"]
        finals = [_track64(ps, _length(case), case["step_mm"] * 1e-3, *_design64(bl.magnets)).cpu().numpy()
                  for bl in sets]
        if kind == "speed":
            return np.stack(finals * case["designs"])
        return np.array([_objectives64(f, st["end"], st["evaluate"].group) for f in finals])
    ds = st["ds"]
    if kind == "field":
        p = torch.as_tensor(st["points"], device="cuda")
        out = torch.cat([_field64(q, ds.kls, ds.p0s, ds.qs) for q in p.split(4096)])
        return out if case["io"] == "device" else out.cpu().numpy()
    if kind == "track":
        return _track64(st["particles"], st["length"], case["step_mm"] * 1e-3, ds.kls, ds.p0s,
                        ds.qs).cpu().numpy()[None]
    J, grads, finals = [], [], []
    for d in range(ds.n_designs):
        a, b = int(ds.h_seg_off[d]), int(ds.h_seg_off[d + 1])
        kl, p0 = (t[a:b].clone().requires_grad_() for t in (ds.kls, ds.p0s))
        qs = ds.qs[int(ds.h_qs_off[d]):int(ds.h_qs_off[d + 1])]
        fin = _track64(st["particles"], st["length"], case["step_mm"] * 1e-3, kl, p0, qs)
        frame = torch.as_tensor(st["frames"][d], device="cuda")
        at = fin[:, 0:3] - frame[0:3]
        j = ((at @ frame[3:6]) ** 2 + (at @ frame[6:9]) ** 2).mean()
        gk, gp = torch.autograd.grad(j, (kl, p0))
        J.append(float(j.detach()))
        grads.append(torch.cat([gk, gp], 1))
        finals.append(fin.detach().cpu().numpy())
    return np.array(J), torch.cat(grads), np.stack(finals)
