"""What a user of the DEM step has it do, as cases that can be timed.

Every case is a bed of spheres that a program builds once and then advances: a pass is one stepping call
(`Simulation.step` or `Simulation.steps`) followed by the read-back of the bed's state into arrays that the program keeps,
which is what a script does between two frames or two log lines. The state goes on from pass to pass, as a simulation does.
The steps of one call are few enough that 64 bits still fix the result: the slip of a sticking contact turns with every
rounding, and in a dense bed with Coulomb friction two exact computations part after some hundred steps.

Scenes (the repository's own workloads at sizes from a thousand to four million spheres):

  box     one walled cube (12 triangles) under gravity: the drop-in's typical script
  bed     a dense periodic bed on a floor, without other walls: the bulk of a packing
  hopper  a conical hopper (about 20,000 triangles) over a floor, periodic in x and z, lognormal radii
  gas     a dilute, fast periodic gas, whose neighbour lists are rebuilt every few tens of steps
  dust    micron-sized adhesive spheres in a periodic cube
  boxes   many walled cubes of uneven size stepped together, each a group with its own surface energy
  drum    a rotating drum (65,536 moving triangles), filled to two fifths

`exact` is the same step in plain torch, in 64 bits: the reference's velocity Verlet, its grid's visit counts, its contact
laws and its sphere-triangle contact, on pairs found by a sort of its own.
"""
import math

import numpy as np
import torch

import rusty_particles_gb300 as rp

VECTORS = ("position", "velocity", "angular_velocity", "acceleration", "torque")
# bytes that a particle's step cannot do without: x, v, omega read and written, radius and mass read
STEP_BYTES = 160.0
# the two half kicks and the drift, and one pair contact
STEP_FLOPS, CONTACT_FLOPS = 60.0, 150.0


def listed():
    return [
        # a script that reads the bed after every step: one call's latency
        dict(name="box-1k-step", scene="box", n=1000, steps=1, normal="hertz", tangential="coulomb"),
        # the same bed run for many steps in one call: launches and gaps
        dict(name="box-1k-run", scene="box", n=1000, steps=100, normal="hertz", tangential="coulomb"),
        # one box of the batched study by itself, an odd number of cohesive spheres
        dict(name="box-23k-sjkr", scene="box", n=23457, steps=50, normal="sjkr", tangential="coulomb"),
        # a sheared bed with tangential springs, at a size that fills the GPU about once
        dict(name="bed-164k-spring", scene="bed", n=163843, steps=20, normal="linear", tangential="linear",
             mode="physical"),
        # the benchmark's bed in the precisions and modes it is run in
        dict(name="hopper-1m", scene="hopper", n=1048576, steps=20, normal="hertz", tangential="mindlin"),
        dict(name="hopper-1m-mixed", scene="hopper", n=1048576, steps=20, normal="hertz", tangential="mindlin",
             precision="mixed"),
        dict(name="hopper-524k-physical", scene="hopper", n=524288, steps=20, normal="hertz", tangential="mindlin",
             mode="physical"),
        # fluidised flow: the rebuild of the lists weighs as much as the steps
        dict(name="gas-1m", scene="gas", n=999983, steps=40, normal="hysteretic", tangential="coulomb"),
        # fine powder: the certified contact-radius solver, and the reference's own iteration
        dict(name="dust-2m-certified", scene="dust", n=2097152, steps=8, normal="jkr", tangential="coulomb",
             solver="certified"),
        dict(name="dust-262k-newton", scene="dust", n=262144, steps=8, normal="jkr", tangential="coulomb"),
        # a parameter study: uneven boxes in one simulation
        dict(name="boxes-96", scene="boxes", n=96, steps=10, normal="sjkr", tangential="coulomb"),
        # the largest bed, in the precision that large beds are run in
        dict(name="drum-4m-mixed", scene="drum", n=4194304, steps=10, normal="hertz", tangential="coulomb",
             precision="mixed"),
    ]


def draw(rng):
    scene = rng.choice(["box", "box", "bed", "hopper", "gas", "dust", "boxes", "drum"])
    lo, hi = {"box": (500, 100_000), "bed": (20_000, 1_500_000), "hopper": (50_000, 1_200_000), "gas": (20_000, 1_500_000),
              "dust": (50_000, 2_000_000), "boxes": (8, 96), "drum": (200_000, 3_000_000)}[scene]
    n = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    case = dict(scene=scene, n=n, precision=rng.choice(["fp64", "fp64", "mixed"]))
    if scene == "dust":
        case["normal"], case["tangential"] = "jkr", "coulomb"
        case["solver"] = "certified" if n > 300_000 else rng.choice(["certified", "newton"])
    elif scene == "boxes":
        case["normal"], case["tangential"] = "sjkr", "coulomb"
    else:
        case["normal"] = rng.choice(["hertz", "hertz", "linear", "hysteretic", "sjkr"])
        case["tangential"] = rng.choice(["coulomb", "coulomb", "mindlin", "linear"])
        if case["normal"] == "sjkr":
            case["tangential"] = "coulomb"
        if case["tangential"] != "coulomb" and scene != "drum":
            case["mode"] = rng.choice(["parity", "physical"])
    case["steps"] = rng.randint(*{"box": (20, 50), "gas": (20, 40), "dust": (4, 8), "boxes": (5, 10), "drum": (5, 10)}.get(scene, (10, 20)))
    return case


# ------------------------------------------------------------------------------------------------------ scenes
def _device():
    return torch.device("cuda")


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, dtype=torch.float64, device=_device())


def _cubic(n, lo, spacing, per_axis):
    """The first n sites of a cubic lattice with per_axis sites a side, layer by layer in y."""
    i = torch.arange(n, device=_device())
    ix, iz, iy = i % per_axis, i // per_axis % per_axis, i // (per_axis * per_axis)
    return torch.stack([ix, iy, iz], 1).double().add_(0.5).mul_(spacing) + torch.tensor(lo, dtype=torch.float64, device=_device())


def _counts(boxes):
    """The spheres of each box: evenly spread over the logarithm of 2,000 to 60,000, large and small ones mixed."""
    order = sorted(range(boxes), key=lambda b: (b * 0.6180339887) % 1.0)
    counts = [0] * boxes
    for k, b in enumerate(order):
        counts[b] = int(2000 * 30.0 ** ((k + 0.5) / boxes))
    return counts


def _spheres(case):
    return sum(_counts(case["n"])) if case["scene"] == "boxes" else case["n"]


def _volume(r):
    return float((4.0 / 3.0 * math.pi * r ** 3).sum())


def _box_triangles(lo, hi):
    """The 12 triangles of a cuboid's faces, normals inward, as [12, 9] vertices."""
    out = []
    for k in range(3):
        a, b = (k + 1) % 3, (k + 2) % 3
        for side in (0, 1):
            c = []
            for u, w in ((0, 0), (1, 0), (1, 1), (0, 1)):
                p = [0.0, 0.0, 0.0]
                p[k], p[a], p[b] = (lo, hi)[side][k], (lo, hi)[u][a], (lo, hi)[w][b]
                c.append(p)
            quad = c if side == 0 else c[::-1]
            out += [quad[0] + quad[1] + quad[2], quad[0] + quad[2] + quad[3]]
    return np.array(out, np.float32)


def _quads(p00, p01, p10, p11, inside):
    """Two triangles a quad, wound so that the normals point at `inside` (a point for each quad)."""
    v = np.concatenate([np.concatenate([p00, p10, p01], 1), np.concatenate([p01, p10, p11], 1)])
    a, b, c = v[:, :3], v[:, 3:6], v[:, 6:]
    flip = (np.cross(b - a, c - a) * (np.concatenate([inside, inside]) - a)).sum(1) < 0
    v[flip] = np.concatenate([a[flip], c[flip], b[flip]], 1)
    return v.astype(np.float32)


def _revolve(radius, height, axis, n_theta):
    """Triangles of the surface of revolution through the profile points (radius, height) about `axis` (1: y, 2: z)."""
    th = np.linspace(0.0, 2.0 * np.pi, n_theta + 1)
    out = []
    for (r0, h0), (r1, h1) in zip(zip(radius[:-1], height[:-1]), zip(radius[1:], height[1:])):
        def ring(r, h, t):
            p = np.empty((n_theta, 3))
            other = (2, 0) if axis == 1 else (0, 1)
            p[:, other[0]], p[:, other[1]], p[:, axis] = r * np.cos(t), r * np.sin(t), h
            return p
        mid = np.zeros((n_theta, 3))
        mid[:, axis] = (min(height) + max(height)) / 2
        v = _quads(ring(r0, h0, th[:-1]), ring(r0, h0, th[1:]), ring(r1, h1, th[:-1]), ring(r1, h1, th[1:]), mid)
        area = np.linalg.norm(np.cross(v[:, 3:6] - v[:, :3], v[:, 6:] - v[:, :3]), axis=1)
        out.append(v[area > 1e-12])
    return np.concatenate(out)


def _settle(x, r, lo, hi, periodic, confine, rounds=120):
    """Pushes overlapping spheres apart, so that a dense start has the light overlaps of a bed at rest. The pushes are
    added as whole numbers, so that the order in which the GPU adds them changes nothing."""
    size = torch.tensor(hi, dtype=torch.float64, device=x.device) - torch.tensor(lo, dtype=torch.float64, device=x.device)
    unit = float(r.max()) * 2.0 ** -40
    for k in range(rounds):
        if k % 15 == 0:
            i, j = _pairs(x, r, 1.0, 0.2 * float(r.max()), lo, hi, periodic)
        d = _image(x[i] - x[j], size, periodic)
        dist = d.norm(dim=1).clamp_min(1e-12)
        over = (r[i] + r[j] - dist).clamp_min(0.0)
        push = (d * (0.4 * over / dist / unit).unsqueeze(1)).round_().to(torch.int64)
        total = torch.zeros_like(x, dtype=torch.int64).index_add_(0, i, push).index_add_(0, j, push, alpha=-1)
        x = confine(x + total.double() * unit)
        for a in range(3):
            if periodic[a]:
                x[:, a] = lo[a] + torch.remainder(x[:, a] - lo[a], float(size[a]))
    return x


def _scene(case, seed):
    """Everything that a program decides before it builds the simulation."""
    g = torch.Generator(device=_device()).manual_seed(int(seed) * 7919 + 17)
    n, kind = case["n"], case["scene"]
    s = dict(dt=2e-6, periodic=(False, False, False), material=(1e7, 0.3, 2500.0, 0.5, 0.5, 0.0), triangles=None, motion=None,
             groups=None, gammas=None, gravity=(0.0, -9.81, 0.0), speed=0.05, skin=None)
    if kind == "box":
        r = _uniform(g, 0.01, 0.02, n)
        side = (_volume(r) / 0.45) ** (1 / 3)
        lo, hi = (-side / 2,) * 3, (side / 2,) * 3
        m = math.ceil(n ** (1 / 3))
        x = _cubic(n, lo, side / m, m)
        gap = r.unsqueeze(1)
        x = _settle(x, r, lo, hi, s["periodic"], lambda p: torch.maximum(torch.minimum(p, side / 2 - gap), gap - side / 2))
        s.update(dt=1e-5, triangles=_box_triangles(lo, hi), speed=0.3)
        if case["normal"] == "sjkr":
            s["material"] = s["material"][:5] + (0.5,)
        lo, hi = tuple(v - 0.05 * side for v in lo), tuple(v + 0.05 * side for v in hi)
    elif kind in ("bed", "gas"):
        r = _uniform(g, 1e-3, 2e-3, n)
        phi = 0.58 if kind == "bed" else 0.2
        side = (_volume(r) / phi) ** (1 / 3)
        lo, hi = (0.0, 0.0, 0.0), (side, side, side)
        m = math.ceil(n ** (1 / 3))
        x = _cubic(n, lo, side / m, m)
        x = x + _uniform(g, -0.1, 0.1, n, 3) * (side / m)
        floor = r.unsqueeze(1)

        def up(p):
            if kind == "bed":
                p[:, 1:2] = torch.maximum(torch.minimum(p[:, 1:2], side - floor), floor)
            return p

        s["periodic"] = (True, kind == "gas", True)
        x = _settle(x, r, lo, hi, s["periodic"], up)
        if kind == "bed":
            s["triangles"] = np.array([[0, 0, 0, 0, 0, side, side, 0, 0], [side, 0, 0, 0, 0, side, side, 0, side]], np.float32)
            hi = (side, side * 1.1, side)
        else:
            s.update(gravity=(0.0, 0.0, 0.0), speed=1.0, material=(1e7, 0.3, 2500.0, 0.3, 0.9, 0.0))
        if case["normal"] == "sjkr":
            s["material"] = s["material"][:5] + (0.05,)
    elif kind == "hopper":
        r = (torch.randn(n, generator=g, dtype=torch.float64, device=_device()) * 0.25).exp_().mul_(2e-3).clamp_(1e-3, 4e-3)
        t, r_out, y_out, bed = math.tan(math.pi / 6), 0.02, 0.15, _volume(r) / 0.55
        h = 0.0
        for _ in range(60):  # the fill height: a cone frustum of the bed's volume
            top = r_out + h * t
            h = max(h + (bed - math.pi / 3 * h * (top * top + top * r_out + r_out * r_out)) / (math.pi * top * top), 1e-3)
        height = 1.15 * h + 0.02
        top = r_out + height * t
        half = round(top + 0.05, 2)
        lo, hi = (-half, 0.0, -half), (half, round(y_out + height + 0.1, 2), half)
        a = (4.0 * bed / n) ** (1 / 3)
        while True:  # face-centred cubic sites inside the cone, from the outlet up
            k = torch.arange(-math.ceil(top / a) - 1, math.ceil(top / a) + 2, device=_device(), dtype=torch.float64)
            ky = torch.arange(0, math.ceil(height / a) + 1, device=_device(), dtype=torch.float64)
            cell = torch.cartesian_prod(ky, k, k)[:, [1, 0, 2]]
            corner = torch.tensor([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], dtype=torch.float64, device=_device())
            sites = ((cell.unsqueeze(1) + corner).reshape(-1, 3) * a)
            sites[:, 1] += y_out + 2e-3
            sites = sites[sites[:, [0, 2]].norm(dim=1) < r_out + (sites[:, 1] - y_out) * t - 2e-3]
            if len(sites) >= n:
                break
            a *= 0.98
        x = sites[torch.sort(sites[:, 1], stable=True).indices[:n]]
        x = x + _uniform(g, -0.02, 0.02, n, 3) * a

        def within(p):
            p[:, 1] = p[:, 1].clamp_min(y_out + 1e-3)
            rho = p[:, [0, 2]].norm(dim=1)
            most = (r_out + (p[:, 1] - y_out) * t - r / math.cos(math.pi / 6)).clamp_min(1e-3)
            p[:, [0, 2]] *= (most / rho.clamp_min(1e-9)).clamp_max(1.0).unsqueeze(1)
            return p

        x = _settle(x, r, lo, hi, (False, False, False), within)
        ys = np.linspace(y_out, y_out + height, 101)
        cone = _revolve(r_out + (ys - y_out) * t, ys, 1, 100)
        ground = np.array([[lo[0], 0, lo[2], lo[0], 0, hi[2], hi[0], 0, lo[2]], [hi[0], 0, lo[2], lo[0], 0, hi[2], hi[0], 0, hi[2]]], np.float32)
        s.update(triangles=np.concatenate([ground, cone]), periodic=(True, False, True), skin=4e-4)
    elif kind == "dust":
        r = _uniform(g, 5e-6, 20e-6, n)
        side = (_volume(r) / 0.35) ** (1 / 3)
        lo, hi = (0.0, 0.0, 0.0), (side, side, side)
        m = math.ceil(n ** (1 / 3))
        x = _cubic(n, lo, side / m, m) + _uniform(g, -0.05, 0.05, n, 3) * (side / m)
        s.update(periodic=(True, True, True), dt=1e-8, material=(5e8, 0.25, 2000.0, 0.5, 0.5, 0.05))
        x = _settle(x, r, lo, hi, s["periodic"], lambda p: p)
    elif kind == "boxes":
        counts = _counts(n)
        s["gammas"] = _uniform(g, 0.0, 0.1, n).tolist()
        per = math.ceil(n ** (1 / 3))
        radii = [_uniform(g, 0.5e-3, 1.5e-3, c) for c in counts]
        sides = [(_volume(q) / 0.45) ** (1 / 3) for q in radii]
        slot = max(sides) + 0.01
        xs, los, his, tris = [], [], [], []
        for b, (c, side) in enumerate(zip(counts, sides)):
            at = [(b % per) * slot + 0.005, (b // per % per) * slot + 0.005, (b // (per * per)) * slot + 0.005]
            m = math.ceil(c ** (1 / 3))
            xs.append(_cubic(c, at, side / m, m))
            los.append(at)
            his.append([v + side for v in at])
            tris.append(_box_triangles(at, [v + side for v in at]))
        r, x = torch.cat(radii), torch.cat(xs)
        group = torch.repeat_interleave(torch.arange(n, device=_device()), torch.tensor(counts, device=_device()))
        low, high = (torch.tensor(v, dtype=torch.float64, device=_device())[group] for v in (los, his))
        lo, hi = (0.0, 0.0, 0.0), (per * slot + 0.01,) * 3
        gap = r.unsqueeze(1)
        x = _settle(x, r, lo, hi, s["periodic"], lambda p: torch.maximum(torch.minimum(p, high - gap), low + gap))
        s.update(dt=1e-6, groups=group, triangles=np.concatenate(tris), material=s["material"][:5] + (s["gammas"][0],))
    else:
        r = _uniform(g, 1e-3, 2e-3, n)
        R = 0.5 if n > 1_000_000 else 0.2
        sp = (_volume(r) / n / 0.52) ** (1 / 3)
        area, yl, yh = 0.4 * math.pi * R * R, -R, R
        for _ in range(60):  # the level of a circular segment of two fifths of the circle
            y = (yl + yh) / 2
            seg = R * R * math.acos(-y / R) + y * math.sqrt(max(R * R - y * y, 0.0))
            yl, yh = (y, yh) if seg < area else (yl, y)
        k = torch.arange(-math.ceil(R / sp), math.ceil(R / sp) + 1, device=_device(), dtype=torch.float64) * sp
        xy = torch.cartesian_prod(k, k)
        xy = xy[(xy.norm(dim=1) < R - 2.5e-3) & (xy[:, 1] < yl)]
        i = torch.arange(n, device=_device())
        z = (i // len(xy)).double().add_(0.5).mul_(sp) + 2e-3
        x = torch.cat([xy[i % len(xy)], z.unsqueeze(1)], 1) + _uniform(g, -0.02, 0.02, n, 3) * sp
        length = math.ceil(n / len(xy)) * sp + 4e-3

        def inside(p):
            p[:, 2] = torch.maximum(torch.minimum(p[:, 2], length - r), r)
            p[:, :2] *= ((R - 1e-4 - r) / p[:, :2].norm(dim=1).clamp_min(1e-9)).clamp_max(1.0).unsqueeze(1)
            return p

        lo, hi = (-R - 0.02, -R - 0.02, -0.02), (R + 0.02, R + 0.02, length + 0.02)
        x = _settle(x, r, lo, hi, s["periodic"], inside)
        ring = np.linspace(0.0, R, 7)
        wall = _revolve(np.concatenate([ring, np.full(116, R), ring[::-1]]),
                        np.concatenate([np.zeros(7), np.linspace(0.0, length, 118)[1:-1], np.full(7, length)]), 2, 256)
        s.update(dt=5e-6, material=(1e7, 0.3, 2500.0, 0.4, 0.3, 0.0), triangles=wall,
                 motion=((0.0, 0.0, 0.0), (0.0, 0.0, math.pi), (0.0, 0.0, 0.0)))
        if case["normal"] == "sjkr":
            s["material"] = s["material"][:5] + (0.05,)
    rho = s["material"][2]
    n = len(r)
    s.update(lo=lo, hi=hi, radius=r, mass=rho * 4.0 / 3.0 * math.pi * r ** 3, position=x,
             velocity=torch.randn(n, 3, generator=g, dtype=torch.float64, device=_device()) * s["speed"],
             angular_velocity=torch.randn(n, 3, generator=g, dtype=torch.float64, device=_device()) * (s["speed"] / float(r.mean())))
    return s


def prepare(case, seed):
    s = _scene(case, seed)
    host = {k: s[k].cpu().numpy() for k in ("position", "radius", "mass", "velocity", "angular_velocity")}
    sim = rp.Simulation.create(s["dt"], *s["lo"], *s["hi"], len(host["radius"]))
    sim.set_particle_material(*s["material"])
    sim.set_contact_models(case["normal"], case["tangential"])
    sim.set_periodic_boundary(*s["periodic"])
    sim.set_gravity(*s["gravity"])
    sim.set_precision(case.get("precision", "fp64"))
    sim.set_interaction_mode(case.get("mode", "parity"))
    if s["skin"]:
        sim.set_skin(s["skin"])
    if case.get("solver", "newton") != "newton":
        sim.set_jkr_solver(case["solver"])
    if s["groups"] is not None:
        for b, v in enumerate(np.split(s["triangles"], case["n"])):
            sim.add_triangles(v, group=b)
    elif s["triangles"] is not None:
        sim.add_triangles(s["triangles"], motion=s["motion"])
    sim.add_particles(host["position"], host["radius"], host["mass"])
    if s["groups"] is not None:
        sim.set_particle_groups(s["groups"].cpu().numpy().astype(np.uint32))
        for b, gamma in enumerate(s["gammas"]):
            sim.set_group_material(b, *s["material"][:5], gamma)
    sim.set_state({k: host[k] for k in ("velocity", "angular_velocity")})
    sim.enable_gpu()
    return dict(sim=sim, steps=case["steps"], out={k: np.zeros((len(host["radius"]), 3)) for k in VECTORS})


def run(state):
    sim = state["sim"]
    if state["steps"] == 1:
        sim.step()
    else:
        sim.steps(state["steps"])
    return sim.get_state(out=state["out"])


def work(case):
    n = _spheres(case)
    contacts = 0.3 if case["scene"] in ("gas", "dust") else 2.5
    return dict(bytes=n * (case["steps"] * STEP_BYTES + 24.0 * len(VECTORS)),
                flops=n * case["steps"] * (STEP_FLOPS + contacts * CONTACT_FLOPS))


# ------------------------------------------------------------------------------------------- the step in 64 bits
def _image(d, size, periodic):
    for a in range(3):
        if periodic[a]:
            d[:, a] -= size[a] * torch.round(d[:, a] / size[a])
    return d


def _expand(first, count):
    """(which, index): `which` repeated count[which] times, with the indices first[which], first[which] + 1, ..."""
    which = torch.repeat_interleave(torch.arange(len(count), device=count.device), count)
    within = torch.arange(len(which), device=count.device) - (torch.cumsum(count, 0) - count)[which]
    return which, first[which] + within


def _pairs(x, r, scale, margin, lo, hi, periodic):
    """Pairs (i, j), each once, nearer than (r_i + r_j) scale + margin."""
    low = torch.tensor(lo, dtype=torch.float64, device=x.device)
    size = torch.tensor(hi, dtype=torch.float64, device=x.device) - low
    reach = 2.0 * float(r.max()) * scale + margin

    def near(i, j):
        d = _image(x[i] - x[j], size, periodic)
        keep = d.square().sum(1) < ((r[i] + r[j]) * scale + margin).square()
        return i[keep], j[keep]

    dims = [max(1, int(float(s) / reach)) for s in size]
    if any(p and d < 3 for p, d in zip(periodic, dims)) or len(x) < 1500:
        return near(*torch.triu_indices(len(x), len(x), 1, device=x.device))
    cell = torch.stack([((x[:, a] - low[a]) / size[a] * dims[a]).floor().long() for a in range(3)], 1)
    for a in range(3):
        cell[:, a] = torch.remainder(cell[:, a], dims[a]) if periodic[a] else cell[:, a].clamp(0, dims[a] - 1)
    key = (cell[:, 0] * dims[1] + cell[:, 1]) * dims[2] + cell[:, 2]
    order = torch.sort(key, stable=True).indices
    count = torch.bincount(key, minlength=dims[0] * dims[1] * dims[2])
    first = torch.cumsum(count, 0) - count
    found = []
    for off in [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if (a, b, c) >= (0, 0, 0)]:
        to, ok = [], torch.ones(len(x), dtype=torch.bool, device=x.device)
        for a in range(3):
            q = cell[:, a] + off[a]
            if periodic[a]:
                q = torch.remainder(q, dims[a])
            else:
                ok &= (q >= 0) & (q < dims[a])
                q = q.clamp(0, dims[a] - 1)
            to.append(q)
        other = (to[0] * dims[1] + to[1]) * dims[2] + to[2]
        i, at = _expand(first[other], count[other] * ok)
        j = order[at]
        if off == (0, 0, 0):
            i, j = i[j > i], j[j > i]
        found.append(near(i, j))
    return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])


def _wall_pairs(x, r, margin, v):
    """Pairs (particle, triangle) nearer than the radius plus margin of the triangle's plane and box."""
    v = v.reshape(-1, 3, 3)
    grow = float(r.max()) + margin
    a, b = v.amin(1) - grow, v.amax(1) + grow
    low, h = x.amin(0), 4.0 * grow
    dims = ((x.amax(0) - low) / h).floor().long() + 1
    ca = ((a - low) / h).floor().long().clamp_min(0)
    cb = torch.minimum(((b - low) / h).floor().long(), dims - 1)
    span = (cb - ca + 1).clamp_min(0)
    t, k = _expand(torch.zeros(len(v), dtype=torch.long, device=x.device), span.prod(1))
    c = ca[t] + torch.stack([k % span[t, 0], k // span[t, 0] % span[t, 1], k // (span[t, 0] * span[t, 1])], 1)
    cell = ((x - low) / h).floor().long()
    key = (cell[:, 0] * dims[1] + cell[:, 1]) * dims[2] + cell[:, 2]
    order = torch.sort(key, stable=True).indices
    count = torch.bincount(key, minlength=int(dims.prod()))
    first = torch.cumsum(count, 0) - count
    at = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
    n = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    n = n / n.norm(dim=1, keepdim=True)
    found = []
    for s in range(0, len(t), 1 << 22):
        w, q = _expand(first[at[s:s + (1 << 22)]], count[at[s:s + (1 << 22)]])
        p, tt = order[q], t[s:s + (1 << 22)][w]
        keep = ((x[p] - v[tt, 0]) * n[tt]).sum(1).abs() < r[p] + margin
        keep &= ((x[p] >= a[tt]) & (x[p] <= b[tt])).all(1)
        found.append(torch.stack([p[keep], tt[keep]]))
    return torch.cat(found, 1)


def _closest(p, v):
    """The point of each triangle that the reference takes for the closest one (its edge regions do not divide)."""
    e0, e1, v0 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0], v[:, 0] - p
    a, b, c, d, e = (e0 * e0).sum(1), (e0 * e1).sum(1), (e1 * e1).sum(1), (e0 * v0).sum(1), (e1 * v0).sum(1)
    det, s, t = a * c - b * b, b * e - c * d, b * d - a * e
    zero, one, side = torch.zeros_like(a), torch.ones_like(a), a - 2 * b + c
    along0, along1 = torch.minimum((-d).clamp_min(0), a), torch.minimum((-e).clamp_min(0), c)
    across = ((c + e - b - d) / side).clamp(0, 1)
    up = c + e > b + d
    edge = (a + d > b + e)
    clip = torch.minimum((-e).clamp_min(0), a)
    first = s + t < det
    sc = torch.where(first, torch.where(s < 0, torch.where((t < 0) & (d < 0), along0, zero), torch.where(t < 0, along0, s / det)),
                     torch.where(s < 0, torch.where(up, across, zero), torch.where(t < 0, torch.where(edge, across, clip), across)))
    tc = torch.where(first, torch.where(s < 0, torch.where((t < 0) & (d < 0), zero, along1), torch.where(t < 0, zero, t / det)),
                     torch.where(s < 0, torch.where(up, one - across, along1), torch.where(t < 0, torch.where(edge, one - across, zero), one - across)))
    return v[:, 0] + sc.unsqueeze(1) * e0 + tc.unsqueeze(1) * e1


def _jkr(ov, es, rs, gamma):
    """The reference's clamped Newton iteration for the contact radius, and its force."""
    C = 8 * math.pi * gamma / es
    a = torch.where(ov > 0, (rs * ov.clamp_min(0)).sqrt(), 0.5 * rs)
    live = torch.ones_like(a, dtype=torch.bool)
    for _ in range(20):
        a = torch.where(live & (a <= 0), torch.full_like(a, 1e-9), a)
        f = a * a / rs - (C * a).sqrt() - ov
        df = 2 * a / rs - 0.5 * C ** 0.5 / a.sqrt()
        live = live & (df.abs() >= 1e-9)
        step = torch.minimum(torch.maximum(f / df, -0.5 * a), 0.5 * a)
        a = torch.where(live, a - step, a)
        live = live & (step.abs() >= 1e-6 * rs)
    off = (a * a / rs - (C * a).sqrt() - ov).abs() > 1e-3 * rs
    fm = 4 * es * a ** 3 / (3 * rs) - (8 * math.pi * gamma * es * a ** 3).sqrt()
    return torch.where(off | (a <= 0) | (fm < -2 / 3 * math.pi * gamma * rs), torch.zeros_like(fm), fm)


def _normal(model, ov, vn, es, rs, ms, beta, gamma, wall):
    hertz = 4 / 3 * es * (rs * ov.clamp_min(0)).sqrt() * ov
    if model == "hertz":
        kt = 2 * es * (rs * ov.clamp_min(0)).sqrt()
        return torch.where(ov > 0, (hertz - 2 * beta * (ms * kt).sqrt() * vn).clamp_min(0), torch.zeros_like(ov))
    if model == "linear":
        return (es * rs * ov - 0.5 * (ms * es * rs).sqrt() * vn).clamp_min(0)
    if model == "hysteretic":
        return (es * rs * ov).clamp_min(0)
    hertz = torch.where(ov > 0, hertz, torch.zeros_like(hertz))
    if model == "jkr":
        return _jkr(ov, es, rs, gamma)
    gone = ov < -(3 * math.pi ** 2 * gamma ** 2 * rs / es ** 2).sqrt()
    return torch.where(gone, torch.zeros_like(ov), torch.where(gamma > 0, hertz - 1.5 * math.pi * gamma * rs * (vn > 0), hertz))


def _coulomb(fn, vt, mu):
    v2 = vt.square().sum(1, keepdim=True)
    return torch.where(v2 < 1e-8, torch.zeros_like(vt), -mu * fn.abs().unsqueeze(1) * vt / v2.clamp_min(1e-30).sqrt())


def exact(case, seed):
    s = _scene(case, seed)
    x, v, w, r, m = s["position"], s["velocity"], s["angular_velocity"], s["radius"], s["mass"]
    dev, dt, per, n = x.device, s["dt"], s["periodic"], len(r)
    low, high = (torch.tensor(s[k], dtype=torch.float64, device=dev) for k in ("lo", "hi"))
    size, grav = high - low, torch.tensor(s["gravity"], dtype=torch.float64, device=dev)
    E, nu, _, mu, rest, gam = s["material"]
    gamma = torch.full_like(r, gam) if s["groups"] is None else torch.tensor(s["gammas"], dtype=torch.float64, device=dev)[s["groups"]]
    beta = abs(math.log(rest) / math.sqrt(math.log(rest) ** 2 + math.pi ** 2))
    soft = (1 - nu * nu) / E
    es, es_wall = 1 / (2 * soft), 1 / (soft + (1 - 0.3 ** 2) / 1e9)  # the wall material keeps its default
    G = E / (2 * (1 + nu))
    physical = case.get("mode", "parity") == "physical"
    spring = case["tangential"] != "coulomb"
    gs = G / (2 * (2 - nu)) if physical else 0.0
    scale = 1.5 if case["normal"] in ("jkr", "sjkr") else 1.0
    inertia = (0.4 * m * r * r).unsqueeze(1)
    acc, tau, dims = torch.zeros_like(x), torch.zeros_like(x), [math.ceil(float(q)) + 1 for q in size]
    tri = None if s["triangles"] is None else torch.tensor(s["triangles"], device=dev).double().reshape(-1, 3, 3)
    start, i = None, None
    margin = 0.04 * float(r.max()) + 3.0 * case["steps"] * dt * float(v.norm(dim=1).max())

    def visits(a, b):
        """How often the reference's 27 cells around cell a list cell b."""
        if physical:
            return torch.ones(len(a), dtype=torch.float64, device=dev)
        k = torch.ones(len(a), dtype=torch.float64, device=dev)
        for c in range(3):
            hits = 0.0
            for d in (-1, 0, 1):
                q = a[:, c] + d
                if per[c]:
                    q = torch.where(q < 0, q + dims[c], torch.where(q >= dims[c], q - dims[c], q))
                hits = hits + (q == b[:, c]).double()
            k = k * hits * ((b[:, c] >= 0) & (b[:, c] < dims[c]))
        return k

    for _ in range(case["steps"]):
        for a in range(3):
            if per[a]:
                x[:, a] = torch.where(x[:, a] < low[a], x[:, a] + size[a], torch.where(x[:, a] >= high[a], x[:, a] - size[a], x[:, a]))
        v = v + acc * (0.5 * dt)
        x = x + v * dt
        w = w + tau / inertia * (0.5 * dt)
        if start is None or float(_image(x - start, size, per).norm(dim=1).max()) > 0.49 * margin:
            pairs = _pairs(x, r, scale, margin, s["lo"], s["hi"], per)
            xi = torch.zeros(len(pairs[0]), 3, dtype=torch.float64, device=dev)
            if start is not None and physical and spring:  # the springs go with their pairs
                old, new = i * n + j, pairs[0] * n + pairs[1]
                back = (pairs[1] * n + pairs[0])
                sort = torch.sort(old)
                for key, sign in ((new, 1.0), (back, -1.0)):
                    at = torch.searchsorted(sort.values, key).clamp_max(len(old) - 1)
                    hit = sort.values[at] == key
                    xi[hit] = sign * springs[sort.indices[at[hit]]]
            (i, j), springs, start = pairs, xi, x.clone()
            walls = None if tri is None else _wall_pairs(x, r, margin, tri)
        F, T = torch.zeros_like(x), torch.zeros_like(x)
        d = _image(x[i] - x[j], size, per)
        on = (d.square().sum(1) < ((r[i] + r[j]) * scale).square()).nonzero().squeeze(1)
        p, q, d = i[on], j[on], d[on]
        dist = d.norm(dim=1)
        nrm, ov, rp_, rq = d / dist.unsqueeze(1), r[p] + r[q] - dist, r[p].unsqueeze(1), r[q].unsqueeze(1)
        rv = v[p] - v[q] - torch.linalg.cross(w[p] * rp_ + w[q] * rq, nrm)
        vn = (rv * nrm).sum(1)
        vt = rv - vn.unsqueeze(1) * nrm
        rs, ms = r[p] * r[q] / (r[p] + r[q]), m[p] * m[q] / (m[p] + m[q])
        fn = _normal(case["normal"], ov, vn, es, rs, ms, beta, gamma[p], False)
        f = fn.unsqueeze(1) * nrm
        if not spring:
            f = f + _coulomb(fn, vt, mu)
        elif physical:
            kt = (8 * gs * (rs * ov.clamp_min(0)).sqrt() if case["tangential"] == "mindlin" else gs * rs).unsqueeze(1)
            z = springs[on]
            z = z - (z * nrm).sum(1, keepdim=True) * nrm + vt * dt
            trial, most = -kt * z, (mu * fn.abs()).unsqueeze(1)
            tm = trial.norm(dim=1, keepdim=True)
            slip = tm > most
            ft = torch.where(slip, torch.where(tm > 1e-6, most * trial / tm.clamp_min(1e-30), torch.zeros_like(trial)), trial)
            z = torch.where(slip, -ft / kt, z)
            touch = (ov > 0).unsqueeze(1)
            f = f + torch.where(touch, ft, torch.zeros_like(ft))
            springs = torch.zeros_like(springs)
            springs[on] = torch.where(touch, z, torch.zeros_like(z))
        cell = ((x - low) / 1.0).floor().long()
        there, back = visits(cell[p], cell[q]).unsqueeze(1), visits(cell[q], cell[p]).unsqueeze(1)
        turn = torch.linalg.cross(nrm, f)
        F.index_add_(0, p, f * there).index_add_(0, q, -f * back)
        T.index_add_(0, p, -rp_ * turn * there).index_add_(0, q, -rq * turn * back)
        if walls is not None:
            p, t = walls
            at = _closest(x[p], tri[t])
            d = x[p] - at
            dist = d.norm(dim=1)
            on = (dist < r[p]).nonzero().squeeze(1)
            p, at, dist, rad = p[on], at[on], dist[on], r[p[on]]
            nrm = d[on] / dist.unsqueeze(1)
            rv = v[p] - torch.linalg.cross(w[p], nrm) * rad.unsqueeze(1)
            if s["motion"] is not None:
                centre, omega, drift = (torch.tensor(q, dtype=torch.float64, device=dev) for q in s["motion"])
                rv = rv - drift - torch.linalg.cross(omega.expand_as(at), at - centre)
            vn = (rv * nrm).sum(1)
            fn = _normal(case["normal"], rad - dist, vn, es_wall, rad, m[p], beta, 0.5 * gamma[p], True)
            f = fn.unsqueeze(1) * nrm + _coulomb(fn, rv - vn.unsqueeze(1) * nrm, mu)
            F.index_add_(0, p, f)
            T.index_add_(0, p, -rad.unsqueeze(1) * torch.linalg.cross(nrm, f))
        acc, tau = grav + F / m.unsqueeze(1), T
        v = v + acc * (0.5 * dt)
        w = w + tau / inertia * (0.5 * dt)
    return dict(position=x, velocity=v, angular_velocity=w, acceleration=acc, torque=tau)
