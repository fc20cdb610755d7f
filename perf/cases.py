"""The calls this library is measured on.

A case is one call, or the short chain of calls, that a user's program makes
through the package's public entry points, at the sizes of the named
workloads (synth.config_cloud, synth.batch_cloud, the drivers' input files and
the tests), from a smoke-sized cloud to one that fills the GPU:

  node_loop      main_portal.x's node loop: the radiation field of every node,
                 then the polarized statistical equilibrium (SE) of every node
  batch          the same over several uneven clouds in one launch
  iterate        the node loop repeated to convergence (local operator + Ng)
  image          finish_portal.x: one Stokes cube (pixel mode)
  image_nodes    the same per bulk node (pix_mod = 0)
  se             the SE alone from a field the caller holds
  mlp_predict, mlp_gradients, mlp_train   the warm start's network

``listed`` names the cases, ``draw`` gives more of the same ranges,
``prepare`` makes what a program holds before the call (clouds and populations
from the seed, contexts with the cloud on the device, networks with their
weights), ``run`` makes the call, ``work`` says what it cannot do without, and
``exact`` restates the call in 64 bits with torch and numpy alone.
"""
import functools
import math

import numpy as np
import torch

import portal_gb300 as pg
from portal_gb300 import synth

TRACE_DX = float(np.float32(1e-6))     # main_portal.x's trace step [r_max]
IMAGE_DX = float(np.float32(1e-4))     # finish_portal.x's
SPI = math.sqrt(math.pi)
MAX_PASSES = 200                       # limit of the iterated node loop


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # the smoke run's cloud: the smallest call, where launches and latency count
        dict(name="node_loop_1k", kind="node_loop", recipe="sphere", points=1024, levels=5, angles=8, nvel=16, kmax=6,
             dust=False, star=False),
        # "sphere4k": the 4,096-point power-law sphere, 16 x 16 directions, 65 channels
        dict(name="node_loop_4k", kind="node_loop", recipe="sphere", points=4096, levels=5, angles=16, nvel=32, kmax=6,
             dust=False, star=False),
        # the benchmark sphere ("sphere262k": 10 levels, 24 x 24 directions, 129 channels, random
        # field component) with a quarter of its points: the largest call
        dict(name="node_loop_65k", kind="node_loop", recipe="sphere_random_b", points=65536, levels=10, angles=24,
             nvel=64, kmax=6, dust=False, star=False),
        # "cube1m", the turbulent cube (20 levels, 32 x 32 directions, 129 channels, kmax 2), scaled down
        dict(name="node_loop_cube", kind="node_loop", recipe="cube", points=8192, levels=20, angles=32, nvel=64, kmax=2,
             dust=False, star=False),
        # a dusty cloud (gas-to-dust ratio 100) of ragged sizes: 41 channels, 7 lines
        dict(name="node_loop_dust", kind="node_loop", recipe="sphere", points=6001, levels=8, angles=12, nvel=20,
             kmax=4, dust=True, star=False),
        # uneven clouds (800 to 12,000 points, 5 to 16 levels) in one launch, 16 x 16 directions, 65 channels
        dict(name="batch_6", kind="batch", clouds=6, min_points=800, max_points=12000, min_levels=5, max_levels=16,
             angles=16, nvel=32, kmax=2),
        # the warm-start study's method: the accelerated iteration to a change of 1e-6 per pass
        dict(name="iterate_cube", kind="iterate", points=2500, levels=10, angles=8, nvel=16, kmax=2, ng=4, local=True),
        # a Stokes cube of 257 x 257 pixels x 129 channels at 45 degrees
        dict(name="image_257", kind="image", points=32768, levels=10, lines=1, nvel=64, pix=128, incl=0.7853981634,
             azim=0.0, dust=False),
        # the per-node maps of a dusty cloud: three lines, 41 channels, all eight quantities
        dict(name="image_nodes_dust", kind="image_nodes", points=9001, levels=8, lines=3, nvel=20, incl=0.6, azim=0.3,
             dust=True),
        # 74 x 74 systems (20 levels, kmax 6) from a field the caller holds
        dict(name="se_74", kind="se", points=8192, levels=20, kmax=6),
        # the warm start: a network fitted for two epochs at its default batch and rate (39 steps each),
        # and evaluated on a cloud's nodes
        dict(name="mlp_train", kind="mlp_train", rows=20001, levels=20, width=256, depth=3, batch=512, epochs=2),
        dict(name="mlp_predict", kind="mlp_predict", rows=16385, levels=20, width=256, depth=3),
    ]


def draw(rng):
    def loguni(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["node_loop", "node_loop", "node_loop", "batch", "iterate", "image", "image_nodes", "se",
                       "mlp_predict", "mlp_gradients", "mlp_train"])
    levels = rng.randint(4, 20)
    if kind == "node_loop":
        star = rng.random() < 0.2      # the reference's run script sets star mode: every node has its own ray set
        case = dict(kind=kind, recipe=rng.choice(["sphere", "sphere_random_b", "cube"]), points=loguni(500, 32768),
                    levels=levels, angles=rng.choice([12, 16, 20, 24] if star else [6, 8, 12, 16, 24]),
                    nvel=rng.choice([8, 16, 20, 25, 32, 40, 64, 100, 128]), kmax=rng.choice([2, 4, 6]),
                    dust=rng.random() < 0.25, star=star)
        if star:
            case["recipe"] = "sphere"
            case["points"] = min(case["points"], 5000)
        top = _updates(next(c for c in listed() if c["name"] == "node_loop_65k"))
        weight = (4.0 if case["dust"] else 1.5)          # dust costs a division per update, padding its share
        if weight * _updates(case) > 0.5 * top:
            case["points"] = max(500, int(case["points"] * (0.5 * top / (weight * _updates(case))) ** 0.75))
        return case
    if kind == "batch":
        return dict(kind=kind, clouds=rng.randint(2, 8), min_points=loguni(400, 1500), max_points=loguni(2000, 12000),
                    min_levels=rng.randint(3, 6), max_levels=rng.randint(7, 16), angles=rng.choice([8, 12, 16]),
                    nvel=rng.choice([12, 16, 20, 32]), kmax=rng.choice([2, 4]))
    if kind == "iterate":
        return dict(kind=kind, points=loguni(800, 4000), levels=rng.randint(5, 12), angles=rng.choice([6, 8]),
                    nvel=rng.choice([8, 12, 16]), kmax=2, ng=rng.choice([3, 4, 5]), local=True)
    if kind == "image":
        return dict(kind=kind, points=loguni(1500, 40000), levels=levels, lines=rng.randint(1, 3),
                    nvel=rng.choice([8, 16, 20, 32, 50]), pix=loguni(16, 110), incl=round(rng.uniform(0.1, 1.4), 4),
                    azim=round(rng.uniform(0.0, 3.0), 4), dust=rng.random() < 0.3)
    if kind == "image_nodes":
        return dict(kind=kind, points=loguni(1500, 20000), levels=levels, lines=rng.randint(1, 3),
                    nvel=rng.choice([8, 16, 20, 32]), incl=round(rng.uniform(0.1, 1.4), 4),
                    azim=round(rng.uniform(0.0, 3.0), 4), dust=rng.random() < 0.5)
    if kind == "se":
        return dict(kind=kind, points=loguni(1000, 16384), levels=levels, kmax=rng.choice([2, 4, 6]))
    if kind == "mlp_train":
        return dict(kind=kind, rows=loguni(2000, 40000), levels=rng.choice([10, 20]), width=256, depth=3,
                    batch=rng.choice([256, 512]), epochs=rng.randint(1, 2))
    if kind == "mlp_gradients":
        return dict(kind=kind, rows=loguni(100, 4096), levels=rng.choice([10, 20]), width=rng.choice([64, 256]),
                    depth=rng.choice([2, 3]))
    return dict(kind=kind, rows=loguni(500, 19000), levels=rng.choice([10, 20]), width=256, depth=3)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _molecule(levels):
    return synth.linear_rotor(levels)


def _cloud(case, seed):
    """The case's cloud and molecule: a named recipe at the case's sizes."""
    mol = _molecule(case["levels"])
    recipe = case.get("recipe", "sphere_random_b")
    if recipe == "cube":
        cloud = synth.turbulent_cube(case["points"], seed, mol, grid=32)
    elif recipe == "sphere":
        cloud = synth.power_law_sphere(case["points"], seed, mol)
    else:
        cloud = synth.power_law_sphere(case["points"], seed, mol, t_law="loglinear", b_random=0.3)
    if case.get("dust"):
        # a gas-to-dust ratio of 100 (eat_lime.f90's dust mass density)
        cloud.dust_p = cloud.h2_dens * float(np.float32(2.32e-27)) / 100.0
    return cloud, mol


def _star(case, cloud):
    """A 2,500 K star of 0.05 r_max at the centre, or no star."""
    return (2500.0, 0.05 * cloud.tx, (0.0, 0.0, 0.0)) if case.get("star") else None


def _run_config(case, seed):
    return synth.RunConfig(nth=case["angles"], nph=case["angles"], nvel=case["nvel"], kmax=case.get("kmax", 2),
                           gvec=synth.gauge_vector(seed))


def _batch_models(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["clouds"]):
        # the batched configuration's recipe; the first and last cloud span the point range
        f = i / max(1, case["clouds"] - 1)
        n = int(case["min_points"] * (case["max_points"] / case["min_points"]) ** f)
        # levels in an order of their own: the largest systems are not the largest cloud's
        f = (i * 3 % case["clouds"]) / max(1, case["clouds"] - 1)
        mol = _molecule(int(round(case["min_levels"] + f * (case["max_levels"] - case["min_levels"]))))
        b = rng.normal(size=3)
        cloud = synth.power_law_sphere(n, seed + 100 + i, mol, density_exp=float(rng.uniform(1.0, 2.0)),
                                       n0_cm3=float(10.0 ** rng.uniform(4.0, 7.0)), b_dir=tuple(b))
        out.append((cloud, mol))
    return out


def _local_field(cloud, mol, seed):
    """A field for the SE alone: local Planck intensity, diluted towards the
    edge, with an anisotropy of a few 1e-3."""
    rng = np.random.default_rng(seed)
    nu = np.asarray(mol.nu)[None, :]
    J0 = 1.4744995e-50 * nu ** 3 / np.expm1(4.79924e-11 * nu / cloud.t_kin[:, None])
    J0 = J0 * rng.uniform(0.2, 1.0, size=J0.shape)
    J2 = 5e-3 * J0 * rng.normal(size=J0.shape)
    return J0, J2


def _pol_pops(cloud, mol, seed):
    """pol_pops as main_portal.x leaves it for finish_portal.x: rho^0_0 of the
    cloud's level populations and an alignment of about a percent."""
    rng = np.random.default_rng(seed)
    pp = np.zeros((cloud.node_num, 2 * mol.nlev))
    frac = cloud.lev_p / cloud.lev_p.sum(axis=1, keepdims=True)
    pp[:, 0::2] = frac / np.sqrt(2.0 * mol.j_lev + 1.0)
    pp[:, 1::2] = pp[:, 0::2] * rng.uniform(0.005, 0.02, size=frac.shape)
    pp[:, 1] = 0.0
    return pp


def _mlp_data(case, seed):
    """(parameters, statistics, X, Y): He-uniform weights, features of the
    warm start's spread, targets a smooth function of them plus noise."""
    rng = np.random.default_rng(seed)
    n_in, n_out = 8, 2 * case["levels"]
    dims = [n_in] + [case["width"]] * case["depth"] + [n_out]
    parts = []
    for i in range(len(dims) - 1):
        bound = math.sqrt(6.0 / dims[i])
        parts += [rng.uniform(-bound, bound, size=dims[i] * dims[i + 1]), rng.normal(size=dims[i + 1]) * 0.05]
    params = np.concatenate(parts).astype(np.float32)
    mx, sx = rng.normal(size=n_in) * 3.0, rng.uniform(0.3, 3.0, size=n_in)
    my, sy = -rng.uniform(0.0, 8.0, size=n_out), rng.uniform(0.1, 2.0, size=n_out)
    if case["kind"] == "mlp_gradients":      # that call takes rows already standardised
        mx, sx, my, sy = np.zeros(n_in), np.ones(n_in), np.zeros(n_out), np.ones(n_out)
    stats = np.concatenate([mx, sx, my, sy]).astype(np.float32)
    z = rng.normal(size=(case["rows"], n_in))
    X = (mx + sx * z).astype(np.float32)
    Y = (my + sy * (np.sin(z @ rng.normal(size=(n_in, n_out))) + 0.1 * rng.normal(size=(case["rows"], n_out))))
    return params, stats, X, Y.astype(np.float32)


def _context(cloud, mol, star=None):
    ctx = pg.Context(0)
    ctx.set_molecule(mol)
    ctx.set_cloud(cloud)
    if star:
        ctx.set_star(star)
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "node_loop":
        cloud, mol = _cloud(case, seed)
        state.update(ctx=_context(cloud, mol, _star(case, cloud)), rc=_run_config(case, seed))
    elif kind == "batch":
        rc = _run_config(case, seed)
        batch = pg.Batch(0)
        for cloud, mol in _batch_models(case, seed):
            batch.add(_context(cloud, mol))
        batch.prepare(rc)
        state.update(batch=batch)
    elif kind == "iterate":
        cloud, mol = _cloud(dict(case, recipe="cube"), seed)
        state.update(ctx=_context(cloud, mol), rc=_run_config(case, seed), lev_p=cloud.lev_p)
    elif kind in ("image", "image_nodes"):
        cloud, mol = _cloud(case, seed)
        state.update(ctx=_context(cloud, mol), pops=_pol_pops(cloud, mol, seed))
    elif kind == "se":
        cloud, mol = _cloud(case, seed)
        J0, J2 = _local_field(cloud, mol, seed)
        state.update(ctx=_context(cloud, mol), J0=J0, J2=J2)
    else:
        params, stats, X, Y = _mlp_data(case, seed)
        mlp = pg.MLP(8, case["width"], case["depth"], 2 * case["levels"], seed=seed)
        mlp.set_params(params, stats)
        state.update(mlp=mlp, X=X, Y=Y, seed=seed)
    return state


# --------------------------------------------------------------------------
# the calls
# --------------------------------------------------------------------------

def _image_args(case):
    lines = list(range(1, case["lines"] + 1))
    return (lines, [k + 1 for k in lines], case["incl"], case["azim"], case["nvel"], 3200.0 / case["nvel"], 0.0)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "node_loop":
        ctx, rc = state["ctx"], state["rc"]
        J0, J2, status, segments = ctx.radiation_field(rc)
        pops, _ = ctx.solve_se(rc.kmax)
        return dict(J0=J0, J2=J2, status=status, segments=segments, pops=pops)
    if kind == "batch":
        segments, _ = state["batch"].run()
        return dict(segments=segments, models=[ctx.results() for ctx in state["batch"].models])
    if kind == "iterate":
        ctx = state["ctx"]
        ctx.set_populations(state["lev_p"])
        pops, lev_p, passes, change, segments = ctx.lambda_iterate(
            state["rc"], tol=1e-6, max_iter=MAX_PASSES, ng_period=case["ng"], local_operator=case["local"])
        change = np.pad(change, (0, MAX_PASSES - passes))
        return dict(pops=pops, lev_p=lev_p, passes=passes, change=change, segments=segments)
    if kind == "image":
        cube, status = state["ctx"].image(*_image_args(case), case["pix"], 0.7, pol_pops=state["pops"],
                                          quantities=8 if case["dust"] else 4)
        return dict(cube=cube, status=status)
    if kind == "image_nodes":
        cube, xy, status = state["ctx"].image_nodes(*_image_args(case), pol_pops=state["pops"],
                                                    quantities=8 if case["dust"] else 4)
        return dict(cube=cube, xy=xy, status=status)
    if kind == "se":
        pops, status = state["ctx"].solve_se(case["kmax"], state["J0"], state["J2"])
        return dict(pops=pops, status=status)
    mlp = state["mlp"]
    if kind == "mlp_predict":
        return dict(y=mlp.predict(state["X"]))
    if kind == "mlp_gradients":
        loss, grads = mlp.gradients(state["X"], state["Y"])
        return dict(loss=loss, grads=grads)
    losses = mlp.train(state["X"], state["Y"], epochs=case["epochs"], batch=case["batch"], lr=1e-3, seed=state["seed"])
    params, stats = mlp.get_params()
    return dict(losses=losses, params=params, stats=stats)


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def _directions(angles):
    """Directions of legendre_all with nth = nph = angles."""
    x, _ = np.polynomial.legendre.leggauss(angles)
    return int(np.ceil(angles * np.sqrt(1.0 - x * x)).sum())


def _system_size(levels, kmax):
    return sum(min(2 * j, kmax) // 2 + 1 for j in range(levels))


def _segments(points, angles):
    # cells a ray crosses grow with N^(1/3): 51 at 262,144 points of the sphere, 78 at 1,048,576 of the cube
    return points * _directions(angles) * 0.78 * points ** (1.0 / 3.0)


def _updates(case, points=None, levels=None):
    """(ray segment, line, channel) transfer updates of one pass."""
    points, levels = points or case["points"], levels or case["levels"]
    return _segments(points, case["angles"]) * (levels - 1) * (2 * case["nvel"] + 1)


def _node_loop_work(case, points, levels):
    # an update: optical depth, 1 - exp(-tau) (a cubic and an exponential), S - I and the step, 10
    # operations; a segment: 16 neighbour faces of 12; an SE solve: an n^3 factorisation and its
    # refinement.  Bytes: the cloud, its neighbour lists (15.5 per node), populations and results
    n = _system_size(levels, case["kmax"])
    flops = (10.0 * _updates(case, points, levels) + 192.0 * _segments(points, case["angles"]) +
             points * (2.0 / 3.0 * n ** 3 + 12.0 * n * n))
    return flops, points * (8.0 * (13 + 3 * levels) + 15.5 * 20 + 16.0 * (levels - 1))


def work(case):
    kind = case["kind"]
    if kind == "node_loop":
        flops, moved = _node_loop_work(case, case["points"], case["levels"])
    elif kind == "batch":
        flops = moved = 0.0
        levels = (case["min_levels"] + case["max_levels"]) // 2
        for i in range(case["clouds"]):
            f = i / max(1, case["clouds"] - 1)
            a, b = _node_loop_work(case, int(case["min_points"] * (case["max_points"] / case["min_points"]) ** f),
                                   levels)
            flops, moved = flops + a, moved + b
    elif kind == "iterate":
        a, b = _node_loop_work(case, case["points"], case["levels"])
        flops, moved = 35.0 * a, 35.0 * b
    elif kind in ("image", "image_nodes"):
        # a ray crosses 0.78 N^(1/3) cells; a (cell, line, channel) step is about 60 operations
        rays = (2 * case["pix"] + 1) ** 2 if kind == "image" else case["points"]
        nch, quantities = 2 * case["nvel"] + 1, 8 if case["dust"] else 4
        cells = rays * 0.78 * case["points"] ** (1.0 / 3.0)
        flops = cells * (60.0 * case["lines"] * nch + 16 * 12)
        moved = 4.0 * quantities * rays * case["lines"] * nch + case["points"] * (8.0 * (13 + 3 * case["levels"]) + 310)
    elif kind == "se":
        n = _system_size(case["levels"], case["kmax"])
        flops = case["points"] * (2.0 / 3.0 * n ** 3 + 12.0 * n * n)
        moved = case["points"] * 8.0 * (2 * (case["levels"] - 1) + 2 * case["levels"] + 3)
    else:
        n_out = 2 * case["levels"]
        weights = 8 * case["width"] + (case["depth"] - 1) * case["width"] ** 2 + case["width"] * n_out
        rows = case["rows"] * case.get("epochs", 1)
        flops = (2.0 if kind == "mlp_predict" else 6.0) * rows * weights
        moved = 4.0 * case["rows"] * (8 + n_out) + 4.0 * weights
    return dict(bytes=float(moved), flops=float(flops))


# --------------------------------------------------------------------------
# the same results in 64 bits
# --------------------------------------------------------------------------

EXACT_UPDATES = 4e10       # transfer updates that 64 bits manage in about 20 seconds


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    a = np.asarray(a)
    return torch.as_tensor(a, dtype=torch.int64 if a.dtype.kind in "iu" else torch.float64, device=_dev())


class _Graph:
    """The cloud's neighbour lists as one padded table, positions, edges."""

    def __init__(self, cloud):
        deg = np.diff(cloud.nb_off)
        table = np.full((cloud.node_num, int(deg.max())), -1, dtype=np.int64)
        slot = np.arange(cloud.nb_idx.shape[0]) - np.repeat(cloud.nb_off[:-1], deg)
        table[np.repeat(np.arange(cloud.node_num), deg), slot] = cloud.nb_idx
        self.nb = _t(table)
        self.pos = _t(cloud.xyz)


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def _quadrature(angles):
    """legendre_all: (mu, phi, weight) rows."""
    x, w = np.polynomial.legendre.leggauss(angles)
    rows = []
    for mu, wm in zip(x, w):
        m = int(math.ceil(angles * math.sin(math.acos(mu))))
        rows += [(mu, k * 2.0 * math.pi / m, wm * 2.0 * math.pi / m / (4.0 * math.pi)) for k in range(m)]
    return np.array(rows)


def _about(axis, g, th, ph):
    """find_dir: the direction at (th, ph) about axis, gauge vector g."""
    u = _unit(np.cross(axis, g))
    v = np.cross(u, axis)
    return (np.cos(th)[..., None] * axis +
            np.sin(th)[..., None] * (np.cos(ph)[..., None] * v + np.sin(ph)[..., None] * u))


def _star_rays(p, k, dist, star_radius, angles):
    """star_all: (th, ph, weight) about the star's direction, number of star rays."""
    d_om = math.pi * (star_radius / dist) ** 2
    dth = d_om / (2.0 * math.pi)
    ths = math.acos(1.0 - dth)
    ns = int(math.ceil(d_om / (4.0 * math.pi / (angles * angles))))
    if ns == 1:      # the reference's stand-in: cos(1) for both entries
        rows = [(math.acos(math.cos(1.0)), math.cos(1.0), 2.0 * math.pi * dth)]
    elif ns < 10:
        rows = [(ths / 2.0, i * 2.0 * math.pi / ns, 2.0 * math.pi / ns * dth) for i in range(ns)]
    else:
        rows = [(ths * math.sqrt((i + 1) / ns), (i + 1) * math.pi * (3.0 - math.sqrt(5.0)), dth * 2.0 * math.pi / ns)
                for i in range(ns)]
    dr = (math.pi - ths) / angles
    thi = ths + dr / 2.0
    for b in range(1, angles + 1):
        th = (b - 1) * dr + thi
        m = int(math.ceil(angles * math.sin(th)))
        lo, hi = math.cos((b - 1.5) * dr + thi), math.cos((b - 0.5) * dr + thi)
        wth = math.cos(ths) - hi if b == 1 else lo + 1.0 if b == angles else lo - hi
        rows += [(th, j * 2.0 * math.pi / m, wth * 2.0 * math.pi / m) for j in range(m)]
    r = np.array(rows)
    r[:, 2] /= 4.0 * math.pi
    return r, ns


def _rays(cloud, nodes, rc, star):
    """Flattened ray sets of the nodes: node, direction, weight of J0, weight
    of J2, whether it is a star ray."""
    g = np.asarray(rc.gvec)
    if star is None:
        q = _quadrature(rc.nth)
        d = _about(cloud.bvec[nodes][:, None, :], g, np.arccos(q[None, :, 0]), q[None, :, 1])
        m = len(q)
        w2 = q[:, 2] * (3.0 * q[:, 0] ** 2 - 1.0) / 2.0 / math.sqrt(2.0)
        return (np.repeat(nodes, m), d.reshape(-1, 3), np.tile(q[:, 2], len(nodes)), np.tile(w2, len(nodes)),
                np.zeros(m * len(nodes), dtype=bool))
    out = [[], [], [], [], []]
    centre, radius = np.asarray(star[2], dtype=np.float64), star[1] / cloud.tx
    for n in nodes:
        to = centre - cloud.xyz[n]
        dist = np.linalg.norm(to)
        r, ns = _star_rays(cloud.xyz[n], to / dist, dist, radius, rc.nth)
        d = _about((to / dist)[None, :], g, r[:, 0], r[:, 1])
        # find_angles in the field frame and find_dir back: the frame's own cos(th)
        mu = np.cos(np.arccos(np.clip(d @ cloud.bvec[n], -1.0, 1.0)))
        for lst, v in zip(out, (np.full(len(r), n), d, r[:, 2], r[:, 2] * (3.0 * mu * mu - 1.0) / 2.0 / math.sqrt(2.0),
                                np.arange(len(r)) < ns)):
            lst.append(v)
    return tuple(np.concatenate(x) for x in out)


def _walk(graph, node, d, exit_len):
    """trace_out: per crossing the cell and its length in trace steps."""
    cells, steps = [], []
    live = torch.arange(node.shape[0], device=_dev())
    c, r, left = node.clone(), torch.zeros_like(d), exit_len.clone()
    count = torch.zeros_like(node)
    while live.numel():
        nb = graph.nb[c[live]]
        e = graph.pos[nb.clamp_min(0)] - graph.pos[c[live]][:, None, :]
        den = (e * d[live][:, None, :]).sum(-1)
        num = 0.5 * (e * e).sum(-1) - (e * r[live][:, None, :]).sum(-1)
        t = torch.where((nb >= 0) & (den > 0), num / den, torch.inf)
        t = torch.where(t > 1e-10, t, torch.inf)
        tmin, j = t.min(dim=1)
        crossing = tmin <= left[live]
        delta = torch.where(crossing, tmin, left[live])
        cell, n = torch.full_like(node, -1), torch.zeros_like(left)
        cell[live], n[live] = c[live], torch.floor(delta / TRACE_DX + 0.5)
        cells.append(cell)
        steps.append(n)
        count[live] += 1
        left[live] -= delta
        r[live] += delta[:, None] * d[live]
        live, j = live[crossing], j[crossing]
        to = graph.nb[c[live], j]
        r[live] -= graph.pos[to] - graph.pos[c[live]]
        c[live] = to
    return torch.stack(cells), torch.stack(steps), count


def _line_table(cloud, mol, lev_p):
    """(opacity per profile value and step, source numerator, dust opacity and
    emissivity per step, background) of every node and line."""
    nu, A, B, kd = (_t(v)[None, :] for v in (mol.nu, mol.A, mol.Bij, mol.kd_v))
    lo, up = _t(mol.r_trans[:, 0] - 1), _t(mol.r_trans[:, 1] - 1)
    g = _t(2.0 * mol.j_lev + 1.0)
    p1, p2 = _t(lev_p)[:, lo], _t(lev_p)[:, up]
    kv = 2.2102191e-42 * nu * B * (p1 - g[lo] * p2 / g[up])
    ev = 5.272859e-35 * nu * A * p2
    phi = 299792458.0 / nu / (SPI * _t(cloud.b_all)[:, None]) * (cloud.tx * TRACE_DX)
    Ad = kd * _t(cloud.dust_p)[:, None] * (cloud.tx * TRACE_DX)
    Td = _t(cloud.t_dust)[:, None]
    planck = 1.4744995e-50 * nu ** 3 / (torch.exp(4.79924e-11 / Td * nu) - 1.0)
    return kv * phi, ev * phi, Ad, Ad * torch.where(Td != 0.0, planck, 0.0)


def _background(nu, T):
    return 1.4744995e-50 * nu ** 3 / (np.exp(4.79924e-11 / T * nu) - 1.0)


def _radiation_field(cloud, mol, rc, star=None):
    """inverse_rt of every bulk node: J0, J2 (N, lines)."""
    graph = _Graph(cloud)
    kv, ev, Ad, Jd = _line_table(cloud, mol, cloud.lev_p)
    v, b = _t(cloud.vel), _t(cloud.b_all)
    N, L, nch = cloud.node_num, mol.r_num, 2 * rc.nvel + 1
    ch = _t(np.arange(nch) - rc.nvel).double()
    wch = torch.exp(-(2.0 * ch / rc.nvel) ** 2) * 2.0 / (SPI * rc.nvel)
    J0, J2 = torch.zeros(N, L, dtype=torch.float64, device=_dev()), torch.zeros(N, L, dtype=torch.float64, device=_dev())
    alive = np.flatnonzero(cloud.ab_all[:cloud.bulk_node_num] > 0.0)
    if star is not None:
        alive = alive[np.linalg.norm(cloud.xyz[alive], axis=1) > star[1] / cloud.tx]
    step = max(1, int(2.5e7 / (L * nch * (_directions(rc.nth) + 1))))
    for at in range(0, len(alive), step):
        node, d, w0, w2, is_star = _rays(cloud, alive[at:at + step], rc, star)
        p = cloud.xyz[node]
        pd = (p * d).sum(1)
        disc = pd * pd - ((p * p).sum(1) - 1.0)
        exit_len = np.where(disc > 0.0, -pd + np.sqrt(np.maximum(disc, 0.0)), 0.0)
        exit_len = np.where(exit_len > 0.0, exit_len, 0.0)
        start = np.tile(_background(np.asarray(mol.nu), 2.73), (len(node), 1))
        if star is not None:
            q = p - np.asarray(star[2])
            qd = (q * d).sum(1)
            disc = qd * qd - ((q * q).sum(1) - (star[1] / cloud.tx) ** 2)
            hit = np.where(disc > 0.0, -qd - np.sqrt(np.maximum(disc, 0.0)), -1.0)
            exit_len = np.where(is_star & (hit > 0.0) & (hit < exit_len), hit, exit_len)
            start = np.where(is_star[:, None], _background(np.asarray(mol.nu), star[0])[None, :], start)
        node, d = _t(node), _t(d)
        cells, steps, count = _walk(graph, node, d, _t(exit_len))
        I = _t(start)[:, :, None].expand(-1, -1, nch).clone()
        vn = (v[node] * d).sum(1)
        for k in range(cells.shape[0] - 1, 0, -1):
            at_k = torch.nonzero(cells[k] >= 0)[:, 0]
            c, n = cells[k][at_k], steps[k][at_k]
            dv = (vn[at_k] - (v[c] * d[at_k]).sum(1))[:, None] + ch[None, :] * (2.0 * b[node[at_k]] / rc.nvel)[:, None]
            prof = torch.exp(-(dv / b[c][:, None]) ** 2)[:, None, :]
            kap = kv[c][:, :, None] * prof + Ad[c][:, :, None]
            tau = kap * n[:, None, None]
            src = (ev[c][:, :, None] * prof + Jd[c][:, :, None]) / kap
            e = torch.exp(-tau)
            I[at_k] = torch.where(tau > 1e-30, I[at_k] * e + src * (1.0 - e), I[at_k])
        prof = torch.exp(-(2.0 * ch / rc.nvel) ** 2)[None, None, :]
        kap = kv[node][:, :, None] * prof + Ad[node][:, :, None]
        e = torch.exp(-kap * steps[0][:, None, None])
        I = I * e + (ev[node][:, :, None] * prof + Jd[node][:, :, None]) / kap * (1.0 - e)
        s = (I * wch).sum(-1)
        J0.index_add_(0, node, _t(w0)[:, None] * s)
        J2.index_add_(0, node, _t(w2)[:, None] * s)
    return J0, J2


@functools.lru_cache(maxsize=None)
def _w3(j1, j2, j3, m1, m2, m3):
    """Wigner 3j symbol of integer arguments (Racah's formula)."""
    if m1 + m2 + m3 or j3 < abs(j1 - j2) or j3 > j1 + j2 or abs(m1) > j1 or abs(m2) > j2 or abs(m3) > j3:
        return 0.0
    f = math.factorial
    pre = f(j1 + j2 - j3) * f(j1 - j2 + j3) * f(-j1 + j2 + j3)
    pre *= f(j1 + m1) * f(j1 - m1) * f(j2 + m2) * f(j2 - m2) * f(j3 + m3) * f(j3 - m3)
    lo, hi = max(0, j2 - j3 - m1, j1 - j3 + m2), min(j1 + j2 - j3, j1 - m1, j2 + m2)
    den = [f(t) * f(j3 - j2 + t + m1) * f(j3 - j1 + t - m2) * f(j1 + j2 - j3 - t) * f(j1 - t - m1) * f(j2 - t + m2)
           for t in range(lo, hi + 1)]
    lcm = math.lcm(*den)
    s = sum((-1) ** t * (lcm // x) for t, x in zip(range(lo, hi + 1), den))
    if not s:
        return 0.0
    val = math.sqrt(s * s * pre / (f(j1 + j2 + j3 + 1) * lcm * lcm))
    return (-1) ** (j1 - j2 - m3) * math.copysign(val, s)


@functools.lru_cache(maxsize=None)
def _w6(a, b, c, d, e, f):
    """Wigner 6j symbol of integer arguments (Racah's formula)."""
    fac = math.factorial

    def tri(x, y, z):
        if z < abs(x - y) or z > x + y:
            return None
        return fac(x + y - z) * fac(x - y + z) * fac(-x + y + z) / fac(x + y + z + 1)

    t = [tri(a, b, c), tri(a, e, f), tri(d, b, f), tri(d, e, c)]
    if any(x is None for x in t):
        return 0.0
    s = 0.0
    for k in range(max(a + b + c, a + e + f, d + b + f, d + e + c), min(a + b + d + e, b + c + e + f, a + c + d + f) + 1):
        s += (-1) ** k * fac(k + 1) / (fac(k - a - b - c) * fac(k - a - e - f) * fac(k - d - b - f) * fac(k - d - e - c) *
                                       fac(a + b + d + e - k) * fac(b + c + e + f - k) * fac(a + c + d + f - k))
    return math.sqrt(t[0] * t[1] * t[2] * t[3]) * s


@functools.lru_cache(maxsize=None)
def _coupling(which, j, k, j2, k2):
    """pop_eqs.f90's rate coefficients (rank-0 and rank-2 part of the field):
    0 transfer by absorption, 1 by stimulated, 2 by spontaneous emission,
    3 relaxation by absorption, 4 by stimulated emission."""
    if abs(j2 - j) > 1:
        return 0.0, 0.0
    if which == 2:
        return ((2 * j2 + 1) * (-1) ** (1 + j + j2 + k) * _w6(j2, j2, k, j, j, 1) if k == k2 else 0.0), 0.0
    if abs(k2 - k) not in (0, 2):
        return 0.0, 0.0
    s0 = s2 = 0.0
    for m in range(-j, j + 1):
        for q in (-1, 0, 1):
            o = m + q if which in (0, 4) else m - q           # the other level's m
            jj, mm = (j2, o) if which in (0, 1) else (j, m)
            w = _w3(j, j, k, m, -m, 0) * _w3(jj, jj, k2, mm, -mm, 0)
            w *= (_w3(j, j2, 1, -m, o, -q) if which in (0, 4) else _w3(j2, j, 1, -o, m, -q)) ** 2
            if which > 2:
                w *= (-1) ** (1 + q)
            s0 += w * _w3(1, 1, 0, q, -q, 0) if k == k2 else 0.0
            s2 += w * _w3(1, 1, 2, q, -q, 0)
    f = math.sqrt(3.0 * (2 * k + 1) * (2 * k2 + 1))
    f *= (2 * j2 + 1) * (-1) ** (1 - j2 + j) if which < 2 else 2 * j + 1
    return s0 * f, s2 * f * math.sqrt(5.0)


def _solve_se(cloud, mol, kmax, J0, J2, alive):
    """make_AC + setup_stateq + get_rhovec + the packing of trace_node for the
    nodes `alive`: pol_pops (N, 2 nlev)."""
    J, nlev = mol.j_lev, mol.nlev
    ranks = [list(range(0, min(2 * int(j), kmax) + 1, 2)) for j in J]
    first = np.concatenate([[0], np.cumsum([len(r) for r in ranks])])
    n = int(first[-1])
    out = torch.zeros(cloud.node_num, 2 * nlev, dtype=torch.float64, device=_dev())
    rad = {(int(a) - 1, int(b) - 1): i for i, (a, b) in enumerate(mol.r_trans)}
    col = {(int(a) - 1, int(b) - 1): i for i, (a, b) in enumerate(mol.c_trans)}
    pairs = sorted(set(rad) | set(col))
    T_all, h2_all = _t(cloud.t_kin), _t(cloud.h2_dens)
    tabT = np.asarray(mol.col_temps)
    for at in range(0, len(alive), max(1, int(6e7 / (n * n)))):
        idx = _t(alive[at:at + max(1, int(6e7 / (n * n)))])
        T, h2 = T_all[idx], h2_all[idx]
        M = torch.zeros(idx.shape[0], n, n, dtype=torch.float64, device=_dev())
        # the first bracket above T (below the table it extrapolates, above the table 0)
        hi = torch.searchsorted(_t(tabT), T, right=True).clamp_min(1)
        inside = hi < len(tabT)
        hi = hi.clamp_max(len(tabT) - 1)
        f = (T - _t(tabT)[hi - 1]) / (_t(tabT)[hi] - _t(tabT)[hi - 1])
        share = [0.25, 0.75] if mol.c_par == 2 else [1.0]
        for lo, up in pairs:
            r, q = rad.get((lo, up)), col.get((lo, up))
            nu = float(mol.e_levs[up] - mol.e_levs[lo])
            A = float(mol.A[r]) if r is not None else 0.0
            B = 6.781962e49 * A / nu ** 3
            b0, b2 = (B * J0[idx, r], B * J2[idx, r]) if r is not None else (0.0 * T, 0.0 * T)
            C = 0.0 * T
            if q is not None:
                for s, part in zip(share, mol.C):
                    tab = _t(part[q])
                    C = C + s * torch.where(inside, tab[hi - 1] + f * (tab[hi] - tab[hi - 1]), 0.0)
                C = C * h2 * 1e-6
            Cup = C * torch.exp(-4.79924e-11 * nu / T)
            gl, gu = 2.0 * J[lo] + 1.0, 2.0 * J[up] + 1.0
            for a, k1 in enumerate(ranks[lo]):
                for b, k2 in enumerate(ranks[up]):           # into the lower level, from the upper
                    ts, te = (_coupling(w, int(J[lo]), k1, int(J[up]), k2) for w in (1, 2))
                    M[:, first[lo] + a, first[up] + b] += ts[0] * b0 + ts[1] * b2 + te[0] * A
                    ta = _coupling(0, int(J[up]), k2, int(J[lo]), k1)       # and the other way
                    M[:, first[up] + b, first[lo] + a] += gu / gl * (ta[0] * b0 + ta[1] * b2)
            M[:, first[lo], first[up]] += math.sqrt(gu / gl) * C
            M[:, first[up], first[lo]] += math.sqrt(gl / gu) * gu / gl * Cup
            for a, k1 in enumerate(ranks[lo]):
                for b, k2 in enumerate(ranks[lo]):
                    ra = _coupling(3, int(J[lo]), k1, int(J[up]), k2)
                    M[:, first[lo] + a, first[lo] + b] -= gu / gl * (ra[0] * b0 + ra[1] * b2)
                M[:, first[lo] + a, first[lo] + a] -= gu / gl * Cup
            for a, k1 in enumerate(ranks[up]):
                for b, k2 in enumerate(ranks[up]):
                    rs = _coupling(4, int(J[up]), k1, int(J[lo]), k2)
                    M[:, first[up] + a, first[up] + b] -= rs[0] * b0 + rs[1] * b2
                M[:, first[up] + a, first[up] + a] -= A + C
        M[:, 0, :] = 0.0
        M[:, 0, _t(first[:-1])] = _t(np.sqrt(2.0 * J + 1.0))[None, :]
        scale = 1.0 / M.abs().amax(dim=2, keepdim=True)
        M = M * scale
        rhs = torch.zeros(idx.shape[0], n, 1, dtype=torch.float64, device=_dev())
        rhs[:, 0, 0] = scale[:, 0, 0]
        lu = torch.linalg.lu_factor(M)
        x = torch.linalg.lu_solve(*lu, rhs)
        x = (x + torch.linalg.lu_solve(*lu, rhs - M @ x))[:, :, 0]
        for i in range(nlev):
            out[idx, 2 * i] = x[:, first[i]]
            if J[i]:
                out[idx, 2 * i + 1] = x[:, first[i] + 1]
    return out


def _rotation(incl, azim):
    ci, si, ca, sa = math.cos(incl), math.sin(incl), math.cos(azim), math.sin(azim)
    rx = np.array([[1, 0, 0], [0, ci, -si], [0, si, ci]])
    rz = np.array([[ca, -sa, 0], [sa, ca, 0], [0, 0, 1]])
    return rz @ rx


def _march(graph, pos, x, y):
    """trace_out_raytrace: along +z in steps of IMAGE_DX, the list of (node,
    step) from the first change of the nearest node to the exit."""
    z0 = -torch.sqrt(1.0 - x * x - y * y)
    start = torch.stack([x, y, z0], dim=1)
    c = torch.empty(x.shape[0], dtype=torch.int64, device=_dev())
    for at in range(0, x.shape[0], 4096):
        # differences, not a Gram matrix: the nearest of two near-equal nodes
        s = start[at:at + 4096]
        d2 = sum((s[:, i, None] - pos[None, :, i]) ** 2 for i in range(3))
        c[at:at + 4096] = d2.argmin(dim=1)
    k = torch.zeros_like(c)
    k_exit = torch.floor(-2.0 * z0 / IMAGE_DX).long() + 1
    cells, steps = [], []
    live = torch.arange(x.shape[0], device=_dev())
    nrm2 = (pos * pos).sum(1)
    while live.numel():
        nb = graph.nb[c[live]]
        ok = nb >= 0
        nb = nb.clamp_min(0)
        pc, pn = pos[c[live]], pos[nb]
        A = (nrm2[nb] - nrm2[c[live]][:, None] - 2.0 * x[live][:, None] * (pn[:, :, 0] - pc[:, None, 0]) -
             2.0 * y[live][:, None] * (pn[:, :, 1] - pc[:, None, 1]))
        dz = pn[:, :, 2] - pc[:, None, 2]
        now = z0[live] + (k[live] + 1) * IMAGE_DX
        nearer = A - 2.0 * now[:, None] * dz < 0.0
        kn = torch.floor((A / (2.0 * dz) - z0[live][:, None]) / IMAGE_DX) + 1.0
        kn = torch.where(nearer, (k[live] + 1)[:, None].double(), torch.where(dz > 0.0, kn, torch.inf))
        kn = torch.maximum(torch.where(ok, kn, torch.inf), (k[live] + 1)[:, None].double())
        kmin = kn.min(dim=1).values
        leaves = kmin >= k_exit[live]
        z = z0[live] + torch.where(leaves, k_exit[live].double(), kmin) * IMAGE_DX
        d2 = (x[live][:, None] - pn[:, :, 0]) ** 2 + (y[live][:, None] - pn[:, :, 1]) ** 2 + (z[:, None] - pn[:, :, 2]) ** 2
        to = torch.gather(nb, 1, torch.where(ok, d2, torch.inf).argmin(dim=1, keepdim=True))[:, 0]
        c[live] = torch.where(leaves, c[live], to)
        k[live] = torch.where(leaves, k_exit[live], kmin.clamp_max(2 ** 30).long())
        cell, step = torch.full_like(c, -1), torch.zeros_like(c)
        cell[live], step[live] = c[live], k[live]
        cells.append(cell)
        steps.append(step)
        live = live[~leaves]
    return torch.stack(cells), torch.stack(steps)


def _phi(x):
    return torch.where(x.abs() > 1e-8, -torch.expm1(-x) / torch.where(x == 0, 1.0, x), 1.0 - 0.5 * x)


def _stokes(case, cloud, mol, pops, alpha=0.15):
    """ray_in_raytrace over the pixels (or the bulk nodes): the (8, lines,
    channels, ...) cube, and the rotated positions."""
    graph = _Graph(cloud)
    R = _rotation(case["incl"], case["azim"])
    pos, vel, fld = (_t(a @ R.T) for a in (cloud.xyz, cloud.vel, cloud.bvec))
    nodes = case["kind"] == "image_nodes"
    if nodes:
        x, y = pos[:cloud.bulk_node_num, 0], pos[:cloud.bulk_node_num, 1]
    else:
        grid = torch.arange(-case["pix"], case["pix"] + 1, device=_dev(), dtype=torch.float64) * 0.7 / case["pix"]
        y, x = (g.reshape(-1) for g in torch.meshgrid(grid, grid, indexing="ij"))
    cells, steps = _march(graph, pos, x, y)
    l1, l2, _, _, nvel, dvel, v0 = _image_args(case)
    nch, rays = 2 * nvel + 1, x.shape[0]
    vch = (torch.arange(nch, device=_dev(), dtype=torch.float64) - nvel) * dvel + v0
    b = _t(cloud.b_all)
    b_xy = torch.sqrt(fld[:, 0] ** 2 + fld[:, 1] ** 2)
    ang = torch.acos((fld[:, 1] / b_xy).clamp(-1, 1))
    al, ph = torch.where(fld[:, 0] > 0, -ang, ang), torch.where(fld[:, 0] < 0, -ang, ang)
    rot = torch.cos(2 * al), torch.sin(2 * al)
    th = torch.acos(fld[:, 2].clamp(-1, 1))
    tki = (3.0 * torch.cos(th) ** 2 - 1.0) / (2.0 * math.sqrt(2.0))
    tkq = -3.0 * torch.sin(th) ** 2 / (2.0 * math.sqrt(2.0))
    nu = float(mol.e_levs[l2[-1] - 1] - mol.e_levs[l1[-1] - 1])    # every line takes the last pair's
    lev, pp, tdx = _t(cloud.lev_p), _t(pops), cloud.tx * IMAGE_DX
    cube = torch.zeros(8, len(l1), nch, rays, dtype=torch.float64, device=_dev())
    part = max(1, int(2e7 / nch))
    for li, (lo, up) in enumerate(zip(l1, l2)):
        lo, up = lo - 1, up - 1
        hit = [i for i, t in enumerate(mol.r_trans) if t[0] == lo + 1 and t[1] == up + 1]
        A, kd = (float(mol.A[hit[0]]), float(mol.kd_v[hit[0]])) if hit else (0.0, 0.0)
        j1, j2 = int(mol.j_lev[lo]), int(mol.j_lev[up])
        if nodes:
            A = float(mol.A[lo])                              # t_Aji(l1(j)), para_finish.f90:303
        g1, g2 = 2.0 * j1 + 1.0, 2.0 * j2 + 1.0
        sgn = (-1) ** (1 + j1 + j2)
        w1, w2 = sgn * math.sqrt(3.0 * g1) * _w6(1, 1, 2, j1, j1, j2), sgn * math.sqrt(3.0 * g2) * _w6(1, 1, 2, j2, j2, j1)
        r1, r2 = lev[:, lo] / math.sqrt(g1), lev[:, up] / math.sqrt(g2)
        a1 = pp[:, 2 * lo + 1] / r1 if lo == 0 else pp[:, 2 * lo + 1] / pp[:, 2 * lo]
        a2 = pp[:, 2 * up + 1] / pp[:, 2 * up]
        Bji = A / (nu ** 3 / 6.781962e49)
        hv = 5.273e-35 * nu
        s1, s2 = math.sqrt(g1) * r1, math.sqrt(g2) * r2
        eI, eQ = hv * A * s2 * (1.0 + w2 * a2 * tki), hv * A * s2 * w2 * a2 * tkq
        nI = hv * g2 / g1 * Bji * (s1 * (1.0 + w1 * a1 * tki) - s2 * (1.0 + w2 * a2 * tki) * g1 / g2)
        nQ = hv * g2 / g1 * Bji * (s1 * w1 * a1 * tkq - s2 * w2 * a2 * tkq * g1 / g2)
        f = float(np.float32(2.99792e8)) / nu / (SPI * b) * tdx
        live = (torch.arange(cloud.node_num, device=_dev()) < cloud.bulk_node_num) & (lev[:, 0] != 0.0)
        coef = [torch.where(live, v * f, 0.0) for v in (nI, nQ, eI, eQ)]
        cmb = float(_background(nu, 2.73))
        Td, dust = _t(cloud.t_dust), _t(cloud.dust_p)
        planck = torch.where(Td != 0.0, 1.4744995e-50 * nu ** 3 / (torch.exp(4.79924e-11 / Td * nu) - 1.0), 0.0)
        for at in range(0, rays, part):
            sl = slice(at, min(rays, at + part))
            m = sl.stop - at
            I = torch.full((m, nch), cmb, dtype=torch.float64, device=_dev())
            Q, U, tau = torch.zeros_like(I), torch.zeros_like(I), torch.zeros_like(I)
            Id = torch.full((m,), cmb, dtype=torch.float64, device=_dev())
            s0, sq, Qd, Ud, td = (torch.zeros_like(Id) for _ in range(5))
            for i in range(cells.shape[0] - 1):
                sel = torch.nonzero((cells[i, sl] >= 0) & (cells[i + 1, sl] >= 0))[:, 0]
                c = cells[i, sl][sel]
                dk = (steps[i + 1, sl][sel] - steps[i, sl][sel]).double()
                prof = torch.exp(-((vch[None, :] - vel[c, 2][:, None]) / b[c][:, None]) ** 2) * dk[:, None]
                ta, tq, ei, eq = (k[c][:, None] * prof for k in coef)
                c2, s2_ = rot[0][c][:, None], rot[1][c][:, None]
                I0, Q0, U0 = I[sel], Q[sel], U[sel]
                Qn, Un = Q0 * c2 + U0 * s2_, U0 * c2 - Q0 * s2_
                p, n_ = ta - tq, ta + tq
                o11, o12 = 0.5 * (_phi(p) + _phi(n_)), -0.5 * (_phi(p) - _phi(n_))
                ch, sh = 0.5 * (torch.exp(-p) + torch.exp(-n_)), 0.5 * (torch.exp(-p) - torch.exp(-n_))
                I1 = o11 * ei + o12 * eq + ch * I0 - sh * Qn
                Q1 = o12 * ei + o11 * eq - sh * I0 + ch * Qn
                U1 = Un * torch.exp(-ta)
                on = ta > 1e-30
                I[sel] = torch.where(on, I1, I0)
                Q[sel] = torch.where(on, Q1 * c2 - U1 * s2_, Q0)
                U[sel] = torch.where(on, U1 * c2 + Q1 * s2_, U0)
                tau[sel] += torch.where(on, ta, 0.0)
                t = kd * dust[c] * tdx * dk
                e = torch.where(t > 1e-30, torch.exp(-t), 1.0)
                mu2 = 1.0 - fld[c, 2] ** 2
                B = planck[c] * (1.0 - e)
                Id[sel] = Id[sel] * e + B
                s0[sel] = s0[sel] * e + B
                sq[sel] = sq[sel] * e + 0.5 * alpha * (mu2 - 2.0 / 3.0) * B
                Qd[sel] = Qd[sel] * e + alpha * mu2 * B * torch.cos(2 * ph[c])
                Ud[sel] = Ud[sel] * e + alpha * mu2 * B * torch.sin(2 * ph[c])
                td[sel] += torch.where(t > 1e-30, t, 0.0)
            Id = Id - cmb
            on = Id != 0.0
            dq, du = (torch.where(on, Id * v / torch.where(on, s0 - sq, 1.0), 0.0) for v in (Qd, Ud))
            for q, v in enumerate((I - cmb, Q, U, tau)):
                cube[q, li, :, sl] = v.T
            for q, v in enumerate((Id, dq, du, torch.where(on, td, 0.0))):
                cube[4 + q, li, :, sl] = v[None, :]
    if not case["dust"]:
        cube[4:] = 0.0                                         # the call asks for four quantities
    if nodes:
        return cube, pos[:cloud.bulk_node_num, :2] * cloud.tx
    npx = 2 * case["pix"] + 1
    return cube.reshape(8, len(l1), nch, npx, npx), None


def _network(case, params):
    """The flat parameters as (weight, bias) per layer."""
    dims = [8] + [case["width"]] * case["depth"] + [2 * case["levels"]]
    p, at, layers = _t(params), 0, []
    for i in range(len(dims) - 1):
        w = p[at:at + dims[i] * dims[i + 1]].reshape(dims[i + 1], dims[i])
        at += w.numel()
        layers.append((w, p[at:at + dims[i + 1]]))
        at += dims[i + 1]
    return layers


def _forward(layers, x):
    for i, (w, b) in enumerate(layers):
        x = x @ w.T + b
        if i + 1 < len(layers):
            x = x * torch.sigmoid(x)
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "node_loop":
        if (4.0 if case["dust"] else 1.0) * _updates(case) > EXACT_UPDATES:
            return None
        cloud, mol = _cloud(case, seed)
        rc, star = _run_config(case, seed), _star(case, cloud)
        J0, J2 = _radiation_field(cloud, mol, rc, star)
        alive = np.arange(cloud.node_num)
        if star is not None:
            alive = alive[np.linalg.norm(cloud.xyz, axis=1) > star[1] / cloud.tx]
        pops = _solve_se(cloud, mol, rc.kmax, J0, J2, alive)
        return dict(J0=J0, J2=J2, status=None, segments=None, pops=pops)
    if kind == "batch":
        models, rc = _batch_models(case, seed), _run_config(case, seed)
        if sum(_updates(case, c.node_num, m.nlev) for c, m in models) > EXACT_UPDATES:
            return None
        out = []
        for cloud, mol in models:
            J0, J2 = _radiation_field(cloud, mol, rc)
            out.append((J0, J2, _solve_se(cloud, mol, rc.kmax, J0, J2, np.arange(cloud.node_num))))
        return dict(segments=None, models=out)
    if kind in ("image", "image_nodes"):
        cloud, mol = _cloud(case, seed)
        cube, xy = _stokes(case, cloud, mol, _pol_pops(cloud, mol, seed))
        return dict(cube=cube, status=None) if xy is None else dict(cube=cube, xy=xy, status=None)
    if kind == "se":
        cloud, mol = _cloud(case, seed)
        J0, J2 = _local_field(cloud, mol, seed)
        return dict(pops=_solve_se(cloud, mol, case["kmax"], _t(J0), _t(J2), np.arange(cloud.node_num)), status=None)
    if kind == "mlp_predict":
        params, stats, X, _ = _mlp_data(case, seed)
        st, n = _t(stats), 2 * case["levels"]
        y = _forward(_network(case, params), (_t(X) - st[:8]) / st[8:16])
        return dict(y=(y * st[16 + n:] + st[16:16 + n]))
    if kind == "mlp_gradients":
        params, _, X, Y = _mlp_data(case, seed)
        layers = [(w.clone().requires_grad_(), b.clone().requires_grad_()) for w, b in _network(case, params)]
        loss = ((_forward(layers, _t(X)) - _t(Y)) ** 2).mean()
        grads = torch.autograd.grad(loss, [p for layer in layers for p in layer])
        return dict(loss=float(loss), grads=torch.cat([g.reshape(-1) for g in grads]))
    # iterate: dozens of passes whose single pass node_loop and batch hold to 64 bits; mlp_train: the order
    # of its minibatches is the library's own
    return None
