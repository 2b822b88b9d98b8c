"""The work that users of capytaine_b200 have it do, as cases that can be timed and compared.

Every case goes through the public entry points: `Delhommeau.evaluate`, the
matrix-engine interface that capytaine's `BEMSolver` calls (`build_matrices`,
`linear_solver`, `build_S_matrix`, `build_fullK_matrix`), and the device
sweeps `solve_frequencies` and `solve_bodies`.  Bodies are the hemispheres,
barges, vertical cylinders and cylinder arrays of the repository's tests and
benchmark; the frequencies are those of ordinary sea states for their size
(below the first irregular frequency of a body without a lid).

`exact` restates Delhommeau's infinite-depth method in float64 with torch:
the tabulated integrals, the Rankine integrals, the dense solve.
"""
import functools
import math
import random

import numpy as np
import torch

from capytaine_b200.bodies import FloatingBody, join_bodies, rigid_body_dofs
from capytaine_b200.engine import B200Engine
from capytaine_b200.green_function import Delhommeau
from capytaine_b200.meshes import mesh_ellipsoid, mesh_parallelepiped, mesh_vertical_cylinder

RHO, G = 1000.0, 9.81
DOFS = ("Surge", "Sway", "Heave", "Roll", "Pitch", "Yaw")
# angular frequencies of interest per shape (rad/s): hemisphere of radius 1 m,
# barge of 80 x 20 x 10 m, vertical cylinder of radius 5 m and draft 20 m
BAND = {"sphere": (0.5, 4.2), "barge": (0.2, 1.2), "cylinder": (0.2, 1.8), "array": (0.3, 1.5)}
DEPTH = {"sphere": 4.0, "barge": 40.0, "cylinder": 60.0}

SWEEP = {"kind": "sweep", "precision": "mixed", "solver": "lu_decomposition", "method": "indirect", "symmetry": False,
         "lid": False, "finite_depth": False, "dofs": 6, "headings": 1, "batch": 8}


def listed():
    return [
        # one small call of the Green function from host code, matrices wanted on the host: latency
        {"name": "evaluate_sphere_100", "kind": "evaluate", "shape": "sphere", "r1": 10, "r2": 20, "r3": 0,
         "float32": False, "variant": "low_freq"},
        # capytaine's own BEMSolver driving the engine: one linear_solver call per right-hand side;
        # an odd resolution whose waterline cells are cut into triangles
        {"name": "dropin_sphere_735", "kind": "dropin", "shape": "sphere", "r1": 27, "r2": 49, "r3": 0, "dofs": 6,
         "headings": 1, "frequencies": 2},
        # free-surface elevation on a 50 x 50 grid and fluid velocities from known sources
        {"name": "points_barge_900", "kind": "points", "shape": "barge", "r1": 40, "r2": 10, "r3": 10,
         "points": 2500, "velocity_points": 300},
        # the small textbook sweep with the default (float64) engine
        {**SWEEP, "name": "sweep_fp64_sphere_800", "shape": "sphere", "r1": 40, "r2": 40, "r3": 0,
         "precision": "fp64", "dofs": 1, "frequencies": 20},
        # a hull with an interior lid, direct method, three headings, float64
        {**SWEEP, "name": "direct_fp64_cylinder_lid", "shape": "cylinder", "r1": 9, "r2": 62, "r3": 60,
         "precision": "fp64", "method": "direct", "lid": True, "headings": 3, "frequencies": 4},
        # float64 GMRES, capytaine's other solver
        {**SWEEP, "name": "gmres_cylinder_2520", "shape": "cylinder", "r1": 10, "r2": 60, "r3": 64,
         "precision": "fp64", "solver": "gmres", "frequencies": 4},
        # one request of a solve server: one frequency of a body of its own
        {**SWEEP, "name": "request_mixed_sphere_3741", "shape": "sphere", "r1": 86, "r2": 87, "r3": 0, "dofs": 3,
         "frequencies": 1},
        # coastal water: finite depth
        {**SWEEP, "name": "finite_depth_barge_2285", "shape": "barge", "r1": 61, "r2": 17, "r3": 16,
         "finite_depth": True, "frequencies": 6},
        # a parametric study: bodies of uneven sizes, a few frequencies of each
        {"name": "bodies_10_mixed", "kind": "bodies", "layout": 3, "bodies": 10, "low": 300, "high": 3000,
         "precision": "mixed", "dofs": 6, "headings": 1, "frequencies": 3},
        # the barge built with its two symmetry planes
        {**SWEEP, "name": "symmetric_barge_6084", "shape": "barge", "r1": 104, "r2": 26, "r3": 26, "symmetry": True,
         "frequencies": 15, "batch": 15},
        # the benchmark's sweep: 15 frequencies of the whole barge in one batch
        {**SWEEP, "name": "sweep_mixed_barge_6084", "shape": "barge", "r1": 104, "r2": 26, "r3": 26,
         "frequencies": 15, "batch": 15},
        # the largest: a 3 x 3 array of cylinders with lids, 54 dofs
        {**SWEEP, "name": "array_mixed_20493", "shape": "array", "r1": 8, "r2": 52, "r3": 64, "lid": True,
         "frequencies": 1},
    ]


def _log_between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _resolution(rng, shape, panels):
    """A resolution of `shape` with about `panels` immersed panels, odd numbers among them."""
    if shape == "sphere":
        a = max(4, int(round(math.sqrt(2 * panels) * rng.uniform(0.8, 1.2))))
        return a, max(4, round(2 * panels / a)), 0
    if shape == "barge":  # nx ny + (nx + ny) nz with ny = nz = nx / 4 (about)
        nx = max(4, round(math.sqrt(panels / 0.5625) * rng.uniform(0.9, 1.1)))
        ny = max(2, round(nx / 4))
        return nx, ny, max(2, 2 * round((panels - nx * ny) / (nx + ny) / 2))
    ntheta = max(8, round(math.sqrt(panels * 1.3) * rng.uniform(0.9, 1.1)))
    rows = max(3, round(panels / ntheta))
    nr = max(1, rows // 4)
    return nr, ntheta, 2 * (rows - nr)


def draw(rng):
    kind = rng.choice(["evaluate", "dropin", "points", "sweep", "sweep", "sweep", "sweep", "bodies"])
    shape = rng.choice(["sphere", "barge", "cylinder"])
    if kind == "bodies":
        return {"kind": "bodies", "layout": rng.randrange(1000), "bodies": rng.randint(3, 10),
                "low": _log_between(rng, 100, 500), "high": _log_between(rng, 1000, 3000),
                "precision": rng.choice(["mixed", "mixed", "fp64"]), "dofs": rng.randint(1, 6),
                "headings": rng.randint(1, 2), "frequencies": rng.randint(1, 3)}
    if kind == "sweep":
        c = dict(SWEEP)
        flavour = rng.choice(["fp64", "mixed", "finite", "gmres", "symmetric"])
        top = {"fp64": 3000, "mixed": 6000, "finite": 2500, "gmres": 3000, "symmetric": 6000}[flavour]
        panels = _log_between(rng, 100 if flavour != "symmetric" else 1000, top)
        c.update(precision="fp64" if flavour in ("fp64", "gmres") else rng.choice(["mixed", "mixed", "fp64"])
                 if flavour != "mixed" else "mixed",
                 solver="gmres" if flavour == "gmres" else "lu_decomposition",
                 method=rng.choice(["indirect", "indirect", "direct"]), symmetry=flavour == "symmetric",
                 finite_depth=flavour == "finite", dofs=rng.randint(1, 6), headings=rng.randint(1, 3),
                 frequencies=rng.randint(1, 6 if panels > 1500 else 15), batch=rng.choice([4, 8, 15]))
        if flavour == "symmetric":
            shape = "barge"
        c["lid"] = shape == "cylinder" and flavour in ("fp64", "mixed") and rng.random() < 0.4
    elif kind == "evaluate":
        panels = _log_between(rng, 50, 1200)
        c = {"kind": kind, "float32": rng.random() < 0.4, "variant": rng.choice(["low_freq", "low_freq", "high_freq"])}
    elif kind == "dropin":
        panels = _log_between(rng, 100, 1500)
        c = {"kind": kind, "dofs": rng.randint(1, 6), "headings": rng.randint(1, 2), "frequencies": rng.randint(2, 3)}
    else:
        panels = _log_between(rng, 200, 2500)
        c = {"kind": kind, "points": _log_between(rng, 300, 4000), "velocity_points": _log_between(rng, 50, 500)}
    r1, r2, r3 = _resolution(rng, shape, panels)
    if c.get("symmetry"):  # whole cells on each side of both planes
        r1, r2 = 2 * (r1 // 2), 2 * max(1, r2 // 2)
    return {**c, "shape": shape, "r1": r1, "r2": r2, "r3": r3}


# ---------------------------------------------------------------------------
# Inputs
def _mesh(case, rng):
    """The immersed mesh of the case, its lengths stretched by up to 5% by the seed."""
    sx, sy, sz = rng.uniform(0.95, 1.05, 3)
    res = (case["r1"], case["r2"], case["r3"])
    if case["shape"] == "sphere":
        return mesh_ellipsoid(semi_axes=(sx, sy, sz), resolution=res[:2]).immersed_part()
    if case["shape"] == "barge":
        return mesh_parallelepiped(size=(80 * sx, 20 * sy, 20 * sz), resolution=res,
                                   reflection_symmetry=case.get("symmetry", False)).immersed_part()
    return mesh_vertical_cylinder(length=40 * sz, radius=5 * sx, resolution=res).immersed_part()


def _body(case, rng):
    dofs = DOFS[:case["dofs"]] if case["dofs"] != 1 else ("Heave",)
    mesh = _mesh(case, rng)
    if case["shape"] != "array":
        return FloatingBody(mesh, rigid_body_dofs(only=dofs), lid_mesh=mesh.generate_lid() if case["lid"] else None)
    lid, bodies = mesh.generate_lid(), []
    for i in range(9):
        x, y = 30.0 * (i // 3 - 1), 30.0 * (i % 3 - 1)
        bodies.append(FloatingBody(mesh.translated((x, y, 0.0)), rigid_body_dofs(rotation_center=(x, y, 0.0)),
                                   lid_mesh=lid.translated((x, y, 0.0)), name=f"cyl{i}"))
    return join_bodies(*bodies)


def _uneven_bodies(case, rng):
    """Ellipsoids and vertical cylinders of uneven sizes; the case's layout fixes their panels."""
    r = random.Random(case["layout"])
    bodies = []
    for i in range(case["bodies"]):
        target = r.uniform(case["low"], case["high"])
        if i % 2 == 0:
            a = max(4, round(math.sqrt(target)))
            mesh = mesh_ellipsoid(semi_axes=[r.uniform(2, 8) for _ in range(3)], resolution=(a, 2 * a))
        else:
            radius, draft = r.uniform(2, 8), r.uniform(3, 15)
            h = math.sqrt((2 * math.pi * radius * draft + 2 * math.pi * radius ** 2) / target)
            mesh = mesh_vertical_cylinder(length=2 * draft, radius=radius, resolution=(
                max(1, round(radius / h)), max(8, round(2 * math.pi * radius / h)), 2 * max(1, round(draft / h))))
        mesh = mesh.immersed_part().scaled(rng.uniform(0.95, 1.05, 3))
        bodies.append(FloatingBody(mesh, rigid_body_dofs(only=DOFS[:case["dofs"]]), name=f"body{i}"))
    return bodies


def _inputs(case, seed):
    """Bodies, meshes, frequencies, headings, points and sources of the case, made from the seed."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "bodies":
        return {"bodies": _uneven_bodies(case, rng), "omegas": np.linspace(0.3, 0.9, case["frequencies"])
                * rng.uniform(0.97, 1.0), "headings": np.linspace(0.0, 1.0, case["headings"])}
    low, high = BAND[case["shape"]]
    if kind in ("evaluate", "points"):
        mesh = _mesh(case, rng)
        d = {"mesh": mesh, "wavenumber": rng.uniform(low, high) ** 2 / G}
        if kind == "points":
            size = np.ptp(mesh.vertices, axis=0)
            t, s = rng.uniform(0, 2 * np.pi, case["points"]), rng.uniform(1.0, 4.0, case["points"])
            d["points"] = np.stack([size[0] * s * np.cos(t), size[1] * s * np.sin(t), 0 * t], axis=1)
            d["fluid"] = d["points"][:case["velocity_points"]] - size * [0, 0, 1] * rng.uniform(
                0.05, 2.0, (case["velocity_points"], 1))
            d["sources"] = rng.standard_normal(mesh.nb_faces) + 1j * rng.standard_normal(mesh.nb_faces)
        return d
    nw = case["frequencies"]
    omegas = np.linspace(low, high, nw) if nw > 1 else np.array([0.5 * (low + high)])
    return {"body": _body({"lid": False, **case}, rng), "omegas": omegas * rng.uniform(0.97, 1.0),
            "headings": np.linspace(0.0, 1.0, case["headings"])}


def _dof_normals(body):
    """(ndof, nf) dof . n on the hull, zero on the lid; pressure weights -(dof . n) area; faces of hull and lid."""
    mesh, mask = body.mesh_including_lid.merged(), body.hull_mask
    vn = np.zeros((len(body.dofs), mesh.nb_faces))
    for d, dof in enumerate(body.dofs.values()):
        vn[d, mask] = np.sum(dof.evaluate_motion(mesh.faces_centers[mask]) * mesh.faces_normals[mask], axis=1)
    return vn, -vn * mesh.faces_areas, mesh, mask


def _boundary_conditions(vn, mesh, mask, omega, k, headings):
    """Columns: radiation -i omega (dof . n), then diffraction -(u_Airy . n) per heading."""
    c, n = mesh.faces_centers, mesh.faces_normals
    cols = list(-1j * omega * vn)
    for b in headings:
        e = G * k / omega * np.exp(k * c[:, 2] + 1j * k * (c[:, 0] * np.cos(b) + c[:, 1] * np.sin(b)))
        cols.append(-1.0 * mask * e * (np.cos(b) * n[:, 0] + np.sin(b) * n[:, 1] - 1j * n[:, 2]))
    return np.array(cols)


def prepare(case, seed):
    """Bodies with their geometry, and an engine whose tabulation is on the device."""
    d = _inputs(case, seed)
    if case["kind"] == "evaluate":
        d["gf"] = Delhommeau(floating_point_precision="float32" if case["float32"] else "float64",
                             gf_singularities=case["variant"], tabulation_cache_dir=None)
    else:
        d["gf"] = Delhommeau(tabulation_cache_dir=None)
        options = {k: case[v] for k, v in (("precision", "precision"), ("linear_solver", "solver"),
                                           ("method", "method"), ("max_batch", "batch")) if v in case}
        d["engine"] = B200Engine(green_function=d["gf"], **options)
    d["gf"].tabulated_integrals
    if case["kind"] == "dropin":
        vn, _, mesh, mask = _dof_normals(d["body"])
        d["rhs"] = [_boundary_conditions(vn, mesh, mask, w, w * w / G, d["headings"]) for w in d["omegas"]]
    d["depth"] = DEPTH[case["shape"]] if case.get("finite_depth") else np.inf
    d["kind"] = case["kind"]
    return d


def _results(r):
    return {"added_mass": r.added_mass, "radiation_damping": r.radiation_damping, "diffraction": r.diffraction,
            "froude_krylov": r.froude_krylov}


def run(d):
    kind = d["kind"]
    if kind == "evaluate":
        return d["gf"].evaluate(d["mesh"], d["mesh"], wavenumber=d["wavenumber"])
    engine = d["engine"]
    if kind == "dropin":  # bem/solver.py's order of calls for the indirect method
        mesh = d["body"].mesh_including_lid
        out = []
        for omega, rhs in zip(d["omegas"], d["rhs"]):
            S, K = engine.build_matrices(mesh, mesh, free_surface=0.0, water_depth=np.inf, wavenumber=omega ** 2 / G,
                                         adjoint_double_layer=True)
            out.append([S @ engine.linear_solver(K, b) for b in rhs])
        return np.array(out)
    if kind == "points":
        k = d["wavenumber"]
        potential = engine.build_S_matrix(d["points"], d["mesh"], wavenumber=k) @ d["sources"]
        gradient = engine.build_fullK_matrix(d["fluid"], d["mesh"], wavenumber=k)
        return {"potential": potential, "velocity": gradient @ d["sources"]}
    if kind == "bodies":
        return [_results(r) for r in engine.solve_bodies(d["bodies"], d["omegas"], wave_directions=d["headings"])]
    return _results(engine.solve_frequencies(d["body"], d["omegas"], wave_directions=d["headings"],
                                             water_depth=d["depth"]))


# ---------------------------------------------------------------------------
# Work: what a pass cannot do without
PAIR_FLOPS = 200  # float64 operations of one panel pair: interpolation of five integrals, two Rankine terms


@functools.lru_cache(maxsize=64)
def _panels(items):
    """Panel counts of a case's bodies (hull and lid)."""
    d = _inputs(dict(items), 0)
    if "bodies" in d:
        return tuple(b.mesh_including_lid.nb_faces for b in d["bodies"])
    return (d["mesh"].nb_faces,) if "mesh" in d else (d["body"].mesh_including_lid.nb_faces,)


def work(case):
    panels = _panels(tuple(sorted(case.items())))
    kind, n = case["kind"], panels[0]
    if kind == "evaluate":
        return {"bytes": 2 * (8 if case["float32"] else 16) * n * n, "flops": PAIR_FLOPS * n * n}
    if kind == "points":
        return {"bytes": 48 * case["velocity_points"] * n + 16 * case["points"],
                "flops": (PAIR_FLOPS + 8) * n * (case["points"] + case["velocity_points"])}
    nrhs = case["headings"] + (54 if case.get("shape") == "array" else case["dofs"])
    flops = bytes_ = 0.0
    for n in panels:
        systems = 4 if case.get("symmetry") else 1
        m = n / systems
        solve = 8 / 3 * m ** 3 if case.get("solver") != "gmres" else 20 * 8 * m * m * nrhs
        per_pair = PAIR_FLOPS + (4 * 60 + 16 * 20 if case.get("finite_depth") else 0)
        flops += case["frequencies"] * (per_pair * n * m + systems * (solve + 3 * 8 * m * m * nrhs))
        bytes_ += 400 * n + case["frequencies"] * 64 * nrhs * nrhs
        if kind == "dropin":
            bytes_ += case["frequencies"] * nrhs * 32 * n
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------
# The same results in float64 by torch
def exp_e1(z):
    """exp(z) E1(z) by the rational approximations of Delhommeau's thesis (p. 367), in complex128."""
    y = 1 / z
    far = y * (1 + y * (-1 + y * (2 + y * (-6 + y * (24 - 120 * y)))))
    side = 0.711093 / (z + 0.415775) + 0.278518 / (z + 2.29428) + 0.010389 / (z + 6.2900)
    p1 = 1 + z * (0.23721365 + z * (0.206543e-01 + z * (0.763297e-03 + z * 0.97087007e-05)))
    p2 = 0.99999207 + z * (-0.149545886e+01 + z * (0.41806426e-01 + z * (
        -0.3000591e-01 + z * (0.19387339e-02 - z * 0.51801555e-03))))
    q = 1 + z * (-0.76273617 + z * (0.28388363 + z * (-0.66786033e-01 + z * (
        0.12982719e-01 + z * (-0.8700861e-03 + z * 0.2989204e-03)))))
    near = -(torch.log(z) * p1 + 0.5772156649 * p2) / q
    a = (1 + 1.3935496e-06j, 15.82958 - 20.14222j, -70.52863 - 227.9511j, -985.4221 - 226.6272j,
         -1202.318 + 1580.907j, 953.2441 + 1342.447j, 417.3716 - 196.6665j, -9.881266 - 24.24952j)
    b = (1 + 0j, 16.83184 - 20.14481j, -55.66969 - 248.1167j, -1068.640 - 434.4707j, -2082.250 + 1522.471j,
         383.3455 + 2730.378j, 1216.791 + 351.7189j, 115.3926 - 161.2647j, -3.777369 - 4.510900j)
    zc = torch.where(z.imag < 0, z, z.conj())  # the approximation is given for one half plane
    num, den = a[0] * zc, b[0] * zc
    for i in range(1, 8):
        num = (num + a[i]) * (zc if i < 7 else 1)
    for i in range(1, 9):
        den = (den + b[i]) * (zc if i < 8 else 1)
    mid = num / den
    mid = torch.where(z.imag < 0, mid, mid.conj())
    return torch.where(z.real < -16, far, torch.where(z.imag.abs() > 10, side, torch.where(z.real > -0.5, near, mid)))


@functools.lru_cache(maxsize=1)
def _table():
    """Default grids (676 x 372) and the five tabulated integrals over theta (Simpson, 1001 points)."""
    nr, nz, one = 676, 372, 81
    i = np.arange(1, nr + 1, dtype=np.float32)
    r = np.where(i < one, np.float32(10) ** (np.float32(-10) * (1 - (i - 1) / np.float32(one - 1))),
                 (100.0 - 1) / (nr - one) * (i.astype(float) - one) + 1)
    r[0] = 0.0
    dz = (math.log10(251.0) + 10) / nz
    z = -np.minimum(10 ** (dz * np.arange(1, nz + 1) - 10), 251.0)
    r, z = (torch.as_tensor(v, dtype=torch.float64, device="cuda") for v in (r, z))
    n = 1001
    out = torch.zeros((5, nr, nz), dtype=torch.float64, device="cuda")
    for k in range(n):
        cos = math.cos(-math.pi / 2 + math.pi * k / (n - 1))
        step = math.pi / (3 * (n - 1)) * (1 if k in (0, n - 1) else 4 if k % 2 else 2)
        zeta = torch.complex(z[None, :].expand(nr, nz), (r * cos)[:, None].expand(nr, nz))
        e = torch.where(zeta.real <= -30, 0, torch.exp(zeta))
        j = exp_e1(zeta) + 1j * math.pi * e
        jm = j - 1 / zeta
        out[0] += step * j.real
        out[1] += step * jm.real
        out[2] += step * e.real
        out[3] -= step * cos * jm.imag
        out[4] -= step * cos * e.imag
    return r, z, out * torch.tensor([2 / math.pi, 2 / math.pi, 2, 2 / math.pi, 2], device="cuda")[:, None, None], dz


def _integrals(r, z):
    """The five integrals at (r, z): 3 x 3 Lagrange interpolation, or their asymptotic form."""
    rg, zg, tab, dz = _table()
    nr, nz, one = len(rg), len(zg), 81
    i = torch.where(r < 1e-10, 1.0, torch.where(
        r < 1, (torch.log10(r) / 10 + 1) * (one - 1) + 1, (r - 1) * (nr - one) / 99.0 + one))
    j = (torch.log10(z.abs()) + 10) / dz

    def node(x, n):  # halves away from zero
        return (torch.floor(x.abs() + 0.5) * torch.sign(x)).nan_to_num(1.0, 2e9, -2e9).clamp(2, n - 1).long() - 1

    def weights(x, u):
        return [(x - u[1]) * (x - u[2]) / ((u[0] - u[1]) * (u[0] - u[2])),
                (x - u[2]) * (x - u[0]) / ((u[1] - u[2]) * (u[1] - u[0])),
                (x - u[0]) * (x - u[1]) / ((u[2] - u[0]) * (u[2] - u[1]))]
    i, j = node(i, nr), node(j, nz)
    wr, wz = weights(r, [rg[i + a] for a in (-1, 0, 1)]), weights(z, [zg[j + a] for a in (-1, 0, 1)])
    flat = tab.reshape(5, -1)
    acc = 0
    for a in range(3):
        for b in range(3):
            acc = acc + (wr[a] * wz[b]) * flat[:, (i + a - 1) * nz + j + b - 1]
    inv_r, inv_r1 = 1 / r.clamp(min=1e-10), 1 / torch.hypot(r, z)
    e, c, s = torch.exp(z) * torch.sqrt(2 * math.pi * inv_r), torch.cos(r - math.pi / 4), torch.sin(r - math.pi / 4)
    far = torch.stack([2 * (-e * s + z * inv_r1 ** 3 - inv_r1), 2 * (-e * s + z * inv_r1 ** 3), 2 * e * c,
                       2 * (-e * (c - s * inv_r / 2) + r * inv_r1 ** 3), -2 * e * (s + c * inv_r / 2)])
    return torch.where((z.abs() < zg[-1].abs()) & (r < rg[-1]), acc, far)


def _norm(*x):
    """Euclidean norm accumulated with scaling, as Fortran's NORM2: the threshold between exact and
    one-point integration meets ties on regular meshes."""
    scale, total = torch.zeros_like(x[0]), torch.ones_like(x[0])
    for v in x:
        a = v.abs()
        big, p, q = scale < a, scale / a, a / scale
        total = torch.where(a == 0, total, torch.where(big, 1 + total * p * p, total + q * q))
        scale = torch.where(big, a, scale)
    return scale * torch.sqrt(total)


def _rankine(M, f, far):
    """Integral over the face of 1 / |M - x| and its gradient at M: (4, rows, faces); one point where far."""
    d = M[:, :, None] - f["c"].T[:, None, :]
    ro = torch.sqrt((d * d).sum(0))
    out = torch.cat([(f["area"] / ro)[None], -d * (f["area"] / ro ** 3)])
    out = torch.where(ro > 1e-7, out, 0)
    row, col = torch.nonzero(~far, as_tuple=True)
    M, n, v, radius = M[:, row], f["n"].T[:, col], f["v"].permute(1, 2, 0)[:, :, col], f["radius"][col]
    gz = ((M - f["c"].T[:, col]) * n).sum(0)
    rr = [(M - v[a]).square().sum(0).sqrt() for a in range(4)]
    sgn, agz = torch.copysign(torch.ones_like(gz), gz), gz.abs()
    g, dg = 0, 0
    for a in range(4):
        b = (a + 1) % 4
        e = v[b] - v[a]
        dk = e.square().sum(0).sqrt()
        gyx = torch.linalg.cross(n, e / dk, dim=0)
        gy = ((M - v[a]) * gyx).sum(0)
        s = rr[a] + rr[b]
        ant, dnt, anl, dnl = 2 * gy * dk, s * s - dk * dk + 2 * agz * s, s + dk, s - dk
        aldn = torch.log(anl / dnl)
        at = torch.where(agz >= 1e-4 * radius, torch.atan(ant / dnt), 0)
        ax = (M - v[a]) / rr[a] + (M - v[b]) / rr[b]
        dntx = 2 * (s + agz) * ax + 2 * sgn * s * n
        keep = dk >= 1e-3 * radius
        g = g + torch.where(keep, torch.where(gy.abs() < 1e-5, 0, gy * aldn) - 2 * at * agz, 0)
        t = (aldn * gyx - 2 * sgn * at * n + gy * (dnl - anl) / (anl * dnl) * ax
             - 2 * agz / (ant ** 2 + dnt ** 2) * (2 * dk * gyx * dnt - dntx * ant))
        dg = dg + torch.where(keep, t, 0)
    out[:, row, col] = torch.cat([g[None], dg])
    return out


def _faces(mesh):
    f = {"c": mesh.faces_centers, "n": mesh.faces_normals, "area": mesh.faces_areas, "radius": mesh.faces_radiuses,
         "v": mesh.vertices[mesh.faces]}
    return {k: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device="cuda") for k, v in f.items()}


def _green(M, f, k, variant):
    """G and its gradient at the points M (3, rows): Rankine terms (the direct one apart) and wave term."""
    c = f["c"].T
    d = M[:, :, None] - c[:, None, :]
    direct = _rankine(M, f, _norm(d[0], d[1], d[2]) > 7 * f["radius"])
    image = M * torch.tensor([1.0, 1.0, -1.0], dtype=torch.float64, device="cuda")[:, None]
    h = _norm(d[0], d[1])
    refl = _rankine(image, f, torch.hypot(h, image[2][:, None] - c[2]) > 7 * f["radius"])
    refl[3] = -refl[3]
    high = variant == "high_freq"
    r, z = k * h, k * (M[2][:, None] + c[2])
    own = (r.abs() < 1e-10) & (z.abs() < 1e-10)  # a panel of the free surface with itself
    z = torch.where(own, -1.0, z)
    i = _integrals(r, z)
    slope = torch.where(r.abs() > 1e-14, k * k / r, 0)
    r1 = torch.hypot(r, z)
    radial, gre = (i[3] - 2 * r / r1 ** 3, i[1]) if high else (i[3], i[0])
    vertical = k * gre - 2 * k * z / r1 ** 3 if high else k * (gre + 2 / r1)
    w = k * f["area"]
    real = w * torch.stack([gre, slope * d[0] * radial, slope * d[1] * radial, vertical])
    imag = w * torch.stack([i[2], slope * d[0] * i[4], slope * d[1] * i[4], k * i[2]])
    zero = torch.zeros_like(gre)
    own_g = w * (1 - torch.log(k * k * f["area"] / math.pi) + 2 * (float(np.float32(0.5772156649)) - math.log(2)))
    own_re = torch.stack([zero + own_g, zero, zero, zero + k * (own_g + 4 * torch.sqrt(math.pi * f["area"]))])
    own_im = torch.stack([zero - 2 * math.pi * w, zero, zero, zero - 2 * math.pi * k * w])
    real, imag = torch.where(own, own_re, real), torch.where(own, own_im, imag)
    return direct, torch.complex(real + (-refl if high else refl), imag)


def _matrices(mesh, k, points=None, normals=None, variant="low_freq", adjoint=True, full=False):
    """S and K (with the dot product, or the gradient's three planes when full) of points (default: the
    mesh's own centres) against the faces of mesh."""
    f = _faces(mesh)
    own = points is None
    P, n = (f["c"], f["n"]) if own else (torch.as_tensor(v, dtype=torch.float64, device="cuda") for v in (points, normals))
    N = len(f["area"])
    S = torch.empty((len(P), N), dtype=torch.complex128, device="cuda")
    K = torch.empty(((3,) if full else ()) + (len(P), N), dtype=torch.complex128, device="cuda")
    step = max(1, 3_000_000 // N)
    for a in range(0, len(P), step):
        rows = slice(a, a + step)
        direct, rest = _green(P[rows].T, f, k, variant)
        if adjoint:
            g = direct + rest
        else:
            sign = torch.tensor([1.0, -1.0, -1.0, 1.0], dtype=torch.float64, device="cuda")[:, None, None]
            g = rest * sign + torch.cat([direct[:1], -direct[1:]])
        S[rows] = g[0]
        if full:
            K[:, rows] = g[1:]
        else:
            m = (n[rows].T[:, :, None] if adjoint else f["n"].T[:, None, :])
            K[rows] = (m * g[1:]).sum(0)
    S *= -1 / (4 * math.pi)
    K *= -1 / (4 * math.pi)
    if not full:
        i = torch.arange(min(len(P), N), device="cuda")
        K[i, i] += torch.where(f["c"][i, 2].abs() < 1e-8, 1.0, 0.5)
    return S, K


def _four_images(cols):
    """The whole matrix of a mesh with two symmetry planes from its first block column."""
    n = cols.shape[1]
    return torch.cat([torch.cat([cols[(i ^ j) * n:(i ^ j) * n + n] for i in range(4)]) for j in range(4)], dim=1)


def _solve(body, omegas, headings, method="indirect", symmetry=False):
    vn, weights, mesh, mask = _dof_normals(body)
    pw = torch.as_tensor(weights, dtype=torch.complex128, device="cuda")
    c = mesh.faces_centers
    nd = len(vn)
    out = {k: [] for k in ("added_mass", "radiation_damping", "diffraction", "froude_krylov")}
    for w in omegas:
        k = w * w / G
        if symmetry:
            quarter = body.mesh.half.half
            S, K = (_four_images(m) for m in _matrices(quarter, k, c, mesh.faces_normals,
                                                             adjoint=method == "indirect"))
        else:
            S, K = _matrices(mesh, k, adjoint=method == "indirect")
        b = torch.as_tensor(_boundary_conditions(vn, mesh, mask, w, k, headings).T.copy(), device="cuda")
        phi = S @ torch.linalg.solve(K, b) if method == "indirect" else torch.linalg.solve(K, S @ b)
        F = (1j * w * RHO * (pw @ phi)).T.cpu().numpy()
        out["added_mass"].append(F[:nd].real / w ** 2)
        out["radiation_damping"].append(F[:nd].imag / w)
        out["diffraction"].append(F[nd:])
        p = RHO * G * np.exp(k * c[:, 2])[None] * np.exp(
            1j * k * (np.outer(np.cos(headings), c[:, 0]) + np.outer(np.sin(headings), c[:, 1])))
        out["froude_krylov"].append(p @ weights.T)
        del S, K
    return {k: np.array(v) for k, v in out.items()}


def exact(case, seed):
    if case.get("finite_depth"):
        return None  # the values hang on a fitted decomposition into exponentials, which has no exact form
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "evaluate":
        S, K = _matrices(d["mesh"], d["wavenumber"], variant=case["variant"])
        return S, K
    if kind == "points":
        k, s = d["wavenumber"], torch.as_tensor(d["sources"], device="cuda")
        S, _ = _matrices(d["mesh"], k, d["points"], 0 * d["points"])
        _, grad = _matrices(d["mesh"], k, d["fluid"], 0 * d["fluid"], full=True)
        return {"potential": S @ s, "velocity": grad @ s}
    if kind == "dropin":
        vn, _, mesh, mask = _dof_normals(d["body"])
        out = []
        for w in d["omegas"]:
            S, K = _matrices(mesh, w * w / G)
            b = _boundary_conditions(vn, mesh, mask, w, w * w / G, d["headings"])
            out.append((S @ torch.linalg.solve(K, torch.as_tensor(b.T.copy(), device="cuda"))).T)
        return torch.stack(out)
    if kind == "bodies":
        return [_solve(b, d["omegas"], d["headings"]) for b in d["bodies"]]
    return _solve(d["body"], d["omegas"], d["headings"], case["method"], case["symmetry"])
