"""Cases of use of the library: what its users' programs call, at sizes from
the smallest to the largest of the repository's configurations.

Families (each case names one as "kind"):

  map        images of query points under a stack of submaps (the flow-map
             evaluation): through the adapter's composite
             (`composite_sphere_diffeomorphism`), through map forms in the
             order given (a driver's sample grid), with the queries grouped
             by coarse cell and tangent Jacobians, or from host buffers
  sht        vorticity samples -> velocity jets (the inversion of every
             barotropic step), FP64 or split-BF16 form
  advect     one RK4 map update through three velocity levels and the
             assembly of the new map
  step       one whole barotropic step through the single calls, as a host
             driver makes it (map update, sample points through the stack,
             vorticity, inversion, velocity records)
  transport  a whole linear-transport run (analytic flow, remapping) and
             the tracer at its end
  gradient   the adjoint: misfit of the final vorticity and its gradient
             with respect to the initial spherical-harmonic coefficients

Every input is made on the GPU from the seed.  `exact` restates the same
results in plain torch FP64.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cmm-s2_gb300"))

F64 = torch.float64
JET_LATS = (-1.1, -0.5, 0.5, 1.1)
JET_PARAMS = (10.0, 0.1, 4.0) + JET_LATS      # amplitude, width, count, latitudes
ROT = 2 * math.pi
EPS = 1e-5


def listed():
    return [
        # a handful of tracer particles or a probe line through a young
        # run's map: the smallest call, launch latency
        {"name": "map_probe_l4", "kind": "map", "route": "adapter", "level": 4, "maps": 2, "n": 1000, "jac": False},
        # a plot or an error norm of a composed map on a coarse mesh, the
        # adapter's default path (coefficient records)
        {"name": "map_records_l5", "kind": "map", "route": "adapter", "level": 5, "maps": 6, "n": 250001,
         "jac": False},
        # the sample grid of a band-limit-512 run through a grown stack
        # with map forms (every step of a long run)
        {"name": "map_grid_l6", "kind": "map", "route": "grid", "level": 6, "maps": 12, "L": 512},
        # the flow-map evaluation configuration: level 7, 8 submaps, 2^24
        # uniform queries, points + ids + Jacobians, grouped by cell
        {"name": "map_jacobian_l7", "kind": "map", "route": "ordered", "level": 7, "maps": 8, "n": 1 << 24,
         "jac": True},
        # the same evaluation from and to host buffers, points and ids
        {"name": "map_host_l7", "kind": "map", "route": "host", "level": 7, "maps": 8, "n": 3000001, "jac": False},
        # the inversion of a small run's step (level 4 / L = 128 runs)
        {"name": "sht_l128", "kind": "sht", "precision": "fp64", "L": 128},
        # the inversion at the adjoint configuration's band-limit, FP64
        {"name": "sht_l512", "kind": "sht", "precision": "fp64", "L": 512},
        # the inversion of the large split-precision run
        {"name": "sht_split_l1024", "kind": "sht", "precision": "split_bf16", "L": 1024},
        # the map update of a level-6 / L = 512 run
        {"name": "advect_l6_L512", "kind": "advect", "level": 6, "L": 512},
        # a host-driven step of a middling run with a grown stack
        {"name": "step_l5_L256", "kind": "step", "level": 5, "L": 256, "maps": 6},
        # the transport test's loop at level 5 and its tracer
        {"name": "transport_l5", "kind": "transport", "level": 5, "steps": 42, "every": 10, "n": 100003},
        # forward and backward of a small data-assimilation gradient
        {"name": "gradient_l4_L96", "kind": "gradient", "level": 4, "L": 96, "steps": 8, "every": 4, "lmax": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.choice(("map", "map", "map", "sht", "sht", "advect", "step", "transport", "gradient"))
    if k == "map":
        route = rng.choice(("adapter", "grid", "ordered", "host"))
        c = {"kind": k, "route": route, "level": rng.randint(3, 7), "maps": rng.randint(1, 14)}
        if route == "grid":
            return {**c, "L": _log_int(rng, 33, 700)}
        hi = {"adapter": 1 << 20, "ordered": 1 << 22, "host": 1 << 21}[route]
        return {**c, "n": _log_int(rng, 500, hi), "jac": rng.random() < 0.4}
    if k == "sht":
        if rng.random() < 0.25:
            return {"kind": k, "precision": "split_bf16", "L": _log_int(rng, 32, 512)}
        return {"kind": k, "precision": "fp64", "L": _log_int(rng, 8, 600)}
    if k == "advect":
        return {"kind": k, "level": rng.randint(3, 6), "L": _log_int(rng, 24, 400)}
    if k == "step":
        return {"kind": k, "level": rng.randint(3, 5), "L": _log_int(rng, 24, 256), "maps": rng.randint(1, 8)}
    if k == "transport":
        return {"kind": k, "level": rng.randint(3, 5), "steps": rng.randint(10, 42), "every": rng.randint(4, 12),
                "n": _log_int(rng, 1000, 200000)}
    return {"kind": k, "level": rng.randint(3, 4), "L": _log_int(rng, 16, 110), "steps": rng.randint(5, 9),
            "every": rng.randint(2, 4), "lmax": rng.randint(6, 16)}


# ------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _d(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_dev())


def _sphere(n, seed):
    g = torch.Generator(device=_dev()).manual_seed(seed)
    x = torch.randn((n, 3), dtype=F64, device=_dev(), generator=g)
    return x / x.norm(dim=1, keepdim=True)


def _ico(level):
    from cmm_gpu.meshgen import icosahedral_mesh, stencil_frames
    verts, tris = icosahedral_mesh(level)
    tan, s_pts = stencil_frames(verts)
    return verts, tris, _d(tan), _d(s_pts)


def _grid(L):
    """Sample points ((L+1) 2L, 3) of band-limit L and the velocity mesh's arrays."""
    from cmm_gpu.meshgen import latlon_mesh_arrays
    theta, phi, grid, verts = latlon_mesh_arrays(L)
    return (theta, phi, grid, verts), _d(np.stack([g.reshape(-1) for g in grid], 1))


def _submaps(tan, s_pts, count, seed):
    """Jets (3,4,Nv) of `count` submaps: random rotations plus harmonic
    perturbations of amplitude 1e-2, as images of the stencil points."""
    rng = np.random.default_rng(seed)
    nv = s_pts.shape[2]
    p = s_pts.permute(1, 2, 0).reshape(-1, 3)
    out = []
    for _ in range(count):
        w, x, y, z = (lambda v: v / np.linalg.norm(v))(rng.standard_normal(4))
        R = _d(np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                         [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                         [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]]))
        k, ph = _d(rng.standard_normal((3, 3))), _d(rng.uniform(0, 2 * math.pi, 3))
        img = p @ R.T
        h = torch.sin(p @ k.T + ph)
        img = img + 1e-2 * (h - (h * img).sum(1, keepdim=True) * img)
        img = (img / img.norm(dim=1, keepdim=True)).reshape(4, nv, 3).permute(2, 0, 1)
        out.append(_stencil_jets(img, tan))
    return out


def _stencil_jets(img, tan):
    """Jets from the images (3,4,Nv) of the four stencil points."""
    m = img.mean(1)
    d1 = (img[:, 1] - img[:, 0] + img[:, 3] - img[:, 2]) / (4 * EPS)
    d2 = (img[:, 2] - img[:, 0] + img[:, 3] - img[:, 1]) / (4 * EPS)
    jets = torch.empty_like(img)
    jets[:, 0] = m / m.norm(dim=0)
    for k in range(3):
        jets[:, 1 + k] = (d1[k][:, None] * tan[0] + d2[k][:, None] * tan[1]).T
    return jets


class _Waves:
    """A smooth random field: a sum of plane waves restricted to the sphere."""

    def __init__(self, seed, count=12, kmax=9.0, amp=1.0):
        rng = np.random.default_rng(seed)
        k = rng.standard_normal((count, 3))
        k *= (rng.uniform(1.0, kmax, count) / np.linalg.norm(k, axis=1))[:, None]
        self.k, self.ph = _d(k), _d(rng.uniform(0, 2 * math.pi, count))
        self.a = _d(amp * rng.standard_normal(count) / np.linalg.norm(k, axis=1))

    def __call__(self, x):
        return torch.sin(x @ self.k.T + self.ph) @ self.a

    def scalar_jets(self, x):
        """(4, N): value and tangent gradient."""
        g = (torch.cos(x @ self.k.T + self.ph) * self.a) @ self.k
        g = g - (g * x).sum(1, keepdim=True) * x
        return torch.cat([self(x)[None], g.T]).contiguous()

    def velocity_jets(self, x):
        """(3,4,N) jets of u = x cross grad f: u_i, and at [c][1 + i] the
        tangent derivative of u_i along c."""
        c, s = torch.cos(x @ self.k.T + self.ph) * self.a, torch.sin(x @ self.k.T + self.ph) * self.a
        g = c @ self.k
        H = -torch.einsum("nw,wc,wk->nck", s, self.k, self.k)        # d_c g_k
        J = torch.zeros((len(x), 3, 3), dtype=F64, device=x.device)  # J[c][i] = d_c u_i
        for i in range(3):
            j, k = (i + 1) % 3, (i + 2) % 3                           # u_i = x_j g_k - x_k g_j
            J[:, :, i] = x[:, j, None] * H[:, :, k] - x[:, k, None] * H[:, :, j]
            J[:, j, i] += g[:, k]
            J[:, k, i] -= g[:, j]
        J = J - x[:, :, None] * (x[:, :, None] * J).sum(1, keepdim=True)
        u = torch.linalg.cross(x, g)
        return torch.stack([torch.cat([u[:, i][None], J[:, i].T]) for i in range(3)]).contiguous()


def _vorticity_in(x, seed):
    lat = torch.asin(x[:, 2].clamp(-1, 1))
    w = _Waves(seed, count=24, kmax=24.0, amp=3.0)(x)
    for l0 in JET_LATS:
        w = w + 10.0 * torch.exp(-((lat - l0) / 0.1) ** 2)
    return w


def _queries(case, seed):
    return _grid(case["L"])[1] if case["route"] == "grid" else _sphere(case["n"], seed + 1)


def _times(seed):
    """ts0, t and dt of a step whose three velocity levels sit at ts0 + k dt."""
    dt = 1.0 / 200
    k = 2 + seed % 7
    return (k - 2) * dt, k * dt, dt


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    return {"map": _prepare_map, "sht": _prepare_sht, "advect": _prepare_advect, "step": _prepare_step,
            "transport": _prepare_transport, "gradient": _prepare_gradient}[case["kind"]](case, seed)


def _prepare_map(case, seed):
    from cmm_gpu import native
    verts, tris, tan, s_pts = _ico(case["level"])
    jets = _submaps(tan, s_pts, case["maps"], seed)
    q = _queries(case, seed)
    s = {"case": case, "q": q}
    if case["route"] == "adapter":
        from cmm_gpu.mesh_functions import spherical_triangulation
        from cmm_gpu.spherical_spline import composite_sphere_diffeomorphism
        mesh = spherical_triangulation(verts, tris)
        comp = composite_sphere_diffeomorphism(mesh, jets, ns=list(range(1, len(jets) + 1)))
        for i, j in enumerate(jets):
            comp.assemble_coefficients(i, j)
        comp.Nc = len(jets)
        return {**s, "comp": comp}
    mesh = native.Mesh(verts, tris, case["level"])
    cs = [mesh.assemble(j) for j in jets]
    fs = [mesh.assemble_forms(c) for c in cs]
    s.update(mesh=mesh, cs=cs, fs=fs)
    if case["route"] == "grid":
        # the driver's current map stays on its coefficient record
        s["fs"] = fs[:-1] + [None]
        return s
    if case["jac"]:
        s["gs"] = [mesh.forms_ff(f) for f in fs]
    if case["route"] == "host":
        n = case["n"]
        s["q"] = q.cpu().pin_memory()
        s["out"] = torch.empty((n, 3), dtype=F64).pin_memory()
        s["tri"] = torch.empty(n, dtype=torch.int32).pin_memory()
        s["jac"] = torch.empty((n, 3, 3), dtype=F64).pin_memory() if case["jac"] else None
        s["scratch"] = s["streams"] = None
        # as on a program's second call: scratch and streams are kept
        s["scratch"], s["streams"] = _host_call(s)
    return s


def _host_call(s):
    from cmm_gpu import native
    return native.compose_host(s["mesh"], s["cs"], s["q"], s["out"], s["tri"], s["jac"], scratch=s["scratch"],
                               streams=s["streams"], forms=s["fs"], forms_ff=s.get("gs"))


def _prepare_sht(case, seed):
    from cmm_gpu import native
    (theta, phi, grid, verts), pts = _grid(case["L"])
    vm = native.VelMesh(case["L"], theta, phi, grid, verts)
    sht = native.Sht(case["L"])
    if case["precision"] == "split_bf16":
        sht.set_precision(native.Sht.SPLIT_BF16)
    return {"case": case, "vm": vm, "sht": sht,
            "omega": _vorticity_in(pts, seed).reshape(case["L"] + 1, 2 * case["L"]),
            "jets": torch.empty((3, 4, vm.nv), dtype=F64, device=_dev())}


def _prepare_advect(case, seed):
    from cmm_gpu import native
    verts, tris, tan, s_pts = _ico(case["level"])
    mesh = native.Mesh(verts, tris, case["level"])
    (theta, phi, grid, vverts), _ = _grid(case["L"])
    vm = native.VelMesh(case["L"], theta, phi, grid, vverts)
    vv = _d(vverts)
    vel = [vm.assemble(_Waves(seed + 100 + k).velocity_jets(vv)) for k in range(3)]
    prev = mesh.assemble(_submaps(tan, s_pts, 1, seed)[0])
    return {"case": case, "mesh": mesh, "vm": vm, "tan": tan, "s_pts": s_pts, "vel": vel, "prev": prev,
            "times": _times(seed), "jets": torch.empty((3, 4, mesh.nv), dtype=F64, device=_dev()),
            "work": torch.empty(native.lib.cmm_advect_workspace(mesh.h), dtype=F64, device=_dev()),
            "cur": mesh.new_coeffs()}


def _prepare_step(case, seed):
    from cmm_gpu import native
    s = _prepare_advect(case, seed)
    L = case["L"]
    mesh, vm = s["mesh"], s["vm"]
    pts = _grid(L)[1]
    from cmm_gpu.meshgen import latlon_mesh_arrays
    vv = _d(latlon_mesh_arrays(L)[3])
    stack = [mesh.assemble(j) for j in _submaps(s["tan"], s["s_pts"], case["maps"], seed + 7)]
    s.update(pts=pts, stack=stack, forms=[mesh.assemble_forms(c) for c in stack], sht=native.Sht(L),
             spline=vm.assemble(_Waves(seed + 200, amp=0.1).scalar_jets(vv)),
             X=torch.empty_like(pts), omega=torch.empty((L + 1, 2 * L), dtype=F64, device=_dev()),
             vjets=torch.empty((3, 4, vm.nv), dtype=F64, device=_dev()), vnew=vm.new_coeffs())
    return s


def _prepare_transport(case, seed):
    from cmm_gpu.mesh_functions import spherical_triangulation
    verts, tris, _, _ = _ico(case["level"])
    return {"case": case, "mesh": spherical_triangulation(verts, tris), "q": _sphere(case["n"], seed)}


def _prepare_gradient(case, seed):
    from cmm_gpu.adjoint import BVEGradient
    from cmm_gpu.workloads import random_sh_vorticity
    G = BVEGradient(case["level"], case["L"], case["steps"], case["steps"] / 200.0, n_maps=case["every"])
    sh = _d(random_sh_vorticity(case["lmax"], seed)[1])
    target = _vorticity_in(G.sample, seed).reshape(case["L"] + 1, 2 * case["L"])
    return {"case": case, "G": G, "sh": sh, "target": target}


# --------------------------------------------------------------------- run
def run(s):
    from cmm_gpu import native
    case = s["case"]
    kind = case["kind"]
    if kind == "map":
        return _run_map(s, case)
    if kind == "sht":
        return {"jets": s["sht"].velocity(s["vm"], s["omega"], jets=s["jets"])}
    if kind in ("advect", "step"):
        ts0, t, dt = s["times"]
        mesh, vm = s["mesh"], s["vm"]
        jets, _ = mesh.advect_project(vm, s["vel"], ts0, native.RK4, t, dt, s["s_pts"], s["tan"], s["prev"],
                                      jets=s["jets"], work=s["work"])
        cur = mesh.assemble(jets, out=s["cur"])
        if kind == "advect":
            return {"jets": jets, "records": cur}
        X = mesh.compose(s["stack"] + [cur], s["pts"], out=s["X"], forms=s["forms"] + [None])[0]
        om = vm.vorticity(native.VORT_GAUSSIAN_JETS, JET_PARAMS, X, ROT, omega=s["omega"], spline=s["spline"])
        vj = s["sht"].velocity(vm, om, jets=s["vjets"])
        return {"jets": jets, "X": X, "omega": om, "vjets": vj, "velocity": vm.assemble(vj, out=s["vnew"])}
    if kind == "transport":
        from cmm_gpu.dynamical_fields import u_deform_rot
        from cmm_gpu.spherical_transport import TransportSolver
        sol = TransportSolver(s["mesh"], u_deform_rot, T=1.0, Nt=case["steps"], remapping=True,
                              n_maps=case["every"]).run()
        return {"X": sol(s["q"]), "tracer": sol.tracer(s["q"]), "jets": sol.maps()[-1].vals}
    J, g = s["G"].gradient(s["sh"], s["target"])
    return {"J": J, "gradient": g}


def _run_map(s, case):
    if case["route"] == "adapter":
        if case["jac"]:
            return {"X": s["comp"](s["q"]), "jac": s["comp"].jacobian(s["q"])}
        return {"X": s["comp"](s["q"])}
    if case["route"] == "host":
        _host_call(s)
        return {k: s[n] for k, n in (("X", "out"), ("tri", "tri"), ("jac", "jac")) if s[n] is not None}
    mesh = s["mesh"]
    if case["route"] == "grid":
        return {"X": mesh.compose(s["cs"], s["q"], forms=s["fs"])[0]}
    perm = mesh.query_order(s["q"])
    X, tri, _, jac = mesh.compose(s["cs"], s["q"], want_tri=True, want_jac=case["jac"], perm=perm, forms=s["fs"],
                                  forms_ff=s.get("gs"))
    return {"X": X, "tri": tri, **({"jac": jac} if case["jac"] else {})}


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: inputs read once, outputs written once (vertex jets of maps and
    velocities, 96 B per vertex; mesh tables are not counted).  Operations:
    24 FP64 multiply-adds per map evaluation (72 with its two tangents), the
    Legendre sums by ring pairs, 100 per velocity evaluation."""
    k = case["kind"]
    nv = 10 * 4 ** case["level"] + 2 if "level" in case else 0
    L = case.get("L", 0)
    nu, ns = 2 + (L - 1) * 2 * L, (L + 1) * 2 * L
    advect = {"bytes": 8.0 * (12 * nv * 3 + 12 * nu * 3 + 57 * 2 * nv), "flops": 2.0 * 100 * 4 * 5 * nv}
    sht = {"bytes": 8.0 * (ns + 12 * nu), "flops": 2.0 * L ** 2 / 2 * (L / 2) * 2 * 13}
    if k == "map":
        n = ns if case["route"] == "grid" else case["n"]
        j = bool(case.get("jac"))
        ids = 4 if case["route"] in ("ordered", "host") else 0
        return {"bytes": float(n * (48 + ids + 72 * j) + 96 * nv * case["maps"]),
                "flops": 2.0 * n * case["maps"] * (72 if j else 24)}
    if k == "sht":
        return sht
    if k == "advect":
        return advect
    if k == "step":
        return {"bytes": advect["bytes"] + sht["bytes"] + 8.0 * (7 * ns + 57 * 2 * nu) + 96.0 * nv * case["maps"],
                "flops": advect["flops"] + sht["flops"] + 2.0 * ns * (24 * (case["maps"] + 1) + 60)}
    if k == "transport":
        maps = -(-case["steps"] // case["every"])
        return {"bytes": case["steps"] * 8.0 * 36 * nv + case["n"] * 2.0 * 80,
                "flops": case["steps"] * 2.0 * 60 * 4 * 5 * nv + 4.0 * case["n"] * 24 * maps}
    steps = case["steps"] + 1                                       # with the bootstrap's
    return {"bytes": 4 * steps * (advect["bytes"] + sht["bytes"]),
            "flops": 4 * steps * (advect["flops"] + sht["flops"] + 2.0 * ns * (case["lmax"] + 1) ** 2)}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    k = case["kind"]
    with torch.no_grad():
        if k == "map":
            verts, tris, tan, s_pts = _ico(case["level"])
            ps = _Patches(_d(verts), _d(tris.astype(np.int64)))
            recs = [ps.records(j) for j in _submaps(tan, s_pts, case["maps"], seed)]
            q = _queries(case, seed)
            loc = _Descent(ps, case["level"])
            X, J = torch.empty_like(q), torch.empty((len(q), 3, 3), dtype=F64, device=q.device)
            jac = bool(case.get("jac"))
            for i in range(0, len(q), 1 << 20):
                X[i:i + (1 << 20)], j = _compose(ps, loc, recs, q[i:i + (1 << 20)], jac)
                if jac:
                    J[i:i + (1 << 20)] = j
            X, J = (X.cpu(), J.cpu()) if case["route"] == "host" else (X, J)
            return {"X": X, **({"jac": J} if jac else {}),
                    **({"tri": None} if case["route"] in ("ordered", "host") else {})}
        if k == "sht":
            om = _vorticity_in(_grid(case["L"])[1], seed).reshape(case["L"] + 1, 2 * case["L"])
            return {"jets": _velocity_jets(om, case["L"])}
        if k in ("advect", "step"):
            return _exact_step(case, seed)
        if k == "transport":
            return _exact_transport(case, seed)
    return None      # the gradient: minutes of automatic differentiation


class _Patches:
    """Powell-Sabin spline patches on the triangles of a mesh."""
    #: ordinates by [argmin][argmax] barycentric, for V^2 E^2 C^2 VE EC VC
    TABLE = [[[0] * 6, [1, 13, 18, 6, 16, 7], [2, 13, 18, 11, 16, 10]],
             [[0, 14, 18, 5, 17, 4], [0] * 6, [2, 14, 18, 9, 17, 10]],
             [[0, 12, 18, 3, 15, 4], [1, 12, 18, 8, 15, 7], [0] * 6]]

    def __init__(self, verts, tris):
        self.verts, self.tris = verts, tris
        self.table = torch.tensor(self.TABLE, device=verts.device)
        v = self.v = [verts[tris[:, k]] for k in range(3)]
        unit = lambda a: a / a.norm(dim=1, keepdim=True)                   # noqa: E731
        dot = lambda a, b: (a * b).sum(1, keepdim=True)                    # noqa: E731
        det = lambda a, b, c: (a * torch.linalg.cross(b, c)).sum(1)        # noqa: E731
        bary = lambda a, b, c, p: [x / det(a, b, c) for x in (det(p, b, c), det(a, p, c), det(a, b, p))]  # noqa: E731
        tang = lambda a, b: unit(a - dot(a, b) * b)                        # noqa: E731
        c = unit(v[0] + v[1] + v[2])
        e = [unit(v[0] + v[1]), unit(v[1] + v[2]), unit(v[2] + v[0])]
        spec = []      # ordinate, its vertex, direction, gamma_vertex, gamma_other
        for o, k, to, mid, at in ((3, 0, v[1], e[0], 1), (5, 0, v[2], e[2], 1), (6, 1, v[2], e[1], 1),
                                  (8, 1, v[0], e[0], 1), (9, 2, v[0], e[2], 1), (11, 2, v[1], e[1], 1),
                                  (4, 0, c, e[0], 2), (7, 1, c, e[1], 2), (10, 2, c, e[2], 2)):
            h = tang(to - v[k], v[k])
            g = bary(v[k], mid, c, h)
            spec.append((o, k, h, g[0], g[at]))
        self.spec = spec
        self.mid = bary(v[0], v[1], v[2], c)
        self.eb = [bary(v[0], v[1], v[2], x) for x in e]
        self.n4 = (v[0] + v[1] + v[2]).norm(dim=1)
        self.ne = torch.stack([(v[1] + v[2]).norm(dim=1), (v[2] + v[0]).norm(dim=1), (v[0] + v[1]).norm(dim=1)], 1)
        # barycentrics relative to the first vertex, b = (1, 0, 0) + R (p - v0)
        a, b = v[1] - v[0], v[2] - v[0]
        d = (v[0] * torch.linalg.cross(a, b)).sum(1, keepdim=True)
        self.R = torch.stack([torch.linalg.cross(a, b) + torch.linalg.cross(v[0], b) + torch.linalg.cross(a, v[0]),
                              -torch.linalg.cross(v[0], b), torch.linalg.cross(v[0], a)], 1)
        self.R = self.R / d[:, :, None]

    def records(self, jets):
        """Ordinates (Nt, 19, C) of jets (3,4,Nv) or scalar jets (4,Nv)."""
        if jets.dim() == 2:
            val, grad = jets[0][:, None], jets[1:].T[:, :, None]
        else:
            val, grad = jets[:, 0].T, jets[:, 1:].permute(2, 0, 1)         # grad[v][j][k] = d_j f_k
        o = [None] * 19
        for k in range(3):
            o[k] = val[self.tris[:, k]]
        for i, k, h, g0, g1 in self.spec:
            o[i] = ((h[:, :, None] * grad[self.tris[:, k]]).sum(1) / 2 - g0[:, None] * o[k]) / g1[:, None]
        E, col = self.eb, lambda x: x[:, None]                             # noqa: E731
        o[12] = col(E[0][0]) * o[3] + col(E[0][1]) * o[8]
        o[13] = col(E[1][1]) * o[6] + col(E[1][2]) * o[11]
        o[14] = col(E[2][2]) * o[9] + col(E[2][0]) * o[5]
        o[15] = col(E[0][0]) * o[4] + col(E[0][1]) * o[7]
        o[16] = col(E[1][1]) * o[7] + col(E[1][2]) * o[10]
        o[17] = col(E[2][0]) * o[4] + col(E[2][2]) * o[10]
        o[18] = col(self.mid[0]) * o[4] + col(self.mid[1]) * o[7] + col(self.mid[2]) * o[10]
        return torch.stack(o, 1)

    def at(self, t, p):
        """The piecewise choice at points p in triangles t."""
        b = self._bary(t, p)
        lo, hi = b.argmin(1), b.argmax(1)
        tie = lo == hi
        return t, torch.where(tie, 1, lo), torch.where(tie, 0, hi)

    def _bary(self, t, p):
        b = torch.einsum("nij,nj->ni", self.R[t], p - self.v[0][t])
        b[:, 0] += 1
        return b

    def _gamma(self, where, b):
        t, lo, hi = where
        pick = lambda i: b.gather(1, i[:, None])[:, 0]                     # noqa: E731
        bl, bm, bh = pick(lo), pick(3 - lo - hi), pick(hi)
        return bh - bm, self.ne[t].gather(1, lo[:, None])[:, 0] * (bm - bl), self.n4[t] * bl

    def value(self, where, rec, p, tangents=()):
        """Patch values (N, C) at p, and the derivatives along `tangents`."""
        t, lo, hi = where
        V, E, C = (x[:, None] for x in self._gamma(where, self._bary(t, p)))
        o = [rec[t, self.table[lo, hi, k]] for k in range(6)]
        P = V * V * o[0] + E * E * o[1] + C * C * o[2] + 2 * (V * E * o[3] + E * C * o[4] + V * C * o[5])
        D = []
        for w in tangents:
            v, e, c = (x[:, None] for x in self._gamma(where, torch.einsum("nij,nj->ni", self.R[t], w)))
            D.append(2 * (v * (V * o[0] + E * o[3] + C * o[5]) + e * (E * o[1] + V * o[3] + C * o[4]) +
                          c * (C * o[2] + E * o[4] + V * o[5])))
        return (P, D) if tangents else P


class _Descent:
    """Triangles of an icosahedral refinement by descent from the 20 faces
    (child c of triangle f is 4 f + c: the three corners, then the middle)."""

    def __init__(self, ps, level):
        self.ps, self.level = ps, level

    def corners(self, f, j):
        k = self.level - j
        at = lambda c: self.ps.verts[self.ps.tris[f * 4 ** k + c * (4 ** k - 1) // 3, c]]   # noqa: E731
        return at(0), at(1), at(2)

    def __call__(self, p):
        side = lambda a, b: (torch.linalg.cross(a, b) * p).sum(1)          # noqa: E731
        best, f = None, None
        for g in range(20):
            a, b, c = (x.expand_as(p) for x in self.corners(torch.tensor(g, device=p.device), 0))
            s = torch.minimum(torch.minimum(side(a, b), side(b, c)), side(c, a))
            best, f = (s, torch.zeros_like(s, dtype=torch.long)) if g == 0 else \
                (torch.maximum(best, s), torch.where(s > best, g, f))
        for j in range(self.level):
            mbc, mca, mab = self.corners(4 * f + 3, j + 1)
            c = torch.where(side(mca, mab) < 0, 0, torch.where(side(mab, mbc) < 0, 1,
                                                               torch.where(side(mbc, mca) < 0, 2, 3)))
            f = 4 * f + c
        return f


def _tangents(q):
    e = torch.zeros_like(q)
    far = q[:, 2].abs() < 0.9
    e[far, 2] = 1
    e[~far, 0] = 1
    t1 = torch.linalg.cross(e, q)
    t1 = t1 / t1.norm(dim=1, keepdim=True)
    return t1, torch.linalg.cross(q, t1)


def _compose(ps, loc, recs, q, jac=False):
    p, base = q, _tangents(q) if jac else ()
    w = list(base)
    for rec in reversed(recs):
        where = ps.at(loc(p), p)
        if jac:
            P, w = ps.value(where, rec, p, w)
        else:
            P = ps.value(where, rec, p)
        r = P.norm(dim=1, keepdim=True)
        p = P / r
        w = [(x - (x * p).sum(1, keepdim=True) * p) / r for x in w]
    J = w[0][:, :, None] * base[0][:, None, :] + w[1][:, :, None] * base[1][:, None, :] if jac else None
    return p, J


def _legendre(L, theta):
    """Pbar_lm(theta) (m = 0..L-1, rings), one degree l at a time."""
    dev = theta.device
    x, s = torch.cos(theta), torch.sin(theta)
    m = torch.arange(L, dtype=F64, device=dev)
    pmm = torch.empty((L, len(theta)), dtype=F64, device=dev)
    pmm[0] = math.sqrt(1 / (4 * math.pi))
    for k in range(1, L):
        pmm[k] = -pmm[k - 1] * math.sqrt((2 * k + 1) / (2 * k)) * s
    p0, p1 = torch.zeros_like(pmm), torch.zeros_like(pmm)
    for l in range(L):
        below = m < l
        d = torch.where(below, l * l - m * m, 1.0)
        a = torch.where(below, torch.sqrt((4.0 * l * l - 1) / d), 0.0)
        b = torch.where(m < l - 1, torch.sqrt(((l - 1.0) ** 2 - m * m).clamp(min=0) / max(4.0 * (l - 1) ** 2 - 1, 1)),
                        0.0)
        p = a[:, None] * (x * p0 - b[:, None] * p1)
        p[l] = pmm[l]
        p1, p0 = p0, p
        yield l, p


def _velocity_jets(om, L):
    """Vorticity samples (L+1, 2L) -> velocity jets (3, 4, Nv)."""
    dev = om.device
    F = torch.fft.rfft(om, dim=1)[:, :L] * (math.pi / L)
    sign = torch.ones(L, dtype=F64, device=dev)
    sign[1::2] = -1
    G = torch.fft.fft(torch.cat([F, sign * F[1:L].flip(0)]), dim=0) / (2 * L)
    z = torch.zeros((2 * L - 1, L), dtype=G.dtype, device=dev)
    fine = torch.fft.ifft(torch.cat([G[:L], G[L:L + 1] / 2, z, G[L:L + 1] / 2, G[L + 1:]]), dim=0)[:2 * L + 1] * 4 * L
    j = torch.arange(2 * L + 1, dtype=F64, device=dev)
    k = torch.arange(1, L + 1, dtype=F64, device=dev)
    w = 1 - (torch.where(k == L, 1.0, 2.0) / (4 * k * k - 1) * torch.cos(math.pi * j[:, None] * k / L)).sum(1)
    w = w * torch.where((j == 0) | (j == 2 * L), 1.0, 2.0) / (2 * L)
    X = (fine * w[:, None]).T.contiguous()
    a = torch.zeros((L, L), dtype=G.dtype, device=dev)                     # [l, m]
    for l, P in _legendre(L, math.pi * j / (2 * L)):
        a[l, :l + 1] = torch.complex((P[:l + 1] * X.real[:l + 1]).sum(1), (P[:l + 1] * X.imag[:l + 1]).sum(1))
    l = torch.arange(L, dtype=F64, device=dev)[:, None]
    m = torch.arange(L, dtype=F64, device=dev)[None]
    psi = a * torch.where(l > 0, -1 / (l * (l + 1)).clamp(min=1), 0.0)

    def momentum(c):
        up = torch.cat([-c[:, 1:2].conj(), c[:, :-1]], 1) * torch.sqrt((l * (l + 1) - m * (m - 1)).clamp(min=0))
        dn = torch.cat([c[:, 1:], torch.zeros_like(c[:, :1])], 1) * torch.sqrt((l * (l + 1) - m * (m + 1)).clamp(min=0))
        keep = m <= l
        return [torch.where(keep, x, 0) for x in (0.5j * (up + dn), 0.5 * (up - dn), 1j * m * c)]

    u = momentum(psi)
    A = torch.stack(u + [g for f in u for g in momentum(f)])               # (12, l, m)
    S = torch.zeros((2, 12, L, L + 1), dtype=F64, device=dev)              # (re/im, field, m, ring)
    for d, P in _legendre(L, math.pi * torch.arange(L + 1, dtype=F64, device=dev) / L):
        S[0].addcmul_(P[None], A[:, d].real[:, :, None])
        S[1].addcmul_(P[None], A[:, d].imag[:, :, None])
    S = torch.complex(S[0], S[1]).permute(0, 2, 1)
    f = torch.fft.irfft(torch.cat([S, torch.zeros_like(S[:, :, :1])], 2), n=2 * L, dim=2) * 2 * L
    f = torch.cat([f[:, 0, :1], f[:, 1:-1].reshape(12, -1), f[:, -1, :1]], 1)
    x = _grid(L)[1].reshape(L + 1, 2 * L, 3)
    x = torch.cat([x[0, :1], x[1:-1].reshape(-1, 3), x[-1, :1]]).T
    jets = torch.empty((3, 4, f.shape[1]), dtype=F64, device=dev)
    for i in range(3):
        jets[i, 0] = f[i]
        c = torch.linalg.cross(f[3 + 3 * i:6 + 3 * i], x, dim=0)
        jets[:, 1 + i] = c - (c * x).sum(0) / x.norm(dim=0) * x
    return jets


class _LatLon:
    """Triangles of the lat-lon velocity mesh: ring and sector from the
    angles, near the rings corrected by the great circles of their edges,
    then the side of the cell's diagonal."""

    def __init__(self, L):
        self.L = L
        (theta, phi, grid, verts), _ = _grid(L)
        self.g = _d(grid).reshape(3, -1).T.contiguous()
        N, rows = 2 * L, L + 1
        k = torch.arange(N, device=_dev())
        k1 = (k + 1) % N
        node = lambda r, p: 1 + (r - 1) * N + p                            # noqa: E731
        tris = [torch.stack([torch.zeros_like(k), node(1, k), node(1, k1)], 1)]
        for r in range(1, rows - 2):
            tris.append(torch.stack([torch.stack([node(r, k), node(r + 1, k1), node(r, k1)], 1),
                                     torch.stack([node(r, k), node(r + 1, k), node(r + 1, k1)], 1)], 1).reshape(-1, 3))
        tris.append(torch.stack([node(L - 1, k), torch.full_like(k, len(verts) - 1), node(L - 1, k1)], 1))
        self.ps = _Patches(_d(verts), torch.cat(tris))

    def __call__(self, q):
        N, M = 2 * self.L, self.L + 1
        phi = torch.remainder(torch.atan2(q[:, 1], q[:, 0]), 2 * math.pi)
        th = torch.atan2(q[:, :2].norm(dim=1), q[:, 2])
        p = torch.floor(phi / (math.pi / self.L)).long() % N
        r = torch.floor(th / (math.pi / self.L)).long().clamp(0, M - 2)
        c = th / (math.pi / self.L) - r
        at = lambda ring, s: self.g[ring.clamp(0, M - 1) * N + s % N]      # noqa: E731
        lo, hi = (c <= 0.03) & (r != 0), (c > 0.85) & (r != M - 2)
        up = (torch.linalg.cross(at(r, p), at(r, p + 1)) * q).sum(1) > 0
        dn = (torch.linalg.cross(at(r + 1, p), at(r + 1, p + 1)) * q).sum(1) < 0
        r = torch.where(lo & up, r - 1, torch.where(hi & dn & ~lo, r + 1, r))
        s = ((torch.linalg.cross(at(r, p), at(r + 1, p + 1)) * q).sum(1) < 0).long()
        return torch.where(r == 0, p, torch.where(r == M - 2, 2 * N * (M - 2) - N + p, N + 2 * (N * (r - 1) + p) + s))


def _rk4(V, x, t, dt):
    unit = lambda y: y / y.norm(dim=1, keepdim=True)                       # noqa: E731
    v1 = V(t + dt, x)
    v2 = V(t + dt / 2, unit(x - dt * v1 / 2))
    v3 = V(t + dt / 2, unit(x - dt / 2 * v2))
    v4 = V(t, unit(x - dt * v3))
    return unit(x - dt / 6 * (v1 + 2 * v2 + 2 * v3 + v4))


def _update(ps, loc, prev, V, t, dt, tan, s_pts):
    """New jets of the map update (prev None: the identity before it)."""
    nv = len(ps.verts)
    y = _rk4(V, ps.verts, t, dt)
    st = _rk4(V, s_pts.permute(1, 2, 0).reshape(-1, 3), t, dt).reshape(4, nv, 3)
    if prev is not None:
        where = ps.at(loc(y), y)
        st = torch.stack([ps.value(where, prev, st[k]) for k in range(4)])
    return _stencil_jets(st.permute(2, 0, 1), tan)


def _exact_step(case, seed):
    L = case["L"]
    verts, tris, tan, s_pts = _ico(case["level"])
    ps = _Patches(_d(verts), _d(tris.astype(np.int64)))
    loc, vm = _Descent(ps, case["level"]), _LatLon(L)
    vel = [vm.ps.records(_Waves(seed + 100 + k).velocity_jets(vm.ps.verts)) for k in range(3)]
    ts0, t, dt = _times(seed)

    def V(at, x):
        a, b, c = at - ts0, at - ts0 - dt, at - ts0 - 2 * dt
        where = vm.ps.at(vm(x), x)
        return sum(w * vm.ps.value(where, r, x) for w, r in zip((b * c / (2 * dt * dt), -a * c / (dt * dt),
                                                                 a * b / (2 * dt * dt)), vel))

    jets = _update(ps, loc, ps.records(_submaps(tan, s_pts, 1, seed)[0]), V, t, dt, tan, s_pts)
    cur = ps.records(jets)
    if case["kind"] == "advect":
        return {"jets": jets, "records": torch.nn.functional.pad(cur.reshape(len(cur), 57), (0, 7))}
    pts = _grid(L)[1]
    X = _compose(ps, loc, [ps.records(j) for j in _submaps(tan, s_pts, case["maps"], seed + 7)] + [cur], pts)[0]
    lat = math.pi / 2 - torch.atan2(X[:, :2].norm(dim=1), X[:, 2])
    w = vm.ps.value(vm.ps.at(vm(X), X), vm.ps.records(_Waves(seed + 200, amp=0.1).scalar_jets(vm.ps.verts)), X)[:, 0]
    for l0 in JET_LATS:
        w = w + JET_PARAMS[0] * torch.exp(-((lat - l0) / JET_PARAMS[1]) ** 2)
    om = (w + 2 * ROT * (X[:, 2] / X.norm(dim=1) - pts[:, 2])).reshape(L + 1, 2 * L)
    vj = _velocity_jets(om, L)
    rec = vm.ps.records(vj)
    return {"jets": jets, "X": X, "omega": om, "vjets": vj,
            "velocity": torch.nn.functional.pad(rec.reshape(len(rec), 57), (0, 7))}


def _exact_transport(case, seed):
    verts, tris, tan, s_pts = _ico(case["level"])
    ps = _Patches(_d(verts), _d(tris.astype(np.int64)))
    loc = _Descent(ps, case["level"])

    def V(at, x):
        c, s = math.cos(2 * math.pi * at), math.sin(2 * math.pi * at)
        a = 4 * math.cos(math.pi * at)
        y = torch.stack([c * x[:, 0] + s * x[:, 1], c * x[:, 1] - s * x[:, 0], x[:, 2]], 1)
        f = torch.zeros_like(y)
        f[:, 1] = a * y[:, 1]
        u = torch.linalg.cross(y, f)
        u = torch.stack([c * u[:, 0] - s * u[:, 1], s * u[:, 0] + c * u[:, 1], u[:, 2]], 1)
        return u + 2 * math.pi * torch.stack([-x[:, 1], x[:, 0], torch.zeros_like(x[:, 0])], 1)

    dt = 1.0 / case["steps"]
    prev, recs, jets = None, [], None
    for k in range(case["steps"]):
        jets = _update(ps, loc, prev, V, k * dt, dt, tan, s_pts)
        prev = ps.records(jets)
        if (k + 1) % case["every"] == 0:
            recs.append(prev)
            prev = None
    X = _compose(ps, loc, recs + ([] if prev is None else [prev]), _sphere(case["n"], seed))[0]
    return {"X": X, "tracer": None, "jets": jets}
