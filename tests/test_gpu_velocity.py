"""GPU parity: lat-lon velocity mesh location, the velocity interpolant, the
backward integrators and the CMM map update against the reference's golden
outputs and the oracle.

Tolerances: lat-lon triangle ids bit-exact; velocities within 1e-12
(relative to max |u|); foot points within 1e-13; new jet values within
1e-12; jet gradients (centred differences with step 1e-5, which amplify
rounding by 1e5) within 1e-9."""
import os

import numpy as np
import pytest
import torch

from conftest import GOLDEN
from oracle import geometry as OG
from oracle import spline as OS
from oracle import evolution as OE

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    import __graft_entry__
    __graft_entry__.build()
    from cmm_gpu import native
    return native


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    return t.cpu().numpy()


def golden(name):
    return np.load(os.path.join(GOLDEN, name))


def velmesh(nat, L):
    from cmm_gpu.meshgen import latlon_mesh_arrays
    theta, phi, grid, verts = latlon_mesh_arrays(L)
    return nat.VelMesh(L, theta, phi, grid, verts), verts


def test_latlon_arrays_match_reference():
    from cmm_gpu.meshgen import latlon_mesh_arrays
    d = golden("velocity_L8.npz")
    theta, phi, grid, verts = latlon_mesh_arrays(8)
    np.testing.assert_array_equal(verts, d["verts"])


def test_latlon_locate_matches_reference(nat):
    """Bit-exact triangle ids, except queries lying on a triangle edge or
    vertex (ring points, meridians), which may resolve to another triangle
    that contains them."""
    d = golden("velocity_L8.npz")
    vm, verts = velmesh(nat, 8)
    tri, bcc = vm.locate(dev(d["q"]))
    tri, bcc = host(tri), host(bcc)
    mu = OG.LatLonMesh(8)
    diff = tri != d["tri"]
    on_edge = OG.edge_distance(mu.vertices, mu.simplices, d["tri"], d["q"]) <= 1e-14
    assert not (diff & ~on_edge).any(), np.nonzero(diff & ~on_edge)
    assert (bcc[diff].min(axis=1) >= -1e-13).all()
    same = ~diff
    np.testing.assert_allclose(bcc[same], d["bcc"][same], rtol=0, atol=1e-13)
    print(f"{diff.sum()} of {len(tri)} edge/vertex queries resolved to another container")


@pytest.mark.parametrize("L", [16, 128, 1024])
def test_latlon_locate_random(nat, L):
    from cmm_gpu.meshgen import random_sphere_points
    q = random_sphere_points(100_000, seed=L)
    vm, _ = velmesh(nat, L)
    tri, _ = vm.locate(dev(q))
    _, ref, _ = OG.LatLonMesh(L).query(q)
    np.testing.assert_array_equal(host(tri), ref)


def vel_coeffs(nat, vm, vals):
    return [vm.assemble(dev(vals[n])) for n in range(3)]


def test_velocity_matches_reference(nat):
    d = golden("velocity_L8.npz")
    vm, _ = velmesh(nat, 8)
    vc = vel_coeffs(nat, vm, d["vals"])
    rec = host(vc[1])[:, :57].reshape(-1, 19, 3).transpose(2, 1, 0)
    np.testing.assert_allclose(rec, d["coeffs"][1], rtol=0, atol=1e-12)
    u = host(vm.velocity(vc, 0.0, float(d["t"]), float(d["dt"]), dev(d["q"].T)))
    scale = np.abs(d["vel"]).max()
    np.testing.assert_allclose(u / scale, d["vel"] / scale, rtol=0, atol=1e-12)
    for nvs in (1, 2):
        u = host(vm.velocity(vc[:nvs], 0.0, 0.17, 0.1, dev(d["q"].T)))
        U = OS.VelocityOracle(OG.LatLonMesh(8), d["vals"], d["ts"])
        for n in range(3):
            U.init_coeffs(n)
        U.nVs = nvs
        np.testing.assert_allclose(u / scale, U(0.17, 0.1, d["q"].T) / scale, rtol=0, atol=1e-12)


@pytest.mark.parametrize("scheme,nvs", [(0, 1), (1, 2), (2, 3)])
def test_integrators_against_oracle(nat, scheme, nvs):
    from cmm_gpu.meshgen import random_sphere_points
    d = golden("velocity_L8.npz")
    vm, _ = velmesh(nat, 8)
    vc = vel_coeffs(nat, vm, d["vals"])[:nvs]
    x = random_sphere_points(5000, seed=scheme).T.copy()
    out = host(vm.integrate(vc, 0.0, scheme, 0.05, 0.1, dev(x)))
    U = OS.VelocityOracle(OG.LatLonMesh(8), d["vals"], d["ts"])
    for n in range(3):
        U.init_coeffs(n)
    U.nVs = nvs
    f = [OE.euler_back, OE.improved_euler_back, OE.rk4_back][scheme]
    ref = f(0.05, 0.1, x, U)
    np.testing.assert_allclose(out, ref, rtol=0, atol=1e-13)


def test_advect_project_matches_reference(nat):
    a, m, v = golden("advect_l3_L8.npz"), golden("mesh_l3.npz"), golden("velocity_L8.npz")
    verts, tris = m["verts"], m["tris"]
    mesh = nat.Mesh(verts, tris, 3)
    vm, _ = velmesh(nat, 8)
    vc = vel_coeffs(nat, vm, v["vals"])
    tan, s_pts = OG.stencil_points(verts)
    prev = mesh.assemble(dev(a["jets_prev"]))
    jets, work = mesh.advect_project(vm, vc, 0.0, nat.RK4, 0.05, 0.1, dev(s_pts), dev(tan), prev)
    jets, yn = host(jets), host(work)[:3 * len(verts)].reshape(3, -1)
    # the reference integrates the same points (RK4_proj) -> foot points
    U = OS.VelocityOracle(OG.LatLonMesh(8), v["vals"], v["ts"])
    for n in range(3):
        U.init_coeffs(n)
    U.nVs = 3
    yref = OE.rk4_back(0.05, 0.1, verts.T, U)
    np.testing.assert_allclose(yn, yref, rtol=0, atol=1e-13)
    # vertices whose foot point lies on a mesh edge may be evaluated in
    # either neighbouring triangle (the reference's Qhull choice is one)
    loc = OG.QhullLocator(verts)
    near = OG.edge_distance(verts, tris, loc.locate(yref.T), yref.T) <= 1e-14
    ok = ~near
    # (1) against the oracle evaluated in closed form (the same linear maps
    #     with the per-triangle inverse vertex matrix the kernels use)
    prev_o = OS.MapOracle(verts, tris, loc, a["jets_prev"], closed=True)
    sn = OE.rk4_back(0.05, 0.1, s_pts.reshape(3, -1), U).reshape(s_pts.shape)
    jo = OE.jets_from_stencil(prev_o.stencil_eval(yref, sn), tan)
    np.testing.assert_allclose(jets[:, 0][:, ok], jo[:, 0][:, ok], rtol=0, atol=1e-12)
    # rounding differences (~1e-15: FMA contraction, summation order) times
    # the 1/(4 eps) = 2.5e4 difference quotient
    np.testing.assert_allclose(jets[:, 1:][..., ok], jo[:, 1:][..., ok], rtol=0, atol=5e-10)
    # (2) against the reference: values within 1e-12; gradients within the
    #     reference's own rounding noise (its four per-point determinant
    #     evaluations round independently and the 1/(4 eps) difference
    #     amplifies that by 2.5e4: the closed-form oracle differs from the
    #     reference by up to ~9e-9 here)
    ref = a["jets_rk4"]
    noise = np.abs(jo[:, 1:][..., ok] - ref[:, 1:][..., ok]).max()
    assert noise < 2e-8
    np.testing.assert_allclose(jets[:, 0][:, ok], ref[:, 0][:, ok], rtol=0, atol=1e-12)
    np.testing.assert_allclose(jets[:, 1:][..., ok], ref[:, 1:][..., ok], rtol=0, atol=2 * noise + 1e-10)
    np.testing.assert_allclose(jets[..., near], ref[..., near], rtol=0, atol=1e-6)
    for scheme, nvs, key in ((nat.EULER, 1, "jets_euler"), (nat.IMPROVED_EULER, 2, "jets_ieuler")):
        j, _ = mesh.advect_project(vm, vc[:nvs], 0.0, scheme, 0.0, 0.1, dev(s_pts), dev(tan), None)
        j = host(j)
        np.testing.assert_allclose(j[:, 0], a[key][:, 0], rtol=0, atol=1e-12)
        np.testing.assert_allclose(j[:, 1:], a[key][:, 1:], rtol=0, atol=1e-9)
    assert mesh.status() == 0 and vm.status() == 0


def test_fp32_velocity_records(nat):
    """cmm_velmesh_set_records(CMM_REC_FP32): FP32 ordinates and FP32
    patches against the FP64 records on the same velocity jets; stated
    error 1e-6 of max |u| (FP32 rounding of ordinates ~1e-7 relative), and
    the RK4 foot points (FP64 accumulation) within dt * 1e-6 * max |u|."""
    from cmm_gpu.meshgen import random_sphere_points
    d = golden("velocity_L8.npz")
    vm64, _ = velmesh(nat, 8)
    vm32, _ = velmesh(nat, 8)
    vm32.set_records(nat.VelMesh.REC_FP32)
    c64 = vel_coeffs(nat, vm64, d["vals"])
    c32 = vel_coeffs(nat, vm32, d["vals"])
    assert c32[0].dtype == torch.float32
    np.testing.assert_allclose(host(c32[1]), host(c64[1]).astype(np.float32), rtol=2e-6, atol=1e-6)
    x = random_sphere_points(20000, seed=11).T.copy()
    u64 = host(vm64.velocity(c64, 0.0, 0.13, 0.1, dev(x)))
    u32 = host(vm32.velocity(c32, 0.0, 0.13, 0.1, dev(x)))
    scale = np.abs(u64).max()
    err = np.abs(u32 - u64).max() / scale
    print(f"FP32 velocity records: relative velocity error {err:.2e}")
    assert 1e-10 < err < 1e-6
    f64 = host(vm64.integrate(c64, 0.0, 2, 0.05, 0.1, dev(x)))
    f32 = host(vm32.integrate(c32, 0.0, 2, 0.05, 0.1, dev(x)))
    assert np.abs(f32 - f64).max() < 0.1 * 1e-6 * scale


@pytest.mark.parametrize("L", [8, 40, 512])
def test_latlon_locate_next_to_cell_boundaries(nat, L):
    """Triangle ids of points 1e-4 .. 1e-12 rad off the rings and meridians
    (inside the FP32 angles' error bound from 2e-6 rad on), and off the 0.03 and
    0.85 thresholds of the row corrections, against the reference's rule."""
    rng = np.random.default_rng(L)
    n = 4000
    off = rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-12, -4, n)
    theta, phi = rng.uniform(0.02, np.pi - 0.02, n), rng.uniform(0, 2 * np.pi, n)
    h = np.pi / L
    ring = (np.rint(theta / h) + rng.choice([0.0, 0.03, 0.85], n)) * h
    pts = [(ring + off, phi), (theta, np.rint(phi / h) * h + off), (ring + off, np.rint(phi / h) * h - off[::-1])]
    q = np.concatenate([np.stack([np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)], 1) for t, p in pts])
    vm, _ = velmesh(nat, L)
    tri = host(vm.locate(dev(q))[0])
    mu = OG.LatLonMesh(L)
    _, ref, _ = mu.query(q)
    diff = tri != ref
    assert (OG.edge_distance(mu.vertices, mu.simplices, ref[diff], q[diff]) <= 1e-13).all()
    assert diff.mean() < 0.02


@pytest.mark.parametrize("nvs", [1, 2, 3])
def test_velocity_scales_exactly_and_at_its_limits(nat, nvs):
    """The velocity evaluation works relative to the largest ordinate of a
    patch, so a power of two in the jets comes out exactly; zero jets, jets
    beyond the scaled range, weights beyond 2 (times far from the levels) and
    points off the unit sphere take the FP64 evaluation.  Against the oracle
    within 1e-12 of max |u| throughout."""
    from cmm_gpu.meshgen import random_sphere_points
    d = golden("velocity_L8.npz")
    vm, _ = velmesh(nat, 8)
    vals = d["vals"][:nvs]
    vc = [vm.assemble(dev(v)) for v in vals]
    x = dev(np.ascontiguousarray(random_sphere_points(5003, seed=3).T))
    V = vm.velocity(vc, 0.0, 0.05, 0.1, x)
    for k in (-300, -40, 7, 300):
        s = [vm.assemble(dev(v * 2.0 ** k)) for v in vals]
        assert torch.equal(vm.velocity(s, 0.0, 0.05, 0.1, x), V * 2.0 ** k)
    scale = float(V.abs().max())
    tiny = [vm.assemble(dev(v * 2.0 ** -1000)) for v in vals]
    assert float((vm.velocity(tiny, 0.0, 0.05, 0.1, x) * 2.0 ** 1000 - V).abs().max()) < 1e-12 * scale
    assert not vm.velocity([torch.zeros_like(c) for c in vc], 0.0, 0.05, 0.1, x).any()
    # a level of another magnitude beside the others
    if nvs > 1:
        mixed = [vc[0] * 2.0 ** -80] + vc[1:]
        z = [torch.zeros_like(vc[0])] + vc[1:]
        a, b = vm.velocity(mixed, 0.0, 0.05, 0.1, x), vm.velocity(z, 0.0, 0.05, 0.1, x)
        assert float((a - b).abs().max()) < 1e-15 * scale
    # weights beyond 2: the same combination of the levels' own velocities
    t = 0.93
    w = {1: [1.0], 2: [1 - t / 0.1, t / 0.1],
         3: [(t - 0.1) * (t - 0.2) / 0.02, -t * (t - 0.2) / 0.01, t * (t - 0.1) / 0.02]}[nvs]
    far = vm.velocity(vc, 0.0, t, 0.1, x)
    ref = sum(c * vm.velocity([v], 0.0, 0.0, 0.1, x) for c, v in zip(w, vc))
    assert float((far - ref).abs().max()) < 1e-12 * scale * max(abs(c) for c in w)
    # off the sphere: homogeneous of degree 2
    out = vm.velocity(vc, 0.0, 0.05, 0.1, 1.5 * x)
    assert float((out / 2.25 - V).abs().max()) < 1e-12 * scale
    assert vm.status() == 0


@pytest.mark.parametrize("width", [0.1, 1e-6, 1e-9])
def test_narrow_gaussian_jets(nat, width):
    """Jets narrower than the FP32 spacing of their latitudes (6e-8 at 0.75), one
    on either side of an FP32 value, at points around them: every term that
    counts is in the sum.  Against numpy on the same coordinates; the
    colatitude's rounding (3e-16) over the width is an error of that size in
    d, at most 1 in the slope of exp(-d^2): 1e-15 + 1e-15 / width."""
    L = 24
    vm, _ = velmesh(nat, L)
    lats = np.array([0.75 + 1e-10, 0.75 - 3e-8, -0.4])
    lat = 0.75 + np.linspace(-5e-8, 5e-8, 2 * L * (L + 1))
    lat[::7] = lats[0] + width * np.linspace(-2, 2, len(lat[::7]))
    lat[::11] = -0.4 + width * np.linspace(-2, 2, len(lat[::11]))
    X = np.stack([np.cos(lat), np.zeros_like(lat), np.sin(lat)], 1)
    got = host(vm.vorticity(nat.VORT_GAUSSIAN_JETS, [1.0, width, 3.0, *lats], dev(X), 0.0)).reshape(-1)
    la = np.pi / 2 - np.arctan2(np.sqrt(X[:, 1]**2 + X[:, 0]**2), X[:, 2])
    ref = np.exp(-((la[:, None] - lats) / width)**2).sum(1)
    assert np.abs(got - ref).max() < 20 * 2.0**-52 + 1e-15 / width
    assert vm.status(clear=True) == 0


def exact_amplitude(verts, p):
    """(b_hi - b_mid + e (b_mid - b_lo) + c b_lo)^2 of the points p (n, 3) in the
    triangles of verts (n, 3, 3): the patch whose ordinates are all 1, in
    50-digit arithmetic from the vertices."""
    import decimal
    ctx = decimal.Context(prec=50)
    out = []
    for V, q in zip(verts, p):
        with decimal.localcontext(ctx):
            V = [[decimal.Decimal(float(x)) for x in v] for v in V]
            q = [decimal.Decimal(float(x)) for x in q]
            det = lambda a, b, c: sum(a[i] * (b[(i + 1) % 3] * c[(i + 2) % 3] - b[(i + 2) % 3] * c[(i + 1) % 3])
                                      for i in range(3))
            norm = lambda *vs: sum(sum(x)**2 for x in zip(*vs)).sqrt()
            D = det(*V)
            b = [det(q, V[1], V[2]) / D, det(V[0], q, V[2]) / D, det(V[0], V[1], q) / D]
            lo, mid, hi = sorted(range(3), key=lambda k: b[k])
            out.append(float((b[hi] - b[mid] + norm(V[hi], V[mid]) * (b[mid] - b[lo]) + norm(*V) * b[lo])**2))
    return np.array(out)


@pytest.mark.parametrize("L,colat", [(512, 1.57), (1024, 1.57), (512, 0.6), (512, 0.02), (128, 1.55), (24, 1.5)])
def test_velocity_barycentrics_no_worse_than_fp64(nat, L, colat):
    """The fixed-point evaluation near the equator, where the triangles are
    largest, and towards the pole, where their inverses are: the patch whose
    ordinates are all 1 (so its value is the barycentrics' error and nothing
    else) at 1500 points, largest error against 50 digits no larger than that
    of the FP64 evaluation, which points of norm 2 take (homogeneous of degree
    2, exactly a factor of 4)."""
    vm, verts = velmesh(nat, L)
    tv = OG.LatLonMesh(L).simplices
    rng = np.random.default_rng(L)
    n = 1500
    th, ph = colat + 0.015 * rng.uniform(-1, 1, n), rng.uniform(0, 2 * np.pi, n)
    p = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], 1)
    ones = vm.new_coeffs()
    ones[:, :57] = 1.0
    tri = host(vm.locate(dev(p))[0])
    ref = exact_amplitude(verts[tv[tri]], p)
    fixed = host(vm.velocity([ones], 0.0, 0.0, 0.1, dev(p.T)))
    wide = host(vm.velocity([ones], 0.0, 0.0, 0.1, dev(2 * p.T))) / 4
    assert np.abs(fixed - ref).max() <= np.abs(wide - ref).max()


@pytest.mark.parametrize("w", [2.0, 3.0, 3.9999999, 4.0, 4.0000001, 5.5])
def test_velocity_weights_either_side_of_the_fixed_range(nat, w):
    """Two levels at a time whose second weight is w (the fixed-point range
    ends at 4): the combination of the levels' own velocities, 1e-14 of the
    largest term (each within 1e-15)."""
    from cmm_gpu.meshgen import random_sphere_points
    d = golden("velocity_L8.npz")
    vm, _ = velmesh(nat, 8)
    vc = [vm.assemble(dev(v)) for v in d["vals"][:2]]
    x = dev(np.ascontiguousarray(random_sphere_points(3001, seed=5).T))
    a, b = (vm.velocity([c], 0.0, 0.0, 0.125, x) for c in vc)
    got = vm.velocity(vc, 0.0, w * 0.125, 0.125, x)
    scale = max(float(a.abs().max()), float(b.abs().max())) * w
    assert float((got - ((1 - w) * a + w * b)).abs().max()) < 1e-14 * scale
