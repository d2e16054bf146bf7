"""GPU parity: point location, assembly, map evaluation, composition,
stencil evaluation and Jacobians of libcmmgpu.so against the oracle and the
reference's golden outputs.

Tolerances: triangle ids bit-exact except for queries within 1e-14 of an
edge of the oracle's triangle (either neighbour contains them; counted);
FP64 map coordinates within 1e-12 (relative to |X| = 1); barycentrics and
ordinates within 1e-13; Jacobians within 1e-10 (relative to |J|)."""
import os

import numpy as np
import pytest
import torch

from conftest import GOLDEN
from oracle import geometry as OG
from oracle import spline as OS

pytestmark = pytest.mark.gpu
EDGE_TOL = 1e-14


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


def coeff_record_to_ref(rec, nt):
    """(nt,64) device record -> reference layout (3,19,nt)."""
    return rec[:, :57].reshape(nt, 19, 3).transpose(2, 1, 0)


@pytest.mark.parametrize("level", [3, 4])
def test_locate_matches_reference_qhull(nat, level):
    d = golden(f"mesh_l{level}.npz")
    m = nat.Mesh(d["verts"], d["tris"], level)
    tri, bcc = m.locate(dev(d["q"]))
    tri, bcc = host(tri), host(bcc)
    diff = tri != d["tri"]
    near = OG.edge_distance(d["verts"], d["tris"], d["tri"], d["q"]) <= EDGE_TOL
    assert not (diff & ~near).any()
    # a disagreement is another container of the query
    assert (OG.edge_distance(d["verts"], d["tris"], tri[diff], d["q"][diff]) <= EDGE_TOL).all()
    same = ~diff
    np.testing.assert_allclose(bcc[same], d["bcc"][same], rtol=0, atol=1e-13)
    assert m.status() == 0
    print(f"level {level}: {diff.sum()} of {len(tri)} near-edge queries resolved to the neighbour")


def qhull_case(level):
    """The Qhull-order fixture of a large level (tests/golden/make_golden.py
    qhull_fixture): the reference's triangle table and find_simplex ids of
    seeded random queries; vertices and queries regenerated here and
    checked against the fixture's digests."""
    import hashlib
    from cmm_gpu.meshgen import icosahedral_mesh, random_sphere_points
    d = golden(f"qhull_l{level}.npz")
    verts, _ = icosahedral_mesh(level)
    assert hashlib.sha256(np.ascontiguousarray(verts).tobytes()).hexdigest() == str(d["verts_sha"])
    qr = random_sphere_points(int(d["nq"]), seed=int(d["seed"]))
    assert hashlib.sha256(np.ascontiguousarray(qr).tobytes()).hexdigest() == str(d["q_sha"])
    return verts, d["tris"], np.concatenate([qr, d["q_special"]]), d["tri"], d["bcc"]


@pytest.mark.parametrize("level", [5, 6])
def test_locate_matches_reference_qhull_large_levels(nat, level):
    """Bit-exact triangle ids in the reference's own (Qhull) row order at
    levels 5 and 6, except within 1e-14 of an edge (counted)."""
    if not os.path.exists(os.path.join(GOLDEN, f"qhull_l{level}.npz")):
        pytest.skip(f"qhull_l{level}.npz not generated")
    verts, tris, q, ref_tri, ref_bcc = qhull_case(level)
    m = nat.Mesh(verts, tris, level)
    tri, bcc = m.locate(dev(q))
    tri, bcc = host(tri), host(bcc)
    diff = tri != ref_tri
    near = OG.edge_distance(verts, tris, ref_tri, q) <= EDGE_TOL
    assert not (diff & ~near).any(), int((diff & ~near).sum())
    assert (OG.edge_distance(verts, tris, tri[diff], q[diff]) <= EDGE_TOL).all()
    # barycentrics: the reference's determinant ratios carry a rounding
    # error ~eps/h^2 (h the edge length), which grows 4x per level: 1e-13
    # at level 4, scaled by 4 per level above it
    same = ~diff
    np.testing.assert_allclose(bcc[same], ref_bcc[same], rtol=0, atol=1e-13 * 4.0 ** (level - 4))
    assert m.status() == 0
    print(f"level {level}: {int(near.sum())} queries within 1e-14 of an edge, "
          f"{int(diff.sum())} resolved to the neighbour, of {len(tri)}")


@pytest.mark.parametrize("level", [5, 7])
def test_locate_large_levels_against_cone_oracle(nat, level):
    from cmm_gpu.meshgen import icosahedral_mesh, random_sphere_points
    verts, tris = icosahedral_mesh(level)
    q = random_sphere_points(200_000, seed=level)
    m = nat.Mesh(verts, tris, level)
    tri, bcc = m.locate(dev(q))
    tri = host(tri)
    ref = OG.ConeLocator(verts, tris).locate(q)
    diff = tri != ref
    near = OG.edge_distance(verts, tris, ref, q) <= EDGE_TOL
    assert not (diff & ~near).any()
    b = host(bcc)
    assert b.min() > -1e-12
    assert m.status() == 0


def test_assemble_matches_reference(nat):
    d, g = golden("map_l3.npz"), golden("mesh_l3.npz")
    m = nat.Mesh(g["verts"], g["tris"], 3)
    rec = host(m.assemble(dev(d["jets"][0])))
    np.testing.assert_allclose(coeff_record_to_ref(rec, len(g["tris"])), d["coeffs0"], rtol=0, atol=1e-13)


def test_map_eval_and_composite_match_reference(nat):
    d, g = golden("map_l3.npz"), golden("mesh_l3.npz")
    m = nat.Mesh(g["verts"], g["tris"], 3)
    cs = [m.assemble(dev(j)) for j in d["jets"]]
    out, tri, _, _ = m.compose(cs[:1], dev(d["q"]), want_tri=True)
    out = host(out)
    # split-centre ties: the reference's three barycentrics are bitwise
    # equal, its tables select the degenerate sub-triangle (v1,v1,v1) and it
    # returns NaN or, when the 0/0 determinants round to finite values, the
    # vertex ordinate c0.  The spline's value there is the centre ordinate,
    # which the library returns (equal to the tie-broken oracle).
    b = g["bcc"]
    tie = (b[:, 0] == b[:, 1]) & (b[:, 1] == b[:, 2])
    assert tie.sum() > 0 and (~np.isfinite(d["img"]).all(0) <= tie).all()
    ok = ~tie
    np.testing.assert_allclose(out[ok], d["img"].T[ok], rtol=0, atol=1e-12)
    orc = OS.MapOracle(g["verts"], g["tris"], OG.ConeLocator(g["verts"], g["tris"]), d["jets"][0],
                       tie_fix=True)
    np.testing.assert_allclose(out[tie], orc(d["q"][tie]).T, rtol=0, atol=1e-12)
    cout, _, _, _ = m.compose(cs, dev(d["q"]))
    cout = host(cout)
    fin = np.isfinite(d["comp_img"]).all(1) & ~tie
    np.testing.assert_allclose(cout[fin], d["comp_img"][fin], rtol=0, atol=1e-12)
    assert np.isfinite(cout).all()
    assert m.status() == 0


def test_stencil_eval_matches_reference(nat):
    d, g = golden("map_l3.npz"), golden("mesh_l3.npz")
    m = nat.Mesh(g["verts"], g["tris"], 3)
    c = m.assemble(dev(d["jets"][0]))
    st = host(m.stencil_eval(c, dev(d["yn"]), dev(d["sp"])))
    np.testing.assert_allclose(st, d["st"], rtol=0, atol=1e-12)


def make_stack(level, S, seed):
    from cmm_gpu.meshgen import icosahedral_mesh
    from cmm_gpu.workloads import submap_stack
    verts, tris = icosahedral_mesh(level)
    tan, s_pts = OG.stencil_points(verts)
    return verts, tris, submap_stack(s_pts, tan, S, seed=seed)


def test_composition_level5_eight_submaps(nat):
    from cmm_gpu.meshgen import random_sphere_points
    verts, tris, jets = make_stack(5, 8, seed=11)
    q = random_sphere_points(20_000, seed=12)
    m = nat.Mesh(verts, tris, 5)
    cs = [m.assemble(dev(j)) for j in jets]
    out, tri, tri_all, _ = m.compose(cs, dev(q), want_tri=True, want_tri_all=True)
    comp = OS.CompositeOracle(verts, tris, OG.ConeLocator(verts, tris), jets, tie_fix=True)
    ref, rtri, pts = comp(q, record=True)
    np.testing.assert_allclose(host(out), ref, rtol=0, atol=1e-12)
    ta = host(tri_all)[::-1]          # application order: submap S-1 first
    np.testing.assert_array_equal(host(tri), ta[0])
    for s in range(8):
        diff = ta[s] != rtri[s]
        near = OG.edge_distance(verts, tris, rtri[s], pts[s]) <= 1e-13
        assert not (diff & ~near).any(), s


def test_jacobian_against_oracle_and_differences(nat):
    from cmm_gpu.meshgen import random_sphere_points
    verts, tris, jets = make_stack(4, 3, seed=21)
    q = random_sphere_points(3000, seed=22)
    m = nat.Mesh(verts, tris, 4)
    cs = [m.assemble(dev(j)) for j in jets]
    out, _, _, jac = m.compose(cs, dev(q), want_jac=True)
    comp = OS.CompositeOracle(verts, tris, OG.ConeLocator(verts, tris), jets, tie_fix=True)
    X, J = OS.composite_jacobian(comp, q)
    J_gpu = host(jac)
    scale = np.abs(J).max(axis=(1, 2))[:, None, None]
    np.testing.assert_allclose(J_gpu / scale, J / scale, rtol=0, atol=1e-10)
    # tangent map: J q = 0 and X . J = 0
    assert np.abs(np.einsum("nij,nj->ni", J_gpu, q)).max() < 1e-12
    assert np.abs(np.einsum("ni,nij->nj", host(out), J_gpu)).max() < 1e-12
    # central differences along a tangent direction (away from edges)
    t = np.cross(q, [0.3, -0.5, 0.8])
    t /= np.linalg.norm(t, axis=1)[:, None]
    h = 1e-6
    qp = q + h * t
    qm = q - h * t
    qp /= np.linalg.norm(qp, axis=1)[:, None]
    qm /= np.linalg.norm(qm, axis=1)[:, None]
    fp, _, tap, _ = m.compose(cs, dev(qp), want_tri_all=True)
    fm, _, tam, _ = m.compose(cs, dev(qm), want_tri_all=True)
    same = (host(tap) == host(tam)).all(0)
    fd = (host(fp) - host(fm)) / (2 * h)
    an = np.einsum("nij,nj->ni", J_gpu, t)
    assert same.mean() > 0.9
    np.testing.assert_allclose(fd[same], an[same], rtol=0, atol=2e-6 * np.abs(an).max())


def test_edge_cases(nat):
    from cmm_gpu.meshgen import icosahedral_mesh
    verts, tris = icosahedral_mesh(2)
    m = nat.Mesh(verts, tris, 2)
    c = m.new_coeffs()
    empty = torch.empty((0, 3), dtype=torch.float64, device="cuda")
    out, tri, _, _ = m.compose([c], empty, want_tri=True)
    assert out.shape == (0, 3)
    q = dev(np.array([[np.nan, 0.0, 1.0], [0.0, 0.0, 1.0]]))
    tri, _ = m.locate(q)
    assert host(tri)[0] == -1
    assert m.status(clear=True) & nat.FLAG_NONFINITE
    assert m.status() == 0
    with pytest.raises(nat.CmmError) as e:
        m.compose([c] * 1025, dev(np.zeros((1, 3))))
    assert e.value.code == 1
    with pytest.raises(TypeError):
        m.locate(torch.zeros((3, 3)))
    # the poles and the 12 base vertices locate without a status flag
    q = dev(verts[[0, -1] + list(range(1, 11))])
    tri, bcc = m.locate(q)
    assert (host(tri) >= 0).all() and m.status() == 0


@pytest.mark.parametrize("level,n", [(2, 1000), (5, 70001), (6, 0)])
def test_ordered_compose_bitwise_equal(nat, level, n):
    """cmm_query_order gives a permutation grouped by coarse cell, and the
    composition processed in that order writes the same bits (points,
    triangles of every submap, Jacobians) as the caller-order composition."""
    from cmm_gpu.meshgen import icosahedral_mesh, random_sphere_points
    from cmm_gpu.workloads import submap_stack
    verts, tris = icosahedral_mesh(level)
    mesh = nat.Mesh(verts, tris, level)
    tan, s_pts = OG.stencil_points(verts)
    coeffs = [mesh.assemble(dev(j)) for j in submap_stack(s_pts, tan, 3, seed=5)]
    q = dev(random_sphere_points(n, seed=6)) if n else torch.empty((0, 3), dtype=torch.float64,
                                                                  device="cuda")
    perm = mesh.query_order(q)
    assert torch.equal(torch.sort(perm.long())[0], torch.arange(n, device="cuda"))
    a = mesh.compose(coeffs, q, want_tri=True, want_tri_all=True, want_jac=True)
    b = mesh.compose(coeffs, q, want_tri=True, want_tri_all=True, want_jac=True, perm=perm)
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    if n and level >= 4:
        # neighbours in the order mostly share a level-4 cell (about 0.05
        # across), against a mean distance near 1.3 between random points
        pts = host(q)[host(perm)]
        step = np.linalg.norm(pts[1:] - pts[:-1], axis=1)
        assert np.median(step) < 0.1, np.median(step)
    assert mesh.status(clear=True) == 0


def test_full_size_composition_properties(nat):
    """The map-evaluation workload at full size (level 7, 8 submaps, 2^24
    queries, ids and Jacobians), through size-independent properties:
    images on the sphere; composing the stack in two launches (submaps 4-7,
    then 0-3) gives the same points to a few ulp (the second launch
    normalises its input point, which the single launch carries
    unnormalised through its deferred projection) and the chain-rule product
    of the two Jacobians (to 1e-10 relative: the tangent pushes run in
    float-float, ~2^-47 per operation, and each push cancels terms ~1/h =
    120 times larger than its result; measured 2.8e-11 over the 2^24
    queries); the ids of the first submap applied equal plain location; and
    a 4096-query sample matches the oracle (1e-12 points, 1e-10 relative
    Jacobians)."""
    from cmm_gpu.meshgen import icosahedral_mesh, random_sphere_points, stencil_frames
    from cmm_gpu.workloads import submap_stack
    verts, tris = icosahedral_mesh(7)
    tan, s_pts = stencil_frames(verts)
    jets = submap_stack(s_pts, tan, 8, seed=1)
    m = nat.Mesh(verts, tris, 7)
    cs = [m.assemble(dev(j)) for j in jets]
    q = dev(random_sphere_points(1 << 24, seed=3))
    X, tri, _, J = m.compose(cs, q, want_tri=True, want_jac=True)
    assert float((X.norm(dim=1) - 1).abs().max()) < 1e-15
    Y, _, _, JB = m.compose(cs[4:], q, want_jac=True)
    X2, _, _, JA = m.compose(cs[:4], Y, want_jac=True)
    assert float((X - X2).abs().max()) < 2e-15
    del X2, Y
    JJ = torch.bmm(JA, JB)
    del JA, JB
    rel = float(((JJ - J).abs().amax(dim=(1, 2)) / J.abs().amax(dim=(1, 2))).max())
    assert rel < 1e-10, rel
    del JJ
    t0, _ = m.locate(q)
    assert torch.equal(t0, tri)
    assert m.status() == 0
    # oracle on a sample
    idx = np.random.default_rng(0).choice(1 << 24, 4096, replace=False)
    qs = host(q[torch.from_numpy(idx).cuda()])
    comp = OS.CompositeOracle(verts, tris, OG.ConeLocator(verts, tris), jets, tie_fix=True)
    np.testing.assert_allclose(host(X)[idx], comp(qs), rtol=0, atol=1e-12)
    _, Jo = OS.composite_jacobian(comp, qs)
    Jg = host(J)[idx]
    scale = np.abs(Jo).max(axis=(1, 2))[:, None, None]
    np.testing.assert_allclose(Jg / scale, Jo / scale, rtol=0, atol=1e-10)
    # the same workload through map forms: ids equal, points within 1e-13
    fs = [m.assemble_forms(c) for c in cs]
    Xf, tf, _, Jf = m.compose(cs, q, want_tri=True, want_jac=True, forms=fs)
    assert torch.equal(tf, tri)
    assert float((Xf - X).abs().max()) < 1e-13
    assert float(((Jf - J).abs().amax(dim=(1, 2)) / J.abs().amax(dim=(1, 2))).max()) < 1e-10
    assert m.status() == 0


def test_ordered_compose_rejects_bad_permutation_entries(nat):
    """Entries outside [0, n) are skipped by the kernel's own bounds check and
    reported as CMM_FLAG_INDEX; every other query is composed as usual."""
    from cmm_gpu.meshgen import icosahedral_mesh, random_sphere_points
    from cmm_gpu.workloads import submap_stack
    verts, tris = icosahedral_mesh(3)
    mesh = nat.Mesh(verts, tris, 3)
    tan, s_pts = OG.stencil_points(verts)
    coeffs = [mesh.assemble(dev(j)) for j in submap_stack(s_pts, tan, 2, seed=5)]
    n = 1000
    q = dev(random_sphere_points(n, seed=8))
    perm = torch.arange(n, dtype=torch.int32, device="cuda")
    perm[3], perm[5] = n + 7, -2          # queries 3 and 5 are then never visited
    ref = mesh.compose(coeffs, q)[0]
    out = torch.full((n, 3), 7.0, dtype=torch.float64, device="cuda")
    mesh.compose(coeffs, q, out=out, perm=perm)
    assert mesh.status(clear=True) == nat.FLAG_INDEX
    keep = torch.ones(n, dtype=torch.bool, device="cuda")
    keep[[3, 5]] = False
    assert torch.equal(out[keep], ref[keep])
    assert bool((out[~keep] == 7.0).all())


def test_map_forms_match_coefficient_records(nat):
    """Composition through map-form records (cmm_assemble_forms /
    cmm_compose_forms: each Powell-Sabin patch as the quadratic form
    p^T Q p, FP32-filtered sub-triangle choice) against the same submaps'
    coefficient records and the oracle, level 5, 8 submaps, 2^16 queries:
    same triangle ids; points within 1e-13 of the records' and 1e-12 of the
    oracle's; Jacobians within 1e-11 (relative) of the records' and 1e-10
    of the oracle's; a stack mixing forms and records; the coarse-cell
    order bitwise equal to caller order."""
    from cmm_gpu.meshgen import icosahedral_mesh, random_sphere_points, stencil_frames
    from cmm_gpu.workloads import submap_stack
    verts, tris = icosahedral_mesh(5)
    tan, s_pts = stencil_frames(verts)
    jets = submap_stack(s_pts, tan, 8, seed=4)
    m = nat.Mesh(verts, tris, 5)
    cs = [m.assemble(dev(j)) for j in jets]
    fs = [m.assemble_forms(c) for c in cs]
    q = dev(random_sphere_points(1 << 16, seed=6))
    Xr, tr, tar, Jr = m.compose(cs, q, want_tri=True, want_tri_all=True, want_jac=True)
    Xf, tf, taf, Jf = m.compose(cs, q, want_tri=True, want_tri_all=True, want_jac=True, forms=fs)
    assert torch.equal(tr, tf) and torch.equal(tar, taf)
    assert float((Xf - Xr).abs().max()) < 1e-13
    scale = Jr.abs().amax(dim=(1, 2), keepdim=True)
    assert float(((Jf - Jr).abs() / scale).max()) < 1e-11
    Xm, _, _, Jm = m.compose(cs, q, want_jac=True, forms=[fs[0], None, fs[2], None, None, fs[5], fs[6], None])
    assert float((Xm - Xr).abs().max()) < 1e-13
    perm = m.query_order(q)
    Xo, to, _, Jo = m.compose(cs, q, want_tri=True, want_jac=True, forms=fs, perm=perm)
    assert torch.equal(Xo, Xf) and torch.equal(to, tf) and torch.equal(Jo, Jf)
    comp = OS.CompositeOracle(verts, tris, OG.ConeLocator(verts, tris), jets, tie_fix=True)
    qs = host(q)[:4096]
    np.testing.assert_allclose(host(Xf)[:4096], comp(qs), rtol=0, atol=1e-12)
    _, Jor = OS.composite_jacobian(comp, qs)
    sc = np.abs(Jor).max(axis=(1, 2))[:, None, None]
    np.testing.assert_allclose(host(Jf)[:4096] / sc, Jor / sc, rtol=0, atol=1e-10)
    # the low floats of the forms' float-float split (cmm_forms_ff): the
    # Jacobian pushes load the same floats they would extract, so every
    # output is bitwise the one without them, in both orders and in a
    # mixed stack
    gs = [m.forms_ff(f) for f in fs]
    assert gs[0].shape == (m.nt, nat.Mesh.FORM_FF_STRIDE) and gs[0].dtype == torch.float32
    assert bool((gs[0][:, 108:] == 0).all())
    Xg, tg, tag, Jg = m.compose(cs, q, want_tri=True, want_tri_all=True, want_jac=True, forms=fs, forms_ff=gs)
    assert torch.equal(Xg, Xf) and torch.equal(tg, tf) and torch.equal(tag, taf) and torch.equal(Jg, Jf)
    Xgo, _, _, Jgo = m.compose(cs, q, want_jac=True, forms=fs, forms_ff=gs, perm=perm)
    assert torch.equal(Xgo, Xf) and torch.equal(Jgo, Jf)
    mixed = [fs[0], None, fs[2], None, None, fs[5], fs[6], None]
    Xgm, _, _, Jgm = m.compose(cs, q, want_jac=True, forms=mixed,
                               forms_ff=[gs[0], None, gs[2], None, None, None, gs[6], None])
    assert torch.equal(Xgm, Xm) and torch.equal(Jgm, Jm)
    # non-finite queries through the forms path
    qn = q[:64].clone()
    qn[3, 1] = float("nan")
    Xn, tn, _, Jn = m.compose(cs, qn, want_tri=True, want_jac=True, forms=fs)
    assert torch.isnan(Xn[3]).all() and int(tn[3]) == -1 and torch.isfinite(Xn[4:]).all()
    assert m.status(clear=True) == nat.FLAG_NONFINITE
    assert m.status() == 0


@pytest.mark.parametrize("scale", [1.0, 1.9, 2.3, 40.0])
@pytest.mark.parametrize("radius", [1.0, 0.51, 1.7, 1e-3, 1e4])
def test_fixed_point_forms_at_the_ends_of_their_range(nat, scale, radius):
    """The points-only composition through map forms (fixed point) against
    the same submaps' coefficient records in FP64: jets scaled by `scale` make
    forms with entries on both sides of 2 (the bound of the fixed-point
    entries; the images are normalised, so the composed map stays the same),
    queries of norm `radius` lie inside and outside the range kept
    unnormalised, and a submap without a form record sits in the stack.  Same
    triangles, points to 1e-13."""
    from cmm_gpu.meshgen import icosahedral_mesh, random_sphere_points
    from cmm_gpu.workloads import submap_stack
    verts, tris = icosahedral_mesh(4)
    tan, s_pts = OG.stencil_points(verts)
    jets = submap_stack(s_pts, tan, 4, seed=8)
    jets[1] *= scale
    jets[3] /= scale
    m = nat.Mesh(verts, tris, 4)
    cs = [m.assemble(dev(j)) for j in jets]
    fs = [m.assemble_forms(c) for c in cs]
    fs[2] = None
    q = dev(random_sphere_points(4099, seed=9) * radius)
    Xr, tr, tar, _ = m.compose(cs, q, want_tri=True, want_tri_all=True)
    Xf, tf, taf, _ = m.compose(cs, q, want_tri=True, want_tri_all=True, forms=fs)
    assert torch.equal(tr, tf) and torch.equal(tar, taf)
    assert float((Xf - Xr).abs().max()) < 1e-13
    for v in (4, 6):
        m.set_variant(nat.Mesh.VARIANT_COMPOSE, v)
        assert torch.equal(m.compose(cs, q, forms=fs)[0], Xf)
    # a form that is not finite: NaN images, the flag, later ids -1
    bad = fs[3].clone()
    bad[:, :6] = float("nan")
    Xn, tn, tan_, _ = m.compose(cs, q, want_tri=True, want_tri_all=True, forms=fs[:3] + [bad])
    hit = torch.isnan(Xn).any(dim=1)
    assert hit.any() and not hit.all() and torch.equal(tn, tf)
    assert torch.equal(Xn[~hit], Xf[~hit]) and bool((tan_[:3, hit] == -1).all())
    assert m.status(clear=True) == nat.FLAG_NONFINITE


@pytest.mark.parametrize("n,spread", [(1, 2.0), (1023, 2.0), (155649, 2.0), ((1 << 20) - 1, 2.0), (1 << 20, 2.0),
                                      ((1 << 20) + 4097, 1e-3), ((1 << 20) + 4097, 0.2)])
def test_query_order_is_a_permutation(nat, n, spread):
    """cmm_query_order either side of its fifth pass and of a block's span,
    with the queries over the whole sphere, within a few cells, and all in
    one or two cells."""
    from cmm_gpu.meshgen import icosahedral_mesh
    verts, tris = icosahedral_mesh(3 if n < 2000 else 5)
    m = nat.Mesh(verts, tris, 3 if n < 2000 else 5)
    g = torch.Generator(device="cuda").manual_seed(n)
    q = torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=g)
    if spread < 2.0:
        q = spread * q + torch.tensor([0.3, -0.5, 0.8], dtype=torch.float64, device="cuda")
    q = (q / q.norm(dim=1, keepdim=True)).contiguous()
    perm = m.query_order(q)
    assert torch.equal(torch.sort(perm.long())[0], torch.arange(n, device="cuda"))
    if spread == 2.0 and n > 1 << 17:
        p = q[perm.long()]
        assert float((p[1:] - p[:-1]).norm(dim=1).median()) < 0.1


def test_host_pipeline_last_chunk_and_reused_scratch(nat):
    """compose_host with a last chunk on the other side of a step of the
    query sort's block count (n = 8 x 155,649 - 7), then a smaller call in the
    same scratch, whose chunks sort in more blocks: both bitwise
    Mesh.compose's."""
    from cmm_gpu.meshgen import icosahedral_mesh
    from cmm_gpu.workloads import submap_stack
    verts, tris = icosahedral_mesh(3)
    tan, s_pts = OG.stencil_points(verts)
    m = nat.Mesh(verts, tris, 3)
    cs = [m.assemble(dev(j)) for j in submap_stack(s_pts, tan, 2, seed=3)]
    n = 1_245_185
    q = torch.randn((n, 3), dtype=torch.float64, generator=torch.Generator().manual_seed(4)).pin_memory()
    out = torch.empty_like(q).pin_memory()
    scratch = streams = None
    for k in (n, 600_000):
        scratch, streams = nat.compose_host(m, cs, q[:k], out[:k], streams=streams, scratch=scratch)
        torch.cuda.synchronize()
        assert torch.equal(out[:k], m.compose(cs, dev(q[:k].numpy()))[0].cpu())
    assert m.status(clear=True) == 0


@pytest.mark.parametrize("n", [38_913, 77_825, 116_737, 311_297, 327_679, 327_681])
def test_composition_variants_bitwise_equal(nat, n):
    """Either side of each rule by which a composition through map forms picks
    its kernel (own or shared fetches, blocks per SM, rolled components), with
    and without an order: points, ids of every submap and Jacobians bitwise
    those of the same queries in calls of 5000, a ragged last warp, queries
    without an image and a form out of the fixed-point range included."""
    from cmm_gpu.meshgen import icosahedral_mesh, stencil_frames, random_sphere_points
    from cmm_gpu.workloads import submap_stack
    verts, tris = icosahedral_mesh(6)
    tan, s_pts = stencil_frames(verts)
    m = nat.Mesh(verts, tris, 6)
    jets = submap_stack(s_pts, tan, 4, seed=12)
    jets[2] *= 3.0
    cs = [m.assemble(dev(j)) for j in jets]
    fs = [m.assemble_forms(c) for c in cs]
    fs[1] = None
    gs = [None if f is None else m.forms_ff(f) for f in fs]
    q = dev(random_sphere_points(n, seed=n))
    q[100:100 + 7] = float("nan")
    q[20_003] = 0.0
    q[n - 2] *= 1e-3
    perm = m.query_order(q)
    for kw in (dict(), dict(want_jac=True), dict(want_jac=True, forms_ff=gs)):
        def call(x, **k):
            X, _, ta, J = m.compose(cs, x, want_tri_all=True, forms=fs, **kw, **k)
            return [X.view(torch.int64), ta.t()] + ([] if J is None else [J.view(torch.int64)])
        parts = [call(q[i:i + 5000]) for i in range(0, n, 5000)]
        ref = [torch.cat([p[k] for p in parts]) for k in range(len(parts[0]))]
        for k in (dict(), dict(perm=perm)):
            for a, b in zip(call(q, **k), ref):
                assert torch.equal(a, b)
    assert m.status(clear=True) == nat.FLAG_NONFINITE


@pytest.mark.parametrize("level", [3, 4, 5])
def test_query_order_on_coarse_meshes(nat, level):
    """cmm_query_order of enough queries for its fifth pass, which meshes whose
    triangles are no smaller than a cell leave out: a permutation, every cell's
    queries together (the composition's triangles change at most once per
    triangle and cell)."""
    from cmm_gpu.meshgen import icosahedral_mesh, random_sphere_points
    verts, tris = icosahedral_mesh(level)
    m = nat.Mesh(verts, tris, level)
    n = (1 << 20) + 4097
    q = dev(random_sphere_points(n, seed=level))
    perm = m.query_order(q).long()
    assert torch.equal(torch.sort(perm)[0], torch.arange(n, device="cuda"))
    tri = m.locate(q, want_bcc=False)[0][perm]
    if level <= 4:
        assert int((tri[1:] != tri[:-1]).sum()) < 2 * m.nt * 4 ** (4 - level)


@pytest.mark.parametrize("n", [1, 31, 33, 40_001, 150_001])
@pytest.mark.parametrize("records", ["-", "r", "rr", "fr", "ffr", "frf", "rfr", "rff", "frrr"])
def test_lists_of_forms_and_records(nat, n, records):
    """Points-only compositions of submaps with forms (f) and without (r), in
    evaluation order from the right (the last is evaluated first): the records
    ahead of the forms, between them, behind them, alone, and "-" no list; own
    and shared fetches and the FP64 kernel.  Ids of every submap those of the
    records alone, points within the bound of forms against records (1e-13);
    every order of the queries bitwise the same; queries without an image."""
    from cmm_gpu.meshgen import icosahedral_mesh, stencil_frames, random_sphere_points
    from cmm_gpu.workloads import submap_stack
    verts, tris = icosahedral_mesh(5)
    tan, s_pts = stencil_frames(verts)
    m = nat.Mesh(verts, tris, 5)
    S = len(records)
    cs = [m.assemble(dev(j)) for j in submap_stack(s_pts, tan, S, seed=21)]
    fs = None if records == "-" else [m.assemble_forms(c) if k == "f" else None for c, k in zip(cs, records)]
    q = dev(random_sphere_points(n, seed=n))
    bad = torch.zeros(n, dtype=torch.bool, device="cuda")
    if n > 40:
        q[7] = float("nan")
        q[n - 3] = 0.0
        bad[7] = bad[n - 3] = True
        q[11] *= 1e-3
        q[12] *= 3.0
    X, _, ta, _ = m.compose(cs, q, want_tri_all=True)
    Y, _, tb, _ = m.compose(cs, q, want_tri_all=True, forms=fs)
    assert torch.equal(ta, tb)
    assert torch.equal(torch.isnan(Y).any(1), bad) and torch.equal(torch.isnan(X).any(1), bad)
    assert bool((tb[:, bad] == -1).all())
    assert float((X - Y)[~bad].abs().max()) < 1e-13
    Z, _, tc, _ = m.compose(cs, q, want_tri_all=True, forms=fs, perm=m.query_order(q))
    assert torch.equal(Z.view(torch.int64), Y.view(torch.int64)) and torch.equal(tc, tb)
    m.status(clear=True)
