"""GPU parity of the triangle-soup fast winding number over the binned binary
tree (tree="binned"; the reference's own 4-wide tree is covered by
tests/test_soup_ref_gpu.py).

Checks, through the C ABI:
  * the tree's stored FP64 moments equal the HDK moments recomputed on the CPU
    from each node's triangles (FWNFS.h:6668-7118);
  * the plain FP64 walk equals the CPU oracle's FP64 walk over the same tree
    (computeSolidAngle semantics, FWNFS.h:7148-7284) to rounding;
  * the mixed walk is within the metric bound |dW| <= 1e-4 of the plain FP64
    walk, with identical inside/outside labels outside 0.5 +- 1e-3;
  * against the reference's own FP32 UT_SolidAngle (committed fixtures from
    tests/golden/make_golden.py): tight where the trees coincide (one
    triangle), within the reference's own approximation error elsewhere;
  * against the exact winding number: within the 1e-2 the reference's own
    test allows (tests/include/igl/fast_winding_number.cpp:76).
"""
import os
import time
from decimal import Decimal, getcontext

import numpy as np
import pytest

import libigl_gb300 as G
from libigl_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
TOL_MIXED = 1e-4


def golden():
    z = np.load(os.path.join(HERE, "golden", "soup_reference.npz"))
    names = sorted({k.split("/")[0] for k in z.files})
    return {n: {k.split("/")[1]: z[k] for k in z.files if k.startswith(n + "/")} for n in names}


@pytest.fixture(scope="module")
def mesh(cuda):
    rng = np.random.default_rng(5)
    V, F = synth.icosphere(5)
    V = synth.sh_deform(V, rng)
    F = synth.delete_random_faces(F, rng, 0.01)
    Q = synth.soup_queries(V, F, seed=6, nq=20000)
    return V, F, Q


def test_tree_moments_match_flat_recomputation(mesh):
    V, F, _ = mesh
    Vs, Fs = V, F[:3000]
    bvh = G.FastWindingNumberBVH(Vs, Fs, order=2, tree="binned")
    nodes, links, tri = bvh.export()
    assert sorted(tri.tolist()) == list(range(Fs.shape[0]))
    ref = O.soup_tree_moments(Vs, Fs, nodes, tri)
    scale = np.abs(ref[:, :23]).max(axis=0) + 1e-300
    rel = np.abs(nodes[:, :23] - ref[:, :23]) / scale
    assert rel.max() < 1e-10, rel.max(axis=0)
    # The reference's SumPermute shift (FWNFS.h:7075) counts the children's
    # first-moment term once; the exact parallel-axis shift counts it twice.
    # Every other moment equals its grouping-independent value.
    flat = O.soup_tree_moments(Vs, Fs, nodes, tri, flat=True)
    relf = np.abs(nodes[:, :23] - flat[:, :23]) / scale
    others = [k for k in range(23) if k != 16]
    assert relf[:, others].max() < 1e-10
    # pre-order skip links: every internal node's subtree is contiguous
    n = nodes.shape[0]
    assert n == 2 * Fs.shape[0] - 1
    internal = links >= 0
    assert np.all(links[internal] > np.nonzero(internal)[0])
    assert np.all(links[internal] <= n)
    assert links[0] == n


def test_fp64_walk_matches_cpu_walk(mesh):
    V, F, Q = mesh
    bvh = G.FastWindingNumberBVH(V, F, order=2, tree="binned")
    nodes, links, tri = bvh.export()
    W64 = bvh.eval(Q, 2.0, precision="fp64")
    Wcpu = O.soup_tree_eval(V, F, nodes, tri, Q, 2.0, order=2)
    assert np.abs(W64 - Wcpu).max() < 1e-11


@pytest.mark.parametrize("tree", ["binned", "reference"])
def test_mixed_within_metric_of_fp64(mesh, tree):
    V, F, Q = mesh
    bvh = G.FastWindingNumberBVH(V, F, order=2, tree=tree)
    for qdt in (np.float64, np.float32):
        Qd = Q.astype(qdt)
        W64 = bvh.eval(Qd, 2.0, precision="fp64", out_dtype=np.float64)
        Wm = bvh.eval(Qd, 2.0, precision="mixed", out_dtype=np.float64)
        err = np.abs(Wm - W64)
        assert err.max() <= TOL_MIXED, err.max()
        out = np.abs(W64 - 0.5) > 1e-3
        assert np.array_equal((Wm > 0.5)[out], (W64 > 0.5)[out])


def test_against_exact_and_orders(mesh):
    V, F, Q = mesh
    Qs = Q[:3000]
    Wex = O.winding_number(V, F, Qs)
    for order, tol in ((2, 1e-2), (1, 2e-1), (0, 5e-1)):
        bvh = G.FastWindingNumberBVH(V, F, order=order, tree="binned")
        W = bvh.eval(Qs, 2.0, precision="fp64")
        assert np.abs(W - Wex).max() < tol, (order, np.abs(W - Wex).max())
        nodes, links, tri = bvh.export()
        Wcpu = O.soup_tree_eval(V, F, nodes, tri, Qs, 2.0, order=order)
        assert np.abs(W - Wcpu).max() < 1e-11


def test_against_reference_fixtures(cuda):
    for name, c in golden().items():
        if "W_exact" not in c:
            continue
        V, F, Q, Wref, Wex = c["V"], c["F"], c["Q"], c["W_ref"], c["W_exact"]
        bvh = G.FastWindingNumberBVH(V, F, order=2, tree="binned")
        W = bvh.eval(Q, 2.0, precision="mixed")
        ref_err = np.abs(Wref - Wex).max()
        if name == "one_tri":
            # same tree (one triangle): only FP32-vs-FP64 arithmetic differs
            assert np.abs(W - Wref).max() < 5e-6, name
        # the reference's own error bound vs exact, with our approximation's
        assert np.abs(W - Wex).max() < max(1e-2, 3 * ref_err), name
        assert np.abs(W - Wref).max() < max(1e-2, 3 * ref_err), name
        far_band = (np.abs(Wex - 0.5) > 0.05)
        assert np.array_equal((W > 0.5)[far_band], (Wex > 0.5)[far_band]), name


def test_single_tet_sign(cuda):
    # tests/include/igl/signed_distance.cpp:4-42: (.5,.5,.5) is outside the unit tet
    V = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)
    F = np.array([[0, 1, 3], [0, 2, 1], [0, 3, 2], [1, 2, 3]], np.int32)
    W = G.fast_winding_number_soup(V, F, np.array([[0.5, 0.5, 0.5], [0.1, 0.1, 0.1]]))
    assert abs(W[0]) < 1e-6 and abs(W[1] - 1) < 1e-6


def test_edge_cases(cuda):
    V = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1], [np.nan, 0, 0]], float)
    F = np.array([[0, 1, 3], [0, 2, 1], [0, 3, 2], [1, 2, 3], [4, 1, 2]], np.int32)
    Q = np.array([[0.1, 0.1, 0.1], [2, 2, 2], [0, 0, 0]])
    # a triangle with a NaN vertex is excluded from the tree (FWNFS.h:4606-4615)
    for tree in ("binned", "reference"):
        b = G.FastWindingNumberBVH(V, F, tree=tree)
        assert b.stats["num_triangles"] == 4
        Wt = b.eval(Q, 2.0, precision="mixed")
        # within the order-2 expansion's error at accuracy 2 of the exact 1 / 0
        assert abs(Wt[0] - 1) < 1e-4 and abs(Wt[1]) < 1e-4 and np.isfinite(Wt[2])
        if tree == "reference":  # and the reference's own values (its tree)
            assert np.abs(Wt[:2] - O.SoupPort(V, F).eval(Q[:2], 2.0)).max() < 1e-6
        with pytest.raises(G.GwnError):
            G.FastWindingNumberBVH(V, np.array([[0, 1, 9]], np.int32), tree=tree)
    bvh = G.FastWindingNumberBVH(V, F)
    assert bvh.stats["num_triangles"] == 4
    W = bvh.eval(Q, 2.0, precision="mixed")
    assert abs(W[0] - 1) < 1e-4 and abs(W[1]) < 1e-4 and np.isfinite(W[2])
    # empty mesh and empty queries
    e = G.FastWindingNumberBVH(V, np.zeros((0, 3), np.int32))
    assert np.all(e.eval(Q) == 0)
    assert bvh.eval(np.zeros((0, 3))).shape == (0,)
    # out-of-range index fails loudly
    with pytest.raises(G.GwnError):
        G.FastWindingNumberBVH(V, np.array([[0, 1, 9]], np.int32))


def test_device_tensors_and_repeatability(mesh, cuda):
    torch = cuda
    V, F, Q = mesh
    bvh = G.FastWindingNumberBVH(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda())
    dQ = torch.from_numpy(Q.astype(np.float32)).cuda()
    W1 = bvh.eval(dQ, 2.0, precision="mixed")
    W2 = bvh.eval(dQ, 2.0, precision="mixed")
    assert W1.is_cuda and torch.equal(W1, W2)  # deterministic
    Wh = bvh.eval(Q.astype(np.float32), 2.0, precision="mixed")
    assert np.array_equal(W1.cpu().numpy(), Wh)
    # a query's value does not depend on the batch it is evaluated in
    sub = Q[::7].astype(np.float32)
    Ws = bvh.eval(sub, 2.0, precision="mixed")
    assert np.abs(Ws - Wh[::7]).max() <= 1e-6
    assert G.device_status() == 0


def _check_tree(V, F, Q):
    bvh = G.FastWindingNumberBVH(V, F, order=2, tree="binned")
    nodes, links, tri = bvh.export()
    n = F.shape[0]
    assert sorted(tri.tolist()) == list(range(n))
    assert nodes.shape[0] == 2 * n - 1
    # pre-order with skip links: an internal node's subtree is [p + 1, link)
    internal = links >= 0
    idx = np.nonzero(internal)[0]
    assert np.all(links[idx] > idx + 1) and np.all(links[idx] <= 2 * n - 1)
    if n > 1:
        assert links[0] == 2 * n - 1
    assert sorted((~links[~internal]).tolist()) == list(range(n))
    W64 = bvh.eval(Q, 2.0, precision="fp64")
    Wcpu = O.soup_tree_eval(V, F, nodes, tri, Q, 2.0, order=2)
    assert np.abs(W64 - Wcpu).max() < 1e-11
    Wm = bvh.eval(Q, 2.0, precision="mixed")
    assert np.abs(Wm - W64).max() <= TOL_MIXED


def test_tree_builder_corner_cases(cuda):
    """The binned top-down builder (soup_tree.cu): sizes around the 32
    triangles one warp finishes, triangles whose centroids all coincide (no
    bin separates them: middle splits), and a flat mesh (zero extent on one
    axis)."""
    rng = np.random.default_rng(71)
    V, F = synth.icosphere(3)
    F = np.ascontiguousarray(F, dtype=np.int32)
    Q = np.ascontiguousarray(rng.uniform(-1.3, 1.3, (500, 3)))
    for m in (2, 3, 31, 32, 33, 34, 64, 65, 200):
        _check_tree(V, np.ascontiguousarray(F[:m]), Q)
    # 300 copies of one triangle, flipped every other time: equal centroids
    Fd = np.ascontiguousarray(np.tile(np.array([[0, 1, 2], [0, 2, 1]], np.int32), (150, 1)))
    _check_tree(V, Fd, Q)
    # a flat grid of triangles in z = 0
    g = np.stack(np.meshgrid(np.linspace(0, 1, 30), np.linspace(0, 1, 30), indexing="ij"), -1)
    Vf = np.concatenate([g.reshape(-1, 2), np.zeros((900, 1))], 1)
    a = (np.arange(29)[:, None] * 30 + np.arange(29)[None, :]).ravel()
    Ff = np.concatenate([np.stack([a, a + 30, a + 1], 1), np.stack([a + 1, a + 30, a + 31], 1)])
    _check_tree(np.ascontiguousarray(Vf), np.ascontiguousarray(Ff, dtype=np.int32), Q * 0.8 + 0.3)



@pytest.mark.parametrize("tree", ["reference", "binned"])
@pytest.mark.parametrize("shape", ["sphere", "nested"])
def test_lanes_per_query_do_not_change_the_result(cuda, tree, shape):
    """Small batches share a query between the lanes of a team, large ones walk
    32 queries per warp: the same queries in batches on either side of each
    rule's edge.  The terms are the same and their sum runs in another order,
    so FP32 sums differ by at most about 150 terms x 2^-24 x the terms' total
    of a few turns (3e-5), FP64 sums by 1e-12.  "nested" puts triangles at
    2^-k, a deep unbalanced tree whose teams run out of stack."""
    if shape == "sphere":
        V, F = synth.icosphere(3)
    else:
        k = 2.0 ** -np.arange(120.0)
        V = (k[:, None, None] * np.array([[1, 0, 0], [1.4, 0, 0.1], [1, 0.4, 0]])).reshape(-1, 3)
        F = np.arange(V.shape[0], dtype=np.int32).reshape(-1, 3)
    rng = np.random.default_rng(41)
    n = 260_000  # past the warp-coherent rule for these trees
    Q = rng.uniform(-1.3, 1.3, (n, 3))
    Q[: n // 2] *= 10.0 ** rng.uniform(-6, 0, (n // 2, 1))
    bvh = G.FastWindingNumberBVH(V, F, tree=tree)
    for prec, tol in (("mixed", 3e-5), ("fp64", 1e-12)):
        W = bvh.eval(Q, 2.0, prec)
        for m in (1, 31, 33, 4096, 4097, 8191, 60_000, 60_001, 70_000):
            w = bvh.eval(Q[:m], 2.0, prec)
            assert np.array_equal(np.isfinite(w), np.isfinite(W[:m])), (prec, m)
            assert np.abs(w - W[:m]).max() <= tol, (prec, m)
            assert np.array_equal(w, bvh.eval(Q[:m], 2.0, prec)), (prec, m)
    bvh.close()


@pytest.mark.parametrize("nq,scales", [(1, (2, 30, 100, 200, 400)), (33, (30, 100, 200, 400)),
                                       (3000, (100, 200)), (30_000, (60, 100, 200)),
                                       (210_000, (60, 80, 100, 200))])
def test_many_small_terms_of_one_sign(cuda, nq, scales):
    """A closed sphere of 327,680 triangles seen from inside: from a scale of
    about 100 a query adds up to 300,000 far terms of one sign, each below 1e-4
    sr.  Up to 3000 queries share a query between 32 lanes, 30,000 between 8,
    210,000 between 4.  W is 1 to the mixed walk's 1e-4 (at scale 2 to the
    expansion's 5e-3), and so is the plain FP64 walk's."""
    V, F = synth.geodesic_sphere(128)
    rng = np.random.default_rng(3)
    Q = rng.normal(size=(nq, 3))
    Q *= 0.05 * rng.uniform(0, 1, (nq, 1)) / np.linalg.norm(Q, axis=1, keepdims=True)
    bvh = G.FastWindingNumberBVH(V, F, 2)
    for scale in scales:
        tol = 5e-3 if scale == 2 else 1e-4
        W = bvh.eval(Q, scale, "mixed", out_dtype=np.float64)
        assert np.abs(W - 1).max() <= tol, scale
        W64 = bvh.eval(Q[:64], scale, "fp64", out_dtype=np.float64)
        assert np.abs(W64 - 1).max() <= tol, scale
        assert np.abs(W[:64] - W64).max() <= 1e-4, scale
    bvh.close()


@pytest.mark.parametrize("nq", [1, 32, 5000, 100_000])
def test_small_sums_keep_their_relative_accuracy(cuda, nq):
    """One triangle of unit size from 1e2 to 1e6 units away, within 45 degrees
    of its normal: W down to 1e-14, in FP32 within the about 50 roundings of a
    far field or a triangle term (50 x 2^-24 = 3e-6 of the value)."""
    V = np.array([[0.1, 0, 0], [1.1, 0.2, 0], [0.3, 0.9, 0.1]])
    F = np.array([[0, 1, 2]], np.int32)
    n = np.cross(V[1] - V[0], V[2] - V[0])
    rng = np.random.default_rng(5)
    d = rng.normal(size=(nq, 3))
    d = 1.5 * n / np.linalg.norm(n) + d / np.linalg.norm(d, axis=1, keepdims=True)
    d *= 10.0 ** rng.uniform(2, 6, (nq, 1)) / np.linalg.norm(d, axis=1, keepdims=True)
    bvh = G.FastWindingNumberBVH(V, F, 2)
    W = bvh.eval(d, 2.0, "mixed", out_dtype=np.float64)
    W64 = bvh.eval(d, 2.0, "fp64", out_dtype=np.float64)
    bvh.close()
    assert (np.abs(W64) > 1e-15).all()
    assert (np.abs(W - W64) <= 3e-6 * np.abs(W64)).all()


def test_coincident_sheets_beyond_forty_thousand_turns(cuda):
    """An 80-triangle sphere 45,000 times over, queries at its centre, at a scale
    that opens every triangle and leaves its term in FP32: W = 45,000, 565,000 sr,
    each term within about 50 roundings."""
    V, F = synth.icosphere(1)
    bvh = G.FastWindingNumberBVH(V, np.tile(F, (45_000, 1)), 2)
    Q = np.array([[0, 0, 0], [1e-3, 2e-3, 0]])
    W = bvh.eval(Q, 6.0, "mixed", out_dtype=np.float64)
    W64 = bvh.eval(Q, 6.0, "fp64", out_dtype=np.float64)
    bvh.close()
    assert np.abs(W64 - 45_000).max() <= 45_000 * 1e-10
    assert np.abs(W - 45_000).max() <= 45_000 * 3e-6


def _solid_angle_50_digits(T, q):
    """Solid angle of triangle T from q (van Oosterom and Strackee), for a
    small angle: the arc tangent by its series."""
    getcontext().prec = 50
    a, b, c = ([Decimal(float(x)) - Decimal(float(y)) for x, y in zip(p, q)] for p in T)

    def dot(u, v):
        return sum((x * y for x, y in zip(u, v)), Decimal(0))

    la, lb, lc = (dot(p, p).sqrt() for p in (a, b, c))
    det = (a[0] * (b[1] * c[2] - b[2] * c[1]) + a[1] * (b[2] * c[0] - b[0] * c[2])
           + a[2] * (b[0] * c[1] - b[1] * c[0]))
    x = det / (la * lb * lc + dot(a, b) * lc + dot(a, c) * lb + dot(b, c) * la)
    return 2 * sum((x ** (2 * k + 1) * (-1) ** k / (2 * k + 1) for k in range(20)), Decimal(0))


@pytest.mark.parametrize("tree", ["reference", "binned"])
def test_distant_opened_triangles_keep_their_digits(cuda, tree):
    """A large accuracy scale opens a triangle d/e = 4 to 1e6 edges away: the
    plain FP64 term is within 4 u e/d sr of the solid angle (u = 2^-53), the
    rounding of differences of unit vectors e/d apart."""
    rng = np.random.default_rng(17)
    F = np.array([[0, 1, 2]], np.int32)
    for _ in range(20):
        T = rng.normal(size=(3, 3))
        e = max(np.linalg.norm(T[i] - T[j]) for i, j in ((0, 1), (1, 2), (2, 0)))
        n = np.cross(T[1] - T[0], T[2] - T[0])
        d = rng.normal(size=(30, 3))
        d = 1.5 * n / np.linalg.norm(n) + d / np.linalg.norm(d, axis=1, keepdims=True)
        far = 10.0 ** rng.uniform(np.log10(4), 6, (30, 1))
        Q = T.mean(0) + far * e * d / np.linalg.norm(d, axis=1, keepdims=True)
        bvh = G.FastWindingNumberBVH(T, F, 2, tree=tree)
        W = bvh.eval(Q, 1e9, "fp64", out_dtype=np.float64)
        bvh.close()
        for q, w, f in zip(Q, W, far[:, 0]):
            err = abs(float(Decimal(float(w)) * Decimal(4 * np.pi) - _solid_angle_50_digits(T, q)))
            # 2 u |value|: the factor 1 / 4 pi and its product here
            assert err <= 2.0 ** -53 * (4 / f + 3 * abs(4 * np.pi * w)), f


def _best_us(cuda, f, reps=7):
    """Shortest of a few passes, waited for."""
    best = float("inf")
    for k in range(reps + 2):
        cuda.cuda.synchronize()
        t = time.perf_counter()
        f()
        cuda.cuda.synchronize()
        if k >= 2:
            best = min(best, time.perf_counter() - t)
    return best * 1e6


@pytest.mark.parametrize("m", [1, 33, 4096, 4097, 50_000, 50_001, 200_000])
def test_results_near_one_half_are_the_fp64_walks(cuda, m):
    """m queries with W within 5e-4 of one half (below the rim of a half sphere)
    among as many others: all m are evaluated again by the plain FP64 walk, with
    32, 8 or one lane each by their number, and the sums differ from that
    walk's own in their order only (1e-12)."""
    V, F = synth.geodesic_sphere(32)
    F = np.ascontiguousarray(F[V[F][:, :, 2].mean(1) > 0])
    bvh = G.FastWindingNumberBVH(V, F, 2)
    rng = np.random.default_rng(m)
    a, r = rng.uniform(0, 2 * np.pi, 400_000), 0.9 * np.sqrt(rng.uniform(0, 1, 400_000))
    Q = np.stack([r * np.cos(a), r * np.sin(a), -2e-3 * rng.uniform(-1, 1, r.size)], 1)
    W = bvh.eval(Q, 2.0, "fp64", out_dtype=np.float64)
    Q = Q[np.abs(W - 0.5) <= 5e-4]
    assert Q.shape[0] > 1000
    Q = np.tile(Q, (m // Q.shape[0] + 1, 1))[:m]
    others = rng.uniform(-3, 3, (m, 3)) + [0, 0, 7]
    B = np.concatenate([Q, others])[rng.permutation(2 * m)]
    W = bvh.eval(B, 2.0, "mixed", out_dtype=np.float64)
    W64 = bvh.eval(B, 2.0, "fp64", out_dtype=np.float64)
    band = np.abs(W64 - 0.5) <= 9e-4
    assert band.sum() == m
    assert np.abs(W - W64)[band].max() <= 1e-12
    bvh.close()


def test_a_batch_near_one_half_costs_its_fp64_walk(cuda):
    """A million queries below the rim of a half sphere of 655,000 triangles, most
    of them near one half: the mixed call takes about the FP64 walk's time (at
    most 1.5 times; with 32 lanes for each, more than twice)."""
    V, F = synth.geodesic_sphere(256)
    F = np.ascontiguousarray(F[V[F][:, :, 2].mean(1) > 0])
    bvh = G.FastWindingNumberBVH(V, F, 2)
    rng = np.random.default_rng(2)
    n = 1_000_000
    a, r = rng.uniform(0, 2 * np.pi, n), 0.9 * np.sqrt(rng.uniform(0, 1, n))
    Q = cuda.from_numpy(np.stack([r * np.cos(a), r * np.sin(a), -1e-4 * rng.random(n)], 1)).cuda()
    W = bvh.eval(Q, 2.0, "fp64", out_dtype=np.float64)
    assert float(((W - 0.5).abs() <= 1e-3).double().mean()) > 0.7
    t = [_best_us(cuda, lambda: bvh.eval(Q, 2.0, p)) for p in ("mixed", "fp64")]
    bvh.close()
    assert t[0] <= 1.5 * t[1], t
