"""Closest triangle and signed distance on the GPU (distance.cu) against the
CPU oracle (oracle/distance.cpp: brute force over all triangles with
Ericson's closest point, and the reference's sign rules,
include/igl/signed_distance.cpp:83-137).

Tolerances: squared distances 1e-12 relative plus 1e-14 |d| (both FP64;
the closest point carries an absolute rounding of a few 1e-16, which
dominates d^2 = |p - c|^2 for points very close to the surface), closest
points 1e-9; the triangle index is checked through its
own distance (a tie may pick another triangle at the same distance); signs
from the exact winding number agree to 1e-9; the fast-winding-number sign is
the reference's soup algorithm on its own tree, so S may differ by
2 |dW| |S| with |dW| <= 2e-2 (the reference's own test tolerance against the
exact winding number is 1e-2)."""
import time

import numpy as np
import pytest

import libigl_gb300 as G
from libigl_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _tet():
    V = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)
    F = np.array([[0, 1, 3], [0, 2, 1], [0, 3, 2], [1, 2, 3]], np.int32)
    return V, F


def test_single_tet_golden(cuda):
    """tests/include/igl/signed_distance.cpp:4-42."""
    V, F = _tet()
    P = np.array([[0.5, 0.5, 0.5]])
    for t, tol in ((G.SIGNED_DISTANCE_TYPE_PSEUDONORMAL, 1e-15),
                   (G.SIGNED_DISTANCE_TYPE_WINDING_NUMBER, 1e-15),
                   (G.SIGNED_DISTANCE_TYPE_DEFAULT, 1e-15),
                   (G.SIGNED_DISTANCE_TYPE_UNSIGNED, 1e-15),
                   (G.SIGNED_DISTANCE_TYPE_FAST_WINDING_NUMBER, 1e-7)):
        S, I, Cp = G.signed_distance(P, V, F, t)
        assert abs(S[0] - np.sqrt(1 / 12)) <= tol, (t, S)
        assert I[0] == 3 and np.allclose(Cp[0], 1 / 3, atol=1e-15)
    # pseudonormal inside / outside / at a vertex region, with its normals
    Q = np.array([[0.5, 0.5, 0.5], [0.1, 0.1, 0.1], [2, 2, 2], [-1, -1, -1], [0.3, -1, 0.3]])
    S, I, Cp, Nn = G.signed_distance(Q, V, F, G.SIGNED_DISTANCE_TYPE_PSEUDONORMAL,
                                     return_normals=True)
    Sr, Ir, Cr, Nr = O.signed_distance(Q, V, F, G.SIGNED_DISTANCE_TYPE_PSEUDONORMAL,
                                       return_normals=True)
    assert np.abs(S - Sr).max() <= 1e-15
    # (0.1, 0.1, 0.1) is equally close to three faces and (-1, -1, -1) to the
    # vertex they share: the closest face (and for the first the normal)
    # follows whichever face each side reached first
    same = I == Ir
    assert same.sum() >= 3 and np.abs(Nn[same] - Nr[same]).max() <= 1e-15


@pytest.fixture(scope="module")
def mesh():
    V, F = synth.soup_mesh(seed=21, subdiv=3, delete_frac=0.02)
    rng = np.random.default_rng(22)
    lo, hi = V.min(0), V.max(0)
    far = rng.uniform(lo - 0.5, hi + 0.5, size=(15000, 3))
    Pn, f = synth.sample_on_faces(V, F, rng, 5000)
    Nn = synth.face_normals(V, F)[f]
    near = Pn + Nn * (rng.choice([-1, 1], (5000, 1)) * 10.0 ** rng.uniform(-7, -1, (5000, 1)))
    return V, F, np.concatenate([far, near, V[:50]])  # and points on vertices (ties)


def _close2(D, Dr):
    return np.abs(D - Dr) <= 1e-12 * Dr + 1e-14 * np.sqrt(Dr) + 1e-300


def _tri_dist2(V, F, P, I):
    out = np.empty(3)
    L = O.lib()
    d = np.empty(len(P))
    for k in range(len(P)):
        t = V[F[I[k]]]
        a, b, c = (np.ascontiguousarray(t[j]) for j in range(3))
        p = np.ascontiguousarray(P[k])
        d[k] = L.oracle_point_triangle(O._ptr(p), O._ptr(a), O._ptr(b), O._ptr(c), O._ptr(out))
    return d


def test_squared_distance_matches_brute_force(mesh, cuda):
    V, F, P = mesh
    bvh = G.FastWindingNumberBVH(V, F)
    D, I, Cp = bvh.squared_distance(P)
    bvh.close()
    Dr, Ir, Cr = O.squared_distance(V, F, P)
    assert np.all(I >= 0)
    assert np.all(_close2(D, Dr))
    # the reported triangle is at the reported distance (tie-safe)
    assert np.all(_close2(_tri_dist2(V, F, P, I), D))
    # a closest edge or vertex is shared by several triangles (ties), so the
    # indices may differ; the closest points agree
    assert np.abs(Cp - Cr).max() <= 1e-9
    # f32 queries: the same up to the query's rounding
    D32, I32, _ = G.FastWindingNumberBVH(V, F).squared_distance(P.astype(np.float32))
    Dr32, _, _ = O.squared_distance(V, F, P.astype(np.float32).astype(np.float64))
    assert np.all(_close2(D32, Dr32))


def test_signed_distance_against_oracle(mesh, cuda):
    V, F, P = mesh
    for t in (G.SIGNED_DISTANCE_TYPE_UNSIGNED, G.SIGNED_DISTANCE_TYPE_WINDING_NUMBER,
              G.SIGNED_DISTANCE_TYPE_DEFAULT):
        S, I, Cp = G.signed_distance(P, V, F, t)
        Sr, Ir, Cr = O.signed_distance(P, V, F, t)
        assert np.abs(S - Sr).max() <= 1e-9 * (1 + np.abs(Sr).max()), t
    # pseudonormal: the sign follows the closest feature, so a tie in the
    # closest triangle may pick another feature's normal; compare where the
    # closest triangles agree, and the magnitude everywhere
    S, I, Cp, Nn = G.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_PSEUDONORMAL,
                                     return_normals=True)
    Sr, Ir, Cr, Nr = O.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_PSEUDONORMAL,
                                       return_normals=True)
    assert np.all(np.abs(np.abs(S) - np.abs(Sr)) <= 1e-12 * (1 + np.abs(Sr)))
    same = I == Ir
    assert same.mean() > 0.5
    assert np.array_equal(np.sign(S[same]), np.sign(Sr[same]))
    assert np.abs(Nn[same] - Nr[same]).max() <= 1e-9
    # and the pseudonormal sign agrees with the exact winding number's
    # away from the surface and the holes' rims
    Sw, _, _ = G.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_WINDING_NUMBER)
    clear = np.abs(Sw) > 1e-3
    assert (np.sign(S[clear]) == np.sign(Sw[clear])).mean() > 0.95
    # fast-winding-number sign
    S, I, Cp = G.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_FAST_WINDING_NUMBER)
    Sr, _, _ = O.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_FAST_WINDING_NUMBER)
    assert np.all(np.abs(S - Sr) <= 2 * 2e-2 * np.abs(Sr) + 1e-12)
    # mixed and plain FP64 exact sign agree to the mixed tolerance
    Sm, _, _ = G.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_WINDING_NUMBER,
                                 precision="mixed")
    S64, _, _ = G.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_WINDING_NUMBER)
    assert np.all(np.abs(Sm - S64) <= 2e-4 * np.abs(S64) + 1e-12)


def test_bounds_empty_and_device(mesh, cuda):
    torch = cuda
    V, F, P = mesh
    lo, hi = -0.05, 0.2
    S, I, Cp = G.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_WINDING_NUMBER, lo, hi)
    Sr, Ir, Cr = O.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_WINDING_NUMBER, lo, hi)
    nan = np.isnan(Sr)
    assert nan.any() and (~nan).any()
    assert np.array_equal(np.isnan(S), nan)
    assert np.all(I[nan] == F.shape[0] + 1) and np.all(Cp[nan] == 0)
    assert np.abs(S[~nan] - Sr[~nan]).max() <= 1e-9
    # empty F (signed_distance.cpp:395-402)
    S0, I0, C0 = G.signed_distance(P[:5], V, np.zeros((0, 3), np.int32))
    assert np.all(np.isnan(S0)) and np.all(I0 == -1) and np.all(np.isnan(C0))
    # device tensors give the host result
    Sd, Id, Cd = G.signed_distance(torch.from_numpy(P).cuda(), torch.from_numpy(V).cuda(),
                                   torch.from_numpy(F).cuda(),
                                   G.SIGNED_DISTANCE_TYPE_WINDING_NUMBER)
    Sh, Ih, Ch = G.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_WINDING_NUMBER)
    assert np.array_equal(Sd.cpu().numpy(), Sh) and np.array_equal(Id.cpu().numpy(), Ih)


def test_squared_distance_random_soup_with_skinny_triangles(cuda):
    """Random triangles (many of them long and thin, some degenerate) and
    queries near and far: the FP32 leaf screen never drops the closest
    triangle (exact brute-force distance)."""
    rng = np.random.default_rng(41)
    nF = 3000
    A = rng.uniform(-1, 1, (nF, 3))
    B = A + rng.normal(0, 0.3, (nF, 3))
    # a third of the triangles nearly collinear, a few exactly degenerate
    t = rng.uniform(0, 1, (nF, 1))
    Cc = A + rng.normal(0, 0.3, (nF, 3))
    thin = rng.random(nF) < 0.33
    Cc[thin] = (A + t * (B - A) + rng.normal(0, 1e-6, (nF, 3)))[thin]
    Cc[:10] = A[:10]
    V = np.concatenate([A, B, Cc])
    F = np.stack([np.arange(nF), nF + np.arange(nF), 2 * nF + np.arange(nF)], 1).astype(np.int32)
    P = np.concatenate([rng.uniform(-1.5, 1.5, (6000, 3)),
                        V[rng.integers(0, len(V), 2000)] + rng.normal(0, 1e-4, (2000, 3))])
    D, I, Cp = G.FastWindingNumberBVH(V, F).squared_distance(P)
    Dr, Ir, Cr = O.squared_distance(V, F, P)
    assert np.all(_close2(D, Dr))
    assert np.all(_close2(_tri_dist2(V, F, P, I), D))


@pytest.mark.parametrize("nq", [1, 31, 33, 400])
@pytest.mark.parametrize("subdiv", [0, 2, 4])
def test_queries_equally_far_from_everything(cuda, subdiv, nq):
    """Queries at and around a sphere's centre reach nearly every triangle:
    the searches a thread hands over to a whole warp.  The surface has
    exactly tied triangles (subdiv 0: the icosahedron), a bounded search and
    float32 queries included."""
    V, F = synth.icosphere(subdiv)
    rng = np.random.default_rng(31)
    Q = rng.normal(size=(nq, 3)) * 10.0 ** rng.uniform(-9, -1, (nq, 1))
    Q[0] = 0
    bvh = G.FastWindingNumberBVH(V, F, tree="binned")
    for q in (Q, Q.astype(np.float32)):
        D, I, Cp = bvh.squared_distance(q)
        Dr, Ir, Cr = O.squared_distance(V, F, q.astype(np.float64))
        assert _close2(D, Dr).all()
        assert (np.abs(((q - Cp) ** 2).sum(1) - D) <= 1e-14).all()
        assert ((I >= 0) & (I < F.shape[0])).all()
    # nothing below the bound: the reference's "not found"
    D, I, _ = bvh.squared_distance(Q, up_sqr_d=0.25)
    Dr, _, _ = O.squared_distance(V, F, Q, 0.25)
    assert np.array_equal(D == 0.25, Dr == 0.25) and (I[D == 0.25] == -1).all()
    bvh.close()


@pytest.mark.parametrize("nf", [1, 2, 8, 9, 10, 33, 300, 4096, 4097, 9000])
@pytest.mark.parametrize("kind", ["sphere", "plane", "soup"])
def test_patches_and_soups_at_any_scale(cuda, nf, kind):
    """From one triangle to more than any search node's own box is made for;
    normals of all directions, one shared direction (an axis, its opposite, and
    a slanted one), and none at all (triangles shrunk to segments and points).
    The bounds never drop the closest triangle (exact brute-force distance),
    and scaling everything by a power of two scales the result exactly."""
    rng = np.random.default_rng([nf, len(kind)])
    if kind == "soup":
        A = rng.uniform(-1, 1, (nf, 3))
        T = A[:, None] + rng.normal(0, 0.1, (nf, 3, 3))
        T[::5, 2] = T[::5, 1]
        T[::7] = T[::7, :1]
    else:
        n = rng.normal(size=(nf, 3))
        n /= np.linalg.norm(n, axis=1, keepdims=True)
        if kind == "plane":
            n[:] = [[0, 0, 1], [0, 0, -1], [0.48, -0.6, -0.64]][nf % 3]
        u = np.cross(n, n[:, [1, 2, 0]] + [0.1, 0.2, 0.3])
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        w = np.cross(n, u)
        c = n if kind == "sphere" else rng.uniform(-1, 1, (nf, 1)) * u + rng.uniform(-1, 1, (nf, 1)) * w
        s = rng.normal(0, 1.5 / np.sqrt(nf), (nf, 3, 2))
        T = c[:, None] + s[..., :1] * u[:, None] + s[..., 1:] * w[:, None]
    V = np.ascontiguousarray(T.reshape(-1, 3))
    F = np.arange(3 * nf, dtype=np.int32).reshape(nf, 3)
    P = np.concatenate([rng.uniform(-1.5, 1.5, (200, 3)), rng.normal(0, 1e-3, (50, 3)),
                        V[rng.integers(0, len(V), 100)] + rng.normal(0, 1e-5, (100, 3))])
    bvh = G.FastWindingNumberBVH(V, F, tree="binned")
    D, I, C = bvh.squared_distance(P)
    Dr, _, _ = O.squared_distance(V, F, P)
    assert _close2(D, Dr).all()
    bvh.close()
    for scale in (2.0 ** -30, 2.0 ** 40):
        bvh = G.FastWindingNumberBVH(V * scale, F, tree="binned")
        Ds, _, Cs = bvh.squared_distance(P * scale)
        assert np.array_equal(Ds, D * scale ** 2)
        bvh.close()
    # the tree of the signed distance, which holds nothing but the search
    S, I2, C2 = G.signed_distance(P, V, F, G.SIGNED_DISTANCE_TYPE_UNSIGNED)
    assert np.array_equal(S, np.sqrt(D)) and np.array_equal(I2, I) and np.array_equal(C2, C)


@pytest.mark.parametrize("far", [0.0, 1e3, 1e6, 1e12])
def test_search_beside_a_far_triangle(cuda, far):
    """The search's pruning does not widen with the extent of the surface: one
    triangle far away, queries next to the rest (distances down to 1e-7, the
    closest triangle as in the exact search) and next to the far one."""
    V, F = synth.icosphere(4)
    rng = np.random.default_rng(77)
    P = np.concatenate([V[rng.integers(0, len(V), 3000)] + 10.0 ** rng.uniform(-7, -1, (3000, 1))
                        * rng.normal(size=(3000, 3)), rng.uniform(-1.2, 1.2, (500, 3)),
                        rng.normal(size=(100, 3)) * 1e-9])
    if far:
        T = far * np.array([[1, 0, 0], [1, 1e-4, 0], [1, 0, 1e-4]])
        F = np.concatenate([F, len(V) + np.arange(3, dtype=np.int32)[None]])
        V = np.concatenate([V, T])
        P = np.concatenate([P, T.mean(0) + far * 1e-4 * rng.normal(size=(200, 3))])
    bvh = G.FastWindingNumberBVH(V, F, tree="binned")
    D, I, C = bvh.squared_distance(P)
    bvh.close()
    Dr, Ir, Cr = O.squared_distance(V, F, P)
    assert _close2(D, Dr).all()
    assert _close2(_tri_dist2(V, F, P, I), D).all()


def test_search_beside_a_far_triangle_takes_no_longer_than_its_bounds_ask(cuda):
    """300,000 queries near an 82,000-triangle sphere with one triangle 10,000
    radii away.  The triangles' own FP32 bounds carry a rounding of 1e-6 of that
    extent, so the search visits more of the sphere than without it: about six
    times the time; with node bounds that carried it too, fifteen times."""
    V, F = synth.geodesic_sphere(64)
    V = synth.sh_deform(V, np.random.default_rng(3))
    rng = np.random.default_rng(1)
    Q = cuda.from_numpy(V[rng.integers(0, len(V), 300_000)]
                        + 1e-3 * rng.normal(size=(300_000, 3))).cuda()
    t = []
    for far in (False, True):
        if far:
            F = np.concatenate([F, len(V) + np.arange(3)[None]]).astype(np.int32)
            V = np.concatenate([V, [[1e4, 0, 0], [1e4, 1, 0], [1e4, 0, 1]]])
        bvh = G.FastWindingNumberBVH(V, F)
        best = float("inf")
        for k in range(8):
            cuda.cuda.synchronize()
            t0 = time.perf_counter()
            bvh.squared_distance(Q)
            cuda.cuda.synchronize()
            if k >= 2:
                best = min(best, time.perf_counter() - t0)
        t.append(best)
        bvh.close()
    assert t[1] <= 10 * t[0], t
