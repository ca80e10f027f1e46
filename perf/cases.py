"""Timed workloads of this package: winding numbers and the queries next to
them, through the public entry points, on CUDA tensors (the server takes host
arrays, as its callers hold them).

A case is a plain dict; ``prepare`` makes its inputs and the handles that a
program keeps between calls, ``run`` is one pass, ``work`` what the pass cannot
do without, and ``exact`` the same outputs summed in 64 bits by plain torch
where that is affordable."""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import libigl_gb300 as G
from libigl_gb300 import synth

DEV = "cuda"

# Triangle counts are 20 nu^2 (a geodesic sphere of frequency nu); nu = 256 is
# the benchmark's 1.31M-triangle sphere, nu = 16 its 5,120-triangle one.
NU_MIN, NU_MAX = 7, 256


def listed():
    return [
        # One short request against a tree that is kept: an interactive
        # probe, a collision test, one step of a solver.
        dict(name="soup_eval_tiny", kind="soup_eval", nu=8, nq=1000, q="f32", precision="mixed",
             order=2),
        # The benchmark's headline: 10M float32 points against 1.3M triangles
        # with 1% of them missing, tree kept.
        dict(name="soup_eval_10M", kind="soup_eval", nu=256, nq=10_000_000, q="f32",
             precision="mixed", order=2),
        # The same evaluation in plain FP64, for a caller that wants the
        # reference's algorithm without mixed precision; odd counts.
        dict(name="soup_eval_fp64", kind="soup_eval", nu=64, nq=300_001, q="f64",
             precision="fp64", order=2),
        # fast_winding_number(V,F,Q,W) as most callers write it: tree built in
        # the call, a scan-sized mesh and as many points as a coarse grid.
        dict(name="soup_oneshot_mid", kind="soup_oneshot", nu=64, nq=100_000, q="f32",
             precision="mixed", order=2),
        # The one-shot call on a large mesh: the tree build carries it.
        dict(name="soup_oneshot_large", kind="soup_oneshot", nu=256, nq=1_000_000, q="f32",
             precision="mixed", order=2),
        # Exact winding number of the benchmark's first configuration.
        dict(name="exact_mixed", kind="exact", nu=16, nq=100_000, q="f32", precision="mixed"),
        # The exact winding number at the reference's own precision.
        dict(name="exact_fp64", kind="exact", nu=32, nq=50_001, q="f64", precision="fp64"),
        # Point cloud, one call: octree, expansions and evaluation, at the
        # benchmark's 2M points and 8M queries.
        dict(name="cloud_oneshot", kind="cloud_oneshot", np=2_000_000, nq=8_000_000, q="f32",
             precision="mixed"),
        # A scan with points and normals only: octree, nearest points, point
        # areas, expansions, evaluation.
        dict(name="cloud_points", kind="cloud_points", np=200_003, nq=500_000, q="f32",
             precision="mixed"),
        # Signed distance to a closed mesh (search tree and pseudonormals
        # built in the call, as in the reference).
        dict(name="signed_distance", kind="signed_distance", nu=128, nq=300_000,
             sign="pseudonormal"),
        # Volume swept by a moving ellipsoid: the benchmark's 64 poses on a
        # grid of 128 points along its longest side.
        dict(name="swept", kind="swept", subdiv=5, poses=64, res=128, sign="pseudonormal"),
        # A burst of mixed requests to a server that keeps its meshes resident.
        dict(name="served_burst", kind="served", meshes=12, nu_max=128, requests=48,
             q_max=262_144, q="f32"),
    ]


def draw(rng):
    def logint(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["soup_eval", "soup_eval", "soup_oneshot", "soup_oneshot", "exact", "exact",
                       "cloud_oneshot", "cloud_oneshot", "cloud_points", "signed_distance",
                       "swept", "served"])
    if kind in ("soup_eval", "soup_oneshot", "exact"):
        fp64 = rng.random() < 0.3
        c = dict(kind=kind, q="f64" if fp64 else "f32", precision="fp64" if fp64 else "mixed")
        if kind == "exact":
            return dict(c, nu=logint(7, 48), nq=logint(100, 60_000 if fp64 else 300_000))
        if kind == "soup_eval" and not fp64:
            c["q"] = rng.choice(["f32", "f64"])
        return dict(c, nu=logint(NU_MIN, NU_MAX), order=rng.choice([2, 2, 1, 0]),
                    nq=logint(500, 500_000 if fp64 else 10_000_000))
    if kind in ("cloud_oneshot", "cloud_points"):
        top = 2_000_000 if kind == "cloud_oneshot" else 400_000
        return dict(kind=kind, np=logint(2000, top), nq=logint(500, 4 * top), q="f32",
                    precision="mixed")
    if kind == "signed_distance":
        exact_sign = rng.random() < 0.4
        return dict(kind=kind, nu=logint(NU_MIN, 64 if exact_sign else 128),
                    nq=logint(500, 100_000 if exact_sign else 300_000),
                    sign="default" if exact_sign else "pseudonormal")
    if kind == "swept":
        return dict(kind=kind, subdiv=rng.choice([3, 4, 5]), poses=logint(4, 64),
                    res=logint(24, 128), sign="pseudonormal")
    return dict(kind=kind, meshes=logint(2, 12), nu_max=logint(16, 128), requests=logint(2, 48),
                q_max=logint(2000, 262_144), q="f32")


# ------------------------------------------------------------------ inputs --
@functools.lru_cache(maxsize=16)
def _sphere(nu):
    """Vertices and faces of the unit geodesic sphere, on the GPU."""
    V, F = synth.geodesic_sphere(nu)
    return torch.from_numpy(np.ascontiguousarray(V)).to(DEV), torch.from_numpy(F).to(DEV)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _bumpy(U, g, lmax=8, sigma=0.05):
    """Unit vectors pushed radially by zonal bumps P_l about random axes (a
    band-limited field of degree 1..lmax, amplitudes falling as 1/l)."""
    r = torch.ones(U.shape[0], device=DEV, dtype=torch.float64)
    for l in range(1, lmax + 1):
        for _ in range(3):
            axis = _randn(g, 3)
            t = U @ (axis / axis.norm())
            a, b = torch.ones_like(t), t
            for k in range(2, l + 1):
                a, b = b, ((2 * k - 1) * t * b - (k - 1) * a) / k
            r = r + _randn(g, 1) * (sigma / l) * b
    return U * r.clamp_min(0.2)[:, None]


def _mesh(nu, g, holes=0.01):
    U, F = _sphere(nu)
    V = _bumpy(U, g)
    if holes:
        F = F[_rand(g, F.shape[0]) >= holes]
    return V.contiguous(), F.contiguous()


def _soup_queries(V, F, g, nq, near=0.1):
    """90% uniform in the box grown 1.2x, 10% at 10^U(-4,-1) along a normal."""
    lo, hi = V.amin(0), V.amax(0)
    n_near = int(nq * near)
    Q = (lo + hi) / 2 + (2 * _rand(g, nq, 3) - 1) * (hi - lo) * 0.6
    f = F[(_rand(g, n_near) * F.shape[0]).long().clamp_max(F.shape[0] - 1)].long()
    a, b, c = V[f[:, 0]], V[f[:, 1]], V[f[:, 2]]
    uv = _rand(g, n_near, 2)
    uv = torch.where(uv.sum(1, keepdim=True) > 1, 1 - uv, uv)
    n = torch.linalg.cross(b - a, c - a)
    n = n / n.norm(dim=1, keepdim=True)
    d = 10.0 ** (-4 + 3 * _rand(g, n_near)) * torch.sign(_rand(g, n_near) - 0.5)
    Q[:n_near] = a + uv[:, :1] * (b - a) + uv[:, 1:] * (c - a) + d[:, None] * n
    return Q[torch.argsort(_rand(g, nq))].contiguous()


def _torus(g, n, R=1.0, r=0.35):
    """Area-uniform torus samples with a radial error, jittered normals and
    uneven areas."""
    u = 2 * math.pi * _rand(g, n)
    y = 2 * math.pi * _rand(g, n)
    v = y
    for _ in range(30):  # v + (r/R) sin v = y: the angle of a uniform area
        v = v - (v + (r / R) * torch.sin(v) - y) / (1 + (r / R) * torch.cos(v))
    rr = r + 0.005 * _randn(g, n)
    cu, su, cv, sv = u.cos(), u.sin(), v.cos(), v.sin()
    P = torch.stack([(R + rr * cv) * cu, (R + rr * cv) * su, rr * sv], 1)
    N = torch.stack([cv * cu, cv * su, sv], 1) + 0.05 * _randn(g, n, 3)
    N = N / N.norm(dim=1, keepdim=True)
    A = (4 * math.pi ** 2 * R * r / n) * (0.8 + 0.4 * _rand(g, n))
    return P.contiguous(), N.contiguous(), A


def _torus_queries(g, nq):
    half = torch.tensor([1.6, 1.6, 0.6], device=DEV, dtype=torch.float64)
    return (2 * _rand(g, nq, 3) - 1) * half


def _as(Q, q):
    return Q.to(torch.float32) if q == "f32" else Q


def _inputs(case, seed):
    """The input arrays of a case (everything but kept handles)."""
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("soup_eval", "soup_oneshot"):
        V, F = _mesh(case["nu"], g)
        return dict(V=V, F=F, Q=_as(_soup_queries(V, F, g, case["nq"]), case["q"]))
    if kind == "exact":
        U, F = _sphere(case["nu"])
        V = (U * (1 + 0.02 * _randn(g, U.shape[0]))[:, None]).contiguous()
        return dict(V=V, F=F, Q=_as(3 * _rand(g, case["nq"], 3) - 1.5, case["q"]))
    if kind in ("cloud_oneshot", "cloud_points"):
        P, N, A = _torus(g, case["np"])
        return dict(P=P, N=N, A=A, Q=_as(_torus_queries(g, case["nq"]), case["q"]))
    if kind == "signed_distance":
        V, F = _mesh(case["nu"], g, holes=0.0)
        return dict(V=V, F=F, Q=_soup_queries(V, F, g, case["nq"]))
    if kind == "swept":
        V, F, T, GV, _, _ = synth.swept_workload(seed, case["subdiv"], case["poses"], 24)
        # a grid of the workload's usual proportions over the sweep's box
        res = np.array([case["res"], round(0.55 * case["res"]), round(0.5 * case["res"])], np.int32)
        lo, hi = GV.min(0), GV.max(0)
        h = float(((hi - lo) / (res - 1)).max())
        x, y, z = (lo[d] + h * torch.arange(int(res[d]), device=DEV, dtype=torch.float64)
                   for d in range(3))
        Z, Y, X = torch.meshgrid(z, y, x, indexing="ij")
        GV = torch.stack([X.reshape(-1), Y.reshape(-1), Z.reshape(-1)], 1).contiguous()
        return dict(V=torch.from_numpy(V).to(DEV), F=torch.from_numpy(F).to(DEV), T=T, GV=GV,
                    res=res, h=h)
    rng = np.random.default_rng(seed)
    meshes, boxes = [], []
    for i in range(case["meshes"]):
        t = i / max(case["meshes"] - 1, 1)
        nu = int(round(NU_MIN * (case["nu_max"] / NU_MIN) ** t))
        V, F = _mesh(nu, g, holes=0.0 if i % 5 else 0.01)
        meshes.append((V.cpu().numpy(), F.cpu().numpy()))
        boxes.append((V.amin(0).cpu().numpy(), V.amax(0).cpu().numpy()))
    requests = []
    sizes = np.random.default_rng(case["requests"])  # of the case, not of the seed
    for _ in range(case["requests"]):
        m = int(sizes.integers(case["meshes"]))
        n = int(np.exp(sizes.uniform(np.log(1000), np.log(case["q_max"]))))
        lo, hi = boxes[m]
        requests.append((m, rng.uniform(lo, hi, (n, 3)).astype(np.float32)))
    return dict(meshes=meshes, requests=requests)


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "soup_eval":
        s["bvh"] = G.FastWindingNumberBVH(s["V"], s["F"], case["order"])
    elif case["kind"] == "served":
        s["server"] = G.Server(hbm_budget_bytes=40 << 30)
        s["ids"] = [s["server"].add_mesh(V, F) for V, F in s.pop("meshes")]
        # a server in use has its meshes resident
        for r in [s["server"].submit(i, s["requests"][0][1][:32]) for i in s["ids"]]:
            r.wait()
    return s


# -------------------------------------------------------------------- pass --
_SIGN = {"pseudonormal": G.SIGNED_DISTANCE_TYPE_PSEUDONORMAL,
         "default": G.SIGNED_DISTANCE_TYPE_DEFAULT}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "soup_eval":
        # a mixed-precision result carries FP32 accuracy, whatever Q's type
        return s["bvh"].eval(s["Q"], 2.0, case["precision"],
                             out_dtype=np.float32 if case["precision"] == "mixed" else np.float64)
    if kind == "soup_oneshot":
        return G.fast_winding_number_soup(s["V"], s["F"], s["Q"], case["order"], 2.0,
                                          case["precision"])
    if kind == "exact":
        return G.winding_number(s["V"], s["F"], s["Q"], case["precision"])
    if kind == "cloud_oneshot":
        return G.fast_winding_number_cloud_oneshot(s["P"], s["N"], s["A"], s["Q"], 2, 2.0,
                                                   case["precision"])
    if kind == "cloud_points":
        return G.fast_winding_number_cloud_points(s["P"], s["N"], s["Q"], 2, 2.0,
                                                  case["precision"])
    if kind == "signed_distance":
        S, I, C = G.signed_distance(s["Q"], s["V"], s["F"], _SIGN[case["sign"]])
        return dict(S=S, I=I, C=C)
    if kind == "swept":
        return G.swept_volume_signed_distance(s["V"], s["F"], s["T"], _SIGN[case["sign"]],
                                              s["GV"], s["res"], s["h"], 0.0)
    sent = [s["server"].submit(s["ids"][m], Q) for m, Q in s["requests"]]
    return [r.wait()[0] for r in sent]


def work(case):
    """Bytes: every input read and every output written once.  Operations: a
    tree search per query, about what one level of an order-2 walk (350), an
    exact cap walk or a closest-point search costs per factor of two in size;
    the sort and moments of a build per primitive."""
    kind = case["kind"]
    if kind == "served":
        lo, hi = math.log(1000), math.log(case["q_max"])
        nq = case["requests"] * ((case["q_max"] - 1000) / (hi - lo) if hi > lo else 1000)
        return dict(bytes=nq * 16, flops=nq * 350 * math.log2(20 * case["nu_max"] ** 2))
    if kind == "swept":
        nf, nq = 20 * 4 ** case["subdiv"], case["res"] ** 3 // 4
        return dict(bytes=nf * 24 + nq * 32, flops=nq * case["poses"] * 100)
    size = 8 if case.get("q", "f64") == "f64" else 4
    nq = case["nq"]
    if "np" in case:
        n, prim = case["np"], 56.0
    else:
        n, prim = 20 * case["nu"] ** 2, 24.0
    out = {"signed_distance": size + 4 + 24}.get(kind, size)
    build = 0 if kind == "soup_eval" else n * 50 * math.log2(n)
    return dict(bytes=n * prim + nq * (3 * size + out),
                flops=nq * 350 * math.log2(n) + build)


# ------------------------------------------------------------------- exact --
_PAIRS = 2.5e10  # pairs that plain torch sums in well under 20 s


def _winding(V, F, Q):
    """The generalized winding number as a plain sum of solid angles."""
    Q = Q.double()
    f = F.long()
    W = torch.zeros(Q.shape[0], device=DEV, dtype=torch.float64)
    step = max(1, 8_000_000 // max(Q.shape[0], 1))
    qx, qy, qz = (Q[:, k, None] for k in range(3))
    for i in range(0, f.shape[0], step):
        T = V[f[i:i + step]]
        (ax, ay, az), (bx, by, bz), (cx, cy, cz) = (
            (T[:, k, 0] - qx, T[:, k, 1] - qy, T[:, k, 2] - qz) for k in range(3))
        la = torch.sqrt(ax * ax + ay * ay + az * az)
        lb = torch.sqrt(bx * bx + by * by + bz * bz)
        lc = torch.sqrt(cx * cx + cy * cy + cz * cz)
        det = ax * (by * cz - bz * cy) + ay * (bz * cx - bx * cz) + az * (bx * cy - by * cx)
        den = (la * lb * lc + (ax * bx + ay * by + az * bz) * lc
               + (bx * cx + by * cy + bz * cz) * la + (cx * ax + cy * ay + cz * az) * lb)
        W += torch.atan2(det, den).sum(1)
    return W / (2 * math.pi)


def _dipoles(P, N, A, Q):
    """The cloud's winding number as a plain sum of its points' dipoles."""
    Q = Q.double()
    W = torch.zeros(Q.shape[0], device=DEV, dtype=torch.float64)
    M = N * A[:, None]
    step = max(1, 16_000_000 // max(Q.shape[0], 1))
    qx, qy, qz = (Q[:, k, None] for k in range(3))
    for i in range(0, P.shape[0], step):
        p, m = P[i:i + step], M[i:i + step]
        x, y, z = p[:, 0] - qx, p[:, 1] - qy, p[:, 2] - qz
        r2 = x * x + y * y + z * z
        W += ((x * m[:, 0] + y * m[:, 1] + z * m[:, 2]) / (r2 * torch.sqrt(r2))).sum(1)
    return W / (4 * math.pi)


def _closest(V, F, Q):
    """Squared distance and closest point of Q over all triangles: the plane's
    foot where it falls inside, else the nearest of the three edges."""
    f = F.long()
    best = torch.full((Q.shape[0],), math.inf, device=DEV, dtype=torch.float64)
    at = torch.zeros(Q.shape[0], device=DEV, dtype=torch.long)
    step = max(1, 4_000_000 // max(Q.shape[0], 1))

    def candidates(a, b, c, q):
        for p0, p1 in ((a, b), (b, c), (c, a)):
            e = p1 - p0
            t = (((q - p0) * e).sum(-1) / (e * e).sum(-1)).clamp(0, 1)
            yield p0 + t[..., None] * e, None
        n = torch.linalg.cross(b - a, c - a)
        n = n / n.norm(dim=-1, keepdim=True)
        foot = q - ((q - a) * n).sum(-1)[..., None] * n
        inside = torch.ones(foot.shape[:-1], device=DEV, dtype=torch.bool)
        for p0, p1 in ((a, b), (b, c), (c, a)):
            inside &= (torch.linalg.cross((p1 - p0).expand_as(foot), foot - p0) * n).sum(-1) >= 0
        yield foot, inside

    def nearest(a, b, c, q):
        d, x = None, None
        for p, ok in candidates(a, b, c, q):
            dd = ((q - p) ** 2).sum(-1)
            if ok is not None:
                dd = torch.where(ok, dd, math.inf)
            if d is None:
                d, x = dd, p
            else:
                x = torch.where((dd < d)[..., None], p, x)
                d = torch.minimum(d, dd)
        return d, x

    for i in range(0, f.shape[0], step):
        T = V[f[i:i + step]][None]
        d, _ = nearest(T[:, :, 0], T[:, :, 1], T[:, :, 2], Q[:, None])
        m, k = d.min(1)
        at = torch.where(m < best, k + i, at)
        best = torch.minimum(best, m)
    T = V[f[at]]
    return nearest(T[:, 0], T[:, 1], T[:, 2], Q)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("swept", "served", "cloud_points"):
        return None
    n = case["np"] if "np" in case else 20 * case["nu"] ** 2
    if n * case["nq"] > (_PAIRS / 12 if kind == "signed_distance" else _PAIRS):
        return None
    s = _inputs(case, seed)
    if kind == "cloud_oneshot":
        return _dipoles(s["P"], s["N"], s["A"], s["Q"])
    if kind == "signed_distance":
        d2, C = _closest(s["V"], s["F"], s["Q"])
        W = _winding(s["V"], s["F"], s["Q"])
        sign = 1 - 2 * (W if case["sign"] == "default" else (W > 0.5).double())
        return dict(S=torch.sqrt(d2) * sign, I=None, C=C)
    return _winding(s["V"], s["F"], s["Q"])
