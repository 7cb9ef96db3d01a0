"""Timing cases of the combined-field layer potentials and their solvers.

Each case is one call, or the short sequence of calls, that a program built
on this package spends its time in, made through the public entry points:
``Plan.solve`` and ``Plan.matvec`` on a resident operator, ``SurfaceBatch``,
``surface.setup`` and the host-buffer entry points of ``layer``.  The surfaces
are smooth closed quad meshes with closed-form charts (tensor Gauss-Legendre
patches, iptype 11): spheres and ellipsoids as six-sided meshes of M x M
patches a side, and the wobbled torus of ``surface.torus_quad``.  Sizes follow
the package's benchmark: the 36,000-node ellipsoid at k = 2, its batch of 64
plane waves at k = 5, the torus with 16 plane waves, batches of uneven
ellipsoids with 4 point sources each, and surfaces above 140,000 nodes whose
far field is hierarchical; small meshes of a few hundred nodes stand for
interactive use and for the inner solves of larger programs.

On the unit sphere the combined-field operator is diagonal on the spherical
harmonics, so ``exact`` gives those cases' outputs in closed form.
"""
import math

import numpy as np
import torch

from fmm3dbie_b200 import Plan, layer
from fmm3dbie_b200 import surface as S
from fmm3dbie_b200.batch import BatchItem, SurfaceBatch

EPS = 1e-7        # quadrature and far-field tolerance of every setup
TOL = 1e-10       # residual of every solve
NUMIT = 200
LMAX = 4          # highest degree of the spherical harmonics used as densities
MODES = 6         # zonal harmonics per density
TERMS = 44        # terms of the expansions of point sources and plane waves on the sphere

# outward-oriented axes (first tangent, second tangent, outward direction)
_FACES = ((1, 2, 0, 1.0), (2, 1, 0, -1.0), (2, 0, 1, 1.0), (0, 2, 1, -1.0), (0, 1, 2, 1.0),
          (1, 0, 2, -1.0))


def quad_ellipsoid(m, norder, axes=(1.0, 1.0, 1.0), center=(0.0, 0.0, 0.0)):
    """Ellipsoid of 6 x m x m quads, tensor Gauss-Legendre nodes of order
    norder: the equiangular map of a cube, scaled by the semi-axes."""
    x, _ = np.polynomial.legendre.leggauss(norder + 1)
    h = 1.0 / m
    u = np.tile(x, norder + 1)
    v = np.repeat(x, norder + 1)
    rows = []
    ax = np.asarray(axes, float)
    for ia, ib, ic, sg in _FACES:
        for j in range(m):
            for i in range(m):
                a = 0.25 * math.pi * (-1.0 + h * (2 * i + 1 + u))
                b = 0.25 * math.pi * (-1.0 + h * (2 * j + 1 + v))
                ta, tb = np.tan(a), np.tan(b)
                c = 0.25 * math.pi * h
                q, qa, qb = (np.zeros((u.size, 3)) for _ in range(3))
                q[:, ia], q[:, ib], q[:, ic] = ta, tb, sg
                qa[:, ia] = c * (1.0 + ta * ta)
                qb[:, ib] = c * (1.0 + tb * tb)
                r = np.sqrt((q * q).sum(1))[:, None]
                p = q / r
                pu = (qa - p * (p * qa).sum(1)[:, None]) / r
                pv = (qb - p * (p * qb).sum(1)[:, None]) / r
                xyz, xu, xv = p * ax, pu * ax, pv * ax
                n = np.cross(xu, xv)
                n /= np.linalg.norm(n, axis=1)[:, None]
                rows.append(np.concatenate([xyz + np.asarray(center, float), xu, xv, n], 1))
    npat = 6 * m * m
    return S.from_srcvals(np.full(npat, norder, np.int64), np.full(npat, 11, np.int64),
                          np.concatenate(rows))


def _surface(case, center=(0.0, 0.0, 0.0)):
    if case["shape"] == "torus":
        s = S.torus_quad(case["m"], case["m2"], case["norder"])
        sv = s.srcvals.copy()
        sv[:, :3] += np.asarray(center, float)
        return S.from_srcvals(s.norders, s.iptype, sv)
    ax = {"sphere": (1.0, 1.0, 1.0), "ellipsoid": (1.0, 2.0, 3.0)}[case["shape"]]
    return quad_ellipsoid(case["m"], case["norder"], ax, center)


def _params(case):
    """(alpha, beta) or (k, -ik, 1): the benchmark's combinations."""
    if case["kind"] == 0:
        return (1.0, 1.0)
    return (case["k"], -1j * case["k"], 1.0)


def _directions(rng, n):
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1)[:, None]


# ---- data ------------------------------------------------------------------
def _harmonics(case, rng):
    """MODES random zonal harmonics: (coefficients, degrees, axes)."""
    c = rng.normal(size=MODES)
    if case["kind"] == 1:
        c = c + 1j * rng.normal(size=MODES)
    return c, rng.integers(0, LMAX + 1, MODES), _directions(rng, MODES)


def _legendre(n, t):
    """P_0 .. P_n at the tensor t, one after the other."""
    a, b = torch.ones_like(t), t
    yield a
    for l in range(1, n + 1):
        yield b
        a, b = b, ((2 * l + 1) * t * b - l * a) / (l + 1)


def _zonal(harm, x, factor=None):
    """sum_q c_q f(l_q, r) P_l_q(x/r . d_q) at the points x (n, 3);
    factor(l, r): radial factor (1 when absent)."""
    x = torch.as_tensor(x, dtype=torch.float64, device="cuda")
    r = x.square().sum(1).sqrt()
    s = 0
    for c, l, d in zip(*harm):
        t = (x @ torch.tensor(d, device="cuda")) / r
        f = 1.0 if factor is None else factor(int(l), r)
        s = s + c.item() * f * list(_legendre(int(l), t))[-1]
    return s


def _sources(case, rng, n):
    """n interior points, inside 0.3 x the semi-axes (near the tube's centre
    line for the torus)."""
    if case["shape"] == "torus":
        t = rng.uniform(0, 2 * math.pi, n)
        return np.stack([2.0 * np.cos(t), 2.0 * np.sin(t), 0.2 * rng.uniform(-1, 1, n)], 1)
    ax = {"sphere": (1.0, 1.0, 1.0), "ellipsoid": (1.0, 2.0, 3.0)}[case["shape"]]
    return 0.3 * np.asarray(ax) * _directions(rng, n) * rng.uniform(0, 1, (n, 1)) ** (1 / 3)


def _point_source(kind, k, xyz, src):
    """Potentials of the interior point sources at the nodes, one per column."""
    x = torch.as_tensor(xyz, device="cuda")
    cols = []
    for s in src:
        r = (x - torch.tensor(s, device="cuda")).square().sum(1).sqrt()
        cols.append((torch.exp(1j * k * r) if kind == 1 else 1.0) / (4 * math.pi * r))
    return torch.stack(cols, 1)


def _plane_waves(k, xyz, d):
    d = torch.tensor(d, device="cuda")
    return -torch.exp(1j * k * (torch.as_tensor(xyz, device="cuda") @ d.T))


def _rhs(case, surf, rng):
    nd = case.get("nd", 1)
    if case["rhs"] == "waves":
        b = _plane_waves(case["k"], surf.xyz, _directions(rng, nd))
    else:
        b = _point_source(case["kind"], case.get("k", 0.0), surf.xyz, _sources(case, rng, nd))
    return b.contiguous() if nd > 1 else b[:, 0].contiguous()


# ---- the sphere's spectra ----------------------------------------------------
def _bessel(l, z):
    """j_l, y_l and their derivatives at the real z (numbers), by series and
    upward recurrence."""
    def series(n):
        s, term, m = 0.0, 1.0, 0
        for i in range(1, n + 1):
            term *= z / (2 * i + 1)
        while abs(term) > 1e-18 * max(abs(s), 1e-300) and m < 200:
            s += term
            m += 1
            term *= -z * z / (2 * m * (2 * n + 2 * m + 1))
        return s

    def y(n):
        a, b = -math.cos(z) / z, -math.cos(z) / z ** 2 - math.sin(z) / z
        for i in range(1, n):
            a, b = b, (2 * i + 1) / z * b - a
        return a if n == 0 else b

    j0, j1 = series(l), series(l + 1)
    y0, y1 = y(l), y(l + 1)
    return j0, y0, l / z * j0 - j1, l / z * y0 - y1


def _hankel(l, z):
    """h_l at the tensor z, by upward recurrence."""
    e = torch.exp(1j * z)
    a, b = -1j * e / z, -e * (1 / z + 1j / z ** 2)
    for i in range(1, l):
        a, b = b, (2 * i + 1) / z * b - a
    return a if l == 0 else b


def _eigenvalue(case, l):
    """alpha S + beta D (principal value) on the degree-l harmonics."""
    p = _params(case)
    if case["kind"] == 0:
        return p[0] / (2 * l + 1) - p[1] / (2.0 * (2 * l + 1))
    k = case["k"]
    j, y, dj, dy = _bessel(l, k)
    h, dh = j + 1j * y, dj + 1j * dy
    return p[1] * 1j * k * j * h + p[2] * 0.5j * k * k * (j * dh + dj * h)


def _outside(case, l, r):
    """alpha S + beta D of a degree-l harmonic at distance r > 1, over the
    harmonic."""
    p = _params(case)
    if case["kind"] == 0:
        return (p[0] + p[1] * l) / (2 * l + 1) * r ** -(l + 1.0)
    k = case["k"]
    j, _, dj, _ = _bessel(l, k)
    return (p[1] * 1j * k * j + p[2] * 1j * k * k * dj) * _hankel(l, k * r)


def _sphere_nodes(case):
    """Nodes of the sphere case's mesh, from the chart alone."""
    x, _ = np.polynomial.legendre.leggauss(case["norder"] + 1)
    m = case["m"]
    t = np.tan(0.25 * math.pi * (-1.0 + (2 * np.arange(m)[:, None] + 1 + x[None, :]) / m))
    out = []
    for ia, ib, ic, sg in _FACES:
        for j in range(m):
            for i in range(m):
                q = np.zeros((x.size ** 2, 3))
                q[:, ia], q[:, ib], q[:, ic] = np.tile(t[i], x.size), np.repeat(t[j], x.size), sg
                out.append(q / np.sqrt((q * q).sum(1))[:, None])
    return np.concatenate(out)


# ---- cases -------------------------------------------------------------------
def listed():
    return [
        # the smallest calls: a coarse mesh solved again and again, where
        # launches and the host loop of GMRES count
        {"name": "lap small solve", "op": "solve", "kind": 0, "shape": "sphere", "m": 3,
         "norder": 3, "mode": 0, "rhs": "points"},
        {"name": "helm small mixed solve", "op": "solve", "kind": 1, "shape": "sphere", "m": 6,
         "norder": 4, "k": 1.5, "mode": 1, "rhs": "points"},
        # one operator application in FP64, as a program with a solver of its
        # own makes it (odd mesh)
        {"name": "helm fp64 matvec", "op": "matvec", "kind": 1, "shape": "sphere", "m": 11,
         "norder": 5, "k": 2.0, "iprec": 0},
        # the benchmark's solve: ellipsoid, one interior point source, k = 2
        {"name": "helm mixed solve", "op": "solve", "kind": 1, "shape": "ellipsoid", "m": 13,
         "norder": 5, "k": 2.0, "mode": 1, "rhs": "points"},
        # the reference method on a torus of ordinary size: FP64 GMRES
        {"name": "helm fp64 solve torus", "op": "solve", "kind": 1, "shape": "torus", "m": 40,
         "m2": 18, "norder": 4, "k": 3.1875, "mode": 0, "rhs": "waves"},
        # 64 plane waves on the ellipsoid at k = 5
        {"name": "helm 64 plane waves", "op": "solve", "kind": 1, "shape": "ellipsoid", "m": 13,
         "norder": 5, "k": 5.0, "mode": 1, "rhs": "waves", "nd": 64},
        # 16 plane waves on the torus (scattering sweeps)
        {"name": "helm 16 plane waves torus", "op": "solve", "kind": 1, "shape": "torus", "m": 48,
         "m2": 24, "norder": 5, "k": 6.6875, "mode": 1, "rhs": "waves", "nd": 16},
        # uneven surfaces with 4 point sources each, one operator
        {"name": "lap uneven batch", "op": "batch", "kind": 0, "shape": "ellipsoid", "nsurf": 9,
         "m": 8, "norder": 6, "nd": 4},
        # a surface whose far field is hierarchical
        {"name": "helm large mixed solve", "op": "solve", "kind": 1, "shape": "ellipsoid", "m": 26,
         "norder": 5, "k": 2.0, "mode": 1, "rhs": "points"},
        {"name": "lap large fp64 matvec", "op": "matvec", "kind": 0, "shape": "sphere", "m": 31,
         "norder": 5, "iprec": 0},
        # a new surface: near list, far orders, oversampling, near quadrature
        {"name": "helm setup", "op": "setup", "kind": 1, "shape": "ellipsoid", "m": 12,
         "norder": 5, "k": 2.0},
        # the field off the surface, from host arrays in one call
        {"name": "helm field from host arrays", "op": "field", "kind": 1, "shape": "sphere",
         "m": 8, "norder": 5, "k": 2.0, "ntarg": 20011},
    ]


def draw(rng):
    op = rng.choice(["solve", "solve", "solve", "batch", "matvec", "matvec", "setup", "field"])
    kind = rng.choice([0, 1, 1])
    shape = rng.choice(["sphere", "ellipsoid", "torus"])
    norder = rng.choice([3, 4, 5, 6, 7])
    c = {"op": op, "kind": kind, "shape": shape, "norder": norder}
    if kind == 1:
        c["k"] = round(rng.uniform(1.0, 6.0), 4)
    if op == "field":
        c["shape"] = "sphere"
        c["ntarg"] = int(round(math.exp(rng.uniform(math.log(500), math.log(60000)))))
    if op == "batch":
        c.update(shape="ellipsoid", nsurf=rng.randint(3, 12), nd=rng.choice([1, 2, 3, 4]))
    # nodes: 400 .. 120,000 for one density, fewer with many or in FP64
    nd = c.get("nd", 1)
    top = {"solve": 40000, "batch": 9000, "matvec": 120000, "setup": 30000, "field": 15000}[op]
    if op == "solve":
        c["mode"] = rng.choice([0, 1, 1])
        nd = rng.choice([1, 1, 1, 2, 4, 5, 8, 16, 24])
        c["rhs"] = "waves" if kind == 1 and rng.random() < 0.5 else "points"
        if nd > 1:
            c["nd"] = nd
            top = 16000
        elif c["mode"] == 0:
            top = 25000
    if op == "matvec":
        c["iprec"] = 0
    npts = math.exp(rng.uniform(math.log(500), math.log(top)))
    per = (norder + 1) ** 2
    if c["shape"] == "torus":
        m2 = max(6, int(round(math.sqrt(npts / per / 2))))
        c["m2"] = m2
        c["m"] = max(12, 2 * m2 + rng.randint(-3, 3))
        size = 17.0 / c["m"]
    else:
        c["m"] = max(3 if norder < 6 else 2, int(round(math.sqrt(npts / per / 6))))
        size = (1.6 if c["shape"] == "sphere" else 4.7) / c["m"]
    if kind == 1:
        # a wave is resolved: its phase over a patch stays below the order
        c["k"] = round(min(c["k"], 0.7 * norder / size), 4)
    return c


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    op, p = case["op"], _params(case)
    if op == "batch":
        # semi-axes, sizes and orders differ from surface to surface
        shape_rng = np.random.default_rng(case["nsurf"])
        items, rhs = [], []
        for q in range(case["nsurf"]):
            ax = shape_rng.uniform(0.5, 3.0, 3)
            m = max(2, int(round(case["m"] * shape_rng.uniform(0.3, 1.2))))
            surf = quad_ellipsoid(m, max(3, case["norder"] - int(shape_rng.integers(0, 3))), ax)
            k = float(shape_rng.uniform(0.5, 1.0)) * case.get("k", 0.0)
            pq = (1.0, 1.0) if case["kind"] == 0 else (k, -1j * k, 1.0)
            items.append(BatchItem(surf, case["kind"], pq, 0.5))
            src = 0.3 * ax * _directions(rng, case["nd"]) * rng.uniform(0, 1, (case["nd"], 1)) ** (1 / 3)
            rhs.append(_point_source(case["kind"], k, surf.xyz, src).contiguous())
        return {"op": op, "batch": SurfaceBatch(items, EPS), "rhs": rhs}
    if op == "setup":
        # the surface stands somewhere else each time
        return {"op": op, "surf": _surface(case, rng.uniform(-1, 1, 3)), "kind": case["kind"], "params": p}
    surf = _surface(case)
    if op == "field":
        sig = _zonal(_harmonics(case, rng), surf.xyz).cpu().numpy()
        d = _directions(rng, case["ntarg"])
        targs = d * rng.uniform(1.05, 4.0, (case["ntarg"], 1))
        return {"op": op, "surf": surf, "kind": case["kind"], "params": p, "sigma": sig,
                "targs": np.ascontiguousarray(targs)}
    st = S.setup(surf, case["kind"], EPS, p)
    plan = Plan(case["kind"], p, surf, st.near, st.over)
    if op == "matvec":
        return {"op": op, "plan": plan, "x": _zonal(_harmonics(case, rng), surf.xyz).contiguous(),
                "iprec": case["iprec"]}
    return {"op": op, "plan": plan, "rhs": _rhs(case, surf, rng), "mode": case["mode"]}


def run(state):
    op = state["op"]
    if op == "solve":
        return state["plan"].solve(state["rhs"], 0.5, mode=state["mode"], numit=NUMIT, eps_gmres=TOL)[0]
    if op == "matvec":
        return state["plan"].matvec(state["x"], state["iprec"])
    if op == "batch":
        return state["batch"].solve(state["rhs"], mode=1, numit=NUMIT, eps_gmres=TOL)[0]
    if op == "setup":
        st = S.setup(state["surf"], state["kind"], EPS, state["params"])
        return {"row_ptr": st.near.row_ptr, "col_ind": st.near.col_ind, "iquad": st.near.iquad,
                "wnear": st.near.wnear, "novers": st.over.novers, "srcover": st.over.srcover,
                "wover": st.over.wover}
    fn = layer.lap_comb_dir_eval if state["kind"] == 0 else layer.helm_comb_dir_eval
    return fn(state["surf"], state["targs"], None, None, EPS, state["params"], state["sigma"])


def _npts(case):
    per = (case["norder"] + 1) ** 2
    return per * (case["m"] * case["m2"] if case["shape"] == "torus" else 6 * case["m"] ** 2)


def work(case):
    """Bytes and operations that the path cannot do without: the densities
    and potentials, the near quadrature and one kernel evaluation per
    (target, oversampled node) pair of each operator application, up to the
    size where a hierarchical method evaluates fewer.  An oversampled surface
    is taken as twice its nodes and a node's near field as 16 patches."""
    n = _npts(case)
    c = 2 if case["kind"] == 1 else 1
    nd = case.get("nd", 1)
    per = (26 + 16 * nd) if case["kind"] == 1 else (15 + 4 * nd)
    near = 16 * n * (case["norder"] + 1) ** 2

    def matvec(nt, ns):
        return min(nt * ns, 4000.0 * (nt + ns)) * per

    op = case["op"]
    if op == "matvec":
        return {"bytes": 8 * c * (2 * n + near), "flops": matvec(n, 2 * n)}
    if op == "solve":
        it = 10 if case["kind"] == 0 else 16
        return {"bytes": it * (8 * c * 2 * n * nd + 4 * c * near), "flops": it * matvec(n, 2 * n)}
    if op == "batch":
        n = 0.55 * n
        return {"bytes": 10 * case["nsurf"] * (8 * c * 2 * n * nd + 2 * c * near),
                "flops": 10 * case["nsurf"] * matvec(n, 2 * n)}
    if op == "setup":
        # about 80 triangles of 64 nodes per near pair at 60 operations each
        return {"bytes": 8.0 * (c * near + 24 * n), "flops": 16.0 * n * 80 * 64 * 60}
    nt = case["ntarg"]
    return {"bytes": 8.0 * (21 * n + 3 * nt + c * (n + nt)),
            "flops": matvec(nt, 2 * n) + 4.0 * nt * 80 * 64 * 60}


def exact(case, seed):
    """Closed form on the sphere: the operator multiplies a degree-l harmonic
    by a number.  None elsewhere."""
    if case["shape"] != "sphere" or case["op"] not in ("solve", "matvec", "field"):
        return None
    rng = np.random.default_rng(seed)
    if case["op"] == "field":
        harm = _harmonics(case, rng)
        d = _directions(rng, case["ntarg"])
        targs = d * rng.uniform(1.05, 4.0, (case["ntarg"], 1))
        return _zonal(harm, targs, lambda l, r: _outside(case, l, r)).cpu().numpy()
    nodes = torch.as_tensor(_sphere_nodes(case), device="cuda")
    if case["op"] == "matvec":
        return _zonal(_harmonics(case, rng), nodes, lambda l, r: _eigenvalue(case, l)).contiguous()
    # the data's expansion in zonal harmonics, each over its eigenvalue
    nd, k = case.get("nd", 1), case.get("k", 0.0)
    if case["rhs"] == "waves":
        src = _directions(rng, nd)
        r0 = np.ones(nd)
    else:
        src = _sources(case, rng, nd)
        r0 = np.linalg.norm(src, axis=1)
    cols = []
    for d, r in zip(src, r0):
        t = nodes @ torch.tensor(d / r, device="cuda")
        x = 0
        for l, pl in enumerate(_legendre(TERMS, t)):
            if case["rhs"] == "waves":
                a = -(1j ** l) * (2 * l + 1) * _bessel(l, k)[0]
            elif case["kind"] == 1:
                j, y, _, _ = _bessel(l, k)
                a = 1j * k / (4 * math.pi) * (2 * l + 1) * _bessel(l, k * r)[0] * (j + 1j * y)
            else:
                a = r ** l / (4 * math.pi)
            x = x + a / (0.5 + _eigenvalue(case, l)) * pl
        cols.append(x)
    x = torch.stack(cols, 1)
    return x if nd > 1 else x[:, 0].contiguous()
