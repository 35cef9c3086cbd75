"""Performance cases: the work a program has this library do.

A case is a dict of plain values; ``prepare`` makes its inputs from a seed
(and the plan a program would keep), ``run`` is one pass through the public
entry points, ``work`` what such a pass cannot do without and ``exact`` the
same outputs from direct sums in 64 bits.  Kinds:

  tria     elfmm3dtriatarg, host arrays in and out (the drop-in call: tree,
           lists, evaluation and both copies in one call)
  total    elhfmm3dtria_total, host arrays (half space: direct arrival plus
           image part)
  part     elfmm3dparttarg, host arrays (point forces and jumps)
  plan     Plan.evaluate on a resident geometry, FP64, one right-hand side
  moving   Plan.set_geometry + Plan.evaluate each pass (geometry that changes
           between passes), resident arrays
  replay   half-space iterative solver: Plan.evaluate and
           Plan.evaluate_image on the stored near fields, FP64, one
           right-hand side
  batch    Plan.evaluate_batch with the analytic near field, several
           right-hand sides, FP64 (precision 0) or mixed (1)
  hsbatch  half-space batch on the stored near fields, both passes replayed
           as CUDA graphs
  forest   Forest.evaluate, many uneven half-space problems in one pass

Surfaces: "sphere" the refined icosahedron cut to its first n triangles,
"fault" a rectangular plane of right triangles dipping 45 degrees.
"""
import functools
import math

import numpy as np
import torch

import elfmmlib3d_b200 as E
from elfmmlib3d_b200 import geometry as G
from elfmmlib3d_b200.batch import fault_problem

LAM, MU = 1.2, 0.9
HALF_SPACE = ("total", "replay", "hsbatch", "forest")


def _case(kind, n, m=0, iprec=2, sl=True, dl=True, strain=True, nrhs=1, precision=0, surface="sphere", **more):
    return dict(kind=kind, surface=surface, n=n, m=m, iprec=iprec, sl=sl, dl=dl, strain=strain, nrhs=nrhs,
                precision=precision, **more)


def listed():
    return [
        # a call on a mesh of a few hundred triangles: launches, allocations and host work
        dict(_case("tria", 317, 41), name="tria-317"),
        # the free-space configuration (sphere refined 4 times, 1,000 targets) through the drop-in call
        dict(_case("tria", 5120, 1000), name="tria-5120"),
        # half-space forward model: slip on a small fault seen at itself and at a station grid
        dict(_case("total", 1702, 301, sl=False, surface="fault"), name="total-1702"),
        # particle sources and targets, drop-in call
        dict(_case("part", 20011, 5003), name="part-20011"),
        # coarse displacement-only evaluation of a single layer while the mesh moves
        dict(_case("moving", 20480, 0, iprec=1, dl=False, strain=False), name="moving-20480"),
        # one right-hand side on a large resident mesh with off-surface targets
        dict(_case("plan", 327680, 250007), name="plan-327680"),
        # one solver iteration on a half-space fault (both stored near fields replayed)
        dict(_case("replay", 49950, 0, sl=False, surface="fault"), name="replay-49950"),
        # several load cases on one mesh at once, both layers, plain FP64
        dict(_case("batch", 9973, 2003, nrhs=16), name="batch16-9973"),
        # the mixed-precision form on a large mesh, one right-hand side
        dict(_case("batch", 81920, 62501, precision=1), name="mixed-81920"),
        # 64 slip vectors of a half-space fault, mixed precision, CUDA graphs (the library's headline use)
        dict(_case("hsbatch", 18034, 0, iprec=3, sl=False, nrhs=64, precision=1, surface="fault"), name="hsbatch64-18034"),
        # a catalogue of uneven faults in one pass, mixed precision
        dict(_case("forest", 4001, 0, sl=False, precision=1, surface="fault", nprob=24, nmin=300), name="forest-24"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["tria", "tria", "total", "part", "moving", "plan", "replay", "batch", "batch", "hsbatch", "forest"])
    sl, dl = rng.choice([(True, True), (True, False), (False, True)])
    strain, iprec = rng.random() < 0.75, rng.choice([1, 2, 2, 3])
    if kind == "tria":
        return _case(kind, size(100, 40000), size(10, 10000) if rng.random() < 0.7 else 0, iprec, sl, dl, strain)
    if kind == "part":
        return _case(kind, size(1000, 40000), size(100, 10000) if rng.random() < 0.7 else 0, iprec, sl, dl, strain)
    if kind == "total":
        return _case(kind, size(200, 4000), size(20, 500), rng.choice([1, 2]), sl, dl, strain, surface="fault")
    if kind == "moving":
        return _case(kind, size(2000, 40000), size(10, 10000) if rng.random() < 0.5 else 0, iprec, sl, dl, strain)
    if kind == "plan":
        return _case(kind, size(2000, 200000), size(100, 100000), rng.choice([1, 2]), sl, dl, strain,
                     surface=rng.choice(["sphere", "fault"]))
    if kind == "replay":
        return _case(kind, size(2000, 40000), 0, rng.choice([1, 2]), False, True, strain, surface="fault")
    if kind == "batch":
        return _case(kind, size(1000, 15000), size(100, 5000) if rng.random() < 0.5 else 0, rng.choice([1, 2]), sl, dl,
                     strain, rng.choice([3, 8, 16, 24]), rng.choice([0, 1]))
    if kind == "hsbatch":
        return _case(kind, size(2000, 15000), 0, rng.choice([2, 3]), False, True, True, rng.choice([9, 16, 40, 64]), 1,
                     surface="fault")
    return _case(kind, size(800, 4000), 0, 2, False, True, True, 1, rng.choice([0, 1]), surface="fault",
                 nprob=rng.randint(3, 24), nmin=300)


# ---- inputs -----------------------------------------------------------------

@functools.lru_cache(maxsize=4)
def _sphere(level):
    return G.sphere_triangles(level)


def _fault_cells(n):
    """Cells (along strike, down dip) of a 2 : 1 fault of about n triangles."""
    nw = max(1, round(math.sqrt(n / 4.0)))
    return max(1, round(n / (2.0 * nw))), nw


def _counts(case):
    rng = np.random.default_rng(case["n"] * 1000 + case["nprob"])  # sizes belong to the case, not to the seed
    return [int(round(c)) for c in np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["n"]), case["nprob"]))]


def _rotation(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    return q * np.sign(np.diag(r)) * np.linalg.det(q * np.sign(np.diag(r)))


def _inputs(case, seed):
    """Host arrays: geometry (tri, nrm, cen), targets, densities (nrhs,n,3) or None."""
    rng = np.random.default_rng(seed)
    kind, n, m, counts = case["kind"], case["n"], case["m"], None
    tgt = np.zeros((0, 3))
    if kind == "part":
        cen, nrm, tri = rng.uniform(-1, 1, (n, 3)), rng.normal(size=(n, 3)), None
        nrm /= np.linalg.norm(nrm, axis=1)[:, None]
        tgt = rng.uniform(-1.2, 1.2, (m, 3))
    elif kind == "forest":
        probs = [fault_problem(c, rng.uniform(0, 360), rng.uniform(15, 90), rng.uniform(0.5, 5), 0)
                 for c in _counts(case)]
        counts = [len(p[2]) for p in probs]
        tri, nrm, cen = (np.concatenate([p[k] for p in probs]) for k in range(3))
    elif case["surface"] == "fault":
        tri, nrm, cen, _ = G.planar_fault(*_fault_cells(n), strike_deg=rng.uniform(0, 360), top_depth=rng.uniform(1, 3))
        tgt = np.stack([rng.uniform(-25, 25, m), rng.uniform(-25, 25, m), -rng.uniform(0, 1, m) ** 2 * 20 - 0.01], axis=1)
    else:
        level = next(k for k in range(12) if 20 * 4 ** k >= n)
        tri, nrm, cen = (a[:n] for a in _sphere(level))
        q = _rotation(rng)
        tri, nrm, cen = (np.ascontiguousarray(a @ q) for a in (tri, nrm, cen))
        tgt = G.shell_targets(m, seed) if m else tgt
    s = (case["nrhs"], len(cen), 3)
    ssl = rng.normal(size=s) if case["sl"] else None
    sdl = rng.normal(size=s) if case["dl"] else None
    return tri, nrm, cen, tgt, ssl, sdl, counts


def _dev(a):
    return None if a is None else torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def prepare(case, seed):
    tri, nrm, cen, tgt, ssl, sdl, counts = _inputs(case, seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("tria", "total", "part"):
        return dict(s, tri=tri, nrm=nrm, cen=cen, tgt=tgt if case["m"] else None,
                    ssl=None if ssl is None else ssl[0], sdl=None if sdl is None else sdl[0])
    R, n, m = case["nrhs"], len(cen), case["m"]
    lead = () if kind in ("plan", "moving", "replay", "forest") else (R,)
    z = lambda *shape: torch.zeros(lead + shape, dtype=torch.float64, device="cuda")  # noqa: E731
    if not lead:
        ssl, sdl = (None if a is None else a[0] for a in (ssl, sdl))
    s.update(tri=_dev(tri), nrm=_dev(nrm), cen=_dev(cen), ssl=_dev(ssl), sdl=_dev(sdl), tgt=_dev(tgt) if m else None)
    s.update(u=z(n, 3), e=z(n, 3, 3) if case["strain"] else None)
    s.update(ut=z(m, 3) if m else None, et=z(m, 3, 3) if m and case["strain"] else None)
    torch.cuda.synchronize()
    if kind == "forest":
        s["forest"] = E.Forest(0)
        s["forest"].set_geometry(counts, s["tri"], s["nrm"], s["cen"], iprec=case["iprec"])
        return s
    s["plan"] = E.Plan(0)
    store = kind in ("replay", "hsbatch")
    if kind != "moving":
        s["plan"].set_geometry(s["tri"], s["nrm"], s["cen"], s["tgt"], iprec=case["iprec"], iter=store)
    if store:
        s.update(ui=z(n, 3), ei=z(n, 3, 3) if case["strain"] else None, refl=_dev(cen * np.array([1.0, 1.0, -1.0])))
        torch.cuda.synchronize()
        s["image"] = E.Plan(0)
        s["image"].set_geometry(s["tri"], s["nrm"], s["cen"], s["refl"], iprec=case["iprec"], iter=True, mindlin=True)
        if kind == "replay":
            s["plan"].evaluate(LAM, MU, s["ssl"], s["sdl"], s["u"], s["e"], mode=1)
        else:
            s["plan"].evaluate_batch(LAM, MU, R, s["ssl"], s["sdl"], s["u"], s["e"], precision=case["precision"], mode=1)
        s["image"].evaluate_image(LAM, MU, R, s["ssl"], s["sdl"], s["ui"], s["ei"], precision=case["precision"], mode=1)
    return s


# ---- one pass ---------------------------------------------------------------

def run(s):
    case = s["case"]
    kind, iprec, R, prec, e1 = case["kind"], case["iprec"], case["nrhs"], case["precision"], int(case["strain"])
    if kind == "part":
        ier, u, e, ut, et = E.elfmm3dparttarg(iprec, LAM, MU, s["cen"], s["ssl"], s["sdl"], s["nrm"], s["tgt"],
                                              ifstrain=e1, ifstraintarg=e1)
    elif kind in ("tria", "total"):
        f = E.elfmm3dtriatarg if kind == "tria" else E.elhfmm3dtria_total
        ier, u, e, ut, et = f(iprec, LAM, MU, s["tri"], s["nrm"], s["cen"], s["ssl"], s["sdl"], s["tgt"],
                              ifstrain=e1, ifstraintarg=e1)
    if kind in ("tria", "total", "part"):
        if ier:
            raise RuntimeError("ier %d" % ier)
        out = dict(u=u, ut=ut, e=e, et=et)
        return {k: v for k, v in out.items() if v.size and (e1 or k in ("u", "ut"))}
    dens, outs = (s["ssl"], s["sdl"]), (s["u"], s["e"], s["ut"], s["et"])
    if kind == "forest":
        s["forest"].evaluate(LAM, MU, *dens, s["u"], s["e"], precision=prec)
    elif kind == "plan":
        s["plan"].evaluate(LAM, MU, *dens, *outs)
    elif kind == "moving":
        s["plan"].set_geometry(s["tri"], s["nrm"], s["cen"], s["tgt"], iprec=iprec)
        s["plan"].evaluate(LAM, MU, *dens, *outs)
    elif kind == "batch":
        s["plan"].evaluate_batch(LAM, MU, R, *dens, *outs, precision=prec)
    elif kind == "replay":
        s["plan"].evaluate(LAM, MU, *dens, s["u"], s["e"], mode=2)
        s["image"].evaluate_image(LAM, MU, 1, *dens, s["ui"], s["ei"], mode=2)
    else:
        s["plan"].evaluate_batch(LAM, MU, R, *dens, s["u"], s["e"], precision=prec, mode=2, graph=True)
        s["image"].evaluate_image(LAM, MU, R, *dens, s["ui"], s["ei"], precision=prec, mode=2, graph=True)
    return {k: s[k] for k in ("u", "ut", "e", "et", "ui", "ei") if s.get(k) is not None}


def work(case):
    """Bytes: geometry and densities read, outputs written (and, on a stored
    near field, its blocks read).  Flops: the terms every such FMM has on a
    surface, at the order and leaf size of iprec: near pairs (9 of the 27
    neighbour leaves hold points) applied to the densities, harmonics of 12
    nodes (1 for a particle) and of every point, and rotated translations."""
    kind, m, R, iprec = case["kind"], case["m"], case["nrhs"], case["iprec"]
    n = case["n"] * case.get("nprob", 1) * (0.5 if kind == "forest" else 1)
    p, leaf = {1: (14, 20), 2: (26, 40), 3: (39, 80)}[iprec]
    store = kind in ("replay", "hsbatch")
    leaf *= 6 if store else 1
    layers, out, pts = case["sl"] + case["dl"], 3 + 9 * case["strain"], n + m
    pairs = pts * min(n, 9 * leaf / 2)
    one = 8 * ((12 + 3 * (kind != "part")) * n + 3 * m)
    data = 8 * R * (3 * layers * n + out * pts)
    blocks = pairs * 3 * layers * (3 + 6 * case["strain"])
    passes = 2 if kind in HALF_SPACE else 1
    boxes = (1.33 * 2 * pts / leaf) if n > leaf else 0
    cols = 4 * R
    far = cols * (p + 1) ** 2 * (n * 2 * (1 if kind == "part" else 12) + pts * 2 * 9) + cols * boxes * 30 * 4 * (p + 1) ** 3 / 3
    near = 2 * blocks * R + (0 if store else 500 * pairs)
    return {"bytes": one + data * (2 if store else 1) + (8 * blocks if store else 0), "flops": near + passes * (far if boxes else 0)}


# ---- the same outputs in 64 bits --------------------------------------------

def _sym(*idx):
    return tuple(sorted(idx))


def _edge_tables(x, a, b, nu, order):
    """Derivatives (up to `order` <= 3, at the target x) of the integral of
    r = |x - y| over the edge a-b, in the frame (tangent, in-plane normal nu,
    triangle normal): {index: value}, and the integral of 1/r.  x, a, b: the
    triangle frame's coordinates, x (P,T,3), a, b (T,2)."""
    d = b - a
    length = d.norm(dim=-1)
    t = d / length[:, None]
    rx, ry, h = x[..., 0] - a[:, 0], x[..., 1] - a[:, 1], x[..., 2]
    v = rx * nu[:, 0] + ry * nu[:, 1]
    u0 = -(rx * t[:, 0] + ry * t[:, 1])
    u1 = u0 + length
    q2 = v * v + h * h
    r0, r1 = (u0 * u0 + q2).sqrt(), (u1 * u1 + q2).sqrt()
    flip = u1 <= 0  # mirror the edge so that both ends lie at u >= 0 where they share a sign
    s0, s1 = torch.where(flip, -u1, u0), torch.where(flip, -u0, u1)
    f0, f1 = torch.where(flip, r1, r0), torch.where(flip, r0, r1)
    inside = s0 < 0
    q2s = torch.where(inside, q2, torch.ones_like(q2))
    log = torch.log(torch.where(inside, (s1 + f1) * (f0 - s0) / q2s, (s1 + f1) / (f0 + s0).clamp_min(1e-300)))
    g0, g1 = 1 / (f0 * (f0 + s0)), 1 / (f1 * (f1 + s1))
    w0, w1 = s0 / f0, s1 / f1
    K3 = torch.where(inside, (w1 - w0) / q2s, g0 - g1)
    c = lambda w: w - w ** 3 / 3  # noqa: E731
    K5 = torch.where(inside, (c(w1) - c(w0)) / (q2s * q2s), (g0 * g0 - g1 * g1) - q2 * (g0 ** 3 - g1 ** 3) / 3)
    # I[n][k] = integral of (-u)^k / r^n
    I1 = [log, -(r1 - r0)]
    I3 = [K3, 1 / r1 - 1 / r0, log - q2 * K3]
    J3 = 1 / (3 * r1 ** 3) - 1 / (3 * r0 ** 3)
    I5 = [K5, J3, K3 - q2 * K5, I3[1] - q2 * J3]
    const = {0: None, 1: v, 2: h}

    def mono(tab, idx):
        k, val = sum(i == 0 for i in idx), 1.0
        for i in idx:
            if i:
                val = val * const[i]
        return tab[k] * val

    T = {(i,): mono(I1, (i,)) for i in range(3)}
    if order >= 2:
        for i in range(3):
            for j in range(i, 3):
                T[(i, j)] = (I1[0] if i == j else 0) - mono(I3, (i, j))
    if order >= 3:
        for i in range(3):
            for j in range(i, 3):
                for k in range(j, 3):
                    val = 3 * mono(I5, (i, j, k))
                    for p, q, o in ((i, j, k), (i, k, j), (j, k, i)):
                        if p == q:
                            val = val - mono(I3, (o,))
                    T[(i, j, k)] = val
    return T, log, v, t


def _triangle_tables(x, xy, order):
    """Target derivatives of orders 2..order (<= 4) of the integral of r over
    the triangles, and of orders 0..order-2 of that of 1/r, in the triangle
    frames: x (P,T,3), xy (T,3,2).  Every derivative with an in-plane index
    goes to the edges; the normal ones follow from laplacian r = 2/r."""
    S, N0, L2 = {}, 0, xy[:, 1, 0]
    for e in range(3):
        a, b = xy[:, e], xy[:, (e + 1) % 3]
        d = b - a
        nu = torch.stack([d[:, 1], -d[:, 0]], dim=-1) / d.norm(dim=-1, keepdim=True)
        T, log, v, t = _edge_tables(x, a, b, nu, order - 1)
        N0 = N0 - v * log
        # frame (tangent, nu, z) -> triangle frame: axis 0, 1 components of each
        ax = [(t[:, 0], nu[:, 0]), (t[:, 1], nu[:, 1])]

        def rot(idx, done=()):
            if not idx:
                return T[_sym(*done)]
            if idx[0] == 2:
                return rot(idx[1:], done + (2,))
            ct, cn = ax[idx[0]]
            return ct * rot(idx[1:], done + (0,)) + cn * rot(idx[1:], done + (1,))

        for k in range(1, order):
            for J in [j for j in _indices(k)]:
                val = rot(J)
                for al in range(2):
                    if J and al <= J[0]:  # one in-plane index taken off: the smallest
                        S[(al,) + J] = S.get((al,) + J, 0) - nu[:, al] * val
    # signed solid angle (Van Oosterom and Strackee), 0 in the plane
    r = [torch.stack([xy[:, k, 0] - x[..., 0], xy[:, k, 1] - x[..., 1], -x[..., 2]], dim=-1) for k in range(3)]
    l = [q.norm(dim=-1) for q in r]  # noqa: E741
    det = (r[0] * torch.linalg.cross(r[1], r[2])).sum(-1)
    den = l[0] * l[1] * l[2] + (r[0] * r[1]).sum(-1) * l[2] + (r[0] * r[2]).sum(-1) * l[1] + (r[1] * r[2]).sum(-1) * l[0]
    h = x[..., 2]
    om = 2 * torch.atan2(det.abs(), den)
    om = torch.where(h.abs() < 1e-11 * L2, torch.zeros_like(om), om) * torch.sign(h)
    N = {(): N0 - h * om}
    S[(2, 2)] = 2 * N[()] - S[(0, 0)] - S[(1, 1)]
    if order >= 3:
        for i in range(2):
            N[(i,)] = None
        N[(2,)] = -om
        S[(2, 2, 2)] = 2 * N[(2,)] - S[(0, 0, 2)] - S[(1, 1, 2)]
        for i in range(2):
            N[(i,)] = sum(S[_sym(i, k, k)] for k in range(3)) / 2
    if order >= 4:
        for i in range(3):
            for j in range(i, 3):
                if (i, j) != (2, 2):
                    N[(i, j)] = sum(S[_sym(i, j, k, k)] for k in range(3)) / 2
        N[(2, 2)] = -N[(0, 0)] - N[(1, 1)]
        S[(2, 2, 2, 2)] = 2 * N[(2, 2)] - S[(0, 0, 2, 2)] - S[(1, 1, 2, 2)]
    return S, N


def _indices(k):
    if k == 0:
        return [()]
    return [(i,) + J for i in range(3) for J in _indices(k - 1) if not J or i <= J[0]]


def _free_triangles(tri, ssl, sdl, x, strain):
    """Kelvin layers by the closed forms above: u (R,P,3), e (R,P,3,3)."""
    R = (ssl if ssl is not None else sdl).shape[0]
    P, n = len(x), len(tri)
    al = (LAM + MU) / (LAM + 2 * MU)
    e1 = tri[:, 1] - tri[:, 0]
    e1 = e1 / e1.norm(dim=1, keepdim=True)
    e3 = torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    e3 = e3 / e3.norm(dim=1, keepdim=True)
    Q = torch.stack([e1, torch.linalg.cross(e3, e1), e3], dim=1)  # rows: local axes
    xy = torch.einsum("tij,tvj->tvi", Q, tri - tri[:, :1])[..., :2].contiguous()
    loc = [None if s is None else torch.einsum("tij,rtj->rti", Q, s) for s in (ssl, sdl)]
    u = torch.zeros(R, P, 3, dtype=torch.float64, device=x.device)
    e = torch.zeros(R, P, 3, 3, dtype=torch.float64, device=x.device)
    step = max(1, 600000 // n)
    for i0 in range(0, P, step):
        rel = x[i0:i0 + step, None, :] - tri[None, :, 0]
        y = torch.einsum("tij,ptj->pti", Q, rel)
        S, N = _triangle_tables(y, xy, 2 + (sdl is not None) + strain)
        ul = torch.zeros(R, *y.shape, dtype=torch.float64, device=x.device)
        gl = torch.zeros(R, *y.shape, 3, dtype=torch.float64, device=x.device) if strain else None

        def add(coef, k, l, J):  # noqa: E741
            """coef (R,T) times (2 delta_ik N_l - al S_ikl) / 2 mu and its gradient, for every i."""
            c = coef[:, None, :] / (2 * MU)
            for i in range(3):
                val = -al * S[_sym(i, k, *l)]
                if i == k:
                    val = val + 2 * N[_sym(*l)]
                ul[..., i] += c * val
                for j in range(3 if strain else 0):
                    val = -al * S[_sym(i, k, j, *l)]
                    if i == k:
                        val = val + 2 * N[_sym(j, *l)]
                    gl[..., i, j] += c * val

        if loc[0] is not None:
            for k in range(3):
                add(loc[0][:, :, k], k, (), None)
        if loc[1] is not None:
            b = loc[1]  # jump; C contracted with the normal (0, 0, 1)
            for k in range(3):
                for l in range(3):  # noqa: E741
                    M = (LAM * b[:, :, 2] if k == l else 0) + (MU * b[:, :, k] if l == 2 else 0) + (MU * b[:, :, l] if k == 2 else 0)
                    if torch.is_tensor(M):
                        add(-M, k, (l,), None)
        u[:, i0:i0 + step] = torch.einsum("tij,rpti->rpj", Q, ul)
        if strain:
            g = torch.einsum("tia,rptij,tjb->rpab", Q, gl, Q)
            e[:, i0:i0 + step] = (g + g.transpose(-1, -2)) / 2
    return u, e


def _image_force(x, s):
    """Image displacement at x of unit forces at s, components first: G[k][i]
    (Mindlin's solution minus Kelvin's, no 1/(4 pi))."""
    al = (LAM + MU) / (LAM + 2 * MU)
    R = [x[0] - s[0], x[1] - s[1], -x[2] - s[2]]
    r = torch.sqrt(R[0] * R[0] + R[1] * R[1] + R[2] * R[2])
    i1, w = 1 / r, 1 / (r + R[2])
    i3 = i1 * i1 * i1
    U = {(2, 2): i1, (0, 2): R[0] * i1 * w, (1, 2): R[1] * i1 * w, (0, 1): R[0] * R[1] * i1 * w * w}
    U[(0, 0)], U[(1, 1)] = R[0] * R[0] * i1 * w * w - w, R[1] * R[1] * i1 * w * w - w
    V2 = {_sym(i, j): 3 * R[i] * R[j] * i3 * i1 * i1 - (i3 if i == j else 0) for i in range(3) for j in range(3)}
    h, sc = -s[2], (1 - al) / al
    G = []
    for k in range(3):
        sign = 1.0 if k == 2 else -1.0
        row = []
        for i in range(3):
            val = (al * i1 if i == k else 0) + (2 - al) * R[k] * R[i] * i3
            val = val / (2 * MU) + sc * sign * U[_sym(i, k)] / MU
            P = h * al * V2[_sym(i, k)]
            if k == 2 and i < 2:
                P = P + (2 - al) * R[i] * i3
            if i == 2:
                P = -P
                if k < 2:
                    P = P + (2 - al) * R[k] * i3
            row.append(val + x[2] * P / MU)
        G.append(row)
    return G


def _image_triangles(tri, nrm, ssl, sdl, x, strain):
    """Image part by a tensor Gauss rule on every triangle: u (P,3), e (P,3,3)."""
    q = 8
    g, w = np.polynomial.legendre.leggauss(q)
    a, b = np.meshgrid((g + 1) / 2, (g + 1) / 2, indexing="ij")
    wt = torch.tensor((np.outer(w, w) / 4 * a).ravel(), device=x.device)
    a, b = (torch.tensor(t.ravel(), device=x.device)[None, :, None] for t in (a, b))
    e1, e2 = (tri[:, k] - tri[:, 0] for k in (1, 2))
    nodes = (tri[:, None, 0] + a * (1 - b) * e1[:, None] + a * b * e2[:, None]).reshape(-1, 3)
    area2 = torch.linalg.cross(e1, e2).norm(dim=1)
    wts = (area2[:, None] * wt).reshape(-1)
    rep = lambda s: s.repeat_interleave(q * q, dim=0)  # noqa: E731
    C = rep(sdl.new_zeros(len(tri), 3) if ssl is None else ssl)
    M = None
    if sdl is not None:
        bn = sdl[:, :, None] * nrm[:, None, :]
        M = rep(LAM * (sdl * nrm).sum(-1)[:, None, None] * torch.eye(3, dtype=x.dtype, device=x.device) + MU * (bn + bn.transpose(1, 2)))
    u, e = torch.zeros_like(x), torch.zeros(len(x), 3, 3, dtype=x.dtype, device=x.device)
    step = max(1, 4000000 // len(nodes))
    jvp = torch.func.jvp
    for i0 in range(0, len(x), step):
        X = x[i0:i0 + step]
        xs = tuple(X[:, None, c].expand(-1, len(nodes)).contiguous() for c in range(3))
        ss = tuple(nodes[None, :, c].expand(len(X), -1).contiguous() for c in range(3))
        zero, one = torch.zeros_like(xs[0]), torch.ones_like(xs[0])

        def field(*xx):
            out = [zero, zero, zero]
            if ssl is not None:
                Gk = _image_force(xx, ss)
                out = [sum(C[:, k] * Gk[k][i] for k in range(3)) for i in range(3)]
            if M is not None:
                for k in range(3):
                    tang = tuple(M[None, :, k, l].expand_as(zero) for l in range(3))  # noqa: E741
                    d = jvp(lambda *s: tuple(_image_force(xx, s)[k]), ss, tang)[1]
                    out = [o + t for o, t in zip(out, d)]
            return tuple(out)

        if not strain:
            val = field(*xs)
        for j in range(3 if strain else 0):
            val, g = jvp(field, xs, tuple(one if c == j else zero for c in range(3)))
            for i in range(3):
                t = (g[i] * wts).sum(1) / 2
                e[i0:i0 + step, i, j] += t
                e[i0:i0 + step, j, i] += t
        for i in range(3):
            u[i0:i0 + step, i] = (val[i] * wts).sum(1)
    return u, e


def _particles(y, ssl, sdl, nu, x, same, strain):
    """Kelvin point forces and jumps, pair by pair: u (P,3), e (P,3,3)."""
    al = (LAM + MU) / (LAM + 2 * MU)
    eye = torch.eye(3, dtype=x.dtype, device=x.device)
    f = torch.zeros_like(y) if ssl is None else ssl
    M = torch.zeros(len(y), 3, 3, dtype=x.dtype, device=x.device)
    if sdl is not None:
        bn = sdl[:, :, None] * nu[:, None, :]
        M = LAM * (sdl * nu).sum(-1)[:, None, None] * eye + MU * (bn + bn.transpose(1, 2))
    trM = M.diagonal(dim1=1, dim2=2).sum(-1)[:, None]
    u, e = torch.zeros_like(x), torch.zeros(len(x), 3, 3, dtype=x.dtype, device=x.device)
    step = max(1, 4000000 // len(y))
    for i0 in range(0, len(x), step):
        d = x[i0:i0 + step, None] - y[None]
        r2 = (d * d).sum(-1)
        if same:
            r2[torch.arange(len(d)), torch.arange(i0, i0 + len(d))] = math.inf
        i2 = (1 / r2)[..., None]
        i1 = i2.sqrt()
        i3, i5 = i1 * i2, i1 * i2 * i2
        df = (d * f).sum(-1, keepdim=True)
        Md = torch.einsum("nij,pnj->pni", M, d)
        dMd = (d * Md).sum(-1, keepdim=True)
        # G_ik = ((2 - al) delta_ik / r + al d_i d_k / r^3) / 2 mu; jumps: -M_kl d_l G_ik
        val = (2 - al) * f * i1 + al * df * d * i3
        val = val + (2 - al) * Md * i3 - al * (trM * d + Md) * i3 + 3 * al * dMd * d * i5
        u[i0:i0 + step] = val.sum(1) / (2 * MU)
        if strain:
            i7 = i5 * i2
            dd = d[..., :, None] * d[..., None, :]
            k = lambda t: t[..., None]  # noqa: E731
            fd, Mdd = f[None, :, :, None] * d[..., None, :], Md[..., :, None] * d[..., None, :]
            g = -(2 - al) * fd * k(i3) + al * (k(df) * eye * k(i3) + d[..., :, None] * f[None, :, None, :] * k(i3) - 3 * k(df) * dd * k(i5))
            g = g + (2 - 2 * al) * (M * k(i3) - 3 * Mdd * k(i5)) - al * k(trM) * (eye * k(i3) - 3 * dd * k(i5))
            g = g + 3 * al * (2 * d[..., :, None] * Md[..., None, :] * k(i5) + k(dMd) * eye * k(i5) - 5 * k(dMd) * dd * k(i7))
            g = g.sum(1) / (2 * MU)
            e[i0:i0 + step] = (g + g.transpose(1, 2)) / 2
    return u, e


def exact(case, seed):
    """Direct sums over all pairs; None where they would take too long."""
    kind = case["kind"]
    pairs = (case["n"] + case["m"]) * case["n"]
    most = 4e6 if kind == "total" else 0 if kind in HALF_SPACE else 1e9 if kind == "part" else 7e8 / (1 + case["nrhs"] / 4)
    if pairs > most:
        return None
    tri, nrm, cen, tgt, ssl, sdl, _ = _inputs(case, seed)
    tri, nrm, cen, tgt, ssl, sdl = (_dev(a) for a in (tri, nrm, cen, tgt, ssl, sdl))
    strain, out = case["strain"], {}
    for name, x in (("", cen), ("t", tgt)):
        if not len(x):
            continue
        if kind == "part":
            u, e = _particles(cen, *(None if a is None else a[0] for a in (ssl, sdl)), nrm, x, not name, strain)
        else:
            u, e = _free_triangles(tri, ssl, sdl, x, strain)
            if kind not in ("batch",):
                u, e = u[0], e[0]
            if kind == "total":
                ui, ei = _image_triangles(tri, nrm, *(None if a is None else a[0] for a in (ssl, sdl)), x, strain)
                u, e = u + ui, e + ei
        out["u" + name] = u
        if strain:
            out["e" + name] = e
    if kind in ("tria", "total", "part"):
        out = {k: v.cpu().numpy() for k, v in out.items()}
    return out
