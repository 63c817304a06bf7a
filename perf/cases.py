"""What a SIMCOFlow time step asks of this library, as measurable cases.

A case is one call (or one stage/run/fetch sequence) of a public entry point:

* ``projection``: the pressure projection on device-resident inputs
  (``Projection.run``), the loop of a host that keeps its fields on the GPU;
* ``update_puvw``: the same through the drop-in call on page-locked Fortran
  arrays, copies included;
* ``loss_grad``: the differentiable harness, loss and gradient of one
  projection through ``ProjectionLoss`` on host arrays;
* ``predictor``: the three implicit momentum solves (``PredictSolves.run``);
* ``geometry``: the cut-cell preprocessing of a moving solid through
  ``GridPreprocess`` on page-locked host arrays;
* ``clsvof``: one interface-transport step (``ClsvofScheme`` stage, run,
  fetch) on page-locked host arrays.

Inputs are analytic two-phase flows around a solid (the configurations of
``simcoflow3d_gb300.workloads``), generated on the GPU; the seed moves the
interface and the solid a little and draws the velocities.  Device arrays here
are (k, j, i) tensors, the memory order of the Fortran arrays (i, j, k).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from simcoflow3d_gb300 import capi
from simcoflow3d_gb300 import geometry as GM
from simcoflow3d_gb300 import predictor as PR
from simcoflow3d_gb300 import workloads as W
from simcoflow3d_gb300.autograd import ProjectionLoss
from simcoflow3d_gb300.projection import Projection
from simcoflow3d_gb300.transport import ClsvofScheme, plane_shapes

EPSI = 1.0e-3
DT = 1.0e-3
F64 = torch.float64


def listed():
    return [
        # the smallest useful grid: a coarse trial run or one block of a
        # parameter study, where launches and latency are the cost
        dict(name="projection_small", kind="projection", scene="bubble", I=40, J=40, K=40, precision="mixed",
             rel_tol=1e-8, degree=3),
        # the 64^3 layered box at the library's default options (FP64, 1e-10)
        dict(name="projection_fp64_64", kind="projection", scene="layers", I=64, J=64, K=64, precision="fp64",
             rel_tol=1e-10, degree=3),
        # an everyday production grid with odd extents and anisotropic cells
        dict(name="projection_odd", kind="projection", scene="sphere", I=147, J=93, K=121, precision="mixed",
             rel_tol=1e-10, degree=3),
        # the benchmark configuration: sphere and gas bubble at 256^3
        dict(name="projection_256", kind="projection", scene="bubble", I=256, J=256, K=256, precision="mixed",
             rel_tol=1e-8, degree=4),
        # the wave tank: z-stretched (line smoother), open top, cylinder
        dict(name="projection_tank", kind="projection", scene="tank", I=256, J=128, K=128, precision="mixed",
             rel_tol=1e-8, degree=8),
        # the Fortran host's drop-in call at 128^3 with default options
        dict(name="update_puvw_128", kind="update_puvw", scene="sphere", I=128, J=128, K=128, precision="fp64",
             rel_tol=1e-10, degree=3),
        # gradient of the pressure force and divergence (forward and backward)
        dict(name="loss_grad_64", kind="loss_grad", scene="sphere", I=64, J=64, K=64, precision="fp64",
             rel_tol=1e-12, degree=3),
        # momentum predictor, mixed precision, even box
        dict(name="predictor_mixed", kind="predictor", I=128, J=112, K=96, precision="mixed", rel_tol=1e-10),
        # momentum predictor in FP64 on an odd box
        dict(name="predictor_fp64_odd", kind="predictor", I=67, J=53, K=75, precision="fp64", rel_tol=1e-10),
        # geometry of a moved solid
        dict(name="geometry_96", kind="geometry", I=96, J=96, K=96),
        # interface transport: the deformation test at twice the reference
        # test's resolution
        dict(name="clsvof_128", kind="clsvof", I=128, J=128, K=128),
        # interface transport on a small odd box, spacings not powers of two
        dict(name="clsvof_odd", kind="clsvof", I=57, J=43, K=51),
    ]


def draw(rng):
    kind = rng.choice(["projection"] * 5 + ["update_puvw", "loss_grad", "predictor", "predictor", "geometry",
                                            "clsvof", "clsvof"])
    fp64 = kind == "loss_grad" or (kind != "geometry" and rng.random() < 0.3)
    lo, hi = {"projection": (32, 256), "update_puvw": (32, 160), "loss_grad": (24, 72), "predictor": (32, 144),
              "geometry": (24, 112), "clsvof": (24, 128)}[kind]
    if fp64 and kind in ("projection", "update_puvw", "predictor"):
        hi = min(hi, 120)
    side = math.exp(rng.uniform(math.log(lo), math.log(hi / 1.26)))
    I, J, K = (int(min(hi, max(lo, round(side * math.exp(rng.uniform(-0.23, 0.23)))))) for _ in range(3))
    case = dict(kind=kind, I=I, J=J, K=K)
    if kind in ("projection", "update_puvw"):
        scene = rng.choice(["bubble", "layers", "sphere", "tank"])
        case.update(scene=scene, precision="fp64" if fp64 else "mixed", rel_tol=rng.choice([1e-8, 1e-10]),
                    degree=8 if scene == "tank" and not fp64 else rng.choice([2, 3, 4]))
    elif kind == "loss_grad":
        case.update(scene="sphere", precision="fp64", rel_tol=1e-12, degree=3)
    elif kind == "predictor":
        case.update(precision="fp64" if fp64 else "mixed", rel_tol=1e-10)
    return case


def work(case):
    n = case["I"] * case["J"] * case["K"]
    kind = case["kind"]
    if kind in ("projection", "update_puvw"):
        # 19 FP64 and 8 int32 arrays in, u, v, w, p out; rows and correction
        return {"bytes": n * (19 * 8 + 8 * 4 + 4 * 8), "flops": n * 150}
    if kind == "loss_grad":
        return {"bytes": n * (21 * 8 + 8 * 4 + 4 * 8), "flops": n * 300}
    if kind == "predictor":
        return {"bytes": 3 * n * (18 * 8 + 2 * 4 + 2 * 8), "flops": 3 * n * 150}
    if kind == "geometry":
        # 9 FP64 arrays in and the outputs (17 FP64, 3 int32 a cell) of the four families
        return {"bytes": 4 * n * (9 * 8 + 17 * 8 + 2 * 4), "flops": 4 * n * 150}
    return {"bytes": n * (14 * 8 + 5 * 8), "flops": 6 * n * 200}   # clsvof


# ---- analytic scenes ----------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _spacing(n, length, stretch=0.0):
    """Cell sizes; with ``stretch`` a uniform middle half and geometric sides."""
    k = np.arange(n, dtype=np.float64)
    out = (1.0 + stretch) ** np.maximum(np.abs(k - 0.5 * (n - 1)) - 0.25 * n, 0.0)
    return out * (length / out.sum())


class _Grid:
    """Centres, sizes and staggered sizes of the tensor grid of a case."""

    def __init__(self, case):
        tank = case.get("scene") == "tank"
        self.n = (case["I"], case["J"], case["K"])
        self.d, self.c, self.s = [], [], []
        for ax in range(3):
            d = _spacing(self.n[ax], 4.0 if tank and ax == 0 else 1.0, 0.02 if tank and ax == 2 else 0.0)
            c = np.cumsum(d) - 0.5 * d
            s = d.copy()
            s[:-1] = c[1:] - c[:-1]
            self.d.append(d), self.c.append(c), self.s.append(s)

    @staticmethod
    def along(a, ax):
        shape = [1, 1, 1]
        shape[2 - ax] = -1
        return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device="cuda").reshape(shape)

    def cells(self, ghost=False):
        idx = [np.clip(np.arange(m + 2) - 1, 0, m - 1) if ghost else np.arange(m) for m in self.n]
        x = [self.along(self.c[a][idx[a]], a) for a in range(3)]
        d = [self.along(self.d[a][idx[a]], a) for a in range(3)]
        return x, d

    def full(self, a, ax):
        I, J, K = self.n
        return self.along(a, ax).expand(K, J, I)


def _cut_volume(n, d, s):
    """Volume fraction of a box on the positive side of a plane (n: |normal|
    components, d: box sizes, s: distance from the box's lowest corner)."""
    a = torch.stack(torch.broadcast_tensors(*(ni.abs() * di for ni, di in zip(n, d))))
    a = torch.sort(a, 0).values
    m1, m2, m3 = a[0], a[1], a[2]
    tot = m1 + m2 + m3
    t = torch.minimum(s, tot - s).clamp(min=0.0)
    eps = 1e-9 * tot
    m1, m2 = torch.maximum(m1, eps), torch.maximum(m2, eps)
    m12 = m1 + m2
    cube = lambda q: q.clamp(min=0.0) ** 3
    poly = (cube(t) - cube(t - m1) - cube(t - m2) - cube(t - m3)) / (6.0 * m1 * m2 * m3)
    sq = t * (t - m1) / (2.0 * m2 * m3) + m1 * m1 / (6.0 * m2 * m3)
    lin = (t - 0.5 * m12) / m3
    f = torch.where(t < m1, t ** 3 / (6.0 * m1 * m2 * m3),
                    torch.where(t < m2, sq, torch.where((m12 <= m3) & (t >= m12), lin, poly)))
    f = torch.where(s <= 0.5 * tot, f, 1.0 - f)
    return torch.where(s >= tot, torch.ones_like(f), torch.where(s <= 0, torch.zeros_like(f), f)).clamp(0.0, 1.0)


def _open_area(a, b, c):
    """Open fraction of a face: a, b = |normal x size| along it, c = level set at its centre."""
    a, b = a.abs(), b.abs()
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    lo = torch.maximum(lo, 1e-6 * hi + 1e-300)
    hi = hi + 1e-300
    s = c + 0.5 * (lo + hi)
    sq = lambda q: q.clamp(min=0.0) ** 2
    f = (sq(s) - sq(s - lo) - sq(s - hi) + sq(s - lo - hi)) / (2.0 * lo * hi)
    return torch.where(s >= lo + hi, torch.ones_like(f), torch.where(s <= 0, torch.zeros_like(f), f)).clamp(0.0, 1.0)


def _solid(scene, x, shift):
    """Level set (positive in the fluid) and unit normal of the solid."""
    if scene == "layers":
        one = torch.ones(torch.broadcast_shapes(*(q.shape for q in x)), dtype=F64, device="cuda")
        return 1.0e3 * one, (0 * one, 0 * one, one)
    tank = scene == "tank"
    cx, cy, cz, r = (2.0, 0.5, None, 0.1) if tank else (0.5, 0.5, 0.3, 0.15)
    dx, dy = x[0] - (cx + shift[0]), x[1] - (cy + shift[1])
    dz = 0.0 * x[2] if tank else x[2] - (cz + shift[2])
    rr = torch.sqrt(dx * dx + dy * dy + dz * dz + 1e-40)
    return rr - r, (dx / rr, dy / rr, dz / rr + 0 * rr)


def _liquid(scene, x, d, shift):
    """Level set (negative in the liquid) and liquid fraction of the box."""
    if scene == "bubble":
        dx, dy, dz = x[0] - 0.5 - shift[0], x[1] - 0.5 - shift[1], x[2] - 0.65 - shift[2]
        rr = torch.sqrt(dx * dx + dy * dy + dz * dz + 1e-40)
        phi, n = 0.1 - rr, (dx / rr, dy / rr, dz / rr)
    else:
        t = 2.0 * math.pi
        if scene == "tank":
            h = 0.5 + shift[2] + 0.03 * torch.cos(t / 0.8 * x[0]) + 0 * x[1]
            hx, hy = -0.03 * t / 0.8 * torch.sin(t / 0.8 * x[0]), 0 * x[1]
        else:
            h = 0.5 + shift[2] + 0.02 * torch.sin(t * x[0]) * torch.sin(t * x[1])
            hx = 0.02 * t * torch.cos(t * x[0]) * torch.sin(t * x[1])
            hy = 0.02 * t * torch.sin(t * x[0]) * torch.cos(t * x[1])
        g = torch.sqrt(1.0 + hx * hx + hy * hy)
        phi, n = (x[2] - h) / g, (hx / g, hy / g, 1.0 / g)
    s = phi + 0.5 * sum(ni.abs() * di for ni, di in zip(n, d))
    return phi, 1.0 - _cut_volume(n, d, s)


def _fill_ghosts(f):
    for a in range(3):
        f.narrow(a, 0, 1).copy_(f.narrow(a, 1, 1))
        f.narrow(a, f.shape[a] - 1, 1).copy_(f.narrow(a, f.shape[a] - 2, 1))
    return f


def _ghosted(f):
    K, J, I = f.shape
    out = torch.empty((K + 2, J + 2, I + 2), dtype=F64, device="cuda")
    out[1:-1, 1:-1, 1:-1] = f
    return _fill_ghosts(out)


def _velocity(gen, n):
    """N(0, 0.1^2) smoothed by three neighbour-average passes."""
    f = _fill_ghosts(0.1 * torch.randn((n[2] + 2, n[1] + 2, n[0] + 2), dtype=F64, device="cuda", generator=gen))
    for _ in range(3):
        g = f.clone()
        g[1:-1, 1:-1, 1:-1] = (f[1:-1, 1:-1, :-2] + f[1:-1, 1:-1, 2:] + f[1:-1, :-2, 1:-1] + f[1:-1, 2:, 1:-1]
                               + f[:-2, 1:-1, 1:-1] + f[2:, 1:-1, 1:-1]) / 6.0
        f = _fill_ghosts(g)
    return f


def _lower(f, ax):
    """The lower neighbour's value along an axis of a ghosted field, on the interior."""
    sl = [slice(1, -1)] * 3
    sl[2 - ax] = slice(0, -2)
    return f[tuple(sl)]


def _upper(f, ax):
    sl = [slice(1, -1)] * 3
    sl[2 - ax] = slice(2, None)
    return f[tuple(sl)]


def _inner(f):
    return f[1:-1, 1:-1, 1:-1]


def _shift(gen, scene):
    return [0.01 * (2.0 * q - 1.0) for q in torch.rand(3, dtype=F64, device="cuda", generator=gen).tolist()]


def _projection_fields(case, seed):
    """All inputs of one projection as device tensors."""
    gen, scene, g = _gen(seed), case["scene"], _Grid(case)
    I, J, K = g.n
    shift = _shift(gen, scene)
    x, d = g.cells()
    phi, nrm = _solid(scene, x, shift)
    vof = _cut_volume(nrm, d, phi + 0.5 * sum(ni.abs() * di for ni, di in zip(nrm, d)))
    phil, vofl = _liquid(scene, *g.cells(ghost=True), shift)
    phil, vofl = phil.expand(K + 2, J + 2, I + 2).clone(), vofl.expand(K + 2, J + 2, I + 2).clone()
    ct = torch.where(vof >= 1.0 - EPSI, 0, torch.where(vof <= EPSI, 2, 1)).expand(K, J, I).clone()
    # apertures of the upper faces, and of the lower boundary face in the ghost layer
    raw = []
    for ax in range(3):
        faces = np.concatenate([[0.0], np.cumsum(g.d[ax])])
        xf = list(x)
        xf[ax] = g.along(faces, ax)
        pf, nf = _solid(scene, xf, shift)
        p, q = [b for b in range(3) if b != ax]
        raw.append(_open_area(nf[p] * d[p], nf[q] * d[q], pf).expand(*[m + (a == 2 - ax) for a, m in enumerate((K, J, I))]))
    for _ in range(3):
        solid = torch.ones((K + 2, J + 2, I + 2), dtype=torch.bool, device="cuda")
        solid[1:-1, 1:-1, 1:-1] = ct == 2
        face, open_sum = [], torch.zeros((K, J, I), dtype=F64, device="cuda")
        for ax in range(3):
            A = torch.ones((K + 2, J + 2, I + 2), dtype=F64, device="cuda")
            sl = [slice(1, -1)] * 3
            sl[2 - ax] = slice(0, -1)
            A[tuple(sl)] = raw[ax]
            up = torch.ones_like(solid)
            up.narrow(2 - ax, 0, A.shape[2 - ax] - 1).copy_(solid.narrow(2 - ax, 1, A.shape[2 - ax] - 1))
            edge = torch.zeros_like(solid)   # a wall face closes only beside a solid cell
            edge.narrow(2 - ax, 0, 1).fill_(True)
            low_solid = solid & ~edge
            up_solid = up.clone()
            up_solid.narrow(2 - ax, A.shape[2 - ax] - 2, 2).fill_(False)
            A = torch.where(low_solid | up_solid, torch.zeros_like(A), A)
            A = torch.where(A < 1e-3, torch.zeros_like(A), A)
            ghost = torch.ones_like(solid)
            ghost[tuple(sl)] = False
            A = torch.where(ghost, torch.ones_like(A), A)
            face.append(A)
            open_sum += _inner(A) + _lower(A, ax)
        stranded = (ct != 2) & (open_sum < 1e-2)
        if not bool(stranded.any()):
            break
        ct[stranded] = 2
    active = ct != 2
    vof = torch.where(ct == 0, torch.ones_like(vof), torch.where(ct == 2, torch.zeros_like(vof), vof)).expand(K, J, I)
    vofl = vofl.clone()
    vofl[1:-1, 1:-1, 1:-1] = torch.where(active, _inner(vofl), torch.zeros_like(vof))
    f = dict(phil=phil, vofl=vofl, vof=_ghosted(vof), ct=ct, face=face, nz=nrm[2].expand(K, J, I), vct=[], vmo=[],
             dp=[], us=[])
    open_top = scene == "tank"
    f["flag"] = (1, 1, 1, 1, 1, 0 if open_top else 1)
    for ax in range(3):
        A = _inner(face[ax])
        vct = torch.where(A <= 0.0, 2, torch.where(A < 1.0, 1, 0))
        nb = torch.zeros((K + 2, J + 2, I + 2), dtype=torch.bool, device="cuda")
        nb[1:-1, 1:-1, 1:-1] = ~active
        f["vct"].append(vct)
        f["vmo"].append((((~active) | _upper(nb, ax)) & (raw[ax].narrow(2 - ax, 1, g.n[ax]) > 0)).to(torch.int64))
        dp = torch.zeros((K + 2, J + 2, I + 2), dtype=F64, device="cuda")
        dp[1:-1, 1:-1, 1:-1] = DT * (vct != 2)
        m = g.n[ax]
        take = lambda i: dp.narrow(2 - ax, i, 1)
        take(m).copy_(take(m - 1))
        f["dp"].append(_fill_ghosts(dp))
        us = _velocity(gen, g.n)
        us[1:-1, 1:-1, 1:-1] *= vct != 2
        if f["flag"][2 * ax] == 1:
            us.narrow(2 - ax, 0, 1).fill_(0.0)
        if f["flag"][2 * ax + 1] == 1:
            us.narrow(2 - ax, m, 2).fill_(0.0)
        f["us"].append(us)
    order = active.permute(2, 1, 0).reshape(-1).cumsum(0).reshape(I, J, K).permute(2, 1, 0) - 1
    f["pos"] = torch.where(active, order, -torch.ones_like(order))
    f["ext"] = int(active.sum()) - 1
    f["grid"] = g
    f["rho"] = {"bubble": (1000.0, 1.0), "tank": (833.0, 1.0)}.get(scene, (1000.0, 1.2))
    return f


def _host(t, dtype=F64):
    """A page-locked Fortran-ordered numpy array with the tensor's values."""
    out = torch.empty(t.shape, dtype=dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy().T


def _host_zeros(shape):
    return _host(torch.zeros(tuple(reversed(shape)), dtype=F64))


def _workload(case, f):
    g = f["grid"]
    I, J, K = g.n
    i32 = torch.int32
    a = {"phil": _host(f["phil"]), "vofl": _host(f["vofl"]), "vof": _host(f["vof"]), "vof_old": _host(f["vof"]),
         "cell_type": _host(f["ct"], i32), "posnu": _host(f["pos"], i32)}
    for ax, (c, v, s) in enumerate((("x", "u", "ee"), ("y", "v", "ne"), ("z", "w", "te"))):
        a["pgrid_d" + c] = _host(g.full(g.d[ax], ax))
        a["%sgrid_d%s" % (v, c)] = _host(g.full(g.s[ax], ax))
        a[s + "area"] = _host(f["face"][ax])
        a["dp_" + v], a[v + "_star"] = _host(f["dp"][ax]), _host(f["us"][ax])
        a["tvar_" + v] = _host(f["us"][ax])
        a[v + "cell_moexcell"], a[v + "cell_cell_type"] = _host(f["vmo"][ax], i32), _host(f["vct"][ax], i32)
    a["tvar_p"] = _host(torch.zeros_like(f["phil"]))
    for key, shape in zip(capi.BCP_KEYS, capi.bc_plane_shapes(I, J, K)):
        a[key] = np.zeros(shape, order="F")
    vflag = tuple(1 - q for q in f["flag"])
    zero = (0.0,) * 6
    return W.Workload(name=case["scene"], imax=I, jmax=J, kmax=K, dt=DT, rho_l=f["rho"][0], rho_g=f["rho"][1],
                      arrays=a, bcp_flag=f["flag"], bcu_flag=vflag, bcv_flag=vflag, bcw_flag=vflag, bcu_const=zero,
                      bcv_const=zero, bcw_const=zero, bcp_const=zero, ext_cell=f["ext"])


class _DeviceField:
    """A library-owned device array as torch sees it; keeps the owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (int(ptr), False),
                                         "version": 3}


def _device_tensor(owner, ptr, shape):
    return torch.as_tensor(_DeviceField(owner, ptr, shape), device="cuda")


# ---- predictor, geometry and transport inputs -----------------------------------

def _geometry_inputs(case, seed):
    gen, g = _gen(seed), _Grid(case)
    I, J, K = g.n
    shift = _shift(gen, "sphere")
    fams = {}
    for fam in GM.FAMILIES:
        c, d = [q.copy() for q in g.c], [q.copy() for q in g.d]
        if fam != "p":
            ax = "uvw".index(fam)
            c[ax], d[ax] = g.c[ax] + 0.5 * g.d[ax], g.s[ax]
        x, dd = [g.along(c[a], a) for a in range(3)], [g.along(d[a], a) for a in range(3)]
        phi, nrm = _solid("sphere", x, shift)
        vof = _cut_volume(nrm, dd, phi + 0.5 * sum(ni.abs() * di for ni, di in zip(nrm, dd)))
        _, vofl = _liquid("bubble", x, dd, shift)
        arr = {"dx": _host(g.full(d[0], 0)), "dy": _host(g.full(d[1], 1)), "dz": _host(g.full(d[2], 2))}
        for key, val in (("phi", phi), ("nx", nrm[0]), ("ny", nrm[1]), ("nz", nrm[2]), ("vof", vof), ("vofl", vofl)):
            arr[key] = _host(_ghosted(val.expand(K, J, I)))
        for key, dt, kind in GM.FIELDS:
            if key not in arr:
                shape = tuple(reversed(GM.field_shape(kind, fam, I, J, K)))
                arr[key] = (_host(torch.full(shape, 7), torch.int32) if dt == np.int32 else
                            _host(torch.randn(shape, dtype=F64, device="cuda", generator=gen)))
        if fam == "p":
            arr["moexcell"] = None
        fams[fam] = GM.GeoFamily(fam, arr)
    return GM.GeoInputs(I, J, K, fams)


def _momentum_inputs(case, seed):
    g = _geometry_inputs(case, seed)
    pre = GM.GridPreprocess(g.imax, g.jmax, g.kmax)
    pre(g)
    pre.close()
    return PR.momentum_inputs(g, seed=seed)


def _momentum_opts(case):
    return PR.default_opts(precision=capi.SCF_PREC_MIXED if case["precision"] == "mixed" else capi.SCF_PREC_FP64,
                           rel_tol=case["rel_tol"])


def _transport_inputs(case, seed):
    """The 3-D deformation test: a liquid sphere in a reversing vortex."""
    gen, g = _gen(seed), _Grid(case)
    I, J, K = g.n
    shift = _shift(gen, "sphere")
    x, d = [], []
    for ax in range(3):
        m, dd = g.n[ax], g.d[ax]
        lo, hi = g.c[ax][0] - dd[0], g.c[ax][-1] + dd[-1]
        x.append(g.along(np.concatenate([[lo], g.c[ax], [hi]]), ax))
        d.append(g.along(np.concatenate([[dd[0]], dd, [dd[-1]]]), ax))
    r = torch.sqrt(sum((q - 0.35 - s) ** 2 for q, s in zip(x, shift)) + 1e-40)
    phi, n = r - 0.15, [(q - 0.35 - s) / r for q, s in zip(x, shift)]
    vof = 1.0 - _cut_volume(n, d, phi + 0.5 * sum(ni.abs() * di for ni, di in zip(n, d)))
    vof = torch.where(vof <= 1e-14, torch.zeros_like(vof), torch.where(vof >= 1 - 1e-14, torch.ones_like(vof), vof))
    s1, s2 = [torch.sin(math.pi * q) for q in x], [torch.sin(2 * math.pi * q) for q in x]
    amp = 1.0 + 0.1 * shift[0]
    vel = [2.0 * amp * s1[0] ** 2 * s2[1] * s2[2], -amp * s2[0] * s1[1] ** 2 * s2[2],
           -amp * s2[0] * s2[1] * s1[2] ** 2]
    fr = torch.sqrt(sum((q - 1000.0) ** 2 for q in x))
    keep = torch.zeros((K + 2, J + 2, I + 2), dtype=F64, device="cuda")
    keep[1:-1, 1:-1, 1:-1] = 1.0
    h = min(float(q.min()) for q in g.d)
    zero = torch.zeros_like(keep)
    return dict(centres=[_host(g.full(g.c[a], a)) for a in range(3)],
                spacings=[_host(g.full(g.d[a], a)) for a in range(3)],
                state={"vofl": _host(vof), "phil": _host(phi), "nxl": _host(zero), "nyl": _host(zero),
                       "nzl": _host(zero)},
                vel=[_host(v * keep) for v in vel], fluid_normals=[_host((q - 1000.0) / fr * keep) for q in x],
                bc_vel=[np.zeros(s, order="F") for s in ((J, K), (I, K), (I, J))],
                lvs_bc=[np.zeros(s, order="F") for s in plane_shapes(I, J, K)], dt=0.15 * h / 2.0,
                lvs_flag=(0,) * 6, vof_flag=(0,) * 6)


# ---- the measured calls ------------------------------------------------------------

def _projection(case, w):
    return Projection.for_workload(
        w, precision=capi.SCF_PREC_MIXED if case["precision"] == "mixed" else capi.SCF_PREC_FP64,
        rel_tol=case["rel_tol"], smoother_degree=case["degree"])


def _density(case, f, seed):
    """Per-cell densities: the phase's, perturbed by up to 5%."""
    gen = _gen(seed + 7)
    phase = torch.where((f["vofl"] >= 0.5), f["rho"][0], f["rho"][1])
    return phase * (1.0 + 0.05 * (2.0 * torch.rand(phase.shape, dtype=F64, device="cuda", generator=gen) - 1.0))


def _weights(f):
    """Weights of the vertical pressure force on the solid (cut cells only)."""
    d = [f["grid"].full(f["grid"].d[a], a) for a in range(3)]
    wet = sum(((_inner(A) - _lower(A, ax)) * (d[0] * d[1] * d[2] / d[ax])) ** 2 for ax, A in enumerate(f["face"]))
    return torch.where(f["ct"] == 1, -f["nz"] * torch.sqrt(wet), torch.zeros_like(wet))


def prepare(case, seed):
    kind, shape = case["kind"], (case["K"] + 2, case["J"] + 2, case["I"] + 2)
    if kind == "projection":
        w = _workload(case, _projection_fields(case, seed))
        p = _projection(case, w)
        p.stage(w)
        out = {k: _device_tensor(p, q, shape) for k, q in p.device_fields().items() if k in ("u", "v", "w", "p")}
        return dict(kind=kind, p=p, out=out)
    if kind == "update_puvw":
        w = _workload(case, _projection_fields(case, seed))
        bc = [[_host_zeros(s) for s in capi.bc_plane_shapes(*w.shape_i)] for _ in range(4)]
        return dict(kind=kind, p=_projection(case, w), w=w, bc=bc,
                    tvar=[w.arrays[k] for k in ("tvar_u", "tvar_v", "tvar_w", "tvar_p")])
    if kind == "loss_grad":
        f = _projection_fields(case, seed)
        w = _workload(case, f)
        runner = ProjectionLoss(w, g=_host(_weights(f)), rel_tol=case["rel_tol"], smoother_degree=case["degree"])
        return dict(kind=kind, runner=runner, us=[w.arrays[v + "_star"] for v in "uvw"],
                    rho=_host(_density(case, f, seed)))
    if kind == "predictor":
        s = PR.PredictSolves(case["I"], case["J"], case["K"])
        s.stage(_momentum_inputs(case, seed))
        return dict(kind=kind, s=s, opts=_momentum_opts(case), shape=shape)
    if kind == "geometry":
        return dict(kind=kind, g=_geometry_inputs(case, seed), pre=GM.GridPreprocess(case["I"], case["J"], case["K"]))
    t = _transport_inputs(case, seed)
    shp = tuple(reversed(shape))
    return dict(kind="clsvof", t=t, s=ClsvofScheme(case["I"], case["J"], case["K"]),
                out={k: _host_zeros(shp) for k in t["state"]},
                planes=[_host_zeros(q) for q in plane_shapes(case["I"], case["J"], case["K"]) * 2])


def run(state):
    kind = state["kind"]
    if kind == "projection":
        state["p"].run()
        return state["out"]
    if kind == "update_puvw":
        u, v, w, p, bc, _ = state["p"].update_puvw(state["w"], tvar=state["tvar"], bc_out=state["bc"])
        return {"u": u, "v": v, "w": w, "p": p, "bc": bc}
    if kind == "loss_grad":
        J, _, _ = state["runner"].forward(*state["us"], rho=state["rho"])
        grads, _ = state["runner"].backward()
        return {"J": J, "u": grads[0], "v": grads[1], "w": grads[2], "rho": grads[3]}
    if kind == "predictor":
        state["s"].run(state["opts"])
        return [_device_tensor(state["s"], q, state["shape"]) for q in state["s"].device_fields()]
    if kind == "geometry":
        state["pre"](state["g"])
        fams = state["g"].fams
        return {f: {k: fams[f].arrays[k] for k in GM.OUTPUTS if fams[f].arrays[k] is not None} for f in GM.FAMILIES}
    t, s = state["t"], state["s"]
    s.stage(**t)
    s.run(1)
    s.fetch(state["out"], state["planes"][:6], state["planes"][6:])
    return {"state": state["out"], "planes": state["planes"]}


# ---- 64-bit values by plain torch -----------------------------------------------------

def _face_coefs(f, rho=None):
    """Face coefficient x spacing ratio of every cell's upper faces: the
    ghost-fluid density weighting, or per-cell densities when given."""
    rho_l, rho_g = f["rho"]
    bp, bm = 1.0, 1.0 / (rho_g / rho_l)   # the reference density is the liquid's
    vof, vofl, phil, g = f["vof"], f["vofl"], f["phil"], f["grid"]
    full, part = vof > 1.0 - EPSI, (vof <= 1.0 - EPSI) & (vof > EPSI)
    wet = ((vofl >= 0.5) & full) | ((phil < 0) & part)
    dry = ((vofl < 0.5) & full) | ((phil >= 0) & part)
    out = []
    for ax in range(3):
        ratio = _inner(f["dp"][ax]) / g.full(g.s[ax], ax)
        pc, pn = _inner(phil).abs(), _upper(phil, ax).abs()
        lam = pc / (pc + pn + 1e-30)
        if rho is not None:
            lam = torch.where(_upper(wet | dry, ax), lam, torch.ones_like(lam))
            c = ratio * rho_l / (lam * _inner(rho) + (1.0 - lam) * _upper(rho, ax))
            c = torch.where(_inner(wet | dry), c, torch.zeros_like(c))
        else:
            wd, dw = _inner(wet) & _upper(dry, ax), _inner(dry) & _upper(wet, ax)
            mix = torch.where(wd, lam * bm + (1.0 - lam) * bp, lam * bp + (1.0 - lam) * bm)
            beta = torch.where(wd | dw, bp * bm / mix, torch.where(_inner(wet), bp, bm))
            c = torch.where(_inner(wet | dry), ratio * beta, torch.zeros_like(ratio))
        out.append(c)
    return out


class _System:
    """The pressure system A p = b of a case: face weights and diagonal."""

    def __init__(self, f, rho=None):
        self.f, g = f, f["grid"]
        self.act = (f["ct"] != 2).to(F64)
        d = [g.full(g.d[a], a) for a in range(3)]
        vol = d[0] * d[1] * d[2]
        self.area = [vol / d[a] for a in range(3)]
        self.coef = _face_coefs(f, rho)
        self.w, self.top = [], 0.0
        for ax in range(3):
            a2 = torch.zeros_like(f["phil"])
            a2[1:-1, 1:-1, 1:-1] = self.act
            w = self.coef[ax] * _inner(f["face"][ax]) * self.area[ax] * self.act * _upper(a2, ax)
            self.w.append(w)
        self.diag = sum(self.w[ax] + self.shift_up(self.w[ax], ax) for ax in range(3))
        if f["flag"][5] == 0:   # open top: its coefficient is the plane below's
            self.top = torch.zeros_like(self.diag)
            self.top[-1] = (self.coef[2][-2] * _inner(f["face"][2])[-1] * self.area[2][-1]) * self.act[-1]
            self.diag = self.diag + self.top
        self.singular = all(q == 1 for q in f["flag"])

    @staticmethod
    def shift_up(a, ax):
        """a of the lower neighbour (0 at the wall)."""
        dim = 2 - ax
        return torch.cat([torch.zeros_like(a.narrow(dim, 0, 1)), a.narrow(dim, 0, a.shape[dim] - 1)], dim)

    @staticmethod
    def diff(p, ax):
        """p of the upper neighbour minus p (0 at the wall)."""
        dim = 2 - ax
        m = p.shape[dim]
        return torch.cat([p.narrow(dim, 1, m - 1) - p.narrow(dim, 0, m - 1), torch.zeros_like(p.narrow(dim, 0, 1))], dim)

    def apply(self, p):
        y = self.top * p if torch.is_tensor(self.top) else torch.zeros_like(p)
        for ax in range(3):
            q = self.w[ax] * self.diff(p, ax)
            y = y - q + self.shift_up(q, ax)
        return y

    def flux_sum(self, us):
        """The divergence sum of the face velocities (ghosted, lower faces included)."""
        return sum(self.area[ax] * (_inner(self.f["face"][ax]) * _inner(us[ax])
                                    - _lower(self.f["face"][ax], ax) * _lower(us[ax], ax)) for ax in range(3))

    def mean_free(self, a):
        return (a - (a * self.act).sum() / self.act.sum()) * self.act

    def solve(self, b, tol=1e-13, most=20000):
        proj = self.mean_free if self.singular else (lambda a: a * self.act)
        b = proj(b)
        x, r = torch.zeros_like(b), b.clone()
        dinv = torch.where(self.act > 0, 1.0 / torch.where(self.diag > 0, self.diag, torch.ones_like(b)),
                           torch.zeros_like(b))
        z = dinv * r
        p, rz, stop = z.clone(), (r * z).sum(), tol * tol * float((b * b).sum())
        for it in range(most):
            q = self.apply(p)
            alpha = rz / (p * q).sum()
            x += alpha * p
            r -= alpha * q
            if it % 25 == 24:
                r = proj(b - self.apply(x)) if it % 500 == 499 else proj(r)
                if float((r * r).sum()) <= stop:
                    break
            z = dinv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        return proj(x)


def _exact_projection(case, seed):
    f = _projection_fields(case, seed)
    s = _System(f)
    b = -s.flux_sum(f["us"]) * s.act
    x = s.solve(b)
    n, fl = f["grid"].n, f["flag"]
    pp = torch.zeros_like(f["phil"])
    pp[1:-1, 1:-1, 1:-1] = x
    for ax in range(3):
        dim, m = 2 - ax, n[ax]
        sl = [slice(1, -1)] * 3
        for at, src, flag in ((0, 1, fl[2 * ax]), (m + 1, m, fl[2 * ax + 1])):
            to, fr = list(sl), list(sl)
            to[dim], fr[dim] = slice(at, at + 1), slice(src, src + 1)
            pp[tuple(to)] = flag * pp[tuple(fr)]
    vel = []
    for ax in range(3):
        u = f["us"][ax].clone()
        c = s.coef[ax].clone()
        dim, m = 2 - ax, n[ax]
        c.narrow(dim, m - 1, 1).copy_(c.narrow(dim, m - 2, 1))
        on = (f["vmo"][ax] != 1) & (f["vct"][ax] != 2)
        u[1:-1, 1:-1, 1:-1] = torch.where(on, _inner(u) - (_upper(pp, ax) - _inner(pp)) * c, torch.zeros_like(c))
        vel.append(u)
    p = torch.zeros_like(pp)
    p[1:-1, 1:-1, 1:-1] = x
    for fld, F in enumerate(vel + [p]):
        for face in range(6):
            ax, high = face // 2, face % 2
            dim, m = 2 - ax, n[ax]
            flag = (1 - fl[face]) if fld < 3 else fl[face]
            src = (m - 1 if fld == ax else m) if high else 1
            plane = F.select(dim, src)
            var = plane[:-2, :-2].clone() if flag else torch.zeros_like(plane[1:-1, 1:-1])
            own = fld == ax
            if own:
                F.select(dim, m if high else 0)[1:-1, 1:-1] = var
            elif fld == 3 and face == 5:
                F.select(dim, m)[1:-1, 1:-1] = var
            if not (own and not high):
                edge = F.select(dim, m if high else 1)[1:-1, 1:-1]
                F.select(dim, m + 1 if high else 0)[1:-1, 1:-1] = (var if flag else 2.0 * var) - edge
    if fl[5] == 0:   # mass correction of the open top
        K = n[2]
        a, (u, v, w) = f["face"], vel
        top = lambda q: _inner(q)[K - 1]
        z = a[2][K, 1:-1, 1:-1]
        num = (-s.area[0][K - 1] * top(a[0]) * (top(u) - _lower(u, 0)[K - 1])   # the cell's own aperture on both sides
               - s.area[1][K - 1] * top(a[1]) * (top(v) - _lower(v, 1)[K - 1])
               + s.area[2][K - 1] * z * w[K - 1, 1:-1, 1:-1])
        w[K, 1:-1, 1:-1] = num / z / s.area[2][K - 1]
    out = {"u": vel[0], "v": vel[1], "w": vel[2], "p": p}
    if case["kind"] == "update_puvw":
        out = {k: v.cpu().numpy().T for k, v in out.items()}
        out["bc"] = [[None] * 6 for _ in range(4)]
    return out


def _exact_loss(case, seed):
    f = _projection_fields(case, seed)
    rho = _density(case, f, seed).requires_grad_(True)
    us = [u.clone().requires_grad_(True) for u in f["us"]]
    s = _System(f, rho)
    b = -s.flux_sum(us) * s.act
    frozen = _System(f, rho.detach())
    p = frozen.solve(b.detach(), 1e-14).requires_grad_(True)
    u = []
    for ax in range(3):
        on = (f["vmo"][ax] != 1) & (f["vct"][ax] != 2)
        keep = torch.zeros_like(us[ax])
        keep.narrow(2 - ax, 0, 1).fill_(1.0)
        keep[1:-1, 1:-1, 1:-1] = on.to(F64)
        corr = torch.zeros_like(us[ax])
        corr[1:-1, 1:-1, 1:-1] = torch.where(on, s.diff(p, ax) * s.coef[ax], torch.zeros_like(p))
        u.append(us[ax] * keep - corr)
    r = s.flux_sum(u) * s.act
    J = (_weights(f) * p * s.act).sum() + 0.5 * (r * r).sum()
    grads = torch.autograd.grad(J, [p] + us + [rho], retain_graph=True, allow_unused=True)
    lam = frozen.solve(grads[0], 1e-14)
    second = torch.autograd.grad((lam * (b - s.apply(p.detach()))).sum(), us + [rho], allow_unused=True)
    zero = torch.zeros_like(rho)
    tot = [(a if a is not None else zero) + (c if c is not None else zero) for a, c in zip(grads[1:], second)]
    g = [q.detach().cpu().numpy().T for q in tot]
    return {"J": float(J.detach()), "u": g[0], "v": g[1], "w": g[2], "rho": g[3]}


def _exact_momentum(case, seed):
    inp, o = _momentum_inputs(case, seed), _momentum_opts(case)
    I, J, K = inp.imax, inp.jmax, inp.kmax
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).to("cuda")
    preds, dps = [], []
    for c in range(3):
        cm = inp.comps[c]
        a = {k: T(v) for k, v in cm.arrays.items()}
        end = [I - (c == 0), J - (c == 1), K - (c == 2)]
        cut = lambda q: q[:end[2], :end[1], :end[0]]
        act = cut(a["cell_type"]) != 2
        vof, vofl = cut(_inner(a["vof"])), cut(_inner(a["vofl"]))
        rho = vofl * o.rho_w_ref + (vof - vofl) * o.rho_a_ref
        rho = torch.where(act, rho, torch.ones_like(rho))
        vol = [cut(a["grid_d" + q]) for q in "xyz"]
        lhs = vof * vol[0] * vol[1] * vol[2]
        aP = lhs / o.dt + cut(a["fric"])
        off, wall = [], []
        for ax, (df, edf, eta) in enumerate((("df_ew", "edf_ew", "eta_e"), ("df_ns", "edf_ns", "eta_n"),
                                             ("df_tb", "edf_tb", "eta_t"))):
            dim, m = 2 - ax, end[ax]
            scale = 1.0 if ax == c else 0.5
            for up in (0, 1):
                # DF(i) lies below cell i: index i (0-based ghosted) = lower face, i + 1 = upper
                lo = 1 + up
                D = (1.0 - o.beta_vis) * cut(a[df].narrow(dim, lo, a[df].shape[dim] - lo)) / rho
                E = cut(a[edf].narrow(dim, lo, a[edf].shape[dim] - lo))
                et = cut(_inner(a[eta]) if up else _lower(a[eta], ax))
                plus, minus = (E * (1.0 - et) / rho, E * et / rho) if up else (E * et / rho, E * (1.0 - et) / rho)
                at = m - 1 if up else 0
                fac = 0.0 if cm.bc_flag[2 * ax + up] == 1 else scale
                for q in (D, plus, minus):
                    q.narrow(dim, at, 1).mul_(fac)
                aP = aP + D + (plus if up else -plus)
                wall.append(D)
                off.append(D - minus if up else D + minus)
        dp0 = 1.0 / (aP - sum(off))
        dp = torch.zeros((K + 2, J + 2, I + 2), dtype=F64, device="cuda")
        dp[1:end[2] + 1, 1:end[1] + 1, 1:end[0] + 1] = torch.where(act, lhs * dp0, torch.zeros_like(lhs))
        U, vo = cut(_inner(a["tvar"])), cut(_inner(a["vof_old"]))
        box = vol[0] * vol[1] * vol[2]
        grav = (o.gx, o.gy, o.gz)[c] / o.g / (o.fr * o.fr)
        b = U * lhs / o.dt - U * (vof - vo) * box / o.dt + grav * lhs - cut(a["flux_div"])
        for face in range(6):
            ax, up = face // 2, face % 2
            dim = 2 - ax
            var = T(cm.bc_var[face])
            keep = [end[q] for q in range(3) if q != ax]
            var = var[:keep[1], :keep[0]]
            at = end[ax] - 1 if up else 0
            b.select(dim, at).add_(wall[face].select(dim, at) * var)
        actf = act.to(F64)
        b = b * actf

        def apply(x):
            y = aP * x
            for face in range(6):
                dim, m = 2 - face // 2, x.shape[2 - face // 2]
                if face % 2:
                    y.narrow(dim, 0, m - 1).sub_(off[face].narrow(dim, 0, m - 1) * x.narrow(dim, 1, m - 1))
                else:
                    y.narrow(dim, 1, m - 1).sub_(off[face].narrow(dim, 1, m - 1) * x.narrow(dim, 0, m - 1))
            return y * actf
        dinv = torch.where(act, 1.0 / aP, torch.zeros_like(aP))
        x = torch.zeros_like(b)
        for _ in range(6):   # BiCGStab with Jacobi scaling, restarted from the true residual
            r = b - apply(x)
            if float(r.norm()) <= 1e-15 * float(b.norm()):
                break
            r0, p, v = r.clone(), torch.zeros_like(r), torch.zeros_like(r)
            rho1 = alpha = om = torch.ones((), dtype=F64, device="cuda")
            stop = max(1e-3 * float(r.norm()) * 1e-6, 1e-16 * float(b.norm()))
            for it in range(200):
                rn = (r0 * r).sum()
                p = r + (rn / rho1) * (alpha / om) * (p - om * v)
                rho1 = rn
                ph = dinv * p
                v = apply(ph)
                alpha = rn / (r0 * v).sum()
                q = r - alpha * v
                sh = dinv * q
                t = apply(sh)
                om = (t * q).sum() / (t * t).sum()
                x = x + alpha * ph + om * sh
                r = q - om * t
                if float(r.norm()) <= stop:
                    break
        pred = torch.zeros((K + 2, J + 2, I + 2), dtype=F64, device="cuda")
        pred[1:end[2] + 1, 1:end[1] + 1, 1:end[0] + 1] = x
        n, dim = (I, J, K)[c], 2 - c
        mid = (slice(1, -1),) * 2
        for lo_hi in (0, 1):
            var = T(cm.bc_var[2 * c + lo_hi])
            if lo_hi == 0:
                pred.select(dim, 0)[mid] = pred.select(dim, 1)[mid] if cm.bc_flag[2 * c] == 1 else var
            else:
                below = pred.select(dim, n - 1)[mid].clone()
                pred.select(dim, n)[mid] = below if cm.bc_flag[2 * c + 1] == 1 else var
                pred.select(dim, n + 1)[mid] = 2.0 * var - below
        pred[1:-1, 1:-1, 1:-1] *= (a["cell_type"] != 2)
        dp.select(dim, n).copy_(dp.select(dim, n - 1))
        for ax in range(3):
            d2 = 2 - ax
            dp.select(d2, 0).copy_(dp.select(d2, 1))
            dp.select(d2, dp.shape[d2] - 1).copy_(dp.select(d2, dp.shape[d2] - 2))
        preds.append(pred)
        dps.append(dp)
    return preds + dps


def exact(case, seed):
    """The geometry and the transport have no solve and no freedom of
    rounding: their results are fixed bit for bit, so no 64-bit value is given
    for them, nor for grids on which plain CG takes too long."""
    kind, n = case["kind"], case["I"] * case["J"] * case["K"]
    if kind in ("projection", "update_puvw"):
        return _exact_projection(case, seed) if n <= 4_500_000 else None
    if kind == "loss_grad":
        return _exact_loss(case, seed)
    if kind == "predictor":
        return _exact_momentum(case, seed)
    return None
