"""Timed cases of the Maxwell time step, as its users' programs call it.

Each case is one program's inner piece of work: set the fields, advance them a
number of RK steps (or evaluate one gradient), take the fields back.  The
sizes are those of the configurations in ``nekcem_gb300.cases`` (cavity,
plane wave, dielectric sphere, adjoint, large box) and of the reference's own
test cases (3dboxpec, 3dboxpml), with ragged and curved meshes between them.
Host arrays are page-locked, as a driver's own field arrays are.

``exact`` is an independent restatement of the same semi-discrete operator and
RK scheme in torch FP64 (torch autograd for the gradient).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import nekcem_gb300
from nekcem_gb300 import MaxwellGPU

WALL = {"pec": 0, "per": 1, "pml": 2}
SLOT_AXIS = (1, 0, 1, 0, 2, 2)  # the reference's face order: s-, r+, s+, r-, t-, t+
SLOT_SIDE = (-1, 1, 1, -1, -1, 1)
SLOT_OPP = (2, 3, 0, 1, 5, 4)
PML = (1, 3.0, 1e-8)  # layers, grading order, reflection error (3dboxpml)
LARGEST = 24 ** 3 * 8 ** 3 * 20 * 5  # node-stages of the largest listed case

# path: "steps" device-resident steps, "host" one call per step on host
# fields, "gradient" the discrete adjoint.  bc: one wall kind per axis.
# eps: "one", "sphere" (eps = 4 inside a sphere) or "smooth".  deform > 0: a
# curved mesh handed over as the reference's arrays.


def _case(name, path, form, N, nel, bc, steps, eps="one", source=False, deform=0.0):
    return {"name": name, "path": path, "form": form, "N": N, "ex": nel[0], "ey": nel[1],
            "ez": nel[2], "bc": bc, "steps": steps, "eps": eps, "source": source,
            "deform": deform}


def listed():
    return [
        # a small PEC cavity, many steps between outputs: each stage is one
        # element's latency and a launch
        _case("cavity_n7_mixed", "steps", "mixed", 7, (4, 4, 4), "pec,pec,pec", 100),
        # the reference's own smallest known-answer test in full FP64
        _case("boxpec_n8_fused64", "steps", "fused64", 8, (3, 3, 3), "pec,pec,pec", 40),
        # the headline configuration: the periodic plane-wave box
        _case("planewave_n7_mixed", "steps", "mixed", 7, (16, 16, 16), "per,per,per", 50),
        # the same box for users who want FP64 throughout
        _case("planewave_n7_fused64", "steps", "fused64", 7, (16, 16, 16), "per,per,per", 20),
        # the same box behind an unchanged driver that keeps its fields on the host
        _case("planewave_n7_host", "host", "mixed", 7, (16, 16, 16), "per,per,per", 40),
        # a dielectric sphere at a lower order on many elements
        _case("dielectric_n5_mixed", "steps", "mixed", 5, (32, 32, 32), "pec,pec,pec", 20, "sphere"),
        # a large box with a graded medium
        _case("large_n7_mixed", "steps", "mixed", 7, (24, 24, 24), "pec,pec,pec", 20, "smooth"),
        # a ragged mesh of stretched elements, odd order, mixed walls, driven
        _case("ragged_n6_mixed", "steps", "mixed", 6, (7, 11, 5), "pec,per,pec", 50, "smooth", True),
        # an antenna in an open domain: PML on all sides, driven
        _case("openbox_n8_mixed", "steps", "mixed", 8, (6, 6, 6), "pml,pml,pml", 50, "one", True),
        # curved elements, in the fast form and in FP64
        _case("curved_n7_mixed", "steps", "mixed", 7, (12, 12, 12), "per,per,per", 20, "one", False, 0.04),
        _case("curved_n5_fused64", "steps", "fused64", 5, (9, 10, 11), "pec,per,pec", 20, "smooth", True, 0.03),
        # the permittivity gradient of a probe energy
        _case("gradient_n7_fused64", "gradient", "fused64", 7, (8, 8, 8), "pec,pec,pec", 100, "smooth", True),
    ]


def draw(rng):
    kind = rng.choice(["mixed", "mixed", "mixed", "fused64", "fused64", "host", "pml", "curved",
                       "curved64", "gradient"])
    N = rng.choice([4, 5, 6, 7, 7, 8])
    if kind in ("curved", "curved64"):
        N = min(N, 7)
    # elements log-uniform over the listed range (in nodes)
    most = {"mixed": 7.0e6, "fused64": 2.1e6, "host": 2.1e6, "pml": 2.0e5, "curved": 8.8e5,
            "curved64": 2.5e5, "gradient": 2.6e5}[kind]
    least = 1.4e5 if kind == "host" else 9.0e3
    nodes = math.exp(rng.uniform(math.log(least), math.log(most)))
    side = (nodes / (N + 1) ** 3) ** (1.0 / 3.0)
    low = 4 if kind == "pml" else 2
    nel = [max(low, int(round(side * f))) for f in (rng.uniform(0.7, 1.3), rng.uniform(0.7, 1.3), 1.0)]
    while nel[0] * nel[1] * nel[2] * (N + 1) ** 3 > most:
        nel[nel.index(max(nel))] -= 1
    bc = ",".join(rng.choice(["pec", "per"]) for _ in range(3))
    if kind == "pml":
        bc = rng.choice(["pml,pml,pml", "per,pml,per", "pec,pml,pec"])
    eps = rng.choice(["one", "sphere", "smooth"])
    if kind in ("curved", "curved64") and eps == "sphere":
        eps = "smooth"
    path = {"host": "host", "gradient": "gradient"}.get(kind, "steps")
    form = "fused64" if kind in ("fused64", "curved64", "gradient") else "mixed"
    steps = rng.choice([10, 20, 40])
    per_step = 5 * nel[0] * nel[1] * nel[2] * (N + 1) ** 3
    weight = {"mixed": 1, "host": 2, "fused64": 5, "pml": 2, "curved": 2.5, "curved64": 8, "gradient": 15}[kind]
    steps = max(2, min(steps, int(LARGEST / (per_step * weight))))
    source = path != "host" and rng.random() < 0.5
    deform = rng.choice([0.02, 0.04]) if kind in ("curved", "curved64") else 0.0
    return {"path": path, "form": form, "N": N, "ex": nel[0], "ey": nel[1], "ez": nel[2], "bc": bc,
            "steps": steps, "eps": eps, "source": source, "deform": deform}


# ---- the mesh, as a driver's set-up leaves it --------------------------------

def _gll(N):
    """GLL points, weights and the derivative matrix D(i, j)."""
    P = np.polynomial.legendre.Legendre.basis(N)
    z = np.concatenate([[-1.0], np.sort(P.deriv().roots().real), [1.0]])
    for _ in range(3):  # Newton on the interior points
        q = z[1:-1]
        z[1:-1] = q - P.deriv()(q) / P.deriv(2)(q)
    z = 0.5 * (z - z[::-1])
    p = P(z)
    w = 2.0 / (N * (N + 1.0) * p * p)
    D = np.zeros((N + 1, N + 1))
    for i in range(N + 1):
        for j in range(N + 1):
            if i != j:
                D[i, j] = p[i] / (p[j] * (z[i] - z[j]))
    D[0, 0], D[N, N] = -N * (N + 1) / 4.0, N * (N + 1) / 4.0
    return z, w, D


class _Mesh:
    """Nodes of a box (x fastest inside an element and over elements), bent
    smoothly inside when deform > 0."""

    def __init__(self, c):
        self.N, self.n = c["N"], c["N"] + 1
        self.nel = (c["ex"], c["ey"], c["ez"])
        self.bc = [WALL[b] for b in c["bc"].split(",")]
        self.deform = c["deform"]
        self.lo = (0.0, 0.0, 0.0)
        m = max(self.nel)
        # the unit cube, or elements stretched a little where the counts differ
        self.hi = tuple(0.75 + 0.25 * k / m for k in self.nel)
        self.z, self.w, self.D = _gll(self.N)
        n, nel = self.n, self.nel
        self.nelt = nel[0] * nel[1] * nel[2]
        self.npts = self.nelt * n ** 3
        line = [((np.arange(nel[d])[:, None] + 0.5 * (self.z + 1.0)[None, :]) * (self.hi[d] / nel[d]))
                for d in range(3)]
        shape = (nel[2], nel[1], nel[0], n, n, n)
        X = np.broadcast_to(line[0][None, None, :, None, None, :], shape)
        Y = np.broadcast_to(line[1][None, :, None, None, :, None], shape)
        Z = np.broadcast_to(line[2][:, None, None, :, None, None], shape)
        if self.deform:
            s = [np.sin(np.pi * A / h) for A, h in zip((X, Y, Z), self.hi)]
            b = self.deform * s[0] * s[1] * s[2]
            X, Y, Z = X + b, Y + 0.7 * b, Z - 0.8 * b
        self.xyz = [np.ascontiguousarray(A).reshape(self.nelt, n, n, n) for A in (X, Y, Z)]

    def spacing(self):
        best = np.inf
        for ax in (1, 2, 3):
            best = min(best, float(np.min(sum(np.diff(A, axis=ax) ** 2 for A in self.xyz))))
        return math.sqrt(best)

    def faces(self):
        """Per face node (e, f, b, a): volume node, partner's volume node (-1
        on a wall), wall kind (-1 inside), and a shared id."""
        n, nel = self.n, np.array(self.nel)
        n2, n3 = n * n, n ** 3
        e = np.arange(self.nelt)
        ec = np.stack([e % nel[0], (e // nel[0]) % nel[1], e // (nel[0] * nel[1])])
        a, b = np.meshgrid(np.arange(n), np.arange(n))  # [b, a]

        def local(f):
            fix = 0 if SLOT_SIDE[f] < 0 else n - 1
            return (fix + n * a + n2 * b, a + n * fix + n2 * b, a + n * b + n2 * fix)[SLOT_AXIS[f]]

        own = np.empty((self.nelt, 6, n, n), dtype=np.int64)
        part, wall, gid = np.empty_like(own), np.empty_like(own), np.empty_like(own)
        first = 0
        base = []
        for ax in range(3):
            o = [q for q in range(3) if q != ax]
            base.append(first)
            first += int((nel[ax] + 1) * nel[o[0]] * nel[o[1]])
        for f in range(6):
            ax, sd = SLOT_AXIS[f], SLOT_SIDE[f]
            o = [q for q in range(3) if q != ax]
            plane = ec[ax] + (1 if sd > 0 else 0)
            edge = (plane == 0) | (plane == nel[ax])
            per = self.bc[ax] == 1
            w = np.where(edge & (not per), self.bc[ax], -1)
            pc = ec.copy()
            pc[ax] = (pc[ax] + sd) % nel[ax]
            pe = pc[0] + nel[0] * (pc[1] + nel[1] * pc[2])
            if per:
                plane = plane % nel[ax]
            fid = base[ax] + (plane * nel[o[0]] + ec[o[0]]) * nel[o[1]] + ec[o[1]]
            own[:, f] = (e * n3)[:, None, None] + local(f)[None]
            part[:, f] = np.where(w[:, None, None] >= 0, -1, (pe * n3)[:, None, None] + local(SLOT_OPP[f])[None])
            wall[:, f] = w[:, None, None]
            gid[:, f] = (fid * n2)[:, None, None] + (a + n * b)[None] + 1
        return own, part, wall, gid

    def metrics(self):
        """Cofactor metrics [d][ax] = jac d(r,s,t)_d/dx_ax and the jacobian."""
        D, n = self.D, self.n
        if not self.deform:
            h = [0.5 * self.hi[d] / self.nel[d] for d in range(3)]
            cof = [[0.0] * 3 for _ in range(3)]
            for d in range(3):
                cof[d][d] = h[(d + 1) % 3] * h[(d + 2) % 3]
            return cof, h[0] * h[1] * h[2]
        J = []  # J[ax][d] = dx_ax/dr_d
        for A in self.xyz:
            J.append([A @ D.T, np.einsum("ij,ekjl->ekil", D, A, optimize=True),
                      (D @ A.reshape(self.nelt, n, n * n)).reshape(A.shape)])
        cof = [[J[(ax + 1) % 3][(d + 1) % 3] * J[(ax + 2) % 3][(d + 2) % 3]
                - J[(ax + 1) % 3][(d + 2) % 3] * J[(ax + 2) % 3][(d + 1) % 3]
                for ax in range(3)] for d in range(3)]
        return cof, sum(J[0][d] * cof[d][0] for d in range(3))

    def face_vectors(self, cof, own):
        """Outward area vectors (3, e, f, b, a), quadrature weights included."""
        n = self.n
        ww = self.w[:, None] * self.w[None, :]
        out = np.zeros((3,) + own.shape)
        for f in range(6):
            d = SLOT_AXIS[f]
            for ax in range(3):
                m = cof[d][ax]
                v = m if np.isscalar(m) else m.reshape(-1)[own[:, f]]
                out[ax, :, f] = SLOT_SIDE[f] * v * ww
        return out

    def pml_sigma(self):
        """Graded conductivity (3, e, k, j, i) of the PML layers, and their elements."""
        thick, order, err = PML
        nel = self.nel
        e = np.arange(self.nelt)
        ec = (e % nel[0], (e // nel[0]) % nel[1], e // (nel[0] * nel[1]))
        sig = np.zeros((3,) + self.xyz[0].shape)
        inside = np.zeros(self.nelt, dtype=bool)
        for d in range(3):
            if self.bc[d] != WALL["pml"]:
                continue
            width = thick * self.hi[d] / nel[d]
            smax = -(order + 1) * math.log(err) / (2 * width)
            for layer, inner, outer in ((ec[d] < thick, width, 0.0),
                                        (ec[d] >= nel[d] - thick, self.hi[d] - width, self.hi[d])):
                sig[d][layer] = smax * np.clip((self.xyz[d][layer] - inner) / (outer - inner), 0, None) ** order
                inside |= layer
        return sig, inside

    def arrays(self, eps):
        """The reference's arrays, as cem_maxwell_init leaves them."""
        own, part, wall, gid = self.faces()
        cof, jac = self.metrics()
        w3 = self.w[:, None, None] * self.w[None, :, None] * self.w[None, None, :]
        bm = (jac * w3[None] * np.ones((self.nelt, 1, 1, 1))).reshape(-1)
        A = self.face_vectors(cof, own)
        area = np.sqrt((A * A).sum(axis=0))
        Z, Y = 1.0 / np.sqrt(eps), np.sqrt(eps)
        imp = {}
        for nm, q in (("Z", Z), ("Y", Y)):
            mine = q[own]
            total = mine + np.where(part >= 0, q[np.maximum(part, 0)], mine)
            imp[nm + "_0"], imp[nm + "_1"] = 0.5 * total, total - mine
        out = {"dxm1": self.D.T.copy(), "w3mn": w3, "bmn": bm, "xmn": self.xyz[0], "ymn": self.xyz[1],
               "zmn": self.xyz[2], "unxm": A[0] / area, "unym": A[1] / area, "unzm": A[2] / area,
               "aream": area, "ebm1": 1.0 / (eps * bm), "hbm1": 1.0 / bm, "cemface": own,
               "cempec": np.nonzero(wall.reshape(-1) >= 0)[0], "glo_face": gid, **imp}
        for d, r in enumerate("rst"):
            for ax, x in enumerate("xyz"):
                out[r + x + "mn"] = cof[d][ax]
        return {k: np.ascontiguousarray(v).reshape(-1) for k, v in out.items()}


# ---- inputs ------------------------------------------------------------------

def _inputs(c, seed):
    rng = np.random.default_rng(seed)
    m = _Mesh(c)
    x, y, z = (A.reshape(-1) for A in m.xyz)
    L = np.array(m.hi)
    # smooth fields: a few low modes per component (a separable product each)
    F = np.empty((6, m.npts))
    n, nel = m.n, m.nel
    for q in range(6):
        f = 0.0
        for _ in range(2):
            k = rng.integers(1, 4, size=3) * 2 * np.pi / L
            ph = rng.uniform(0, 2 * np.pi, size=3)
            if m.deform:
                f = f + rng.standard_normal() * np.cos(k[0] * x + k[1] * y + k[2] * z + ph[0])
                continue
            l = [np.cos(k[d] * (np.arange(nel[d])[:, None] + 0.5 * (m.z + 1.0)) * (L[d] / nel[d]) + ph[d])
                 for d in range(3)]
            f = f + rng.standard_normal() * (l[2][:, None, None, :, None, None] * l[1][None, :, None, None, :, None]
                                             * l[0][None, None, :, None, None, :]).reshape(-1)
        F[q] = f
    eps = np.ones(m.npts)
    if c["eps"] == "sphere":
        ctr = L * rng.uniform(0.45, 0.55, size=3)
        eps[(x - ctr[0]) ** 2 + (y - ctr[1]) ** 2 + (z - ctr[2]) ** 2 < (0.25 * L.min()) ** 2] = 4.0
    elif c["eps"] == "smooth":
        p = rng.uniform(0, 2 * np.pi, size=3)
        eps = 2.5 + 0.5 * (np.cos(2 * np.pi * x / L[0] + p[0]) + np.cos(2 * np.pi * y / L[1] + p[1])
                           + np.cos(2 * np.pi * z / L[2] + p[2]))
    pml = WALL["pml"] in m.bc
    if pml:
        eps = np.ones(m.npts)  # the layers absorb into the same medium
        F *= 0.0               # an empty domain, driven by its source
    dt = (0.1 if pml else (0.25 if m.deform else 0.5)) * m.spacing()
    src = None
    if c["source"]:
        src = {"xc": tuple(L * rng.uniform(0.35, 0.65, size=3)), "sigma": 0.08 * float(L.min()), "amp": 1.0,
               "f0": 2.0, "t0": 0.1}
    jw = None
    if c["path"] == "gradient":  # the field energy in a probe box
        w3 = (m.w[:, None, None] * m.w[None, :, None] * m.w[None, None, :]).reshape(-1)
        probe = np.ones(m.npts, dtype=bool)
        for A, h in zip((x, y, z), L):
            probe &= (A > 0.6 * h) & (A < 0.95 * h)
        jw = np.where(probe, np.tile(w3, m.nelt) * m.metrics()[1], 0.0)
    return m, F, eps, dt, src, jw


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t.numpy()


class _State:
    def close(self):
        self.gpu.close()

    def __del__(self):
        self.close()


def prepare(case, seed):
    s = _State()
    m, F, eps, dt, src, jw = _inputs(case, seed)
    uniform = case["eps"] == "one" or WALL["pml"] in m.bc
    if m.deform:
        s.gpu = MaxwellGPU.from_arrays(m.arrays(eps), m.n, m.nelt, form=case["form"])
    else:
        s.gpu = MaxwellGPU.from_box(m.N, m.nel, m.lo, m.hi, m.bc, form=case["form"],
                                    permittivity=None if uniform else eps,
                                    pml=PML if WALL["pml"] in m.bc else None)
    if src is not None:
        s.gpu.set_source(**src)
    s.H0, s.E0 = _pinned(F[:3]), _pinned(F[3:])
    s.H, s.E = _pinned(F[:3]), _pinned(F[3:])
    s.dt, s.steps, s.jw, s.path = dt, case["steps"], jw, case["path"]
    s.aux = np.zeros((3, m.npts)) if WALL["pml"] in m.bc else None
    return s


def _fields(s):
    """The state into the program's own arrays, as userchk takes it."""
    dp = ctypes.POINTER(ctypes.c_double)
    st = nekcem_gb300.load().nekgpu_get_state(s.gpu._h, s.H.ctypes.data_as(dp), s.E.ctypes.data_as(dp),
                                              s.gpu.npts)
    if st:
        raise RuntimeError("nekgpu_get_state: %d" % st)
    return [s.H, s.E]


def run(state):
    s, g = state, state.gpu
    if s.path == "host":
        np.copyto(s.H, s.H0)
        np.copyto(s.E, s.E0)
        for i in range(s.steps):
            g.op_rk_host(s.H, s.E, i * s.dt, s.dt)
        return [s.H, s.E]
    g.set_state(s.H0, s.E0)
    if s.path == "gradient":
        J, grad, _, _ = g.adjoint_gradient(s.steps, 0.0, s.dt, s.jw)
        return [*_fields(s), J, grad]
    if s.aux is not None:
        g.set_array("pmlbn", s.aux)
        g.set_array("pmldn", s.aux)
    g.run(s.steps, 0.0, s.dt)
    return _fields(s)


def work(case):
    n = case["N"] + 1
    npts = case["ex"] * case["ey"] * case["ez"] * n ** 3
    stages = 5 * case["steps"]
    # per node and stage: state and RK register read and written, two
    # inverse-mass coefficients; curved meshes add nine metrics per node
    node = 208.0 + (72.0 if case["deform"] else 0.0)
    deriv = 18 if case["deform"] else 12
    flop = deriv * 2.0 * n + 48.0 + 6.0 / n * 60.0
    if case["path"] == "gradient":
        # forward twice (stage states are recomputed from checkpoints) and one
        # reverse stage: two adjoint fields read and written, the stage's state
        # and register read, coefficients, gradient
        node = 2 * node + 192.0 + 96.0 + 32.0
        flop = 3.5 * flop
    return {"bytes": node * npts * stages, "flops": flop * npts * stages}


# ---- the same scheme in torch FP64 -------------------------------------------

RK_A = (0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
        -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0)
RK_B = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
        1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
        2277821191437.0 / 14882151754819.0)
RK_C = (0.0, 1432997174477.0 / 9575080441755.0, 2526269341429.0 / 6820363962896.0,
        2006345519317.0 / 3224310063776.0, 2802321613138.0 / 2924317926251.0)


class _Exact:
    def __init__(self, m, eps, src):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        self.T, self.m = T, m
        self.D = T(m.D)
        cof, jac = m.metrics()
        self.cof = [[v if np.isscalar(v) else T(v) for v in r] for r in cof]
        w3 = m.w[:, None, None] * m.w[None, :, None] * m.w[None, None, :]
        self.w3 = T(w3)
        self.bm = T(jac * w3[None] * np.ones((m.nelt, 1, 1, 1)))
        own, part, wall, _ = m.faces()
        A = m.face_vectors(cof, own)
        area = np.sqrt((A * A).sum(axis=0))
        self.normal = [T(A[q] / area).reshape(-1) for q in range(3)]
        self.area = T(area).reshape(-1)
        self.own, self.part = T(own).reshape(-1), T(part).reshape(-1)
        self.inner = self.part >= 0
        self.part = self.part.clamp(min=0)
        self.pmlwall = T(wall == WALL["pml"]).reshape(-1)
        self.set_eps(T(eps))
        self.src = src
        if src is not None:
            d2 = sum((A_ - c_) ** 2 for A_, c_ in zip(m.xyz, src["xc"]))
            self.shape = self.bm * T(np.exp(-d2 / (2 * src["sigma"] ** 2)))
        self.pml = None
        if WALL["pml"] in m.bc:
            sig, inside = m.pml_sigma()
            self.pml = T(sig), T(inside)

    def set_eps(self, eps):
        """Impedance factors and inverse mass of a permittivity (mu = 1)."""
        Z, Y = 1.0 / eps.sqrt(), eps.sqrt()
        f = []
        for q, sign in ((Y, -0.5), (Z, 0.5)):
            mine = q[self.own]
            other = torch.where(self.inner, q[self.part], mine)
            total = torch.where(self.pmlwall, mine, mine + other)
            f += [sign * (total - mine) / (0.5 * total), 0.5 / (0.5 * total)]
        self.Y02, self.C02Y, self.Z02, self.C02Z = f
        self.inv = [1.0 / self.bm, 1.0 / (eps.reshape(self.bm.shape) * self.bm)]

    def curl(self, u):
        m, D = self.m, self.D
        g = [[0.0] * 3 for _ in range(3)]  # jac du_q/dx_ax
        for q in range(3):
            ds = (u[q] @ D.T, D @ u[q], (D @ u[q].reshape(m.nelt, m.n, -1)).reshape(u[q].shape))
            for ax in range(3):
                if ax == q:
                    continue
                for d in range(3):
                    c = self.cof[d][ax]
                    if torch.is_tensor(c) or c != 0.0:
                        g[q][ax] = g[q][ax] + ds[d] * c
        return [self.w3 * (g[2][1] - g[1][2]), self.w3 * (g[0][2] - g[2][0]), self.w3 * (g[1][0] - g[0][1])]

    def rhs(self, u, t):
        H, E = u[:3], u[3:]
        res = [-v for v in self.curl(E)] + self.curl(H)
        flat = [v.reshape(-1) for v in u]
        mine = [v[self.own] for v in flat]
        dH = [torch.where(self.inner, flat[q][self.part] - mine[q], 0.0) for q in range(3)]
        dE = [torch.where(self.inner, flat[3 + q][self.part] - mine[3 + q], -2.0 * mine[3 + q]) for q in range(3)]
        n = self.normal

        def cross(a, b):
            return [a[(q + 1) % 3] * b[(q + 2) % 3] - a[(q + 2) % 3] * b[(q + 1) % 3] for q in range(3)]

        nE, nH = cross(n, dE), cross(n, dH)
        fu, fw = cross(n, nH), cross(n, nE)
        out = []
        for q in range(6):
            f = (self.Y02 * nE[q] - self.C02Y * fu[q]) if q < 3 else (self.Z02 * nH[q - 3] - self.C02Z * fw[q - 3])
            out.append(res[q].reshape(-1).index_add(0, self.own, self.area * f).reshape(res[q].shape))
        return out

    def drive(self, res, t):
        if self.src is not None:
            a = math.pi * self.src["f0"] * (t - self.src["t0"])
            res[5] = res[5] + self.shape * (self.src["amp"] * (1 - 2 * a * a) * math.exp(-a * a))
        return res

    def step(self, u, t, dt, aux=None):
        k, ka = [0.0] * 6, [0.0] * 6
        for i in range(5):
            res = self.rhs(u, t)
            if aux is not None:
                s, inside = self.pml
                new = []
                for q in range(6):
                    x, y, z = q % 3, (q + 1) % 3, (q + 2) % 3  # sigma of own, next, previous axis
                    f = aux[q]
                    ra = res[q] / self.bm - s[y] * f
                    res[q] = res[q] + self.bm * ((s[x] - s[y]) * f - s[z] * u[q])
                    ka[q] = RK_A[i] * ka[q] + dt * ra
                    new.append(torch.where(inside[:, None, None, None], f + RK_B[i] * ka[q], 0.0))
                aux = new
            res = self.drive(res, t + dt * RK_C[i])
            k = [RK_A[i] * k[q] + dt * (res[q] * self.inv[q // 3]) for q in range(6)]
            u = [u[q] + RK_B[i] * k[q] for q in range(6)]
        return u, aux


def exact(case, seed):
    m, F, eps, dt, src, jw = _inputs(case, seed)
    X = _Exact(m, eps, src)
    shape = (m.nelt, m.n, m.n, m.n)
    u = [X.T(F[q]).reshape(shape) for q in range(6)]

    def fields(u):
        return [torch.stack([u[q].reshape(-1) for q in r]).detach() for r in ((0, 1, 2), (3, 4, 5))]

    if case["path"] == "gradient":
        from torch.utils.checkpoint import checkpoint
        e = X.T(eps).clone().requires_grad_(True)

        def one(t, e, *u):
            X.set_eps(e)
            return tuple(X.step(list(u), t, dt)[0])

        for i in range(case["steps"]):
            u = checkpoint(one, i * dt, e, *u, use_reentrant=False)
        w = X.T(jw).reshape(shape)
        J = sum((w * u[q] * u[q]).sum() for q in (3, 4, 5))
        J.backward()
        return [*fields(u), J.detach(), e.grad]
    with torch.no_grad():
        aux = [torch.zeros_like(u[0]) for _ in range(6)] if X.pml is not None else None
        for i in range(case["steps"]):
            u, aux = X.step(u, i * dt, dt, aux)
    return fields(u)
