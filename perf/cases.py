"""Timed cases of the QBX-FMM layer-potential apply.

Each case is one call that a program using this package makes over and over: a layer
potential applied to densities on the GPU, a wrangler driven stage by stage, a forward
and backward pass of a loss through the single layer, a batched solve.  The surface, the
targets, the orders and the plan are in hand before the call; a pass starts from densities
in device memory and ends with potentials (or gradients, or solutions) there.

Surfaces: the 5-arm starfish in 2D (16 nodes per element upsampled to 64) and the
ellipsoid (1, 1.5, 2) in 3D (``20 nu^2`` triangles, 15 nodes each upsampled to 45).
``exact`` sums the same QBX expansions over all sources directly in 64 bits (no tree, no
translations), so an apply differs from it by its FMM truncation.
"""

import functools
import math

import numpy as np
import torch


# {{{ the cases

def listed():
    return [
        # the smallest ordinary call: a 2D boundary of 1024 nodes and points to plot at
        dict(name="laplace2d_s_small", call="apply", family="laplace", dim=2, op="S", size=64,
             extra=1000, nrhs=1, q=4, p=10, k=0.0, mixed=False),
        # a 3D double layer of ordinary size, with evaluation points off the surface
        dict(name="laplace3d_d", call="apply", family="laplace", dim=3, op="D", size=8,
             extra=2000, nrhs=1, q=3, p=10, k=0.0, mixed=False),
        # the mixed-precision option on a larger surface
        dict(name="laplace3d_d_mixed", call="apply", family="laplace", dim=3, op="D", size=16,
             extra=2000, nrhs=1, q=3, p=10, k=0.0, mixed=True),
        # a large surface: 307 200 nodes, 921 600 sources
        dict(name="laplace3d_s_large", call="apply", family="laplace", dim=3, op="S", size=32,
             extra=0, nrhs=1, q=4, p=12, k=0.0, mixed=False),
        # the wrangler driven stage by stage, as pytential's driver calls it
        dict(name="laplace3d_s_drive", call="drive", family="laplace", dim=3, op="S", size=7,
             extra=1333, nrhs=1, q=3, p=10, k=0.0, mixed=False),
        # an inverse problem's step: loss at far points, gradients in density and points
        dict(name="laplace3d_gradient_far", call="gradient", family="laplace", dim=3, op="S",
             size=16, extra=5000, nrhs=1, q=4, p=12, k=0.0, mixed=False),
        # the same on the surface itself (every target through QBX): density gradient
        dict(name="laplace3d_gradient_surface", call="gradient", family="laplace", dim=3, op="S",
             size=11, extra=0, nrhs=1, q=4, p=12, k=0.0, mixed=False),
        # scattering in 2D from many incident angles at once: 64 densities
        dict(name="helmholtz2d_bw_64", call="apply", family="helmholtz", dim=2, op="BW", size=2048,
             extra=0, nrhs=64, q=5, p=20, k=20.0, mixed=False),
        # the exterior Dirichlet problem solved for a few incident angles
        dict(name="helmholtz2d_solve", call="solve", family="helmholtz", dim=2, op="BW", size=389,
             extra=0, nrhs=7, q=5, p=20, k=20.0, mixed=False),
        # scattering in 3D from one incident wave, with near-field evaluation points
        dict(name="helmholtz3d_cf_single", call="apply", family="helmholtz", dim=3, op="CF", size=9,
             extra=1500, nrhs=1, q=5, p=15, k=5.0, mixed=False),
        # some incident waves in the other truncation (spherical waves, as pytential's fmmlib
        # backend), on a surface of ordinary size
        dict(name="helmholtz3d_cf_fmmlib", call="apply", family="helmholtz", dim=3, op="CF", size=8,
             extra=0, nrhs=6, q=4, p=13, k=6.0, mixed=False, backend="fmmlib"),
        # 16 incident waves on the largest surface: 307 200 nodes
        dict(name="helmholtz3d_cf_16", call="apply", family="helmholtz", dim=3, op="CF", size=32,
             extra=0, nrhs=16, q=5, p=15, k=10.0, mixed=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["laplace2d", "laplace3d", "laplace3d", "gradient", "drive", "helmholtz2d",
                       "helmholtz2d", "solve", "helmholtz3d", "helmholtz3d"])
    if kind == "laplace2d":
        return dict(call="apply", family="laplace", dim=2, op=rng.choice("SD"),
                    size=_log_int(rng, 48, 4096), extra=_log_int(rng, 100, 20000),
                    nrhs=rng.choice([1, 1, 2, 5]), q=rng.randint(3, 6), p=rng.randint(8, 18),
                    k=0.0, mixed=False)
    if kind in ("laplace3d", "drive"):
        mixed = kind == "laplace3d" and rng.random() < 0.4
        return dict(call="drive" if kind == "drive" else "apply", family="laplace", dim=3,
                    op=rng.choice("SD"), size=_log_int(rng, 4, 14 if kind == "drive" else 24),
                    extra=rng.choice([0, _log_int(rng, 50, 8000)]), nrhs=rng.choice([1, 1, 2, 3]),
                    q=rng.randint(2, 5), p=rng.randint(8, 13), k=0.0, mixed=mixed)
    if kind == "gradient":
        return dict(call="gradient", family="laplace", dim=3, op="S", size=_log_int(rng, 4, 14),
                    extra=rng.choice([0, _log_int(rng, 200, 8000)]), nrhs=1, q=rng.randint(2, 5),
                    p=rng.randint(8, 13), k=0.0, mixed=False)
    if kind == "solve":      # orders that let the residual fall to the solve's tolerance
        return dict(call="solve", family="helmholtz", dim=2, op="BW", size=_log_int(rng, 390, 640),
                    extra=0, nrhs=_log_int(rng, 1, 16), q=5, p=20,
                    k=round(rng.uniform(12.0, 22.0), 2), mixed=False)
    if kind == "helmholtz2d":
        return dict(call="apply", family="helmholtz", dim=2, op=rng.choice(["BW", "S", "D"]),
                    size=_log_int(rng, 150, 2048), extra=rng.choice([0, _log_int(rng, 100, 5000)]),
                    nrhs=_log_int(rng, 1, 64), q=rng.randint(3, 6), p=rng.randint(15, 20),
                    k=round(rng.uniform(5.0, 25.0), 2), mixed=False)
    nrhs, extra = _log_int(rng, 1, 20), rng.choice([0, _log_int(rng, 50, 3000)])
    return dict(call="apply", family="helmholtz", dim=3, op=rng.choice(["CF", "CF", "S", "D"]),
                size=_log_int(rng, 4, 13), extra=extra, nrhs=nrhs, q=rng.randint(3, 5),
                p=rng.randint(10, 16), k=round(rng.uniform(2.0, 5.0 if extra else 10.0), 2), mixed=False,
                backend=rng.choice(["sumpy", "sumpy", "fmmlib"]))

# }}}


# {{{ surfaces

def _lagrange(xs, xt):
    w = np.array([1.0 / np.prod(np.delete(x - xs, j)) for j, x in enumerate(xs)])
    t = w / (xt[:, None] - xs[None, :])
    return t / t.sum(1, keepdims=True)


def _starfish(nel):
    def curve(t):
        r, dr = 1 + 0.25 * np.cos(5 * t), -1.25 * np.sin(5 * t)
        c, s = np.cos(t), np.sin(t)
        dx = np.array([dr * c - r * s, dr * s + r * c])
        sp = np.linalg.norm(dx, axis=0)
        return np.array([r * c, r * s]), np.array([dx[1], -dx[0]]) / sp, sp

    h = np.pi / nel
    out = {}
    for pre, n in (("", 16), ("quad_", 64)):
        x, w = np.polynomial.legendre.leggauss(n)
        t = (2 * h * np.arange(nel)[:, None] + (x + 1) * h).ravel()
        pts, nrm, sp = curve(t)
        out |= {pre + "nodes": pts, pre + "normals": nrm, pre + "weights": np.tile(w, nel) * h * sp}
        if n == 16:
            x16, out["param"] = x, t[:, None]
            out["element_stretch"] = (2 * h * sp).reshape(nel, n).max(1)
    out["upsample"] = _lagrange(x16, x)
    return dict(out, ambient_dim=2, nelements=nel, nodes_per_element=16, quad_nodes_per_element=64)


def _triangles(nu):
    """The icosahedron's faces cut into nu^2 triangles each, on the unit sphere:
    three corner arrays (20 nu^2, 3), counterclockwise seen from outside."""
    g = (1 + 5 ** 0.5) / 2
    v = np.array([(s * a, t * b * g, 0.0) for s in (1, -1) for t in (1, -1) for a, b in [(1, 1)]])
    v = np.concatenate([v, v[:, [2, 0, 1]], v[:, [1, 2, 0]]])
    d = np.linalg.norm(v[:, None] - v[None], axis=2)
    faces = [(i, j, l) for i in range(12) for j in range(i + 1, 12) for l in range(j + 1, 12)
             if max(d[i, j], d[j, l], d[i, l]) < 2.1]
    up = [((i, j), (i + 1, j), (i, j + 1)) for i in range(nu) for j in range(nu - i)]
    down = [((i + 1, j), (i + 1, j + 1), (i, j + 1)) for i in range(nu) for j in range(nu - 1 - i)]
    lat = np.array(up + down, float) / nu                             # (nu^2, 3, 2)
    corners = []
    for i, j, l in faces:
        A, B, C = v[i], v[j], v[l]
        if np.dot(np.cross(B - A, C - A), A) < 0:
            B, C = C, B
        corners.append(A + lat[..., :1] * (B - A) + lat[..., 1:] * (C - A))
    w = np.concatenate(corners)
    w /= np.linalg.norm(w, axis=2, keepdims=True)
    return w[:, 0], w[:, 1], w[:, 2]


def _ellipsoid(nu):
    axes2 = np.array([1.0, 1.5, 2.0]) ** 2
    A, B, C = _triangles(nu)
    nel = len(A)
    lat = [(i, j) for j in range(5) for i in range(5 - j)]
    ref1 = (np.array(lat) + 0.5) / 5.5
    xa, wa = np.polynomial.legendre.leggauss(9)
    xb, wb = np.polynomial.legendre.leggauss(5)
    a, b = np.meshgrid((xa + 1) / 2, (xb + 1) / 2, indexing="ij")
    refq = np.stack([(a * (1 - b)).ravel(), b.ravel()], 1)
    wq = (np.outer(wa / 2, wb / 2) * (1 - b)).ravel()

    def mono(uv):
        return np.stack([uv[:, 0] ** (t - j) * uv[:, 1] ** j for t in range(5) for j in range(t + 1)], 1)

    upsample = mono(refq) @ np.linalg.inv(mono(ref1))
    M = np.linalg.inv(np.array([[2.0, 1.0], [0.0, np.sqrt(3.0)]]))
    out = {}
    for pre, ref, wref in (("", ref1, wq @ upsample), ("quad_", refq, wq)):
        u, v = ref[:, 0][:, None], ref[:, 1][:, None]
        e1, e2 = (B - A)[:, None], (C - A)[:, None]
        w = A[:, None] + u * e1 + v * e2                              # (nel, n, 3)
        wn = np.linalg.norm(w, axis=2, keepdims=True)
        s = w / wn
        rho = np.sqrt((s * s / axes2).sum(2, keepdims=True))
        x, grho = s / rho, s / axes2 / rho

        def dx(dw):
            ds = (dw - s * (s * dw).sum(2, keepdims=True)) / wn
            return ds / rho - s * (grho * ds).sum(2, keepdims=True) / rho ** 2

        xu, xv = dx(e1), dx(e2)
        cr = np.cross(xu, xv)
        area = np.linalg.norm(cr, axis=2, keepdims=True)
        out |= {pre + "nodes": x.reshape(-1, 3).T.copy(),
                pre + "normals": (cr / area).reshape(-1, 3).T.copy(),
                pre + "weights": (wref * area[..., 0]).ravel()}
        if not pre:      # the longest stretch of a side-2 triangle, as a singular value
            ju, jv = xu * M[0, 0] + xv * M[1, 0], xu * M[0, 1] + xv * M[1, 1]
            uu, vv, uv = (ju * ju).sum(2), (jv * jv).sum(2), (ju * jv).sum(2)
            sv = np.sqrt((uu + vv) / 2 + np.sqrt(((uu - vv) / 2) ** 2 + uv ** 2))
            out["element_stretch"] = 2 * sv.max(1)
    return dict(out, ambient_dim=3, nelements=nel, nodes_per_element=15, quad_nodes_per_element=45,
                upsample=upsample, param=np.tile(ref1, (nel, 1)))


@functools.lru_cache(maxsize=None)
def _surface(dim, size):
    return (_starfish if dim == 2 else _ellipsoid)(size)

# }}}


# {{{ inputs made from the seed

def _far_points(rng, dim, n, lo, hi):
    v = rng.normal(size=(dim, n))
    v /= np.linalg.norm(v, axis=0)
    return v * rng.uniform(lo ** dim, hi ** dim, n) ** (1 / dim)


def _coefficients(case):
    """(single-layer coefficient, double-layer coefficient)."""
    k = case["k"]
    return {"S": (1.0, 0.0), "D": (0.0, 1.0), "BW": (-1j * k, 1.0), "CF": (-1j * k, 1.0)}[case["op"]]


def _inputs(case, seed):
    """(surface, [(points, side)], data): the seeded host arrays of one case."""
    rng = np.random.default_rng(seed)
    srf = _surface(case["dim"], case["size"])
    x, dim, nrhs, k = srf["nodes"], case["dim"], case["nrhs"], case["k"]
    if case["call"] == "gradient":
        # targets far from the surface, or the surface's nodes; the field of a few charges
        # inside the ellipsoid is what the potential should match
        pts = _far_points(rng, 3, case["extra"], 3.0, 3.0) if case["extra"] else x
        charges = _far_points(rng, 3, 8, 0.05, 0.5)
        g = (1 / (4 * np.pi * np.linalg.norm(pts[:, :, None] - charges[:, None], axis=0))).sum(1)
        return srf, [(pts, 0 if case["extra"] else 1)], {"density": rng.normal(size=x.shape[1]), "g": g}
    targets = [(x, +1)]
    if case["extra"]:
        if dim == 2:      # a plot's points all over the square, some of them close to the curve
            v = rng.uniform(-2, 2, size=(2, 2 * case["extra"] + 100))
            off = np.abs(np.hypot(*v) - (1 + 0.25 * np.cos(5 * np.arctan2(v[1], v[0]))))
            v = v[:, off > 0.025 * srf["element_stretch"].max()]      # none on the curve itself
            targets.append((v[:, :case["extra"]], 0))
        else:             # a shell around the ellipsoid
            targets.append((_far_points(rng, 3, case["extra"], 2.5, 3.5), 0))
    if case["family"] == "laplace":
        s = x / np.linalg.norm(x, axis=0)
        base = np.cos(3 * srf["param"][:, 0]) if dim == 2 else s[2] * (s[0] ** 2 - s[1] ** 2)
        dens = base + 0.05 * rng.normal(size=(nrhs, x.shape[1]))
    else:                 # incident plane waves on the surface
        dirs = rng.normal(size=(dim, nrhs))
        dens = -np.exp(1j * k * ((dirs / np.linalg.norm(dirs, axis=0)).T @ x))
    return srf, targets, {"density": dens}

# }}}


# {{{ prepare and run

def prepare(case, seed):
    from pytential_b200 import adjoint, fmm
    from pytential_b200.discretization import Discretization
    from pytential_b200.geometry import QBXFMMGeometryData
    srf, targets, data = _inputs(case, seed)
    discr = Discretization(**srf)
    st = {"case": case, "density": torch.from_numpy(np.ascontiguousarray(data["density"])).cuda()}
    precision = fmm.PRECISION_MIXED if case["mixed"] else fmm.PRECISION_FP64
    if case["call"] == "gradient":
        pts, side = targets[0]
        if side:
            st["op"] = adjoint.SingleLayer(discr, pts, case["q"], case["p"], qbx_side=side)
        else:
            st["op"] = adjoint.FarFieldSingleLayer(discr, pts, case["q"], case["p"])
            st["points"] = torch.from_numpy(np.ascontiguousarray(pts)).cuda()
        st["g"] = torch.from_numpy(data["g"]).cuda()
        return st
    cq, cd = _coefficients(case)
    kern = (fmm.LaplaceKernel(case["dim"]) if case["family"] == "laplace"
            else fmm.HelmholtzKernel(case["dim"], case["k"]))
    spec = fmm.SourceKernelSpec(kern, charge_coeff=cq, dipole_coeff=cd)
    geo = QBXFMMGeometryData(discr, targets)
    if case["call"] == "drive":
        st["wrangler"] = fmm.B200QBXExpansionWrangler(
            fmm.B200TreeIndependentDataForWrangler(spec), geo, np.float64, case["q"],
            lambda kernel, kernel_args, tree, level: case["p"], nrhs=case["nrhs"])
        up = torch.from_numpy(np.ascontiguousarray(srf["upsample"])).cuda()
        d = st["density"].reshape(case["nrhs"], srf["nelements"], -1) @ up.T
        st["strengths"] = d.reshape(case["nrhs"], -1) * torch.from_numpy(srf["quad_weights"]).cuda()
    else:
        st["apply"] = fmm.QBXApply(geo, spec, case["q"], case["p"], nrhs=case["nrhs"],
                                   precision=precision, fmm_backend=case.get("backend", "sumpy"))
    return st


def run(st):
    call = st["case"]["call"]
    if call == "apply":
        return st["apply"](st["density"])
    if call == "drive":
        from pytential_b200.fmm import drive_fmm
        return drive_fmm(None, st["wrangler"], [st["strengths"]])
    if call == "solve":
        from pytential_b200.gmres import gmres
        return gmres(st["apply"], st["density"], tol=1e-8, restart=50, maxiter=300).solution
    from pytential_b200.adjoint import single_layer
    sigma = st["density"].clone().requires_grad_(True)
    points = st["points"].clone().requires_grad_(True) if "points" in st else None
    u = single_layer(st["op"], sigma, points)
    (0.5 * ((u - st["g"]) ** 2).sum()).backward()
    out = {"u": u.detach(), "density_grad": sigma.grad}
    if points is not None:
        out["points_grad"] = points.grad
    return out

# }}}


# {{{ work

#: about the iterations that the solve takes over its range
_ITERATIONS = 20


def work(case):
    dim, nrhs, p, q = case["dim"], case["nrhs"], case["p"], case["q"]
    n = case["size"] * 16 if dim == 2 else 300 * case["size"] ** 2      # nodes
    ns = n * (4 if dim == 2 else 3)                                     # sources
    far = case["call"] == "gradient" and case["extra"]
    nt = case["extra"] if far else n + case["extra"]
    val = 16 if case["family"] == "helmholtz" else 8
    cx = val // 8 * (val // 8)                # real products per product of two values
    cf = 2 * p + 1 if dim == 2 else (p + 1) ** 2
    # densities in, potentials out; source positions, normals and weights, target
    # positions and centers once for all densities
    byts = val * nrhs * (n + nt) + 8 * (ns * (2 * dim + 1) + nt * (2 * dim + 1))
    # per source and per target one expansion of the box around it, and per target the
    # sources around it (three leaves of 64 in 2D, nine of 256 in 3D) to order q
    near = 0 if far else n * (192 if dim == 2 else 2304)
    flops = 2 * cx * nrhs * ((ns + nt) * cf + near) + near * (q + 1) * 8
    passes = {"gradient": 2, "solve": _ITERATIONS}.get(case["call"], 1)
    return {"bytes": byts * passes, "flops": flops * passes}

# }}}


# {{{ the values in 64 bits: QBX expansions of every source, summed directly

def _series_mul(a, b):
    return [sum(a[i] * b[n - i] for i in range(n + 1)) for n in range(len(a))]


def _laplace2d(a, b, nb, q):
    """log|b - a| expanded about a = 0 to order q, and its derivative in b along nb."""
    z, t, s = a / b, torch.ones_like(b), torch.ones_like(b)
    lg = torch.log(b.abs())
    for n in range(1, q + 1):
        t = t * z
        lg = lg - t.real / n
        s = s + t
    return lg, (nb / b * s).real


def _laplace3d(a, b, nb, q):
    """1/|b - a| to order q in a: the terms |a|^n |b|^(-n-1) P_n, and their derivative."""
    A, B, S = (a * a).sum(0), (b * b).sum(0), (a * b).sum(0)
    dB, dS = 2 * (b * nb).sum(0), (a * nb).sum(0)
    g, dg = [B ** -0.5], [-0.5 * B ** -1.5 * dB]
    for n in range(1, q + 1):
        t, dt = (2 * n - 1) * S * g[-1], (2 * n - 1) * (dS * g[-1] + S * dg[-1])
        if n > 1:
            t, dt = t - (n - 1) * A * g[-2], dt - (n - 1) * A * dg[-2]
        g.append(t / (n * B))
        dg.append(dt / (n * B) - g[-1] * dB / B)
    return sum(g), sum(dg)


def _helmholtz3d(a, b, nb, q, k):
    """Degree-q Taylor polynomial in a of e^(ikr)/r, r = |b - a|: power series along a."""
    zero = torch.zeros_like(b[0])
    r2 = [(b * b).sum(0), -2 * (a * b).sum(0), (a * a).sum(0) + zero] + [zero] * (q + 1)
    r = [r2[0].sqrt()]
    for n in range(1, q + 1):
        r.append((r2[n] - sum(r[i] * r[n - i] for i in range(1, n))) / (2 * r[0]))
    e = [torch.exp(1j * k * r[0])]
    for n in range(1, q + 1):
        e.append(sum((1j * k * i / n) * r[i] * e[n - i] for i in range(1, n + 1)))
    g = []
    for n in range(q + 1):
        g.append((e[n] - sum(r[i] * g[n - i] for i in range(1, n + 1))) / r[0])
    h = _series_mul(g, [1j * k * r[0] - 1] + [1j * k * x for x in r[1:]])
    h2 = []
    for n in range(q + 1):
        h2.append((h[n] - sum(r2[i] * h2[n - i] for i in range(1, min(n, 2) + 1))) / r2[0])
    d = _series_mul(h2, [(b * nb).sum(0), -(a * nb).sum(0)] + [zero] * (q - 1))
    return sum(g), sum(d[:q + 1])


def _helmholtz3d_waves(a, b, nb, q, k):
    """ik sum (2n + 1) j_n(k|a|) h_n(k|b|) P_n, n <= q, and its derivative in b along nb."""
    la, lb = (a * a).sum(0).sqrt(), (b * b).sum(0).sqrt()
    ah, bh = a / la.clamp(min=1e-300), b / lb
    c, db = (ah * bh).sum(0), (bh * nb).sum(0)
    dc = ((ah * nb).sum(0) - c * db) / lb
    xa, xb = k * la, k * lb
    h = [torch.exp(1j * xb) / (1j * xb)]
    h.append(h[0] * (1 / xb - 1j))
    for n in range(1, q + 1):
        h.append((2 * n + 1) / xb * h[n] - h[n - 1])
    s, d, p, dp = 0, 0, [torch.ones_like(c)], [torch.zeros_like(c)]
    for n in range(q + 1):
        if n:
            p.append(c if n == 1 else ((2 * n - 1) * c * p[-1] - (n - 1) * p[-2]) / n)
            dp.append(n * p[n - 1] + c * dp[-1])
        odd = float(math.prod(range(1, 2 * n + 2, 2)))
        j, t = 0, xa ** n / odd
        for i in range(30):
            j, t = j + t, t * (-xa * xa / 2) / ((i + 1) * (2 * n + 2 * i + 3))
        w = 1j * k * (2 * n + 1) * j
        s = s + w * h[n] * p[n]
        d = d + w * (k * db * (n / xb * h[n] - h[n + 1]) * p[n] + h[n] * dp[n] * dc)
    return s, d


_EULER, _STEP, _TERMS = 0.57721566490153286, 0.5, 30


def _small_hankel(x):
    """H_0 and H_1 by their series about 0, for x <= 1."""
    h, ln = x * x / 4, torch.log(x / 2) + _EULER
    j0, j1, s0, s1 = 0, 0, 0, 0
    for m in range(12):
        har = sum(1 / i for i in range(1, m + 1))
        t = (-1) ** m / math.factorial(m) ** 2 * h ** m
        j0, s0 = j0 + t, s0 - har * t
        t = t * x / (2 * (m + 1))
        j1, s1 = j1 + t, s1 + (2 * har + 1 / (m + 1)) * t
    y0 = (ln * j0 + s0) * 2 / math.pi
    y1 = (2 * ln * j1 - s1 - 2 / x) / math.pi
    return torch.complex(j0, y0), torch.complex(j1, y1)


def _taylor(x, f, df, terms):
    """Taylor coefficients at x of the solution of x f'' + f' + x f = 0."""
    a = [f, df]
    for j in range(terms - 2):
        a.append(-((j + 1) ** 2 * a[j + 1] + x * a[j] + (a[j - 1] if j else 0))
                 / (x * (j + 1) * (j + 2)))
    return a


@functools.lru_cache(maxsize=None)
def _hankel_table(n):
    """Taylor coefficients of H_0 at 1, 1 + _STEP, ...: each from those before it."""
    h0, h1 = _small_hankel(torch.ones(1, dtype=torch.float64))
    f, df, rows = complex(h0), -complex(h1), []
    for i in range(n):
        a = _taylor(1 + i * _STEP, f, df, 80)
        rows.append(a[:_TERMS])
        f = sum(c * _STEP ** j for j, c in enumerate(a))
        df = sum(j * c * _STEP ** (j - 1) for j, c in enumerate(a) if j)
    return torch.tensor(rows, dtype=torch.complex128)


def _hankel(x, n):
    """H_0(x) .. H_n(x)."""
    at = torch.round((x - 1) / _STEP).clamp(min=0)
    tab = _hankel_table(int(at.max()) + 1).to(x.device)
    d, at = x - 1 - at * _STEP, at.long()
    f, df = torch.zeros_like(x, dtype=tab.dtype), torch.zeros_like(x, dtype=tab.dtype)
    for j in range(_TERMS - 1, -1, -1):
        df = df * d + f
        f = f * d + tab[:, j][at]
    h = [torch.where(x < 1, s, t) for s, t in zip(_small_hankel(x.clamp(max=1.0)), (f, -df))]
    for l in range(1, n):
        h.append(2 * l / x * h[l] - h[l - 1])
    return h


def _helmholtz2d(a, b, nb, q, k):
    """H_0(k|b - a|) by Graf's theorem to order q, and its derivative in b along nb."""
    h = _hankel(k * b.abs(), q + 1)
    e = b / b.abs()
    G = {}
    for m, hm in enumerate(h):                       # G_m = H_m(k|b|) e^(i m arg b)
        G[m] = hm * e ** m
        G[-m] = (-1) ** m * hm * e ** -m
    x = k * a.abs()
    ea = torch.where(a.abs() > 0, a / a.abs(), torch.ones_like(a))
    s, d = 0, 0
    for l in range(-q, q + 1):
        n = abs(l)
        j = sum((-1) ** m / (math.factorial(m) * math.factorial(m + n)) * (x / 2) ** (2 * m + n)
                for m in range(25)) * ((-1) ** n if l < 0 else 1)
        c = (-1) ** n * j * ea ** l
        s = s + c * G[-l]
        d = d + c * (0.5 * k) * (nb * G[-l - 1] - nb.conj() * G[-l + 1])
    return s, d


def _block(case, t, c, y, ny):
    """Kernel of the targets t (dim, n) against the sources y (dim, m), (n, m): expanded about
    c where it is not nan, summed as it is where it is."""
    near = ~torch.isnan(c[0])
    a = torch.where(near, t - c, torch.zeros_like(t))
    b0 = torch.where(near, c, t)
    q, k, cq, cd = case["q"], case["k"], *_coefficients(case)
    if case["dim"] == 2:
        a, b = torch.complex(a[0], a[1])[:, None], y[:, None, :] - b0[:, :, None]
        b, nb = torch.complex(b[0], b[1]), torch.complex(ny[0], ny[1])[None]
    else:
        a, b, nb = a[:, :, None], y[:, None, :] - b0[:, :, None], ny[:, None, :]
    if case["family"] == "laplace":
        f = _laplace2d if case["dim"] == 2 else _laplace3d
        s, d = f(a, b, nb, q)
        return (-0.5 / math.pi if case["dim"] == 2 else 0.25 / math.pi) * (cq * s + cd * d)
    f = (_helmholtz2d if case["dim"] == 2 else
         _helmholtz3d_waves if case.get("backend") == "fmmlib" else _helmholtz3d)
    s, d = f(a, b, nb, q, k)
    if case["dim"] == 3 and case.get("backend") == "fmmlib":
        s, d = (torch.where(near[:, None], v, w) for v, w in
                zip((s, d), _helmholtz3d(torch.zeros_like(a), b, nb, 0, k)))
    return (0.25j if case["dim"] == 2 else 0.25 / math.pi) * (cq * s + cd * d)


def _distances(x, y):
    return torch.cdist(x.T.contiguous(), y.T.contiguous(), compute_mode="donot_use_mm_for_euclid_dist")


def _centers(case, srf, targets, dev):
    """Points and, for each, the center of its expansion (nan: summed as it is)."""
    def on(x):
        return torch.from_numpy(np.ascontiguousarray(x)).to(dev)
    rad = 0.5 * (0.5 if case["dim"] == 3 else 1.0) * on(srf["element_stretch"])
    r1, rq = (rad.repeat_interleave(srf[n]) for n in ("nodes_per_element", "quad_nodes_per_element"))
    x, nrm, src = on(srf["nodes"]), on(srf["normals"]), on(srf["quad_nodes"])
    pts, ctr = [], []
    for p, side in targets:
        p = on(p)
        for i in range(0, p.shape[1], 512):
            t = p[:, i:i + 512]
            sides = (side,) if side else (-1, 1)
            close = (torch.ones_like(t[0], dtype=torch.bool) if side else
                     (_distances(t, src) <= 0.5 * rq).any(1))
            best, dist = torch.full_like(t, math.nan), torch.full_like(t[0], math.inf)
            for s in sides:                          # interior first: it wins ties
                cs = x + s * r1 * nrm
                d = _distances(t, cs)
                rel, j = (d / (r1 * (1 + 1e3 * 2.0 ** -52))).min(1)
                d = d.gather(1, j[:, None])[:, 0]
                take = close & (rel <= 1) & (d < dist)
                best, dist = torch.where(take, cs[:, j], best), torch.where(take, d, dist)
            pts.append(t)
            ctr.append(best)
    return torch.cat(pts, 1), torch.cat(ctr, 1)


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    srf, targets, data = _inputs(case, seed)
    if case["dim"] == 3 and case["size"] > (12 if case["family"] == "helmholtz" else 24):
        return None                                  # pairs of every node and source: too many
    if case["call"] == "solve":
        # the iteration's own: it leaves what the matrix nearly annihilates out of the solution
        return None
    t, c = _centers(case, srf, targets, dev)
    y, ny, w, U = (torch.from_numpy(np.ascontiguousarray(srf[n])).to(dev)
                   for n in ("quad_nodes", "quad_normals", "quad_weights", "upsample"))
    ns = y.shape[1]
    rows = max(1, (1 << 23) // ns)
    blocks = [(i, min(i + rows, t.shape[1])) for i in range(0, t.shape[1], rows)]

    def kernel(i, j):
        return _block(case, t[:, i:j], c[:, i:j], y, ny)

    dens = torch.from_numpy(np.ascontiguousarray(data["density"])).to(dev)
    lead = dens.reshape(-1, srf["nelements"], srf["nodes_per_element"])
    Uc = U.to(dens.dtype)
    strengths = (lead @ Uc.T).reshape(lead.shape[0], ns) * w
    u = torch.cat([kernel(i, j) @ strengths.T for i, j in blocks]).T
    if case["call"] != "gradient":
        return u
    u = u[0]
    res = u - torch.from_numpy(data["g"]).to(dev)
    back = sum(res[i:j] @ kernel(i, j) for i, j in blocks) * w
    out = {"u": u, "density_grad": (back.reshape(srf["nelements"], -1) @ U).reshape(-1)}
    if case["extra"]:
        grad = []
        for i, j in blocks:
            b = t[:, i:j, None] - y[:, None, :]
            f = -strengths[0] * (b * b).sum(0) ** -1.5 / (4 * math.pi)
            grad.append((b * f).sum(2))
        out["points_grad"] = res * torch.cat(grad, 1)
    return out

# }}}
