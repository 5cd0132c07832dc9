"""The calls that users of this framework make, as timed cases.

A case names a public entry point and its sizes; `prepare` makes what a program holds before
the call (bodies, operands, handles) from a seed, `run` is one call, `work` its unavoidable
bytes and operations, and `exact` the same outputs in 64 bits from plain torch.  Complex
matrices on the device are column-major for the library, so a torch tensor of one is its
transpose; `exact` returns them in that layout.
"""
import ctypes
import math
from fractions import Fraction

import numpy as np
import torch
import torch.autograd.forward_ad as fwad

import __graft_entry__

mh = __graft_entry__.load_package()

RHO, G = 1025.0, 9.81
SIX = ("Surge", "Sway", "Heave", "Roll", "Pitch", "Yaw")
PREC = {"fp64": 0, "mixed": 1, "fp64_tc": 2}


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def listed():
    return [
        # a single frequency of the 200-panel hemisphere, heave and one heading, every option at
        # its default: the first call anyone makes, and an optimiser's inner loop on a coarse mesh
        {"name": "one-frequency", "kind": "sweep", "shape": "hemisphere", "panels": 200, "omegas": 1, "dofs": 1,
         "headings": 1, "direct": True, "wave": "Wu", "precision": "fp64"},
        # a small design sweep of a coarse barge by the indirect method with several headings
        {"name": "coarse-sweep", "kind": "sweep", "shape": "barge", "panels": 430, "omegas": 12, "dofs": 3,
         "headings": 4, "direct": False, "wave": "Wu", "precision": "mixed"},
        # the default formulation (plain FP64) on a mesh of ordinary size, all rigid dofs
        {"name": "default-sweep", "kind": "sweep", "shape": "cylinder", "panels": 1000, "omegas": 5, "dofs": 6,
         "headings": 1, "direct": True, "wave": "Wu", "precision": "fp64"},
        # the benchmark's frequency sweep: 2000-panel truncated cylinder, 30 frequencies, 6 dofs and
        # one heading, the LU's update on the tensor cores
        {"name": "cylinder-sweep", "kind": "sweep", "shape": "cylinder", "panels": 2000, "omegas": 30, "dofs": 6,
         "headings": 1, "direct": True, "wave": "Wu", "precision": "fp64_tc"},
        # the exact Guevel-Delhommeau term in a sweep, indirect (what forward speed needs)
        {"name": "exact-sweep", "kind": "sweep", "shape": "cylinder", "panels": 640, "omegas": 3, "dofs": 3,
         "headings": 2, "direct": False, "wave": "ExactGuevelDelhommeau", "precision": "fp64_tc"},
        # the 8000-panel barge of the learned-surrogate benchmark (4 of its 40 frequencies)
        {"name": "large-barge", "kind": "sweep", "shape": "barge", "panels": 8000, "omegas": 4, "dofs": 3,
         "headings": 1, "direct": True, "wave": "Surrogate", "precision": "mixed"},
        # many bodies of uneven size at many frequencies, heave and pitch radiation, one graph
        {"name": "bodies-batch", "kind": "batch", "bodies": 10, "low": 300, "high": 2400, "omegas": 8,
         "direct": True, "precision": "mixed"},
        # gradient of the summed heave added mass and damping of two cylinders with respect to
        # every mesh vertex (a shape-optimisation step)
        {"name": "shape-gradient", "kind": "gradient", "panels": 1400, "omegas": 4, "wave": "Wu",
         "direct": True, "precision": "mixed"},
        # coefficients with their derivative in the wave frequency (FP64 only)
        {"name": "frequency-derivative", "kind": "derivative", "shape": "hemisphere", "panels": 450, "omegas": 3,
         "dofs": 2, "headings": 1, "direct": True, "wave": "Wu"},
        # S and D into a caller's device buffers, stream-ordered (a program with its own memory pool)
        {"name": "assemble-wu", "kind": "assemble", "shape": "barge", "panels": 1750, "direct": True, "wave": "Wu"},
        # S and D of the exact term into device buffers
        {"name": "assemble-exact", "kind": "assemble", "shape": "hemisphere", "panels": 900, "direct": True,
         "wave": "ExactGuevelDelhommeau"},
        # a dense complex solve of device operands (the linear solve of a user's own pipeline)
        {"name": "linsolve", "kind": "linsolve", "n": 2999, "rhs": 9, "precision": "fp64_tc"},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("sweep", "sweep", "sweep", "batch", "gradient", "derivative", "assemble", "linsolve"))
    shape = rng.choice(("hemisphere", "cylinder", "barge"))
    direct = rng.random() < 0.6
    if kind == "sweep":
        wave = rng.choice(("Wu", "Wu", "Wu", "ExactGuevelDelhommeau", "Surrogate"))
        precision = rng.choice(("fp64", "mixed", "fp64_tc")) if wave != "Surrogate" else "mixed"
        high = {"Wu": {"fp64": 1400, "mixed": 4000, "fp64_tc": 3000}[precision], "ExactGuevelDelhommeau": 800,
                "Surrogate": 6000}[wave]
        panels = _log(rng, 60, high)
        omegas = _log(rng, 1, max(1, min(32, int(3e4 / panels), int((high / panels) ** 3 * 2))))
        return {"kind": kind, "shape": shape, "panels": panels, "omegas": omegas, "dofs": rng.randint(1, 6),
                "headings": rng.randint(1, 5), "direct": direct, "wave": wave, "precision": precision}
    if kind == "batch":
        low = _log(rng, 100, 400)
        return {"kind": kind, "bodies": rng.randint(3, 10), "low": low, "high": _log(rng, 600, 2400),
                "omegas": rng.randint(2, 8), "direct": direct, "precision": rng.choice(("mixed", "fp64_tc"))}
    if kind == "gradient":
        return {"kind": kind, "panels": _log(rng, 120, 1400), "omegas": rng.randint(1, 4),
                "wave": "Wu", "direct": direct, "precision": rng.choice(("mixed", "fp64_tc"))}
    if kind == "derivative":
        return {"kind": kind, "shape": shape, "panels": _log(rng, 60, 900), "omegas": rng.randint(1, 4),
                "dofs": rng.randint(1, 6), "headings": rng.randint(1, 3), "direct": direct, "wave": "Wu"}
    if kind == "assemble":
        wave = rng.choice(("Wu", "ExactGuevelDelhommeau"))
        return {"kind": kind, "shape": shape, "panels": _log(rng, 60, 3000 if wave == "Wu" else 900),
                "direct": direct, "wave": wave}
    precision = rng.choice(("fp64", "mixed", "fp64_tc"))
    return {"kind": kind, "n": _log(rng, 30, 1500 if precision == "fp64" else 4000), "rhs": _log(rng, 1, 24),
            "precision": precision}


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _mesh(shape, panels, rng, x0=0.0):
    """A body's mesh: the resolution follows from `panels`, the dimensions from the seed."""
    s = rng.uniform(0.85, 1.15, 3)
    if shape == "hemisphere":
        return mh.hemisphere_mesh(2.0 * s[0], *mh.meshes.hemisphere_resolution(panels), center=(x0, 0.0, 0.0))
    if shape == "cylinder":
        return mh.vertical_cylinder_mesh(5.0 * s[0], 10.0 * s[1], *mh.meshes.cylinder_resolution(5.0, 10.0, panels),
                                         center=(x0, 0.0))
    return mh.barge_mesh(60.0 * s[0], 12.0 * s[1], 6.0 * s[2], *mh.meshes.barge_resolution(60.0, 12.0, 6.0, panels))


def _panels(shape, panels):
    if shape == "hemisphere":
        a, b = mh.meshes.hemisphere_resolution(panels)
        return a * b
    if shape == "cylinder":
        t, z, r = mh.meshes.cylinder_resolution(5.0, 10.0, panels)
        return t * (z + r)
    a, b, d = mh.meshes.barge_resolution(60.0, 12.0, 6.0, panels)
    return a * b + 2 * a * d + 2 * b * d


def _omegas(rng, count, low=0.25, high=2.8):
    step = (high - low) / count
    return low + step * (np.arange(count) + rng.uniform(0.1, 0.9, count))


def _formulation(case):
    greens = mh.default_greens_functions(case["wave"]) if "wave" in case else None
    make = mh.DirectBEM if case["direct"] else mh.IndirectBEM
    return make(greens, precision=case.get("precision", "fp64"))


def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 20260])
    kind = case["kind"]
    s = {"case": dict(case)}
    if kind in ("sweep", "derivative"):
        mesh = _mesh(case["shape"], case["panels"], rng)
        names = ["Heave"] if case["dofs"] == 1 else list(SIX[:case["dofs"]])
        s["body"] = mh.FloatingBody(mesh, names)
        s["params"] = {"wave_frequencies": _omegas(rng, case["omegas"]), "radiating_dofs": names,
                       "influenced_dofs": names, "wave_directions": list(rng.uniform(0.0, 3.0, case["headings"])),
                       "rho": RHO, "g": G}
        s["formulation"] = _formulation(case)
        if case["wave"] == "Surrogate":
            mh.load_surrogate()
    elif kind == "batch":
        # sizes spread over [low, high] whatever the seed, kinds in turn; the context that holds
        # the captured graph is kept, as the batch call is made to be replayed
        shapes = ("hemisphere", "cylinder", "barge")
        s["bodies"] = []
        for b, n in enumerate(_batch_sizes(case)):
            s["bodies"].append(mh.FloatingBody(_mesh(shapes[b % 3], n, rng), ["Heave", "Pitch"]))
        s["params"] = [{"wave_frequencies": np.exp(np.sort(rng.uniform(math.log(0.3), math.log(2.5), case["omegas"]))),
                        "radiating_dofs": ["Heave", "Pitch"], "rho": RHO, "g": G} for _ in s["bodies"]]
        s["formulation"] = _formulation(case)
        s["ctx"] = mh.Context(0)
    elif kind == "gradient":
        t, z, r = mh.meshes.cylinder_resolution(3.0, 6.0, case["panels"] // 2)
        a = rng.uniform(0.9, 1.1, 4)
        one = mh.FloatingBody(mh.vertical_cylinder_mesh(3.0 * a[0], 6.0 * a[1], t, z, r), ["Heave"], body_name="a")
        two = mh.FloatingBody(mh.vertical_cylinder_mesh(3.0 * a[2], 6.0 * a[3], t, z, r, center=(30.0, 0.0)),
                              ["Heave"], body_name="b")
        s["body"] = one + two
        s["omegas"] = _omegas(rng, case["omegas"], 0.4, 2.0)
        s["formulation"] = _formulation(case)
    elif kind == "assemble":
        s["mesh"] = mesh = _mesh(case["shape"], case["panels"], rng)
        s["k"] = float(rng.uniform(0.05, 0.6))
        dev = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).cuda()  # noqa: E731
        s["V"], s["C"], s["N"] = dev(mesh.panel_vertices), dev(mesh.centers), dev(mesh.normals)
        s["A"], s["R"] = dev(mesh.areas), dev(mesh.radii)
        s["S"] = torch.empty((mesh.nfaces, mesh.nfaces), dtype=torch.complex128, device="cuda")
        s["D"] = torch.empty_like(s["S"])
        s["gfs"] = mh.gf_flags(mh.default_greens_functions(case["wave"]))
        s["ctx"] = mh.default_context(0)
        if case["wave"] != "Wu":
            s["handle"] = mesh.device_mesh(s["ctx"])
    else:
        n, m = case["n"], case["rhs"]
        gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)
        rand = lambda *d: torch.view_as_complex(torch.randn(*d, 2, dtype=torch.float64, device="cuda", generator=gen))  # noqa: E731
        # a second-kind boundary operator: half the identity, a kernel that decays along the
        # surface, and an unsymmetric remainder
        x = torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=gen)
        dist = torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist") + 0.05
        A = torch.exp(1j * 4.0 * dist) / dist * (0.6 / n) + rand(n, n) * (0.2 / math.sqrt(n))
        A += 0.5 * torch.eye(n, dtype=torch.complex128, device="cuda")
        s["A"], s["B"] = A, rand(m, n)
        s["X"] = torch.empty_like(s["B"])
        s["ctx"] = mh.default_context(0)
    torch.cuda.synchronize()
    return s


def _batch_sizes(case):
    b = case["bodies"]
    r = (case["high"] / case["low"]) ** (1.0 / max(1, b - 1))
    return [int(round(case["low"] * r ** q)) for q in range(b)]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "sweep":
        return mh.hydrodynamic_coefficients(s["body"], s["params"], s["formulation"])
    if kind == "derivative":
        return mh.hydrodynamic_coefficients_derivative(s["body"], s["params"], s["formulation"])
    if kind == "batch":
        res = mh.batch_hydrodynamic_coefficients(s["bodies"], s["params"], s["formulation"], ctx=s["ctx"])
        return [{"added_mass": r["added_mass"], "radiation_damping": r["radiation_damping"]} for r in res]
    if kind == "gradient":
        return mh.hydro_gradient(s["body"], s["omegas"], list(s["body"].dofs), s["formulation"], rho=RHO, g=G)
    L, ctx = mh.load_library(), s["ctx"]
    if kind == "assemble" and case["wave"] == "Wu":
        rc = L.mh_assemble_matrices_noalloc(torch.cuda.current_stream().cuda_stream, s["mesh"].nfaces,
                                            s["V"].data_ptr(), s["C"].data_ptr(), s["N"].data_ptr(),
                                            s["A"].data_ptr(), s["R"].data_ptr(), s["k"], s["gfs"],
                                            int(case["direct"]), 1, None, s["S"].data_ptr(), s["D"].data_ptr())
        ctx.check(rc, "assemble")
        return s["S"], s["D"]
    if kind == "assemble":
        ctx.check(L.mh_assemble_matrices(ctx.handle, s["handle"].handle, s["k"], s["gfs"], int(case["direct"]), 1,
                                         None, ctypes.c_void_p(s["S"].data_ptr()), ctypes.c_void_p(s["D"].data_ptr()),
                                         1), "assemble")
        return s["S"], s["D"]
    ctx.check(L.mh_linsolve(ctx.handle, case["n"], case["rhs"], s["A"].data_ptr(), s["B"].data_ptr(),
                            s["X"].data_ptr(), PREC[case["precision"]], 1), "linsolve")
    return s["X"]


# ---------------------------------------------------------------------------------------
# the work of one call: what any implementation reads, writes and computes
# ---------------------------------------------------------------------------------------
def _wave_flops(case):
    # per unordered pair: fits, Bessel and elementary functions of the wave term, two entries
    return 300.0


def work(case):
    kind = case["kind"]
    if kind in ("sweep", "derivative"):
        n, w = _panels(case["shape"], case["panels"]), case["omegas"]
        m = case["dofs"] + case["headings"]
        flops = w * (8 / 3 * n ** 3 + 16.0 * n * n * m + n * n / 2 * _wave_flops(case)) + 200.0 * n * n
        if kind == "derivative":
            flops += w * n * n * (24.0 * m + _wave_flops(case) / 2)
        return {"bytes": 8.0 * n * (20 + 3 * case["dofs"]) + 16.0 * w * case["dofs"] * m, "flops": flops}
    if kind == "batch":
        shapes = ("hemisphere", "cylinder", "barge")
        sizes = [_panels(shapes[b % 3], p) for b, p in enumerate(_batch_sizes(case))]
        w = case["omegas"]
        flops = sum(w * (8 / 3 * n ** 3 + 32.0 * n * n + n * n / 2 * _wave_flops(case)) + 200.0 * n * n for n in sizes)
        return {"bytes": sum(8.0 * n * 26 for n in sizes) + 64.0 * w * len(sizes), "flops": flops}
    if kind == "gradient":
        t, z, r = mh.meshes.cylinder_resolution(3.0, 6.0, case["panels"] // 2)
        n, w = 2 * t * (z + r), case["omegas"]
        flops = w * (8 / 3 * n ** 3 + 16.0 * n * n * 6 + n * n / 2 * _wave_flops(case) * 3) + 1000.0 * n * n
        return {"bytes": 8.0 * n * 26 + 24.0 * n, "flops": flops}
    if kind == "assemble":
        n = _panels(case["shape"], case["panels"])
        return {"bytes": 8.0 * 20 * n + 32.0 * n * n, "flops": n * n / 2 * _wave_flops(case) + 200.0 * n * n}
    n, m = case["n"], case["rhs"]
    return {"bytes": 16.0 * n * n + 32.0 * n * m, "flops": 8 / 3 * n ** 3 + 8.0 * n * n * m}


# ---------------------------------------------------------------------------------------
# the same outputs in 64 bits, from plain torch
# ---------------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if case.get("wave") == "Surrogate":
        return None  # a trained network's values, not a formula's
    s = prepare(case, seed)
    if kind == "linsolve":
        return torch.linalg.solve(s["A"].T, s["B"].T).T.contiguous()
    if kind == "assemble":
        S, D = _Influence(s["mesh"], case["direct"], case["wave"]).at(s["k"])
        return S.T.contiguous(), D.T.contiguous()
    if kind == "sweep":
        return _coefficients(s["body"], s["params"], case["direct"], case["wave"])
    if kind == "batch":
        out = []
        for body, p in zip(s["bodies"], s["params"]):
            r = _coefficients(body, {**p, "influenced_dofs": ["Heave", "Pitch"], "wave_directions": []},
                              case["direct"], "Wu")
            out.append({"added_mass": r["added_mass"], "radiation_damping": r["radiation_damping"]})
        return out
    if kind == "derivative":
        return _with_derivative(s["body"], s["params"], case["direct"], case["wave"])
    names = list(s["body"].dofs)
    r = _coefficients(s["body"], {"wave_frequencies": s["omegas"], "radiating_dofs": names, "influenced_dofs": names,
                                  "wave_directions": []}, case["direct"], case["wave"])
    J = sum(float((r[key][h, h]).sum()) for h in range(len(names)) for key in ("added_mass", "radiation_damping"))
    return J, None


def _t(x):
    return torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).cuda()


class _Influence:
    """S and D of a mesh at any wavenumber (Rankine, its image, and one wave term)."""

    def __init__(self, mesh, direct, wave):
        self.direct, self.wave, self.n = direct, wave, mesh.nfaces
        self.c, self.nrm, self.area = _t(mesh.centers), _t(mesh.normals), _t(mesh.areas)
        self.S0, self.D0 = self._static(_t(mesh.panel_vertices), _t(mesh.radii))
        self.dx = self.c[:, None, :2] - self.c[None, :, :2]  # field - source
        self.h = torch.sqrt(self.dx[..., 0] ** 2 + self.dx[..., 1] ** 2)
        self.z = self.c[:, None, 2] + self.c[None, :, 2]

    def _static(self, V, radius):
        # panel frames: s along the mid-edge line, n normal, origin at the area centroid
        mid = (V + V.roll(-1, 1)) / 2
        org = (mid[:, 1] + mid[:, 3]) / 2
        unit = lambda v: v / v.norm(dim=-1, keepdim=True)  # noqa: E731
        s = unit(mid[:, 1] - mid[:, 3])
        n = unit(torch.linalg.cross(s, mid[:, 2] - mid[:, 0]))
        t = unit(torch.linalg.cross(n, s))
        d = V - org[:, None]
        x, y = (d * s[:, None]).sum(-1), (d * t[:, None]).sum(-1)
        x1, y1 = x.roll(-1, 1), y.roll(-1, 1)
        area = ((y1 - y) * (x + x1) / 2).sum(1)
        cx = ((y1 - y) * (x * x + x * x1 + x1 * x1) / 6).sum(1) / area
        cy = -((x1 - x) * (y * y + y * y1 + y1 * y1) / 6).sum(1) / area
        org = org + cx[:, None] * s + cy[:, None] * t
        lx, ly = x - cx[:, None], y - cy[:, None]
        S = torch.zeros(self.n, self.n, dtype=torch.float64, device="cuda")
        D = torch.zeros_like(S)
        for image in (False, True):
            p = self.c * torch.tensor([1.0, 1.0, -1.0 if image else 1.0], dtype=torch.float64, device="cuda")
            phi, g = self._panel(p, s, t, n, org, lx, ly, radius, image)
            if self.direct:
                d = (g * self.nrm[None]).sum(-1)
            else:
                g = -g
                if image:
                    g[..., 2] = -g[..., 2]
                d = (g * self.nrm[:, None]).sum(-1)
            S += phi
            D += d
        S, D = -S / (4 * math.pi), -D / (4 * math.pi)
        return S, D + 0.5 * torch.eye(self.n, dtype=torch.float64, device="cuda")

    def _panel(self, p, s, t, n, org, lx, ly, radius, image):
        """Integral of 1/r over every panel seen from every point, and its source gradient."""
        rb = p[:, None] - self.c[None]
        r = rb.norm(dim=-1)
        far = r > 7 * radius[None]
        rr = torch.where(far, r, torch.ones_like(r))
        phi_far = self.area[None] / rr
        g_far = rb * (self.area[None] / rr ** 3)[..., None]
        d = p[:, None] - org[None]
        fx, fy, fz = ((d * a[None]).sum(-1) for a in (s, t, n))
        if not image:
            fz.fill_diagonal_(0.0)  # a flat panel's own centre lies in its plane
        plane = fz.abs() <= 1e-14
        s0 = torch.zeros_like(r)
        s1, s2, s3 = (torch.zeros_like(r) for _ in range(3))
        for k in range(4):
            q = (k + 1) & 3
            dx, dy = (lx[:, q] - lx[:, k])[None], (ly[:, q] - ly[:, k])[None]
            edge = torch.hypot(dx, dy)
            ok = (edge > 1e-14).expand_as(r)
            ex = [fx - lx[None, :, j] for j in (k, q)]
            ey = [fy - ly[None, :, j] for j in (k, q)]
            rk = [torch.sqrt(a * a + b * b + fz * fz) for a, b in zip(ex, ey)]
            rs = rk[0] + rk[1]
            lt = torch.where(ok, torch.log((rs - edge) / (rs + edge)) / torch.where(edge > 1e-14, edge, 1.0), 0.0)
            at = []
            for a, b, rad in zip(ex, ey, rk):
                num, den = dy * (a * a + fz * fz) - dx * (a * b), dx * fz * rad
                at.append(torch.atan2(torch.where(den < 0, -num, num), den.abs()))
            vz = torch.where(plane | ~ok, 0.0, at[0] - at[1])
            s0 += (ex[0] * dy - ey[0] * dx) * lt + fz * vz
            s1 += dy * lt
            s2 -= dx * lt
            s3 += vz
        g_near = -(s1[..., None] * s[None] + s2[..., None] * t[None] + s3[..., None] * n[None])
        return torch.where(far, phi_far, s0), torch.where(far[..., None], g_far, g_near)

    def at(self, k):
        hh, vv = k * self.h, k * self.z
        val, dh, dv = (_wu if self.wave == "Wu" else _delhommeau)(hh, vv)
        sgn = -1.0 if self.direct else 1.0  # gradient in the source (direct) or the field point
        a = torch.where(hh > 1e-6, k * k / torch.where(hh > 1e-6, hh, 1.0), 0.0) * sgn * k
        nrm = self.nrm[None] if self.direct else self.nrm[:, None]
        proj = (nrm[..., 0] * self.dx[..., 0] + nrm[..., 1] * self.dx[..., 1]) * a
        w = -self.area[None] / (4 * math.pi)
        S = self.S0 + w * k * val
        D = self.D0 + w * (proj * dh + nrm[..., 2] * (k * k) * dv)
        return S, D


def _cheb(coeffs):
    """Chebyshev coefficients on [0, 1] of the polynomial with these power coefficients."""
    a = [Fraction(c) for c in coeffs]
    n = len(a)
    p = [Fraction(0)] * n  # powers of t = 2 rho - 1
    for i, c in enumerate(a):
        for j in range(i + 1):
            p[j] += c * math.comb(i, j) / 2 ** i
    out = [Fraction(0)] * n
    for i, c in enumerate(p):  # t^i = 2^(1-i) sum_j C(i, j) T_(i-2j), the T_0 term halved
        for j in range(i // 2 + 1):
            w = Fraction(math.comb(i, j) * 2, 2 ** i)
            out[i - 2 * j] += c * (w / 2 if i == 2 * j else w)
    return [float(c) for c in out]


_FITS = {
    "A": _cheb([1.21, -13.328, 215.896, -1763.96, 8418.94, -24314.21, 42002.57, -41592.9, 21859.0, -4838.6]),
    "B": _cheb([0.938, 5.737, -67.92, 796.534, -4780.77, 17137.74, -36618.81, 44894.06, -29030.24, 7671.22]),
    "C": _cheb([1.268, -9.747, 209.653, -1397.89, 5155.67, -9844.35, 9136.4, -3272.62]),
    "D": _cheb([0.632, -40.97, 667.16, -6072.07, 31127.39, -96293.05, 181856.75, -205690.43, 128170.2, -33744.6]),
    "dA": _cheb([2.948, -24.53, 249.69, -754.85, -1187.71, 16370.75, -48811.41, 68220.87, -46688.0, 12622.25]),
    "dB": _cheb([1.11, 2.894, -76.765, 1565.35, -11336.19, 44270.15, -97014.11, 118879.26, -76209.82, 19923.28]),
    "dC": _cheb([14.19, -148.24, 847.8, -2318.58, 3168.35, -1590.27]),
}


def _fit(name, rho):
    t = 2.0 * (2.0 * rho - 1.0)
    b1 = b2 = torch.zeros_like(rho)
    c = _FITS[name]
    for v in reversed(c[1:]):
        b1, b2 = v + t * b1 - b2, b1
    return c[0] + t / 2 * b1 - b2


def _poly(c, x):
    v = torch.full_like(x, c[-1])
    for a in reversed(c[:-1]):
        v = v * x + a
    return v


_NODES = [tuple(_x) for _x in zip(*np.polynomial.legendre.leggauss(40))]


class _Bessel(torch.autograd.Function):
    """J0, J1, Y0, Y1 of _bessel with their forward-mode derivatives."""

    @staticmethod
    def forward(ctx, x):
        out = _bessel(x)[:4]
        ctx.save_for_forward(x, *out)
        return out

    @staticmethod
    def jvp(ctx, dx):
        x, J0, J1, Y0, Y1 = ctx.saved_tensors
        return -J1 * dx, (J0 - J1 / x) * dx, -Y1 * dx, (Y0 - Y1 / x) * dx


def _bessel(x):
    """J0, J1, Y0, Y1, H0 and H0' of x > 0 in 64 bits (torch's own hold 32 bits above x = 5):
    J and Struve's H0 from their integrals over an angle, Y0 above x = 4 from
    H0 - Y0 = (2 / pi) int_0^inf e^-u / sqrt(x^2 + u^2) du."""
    top = float(x.max())
    n = int(top / 2) + 24
    J0, J1, H0, H0d, P, Q = (torch.zeros_like(x) for _ in range(6))
    for q in range(n):  # the midpoint rule converges exponentially on these periodic integrands
        cs = math.cos(math.pi / 2 * (q + 0.5) / n)
        J0 += torch.cos(x * cs) / n
        J1 += torch.sin(x * cs) * cs / n
    cells = max(1, int(math.ceil(top / 25)))
    for c in range(cells):
        for t, w in _NODES:
            cs = math.cos(math.pi / 2 * (c + (t + 1) / 2) / cells)
            H0 += w / (2 * cells) * torch.sin(x * cs)
            H0d += w / (2 * cells) * torch.cos(x * cs) * cs
    xb = torch.clamp(x, min=4.0)
    for c in range(4):
        for t, w in _NODES:
            u = 10 * (c + (t + 1) / 2)
            s = torch.rsqrt(xb * xb + u * u)
            P += (5 * w * math.exp(-u)) * s
            Q += (5 * w * math.exp(-u)) * s ** 3
    low = x <= 4.0
    xl = torch.where(low, x, 1.0)
    Y0 = torch.where(low, torch.special.bessel_y0(xl), H0 - 2 / math.pi * P)
    Y1 = torch.where(low, torch.special.bessel_y1(xl), -H0d - 2 / math.pi * xb * Q)
    return J0, J1, Y0, Y1, H0, H0d


def _wu(h, v):
    """The wave term of Wu et al. by its published fits, and its derivatives in h and v."""
    d = torch.sqrt(h * h + v * v)
    alpha, beta, rho, ev = -v / d, h / d, d / (1 + d), torch.exp(v)
    J0, J1, Y0, Y1 = _Bessel.apply(torch.clamp(h, min=1e-30))
    low = h <= 3.0
    y = (h / 3.0) ** 2
    H0 = _poly([1.909859164, -1.909855001, 0.687514637, -0.126164557, 0.013828813, -0.000876918], y) * (h / 3.0)
    H1 = y * _poly([1.909859286, -1.145914713, 0.294656958, -0.042070508, 0.003785727, -0.000207183], y)
    hb = torch.where(low, 3.0, h)
    y = (3.0 / hb) ** 2
    c1 = 2 * _poly([0.99999906, 4.77228920, 3.85542044, 0.32303607], y)
    c2 = math.pi * hb * _poly([1.0, 4.88331068, 4.28957333, 0.52120508], y)
    d1 = 2 * _poly([1.00000004, 3.92205313, 2.64893033, 0.27450895], y)
    d2 = math.pi * _poly([1.0, 3.81095112, 2.26216956, 0.10885141], y)
    H0 = torch.where(low, H0, c1 / c2 + Y0)
    H1 = torch.where(low, H1, d1 / d2 + Y1)
    r3 = rho * (1 / (1 + d)) ** 3
    R = ((1 - beta) * _fit("A", rho) - beta * _fit("B", rho)
         - alpha * _fit("C", rho) / (1 + 6 * alpha * rho * (1 - rho)) + beta * (1 - beta) * _fit("D", rho))
    P = ev * (torch.log(0.5 * (d - v)) + 0.5772156649 - 2 * d * d) + d * d - v
    L0 = 2 * P / (1 + d ** 3) + 2 * r3 * R
    val = torch.complex(-L0 - 2 * math.pi * H0 * ev, 2 * math.pi * J0 * ev)
    R = (beta * _fit("dA", rho) - (1 - alpha) * _fit("dB", rho)
         + beta * (1 - beta) * rho * (1 - 2 * rho) * _fit("dC", rho))
    P = (beta + h) / (d - v) - 2 * beta + 2 * ev * d - h
    Q = torch.exp(-d) * (1 - beta) * (1 + d / (1 + d ** 3))
    Ls = 2 * P / (1 + d ** 3) - 4 * Q + 2 * r3 * R
    dh = torch.complex(-Ls - 2 * math.pi * (2 / math.pi - H1) * ev, -2 * math.pi * J1 * ev)
    return val, dh, val + 2 / d


def _delhommeau(h, v):
    """The exact infinite-depth wave term and its derivatives, one row of pairs at a time:
    Re G = 2 int_0^inf e^-u sgn(u + v) / sqrt((u + v)^2 + h^2) du - 2 pi e^v H0(h), with the
    singular point u = -v split off in t = h sinh(s), and Struve's integral by quadrature."""
    val, dh, dv = (torch.empty(h.shape, dtype=torch.complex128, device="cuda") for _ in range(3))
    for i in range(0, h.shape[0], 64):
        sl = slice(i, i + 64)
        val[sl], dh[sl], dv[sl] = _delhommeau_rows(h[sl], v[sl])
    return val, dh, dv


def _delhommeau_rows(h, v):
    Y, r = -v, torch.clamp(h, min=1e-9)
    d = torch.sqrt(Y * Y + r * r)
    e = torch.exp(-Y)
    I, K = torch.zeros_like(r), torch.zeros_like(r)
    # int e^(t - Y) / sqrt(t^2 + r^2) dt over [0, Y], t = r sinh(s), and r times its -3/2 form
    # less 1/r: cells that halve the distance to s_max, where e^t varies fastest
    smax = torch.asinh(Y / r)
    edges = [1 - 2.0 ** -q for q in range(0, 8)] + [1.0]
    for a, b in zip(edges[:-1], edges[1:]):
        for x, w in _NODES:
            u = smax * (a + (b - a) * (x + 1) / 2)
            wt = smax * w * (b - a) / 2
            t = r * torch.sinh(u)
            ex = torch.exp(t - Y)
            I += wt * ex
            # e^t - 1 - t over r cosh^2, which vanishes like t^2
            em = torch.where(t < 1e-2, t * t * (0.5 + t * (1 / 6 + t * (1 / 24 + t * (1 / 120 + t / 720)))),
                             torch.expm1(t) - t) * e
            em = torch.where(t < 1e-2, em, torch.where(t > 30, ex - (1 + t) * e, em))
            K += wt * em / (r * torch.cosh(u) ** 2)
    # -r int e^t (t^2 + r^2)^(-3/2) dt = -Y/(r d) - (1 - r/d) - K e^Y
    J0, J1, Y0, Y1, H0, H1 = _bessel(r)  # H1: the derivative of H0
    val = torch.complex(-e * math.pi * (H0 + Y0) - 2 * I, 2 * math.pi * e * J0)
    # Y1's pole against Y/(r d): both as 1/r less a regular part
    pole = -math.pi * Y1 - 2 / r + 2 * r / (d * (d + Y))
    re = -e * (math.pi * H1 + pole - 2 * (1 - r / d)) + 2 * K
    dh = torch.complex(re, -2 * math.pi * e * J1)
    return val, dh, val + 2 / torch.sqrt(v * v + h * h)


class _Sweep:
    """Forces on a body at one frequency at a time (a number, or a tensor to differentiate)."""

    def __init__(self, body, params, direct, wave):
        mesh = body.mesh
        self.C, self.N, A = _t(mesh.centers), _t(mesh.normals), _t(mesh.areas)
        self.influence, self.direct, self.betas = _Influence(mesh, direct, wave), direct, params["wave_directions"]
        motion = lambda d: (self.N * _t(body.dofs[d])).sum(1)  # noqa: E731
        self.disp = torch.stack([motion(d) for d in params["radiating_dofs"]], 1)
        self.pull = torch.stack([-motion(d) * A for d in params["influenced_dofs"]], 0).to(torch.complex128)

    def at(self, om):
        """(influenced, rhs) forces and (influenced, heading) Froude-Krylov forces."""
        C, N, k = self.C, self.N, om * om / G
        S, D = self.influence.at(k)
        cols, inc = [(-1j * om) * self.disp], []
        for b in self.betas:
            wb = C[:, 0] * math.cos(b) + C[:, 1] * math.sin(b)
            wv = torch.exp(k * C[:, 2]) * torch.exp(1j * k * wb)
            cols.append(-((G * k / om) * wv * (math.cos(b) * N[:, 0] + math.sin(b) * N[:, 1] - 1j * N[:, 2]))[:, None])
            inc.append(RHO * G * wv)
        bc = torch.cat([c.to(torch.complex128) for c in cols], 1)
        phi = torch.linalg.solve(D, S @ bc) if self.direct else S @ torch.linalg.solve(D, bc)
        F = self.pull @ (1j * RHO * om * phi)
        FK = self.pull @ torch.stack(inc, 1) if inc else F[:, :0]
        return F, FK


def _pack(F, FK, omegas, n_rad):
    om = np.asarray(omegas)[:, None, None]
    Fr, Fd = F[:, :, :n_rad], F[:, :, n_rad:]
    turn = lambda x: np.ascontiguousarray(np.moveaxis(x, 0, 1))[..., None]  # noqa: E731
    rad = lambda x: np.ascontiguousarray(np.moveaxis(x, 0, 2))[..., None]  # noqa: E731
    return {"added_mass": rad(Fr.real / om ** 2), "radiation_damping": rad(Fr.imag / om),
            "diffraction_force": turn(Fd) if Fd.shape[2] else np.zeros(0),
            "Froude_Krylov_force": turn(FK) if Fd.shape[2] else np.zeros(0),
            "excitation_force": turn(Fd + FK) if Fd.shape[2] else np.zeros(0)}


def _stack(parts):
    return torch.stack(parts).cpu().numpy()


def _coefficients(body, params, direct, wave):
    sweep, oms = _Sweep(body, params, direct, wave), params["wave_frequencies"]
    parts = [sweep.at(float(om)) for om in oms]
    return _pack(_stack([p[0] for p in parts]), _stack([p[1] for p in parts]), oms, len(params["radiating_dofs"]))


def _with_derivative(body, params, direct, wave):
    """The coefficients and their derivatives in omega, by forward-mode differentiation."""
    sweep, oms, n_rad = _Sweep(body, params, direct, wave), params["wave_frequencies"], len(params["radiating_dofs"])
    parts = []
    for om in oms:
        with fwad.dual_level():
            x = torch.tensor(float(om), dtype=torch.float64, device="cuda")
            F, FK = sweep.at(fwad.make_dual(x, torch.ones_like(x)))
            parts.append([t for y in (F, FK) for t in fwad.unpack_dual(y)])
    F, dF, FK, dFK = (_stack([p[q] for p in parts]) for q in range(4))
    out = _pack(F, FK, oms, n_rad)
    d = _pack(dF, dFK, oms, n_rad)
    om = np.asarray(oms)[None, None, :, None]
    d["added_mass"] = d["added_mass"] - 2 * out["added_mass"] / om
    d["radiation_damping"] = d["radiation_damping"] - out["radiation_damping"] / om
    out.update({"d_" + key: value for key, value in d.items()})
    return out
