"""The reference's public solve path, re-targeted at libmarinehydro_cuda.so.

Mirrors (names, argument meaning, errors):
  assemble_matrices(gfs, mesh, k; direct, include_identity, all_normals)   matrix_assembly.jl:164-222
  linsolve(A, b) / gpu_linsolve                                            matrix_assembly.jl:396-434
  solve(D, S, bc; direct) -> (phi, sources)                                matrix_assembly.jl:436-449
  solve(problem, formulation)                                              solve.jl:47-65
  radiation_bc / airy_bc / integrate_pressure / froude_krylov_force       waves.jl:154-303
  problems_from_data / hydrodynamic_coefficients                          problems_and_results.jl:242-495
Assembly and dense solves always run on the GPU; there is no CPU fallback.  The
O(N) boundary conditions and force sums of `solve(problem, ...)` run in numpy
exactly where the reference runs them on the host; `hydrodynamic_coefficients`
keeps everything on the device.
"""
from __future__ import annotations

import os

import numpy as np

from . import _device, _lib
from .bodies import FloatingBody, evaluate_gradient_of_motion
from .formulations import BEMFormulation, DirectBEM, SurrogateDelhommeau, bem_formulation, gf_flags, is_direct
from .meshes import StaticArraysMesh, face_fields, face_fields_pullback
from .problems import (DiffractionProblem, DiffractionResult, RadiationProblem, RadiationResult, SETTINGS,
                       added_mass, compute_wavenumber, make_result, radiation_damping)


def _ctx(ctx=None):
    return ctx if ctx is not None else _lib.default_context(0)


def _prec(precision):
    if precision in (None, "fp64", _lib.MH_PREC_FP64):
        return _lib.MH_PREC_FP64
    if precision in ("mixed", _lib.MH_PREC_MIXED):
        return _lib.MH_PREC_MIXED
    if precision in ("fp64_tc", _lib.MH_PREC_FP64_TC):
        return _lib.MH_PREC_FP64_TC
    raise ValueError('precision must be "fp64", "mixed" or "fp64_tc"')


# ---------------------------------------------------------------------------
# matrix level
# ---------------------------------------------------------------------------
def assemble_matrices(green_functions, mesh: StaticArraysMesh, wavenumber, direct=True, include_identity=True,
                      all_normals=None, ctx=None):
    """(S, D) influence matrices, n x n complex (matrix_assembly.jl:167-222)."""
    c = _ctx(ctx)
    return _device.assemble(c, mesh.device_mesh(c), wavenumber, gf_flags(green_functions), direct,
                            include_identity, all_normals)


def assemble_matrix_wu(mesh, wavenumber, direct=True, all_normals=None, ctx=None):
    """assemble_matrix_wu (matrix_assembly.jl:372-374)."""
    from .formulations import GFWu, Rankine, RankineReflected

    return assemble_matrices((Rankine(), RankineReflected(), GFWu()), mesh, wavenumber, direct=direct,
                             all_normals=all_normals, ctx=ctx)


def linsolve(A, b, precision="fp64", ctx=None):
    """A \\ b (matrix_assembly.jl:396-416); raises numpy.linalg.LinAlgError on an exactly singular A."""
    return _device.linsolve(_ctx(ctx), A, b, _prec(precision))


gpu_linsolve = linsolve


def linsolve_adjoint(A, ybar, precision="fp64", ctx=None):
    """lambda = A^H \\ ybar, the adjoint solve of the IFT rule (ad_rules.jl:360-414)."""
    return _device.linsolve(_ctx(ctx), A, ybar, _prec(precision), adjoint=True)


def solve_pullback(D, S, bc, phi_bar, direct=True, sources_bar=None, precision="fp64", ctx=None):
    """The reverse-mode pullback of solve(D, S, bc; direct) (matrix_assembly.jl:436-449) through
    the _mulvec and _linearsolve rules (ad_rules.jl:300-414), on the device
    (mh_solve_pullback).  Given the cotangent phi_bar of the potential (and, indirect,
    sources_bar of the sources) returns (phi, sources, D_bar, S_bar, bc_bar) with Julia's
    complex conventions: direct lambda = D^-H phi_bar, D_bar = -lambda phi^H,
    S_bar = lambda bc^H, bc_bar = S^H lambda; indirect lambda = K^-H (S^H phi_bar +
    sources_bar), S_bar = phi_bar sources^H, D_bar = -lambda sources^H, bc_bar = lambda."""
    return _device.solve_pullback(_ctx(ctx), D, S, bc, phi_bar, direct, sources_bar, _prec(precision))


def solve_linear(D, S, bc, direct=True, precision="fp64", ctx=None):
    """solve(D, S, bc; direct) -> (phi, sources) (matrix_assembly.jl:436-449)."""
    return _device.solve_linear(_ctx(ctx), D, S, bc, direct, _prec(precision))


# ---------------------------------------------------------------------------
# physics around the solve (waves.jl)
# ---------------------------------------------------------------------------
def _normal_displacement(mesh, dof):
    return np.einsum("ij,ij->i", mesh.normals, dof)


def radiation_bc(problem: RadiationProblem) -> np.ndarray:
    """radiation_bc(problem) (waves.jl:183-199)."""
    mesh = problem.floatingbody.mesh
    dof = problem.floatingbody.dofs[problem.radiating_dof]
    bc = (-1j * problem.encountered_omega) * _normal_displacement(mesh, dof)
    if problem.forward_speed != 0:
        ddx = evaluate_gradient_of_motion(mesh, problem.radiating_dof)
        bc = bc + problem.forward_speed * _normal_displacement(mesh, ddx)
    return bc


def _airy_vel(centers, problem):
    """_airy_vel (waves.jl:266-273)."""
    k = problem.wavenumber
    wbar = centers[:, 0] * np.cos(problem.encountered_beta) + centers[:, 1] * np.sin(problem.encountered_beta)
    cih = np.exp(k * centers[:, 2])
    amp = problem.g * k / problem.omega * np.exp(1j * k * wbar)
    return np.stack([amp * np.cos(problem.beta) * cih, amp * np.sin(problem.beta) * cih, -1j * amp * cih], axis=1)


def airy_bc(problem: DiffractionProblem) -> np.ndarray:
    """_airy_bc(::StaticArraysMesh) (waves.jl:275-282)."""
    mesh = problem.floatingbody.mesh
    v = _airy_vel(mesh.centers, problem)
    n = mesh.normals
    return -(v[:, 0] * n[:, 0] + v[:, 1] * n[:, 1] + v[:, 2] * n[:, 2])


def compute_bc(problem):
    return radiation_bc(problem) if isinstance(problem, RadiationProblem) else airy_bc(problem)


def airy_pressure(problem: DiffractionProblem) -> np.ndarray:
    """_airy_pressure(::StaticArraysMesh) (waves.jl:259-264, 301-303)."""
    c = problem.floatingbody.mesh.centers
    k = problem.wavenumber
    wbar = c[:, 0] * np.cos(problem.encountered_beta) + c[:, 1] * np.sin(problem.encountered_beta)
    phi = -1j * problem.g / problem.omega * np.exp(k * c[:, 2]) * np.exp(1j * k * wbar)
    return 1j * problem.omega * problem.rho * phi


def integrate_pressure(body: FloatingBody, influenced_dofs, pressure) -> dict:
    """integrate_pressure (waves.jl:154-178): {dof: sum p_i * -(dof_i . n_i) * a_i}."""
    mesh = body.mesh
    out = {}
    for d in influenced_dofs:
        disp = _normal_displacement(mesh, body.dofs[d])
        out[d] = complex(np.sum(pressure * -disp * mesh.areas))
    return out


def froude_krylov_force(problem_or_result, influenced_dofs=None) -> dict:
    """froude_krylov_force (waves.jl:294-298; problems_and_results.jl:216-217)."""
    prob = problem_or_result.problem if isinstance(problem_or_result, DiffractionResult) else problem_or_result
    inf = prob.influenced_dofs if influenced_dofs is None else influenced_dofs
    return integrate_pressure(prob.floatingbody, inf, airy_pressure(prob))


def excitation_force(res: DiffractionResult) -> dict:
    """diffraction + Froude-Krylov (problems_and_results.jl:218-219)."""
    fk = froude_krylov_force(res)
    return {k: v + fk[k] for k, v in res.forces.items()}


# ---------------------------------------------------------------------------
# problem level
# ---------------------------------------------------------------------------
def solve(problem, formulation: BEMFormulation | None = None, ctx=None):
    """solve(problem, formulation) (solve.jl:59-65) or, for arrays, solve(D, S, bc; direct)."""
    if isinstance(problem, (list, tuple)):
        return [solve(p, formulation, ctx=ctx) for p in problem]
    if isinstance(problem, np.ndarray):
        raise TypeError("use solve_linear(D, S, bc, direct=...) for the matrix-level solve")
    return _solve_group([problem], formulation or DirectBEM(), _ctx(ctx))[0]


def _solve_group(problems, f: BEMFormulation, c):
    """solve(problem, f) for problems of one body that share the encountered frequency,
    wavenumber and forward speed: one assembly and one factorization for all of their
    right-hand sides, the rest as the reference's per-problem path (solve.jl:20-65):
    hull + lid mesh with the hull conditions padded by zeros, pressure i rho omega phi on
    the hull, plus rho U (K sigma) with K assembled for the normal [1, 0, 0] when U != 0."""
    p0 = problems[0]
    body = p0.floatingbody
    direct = is_direct(f)
    U = p0.forward_speed
    omega = p0.omega if U == 0 else p0.encountered_omega
    k = p0.wavenumber if U == 0 else p0.encountered_wavenumber
    for p in problems[1:]:
        if (p.floatingbody is not body or p.forward_speed != U or p.rho != p0.rho
                or (p.omega if U == 0 else p.encountered_omega) != omega
                or (p.wavenumber if U == 0 else p.encountered_wavenumber) != k):
            raise ValueError("problems solved together must share body, frequency, wavenumber and forward speed")
    if U != 0 and direct:
        raise ValueError("nonzero forward speed is not supported with the direct method; use IndirectBEM "
                         "(direct = false)")
    mesh, n_hull = body.mesh_including_lid()
    bc = np.zeros((mesh.nfaces, len(problems)), dtype=np.complex128)
    for q, p in enumerate(problems):
        bc[:n_hull, q] = compute_bc(p)
    S, D = assemble_matrices(f.greens, mesh, k, direct=direct, ctx=c)
    potential, sources = _device.solve_linear(c, D, S, bc, direct, f.precision_code)
    pressure = 1j * p0.rho * omega * potential
    if U != 0:
        # _maybe_forward_speed_pressure (solve.jl:35-45)
        _, K = assemble_matrices(f.greens, mesh, k, direct=False, all_normals=[1.0, 0.0, 0.0], ctx=c)
        pressure = pressure + p0.rho * U * (K @ sources)
    pressure = pressure[:n_hull]
    return [make_result(p, integrate_pressure(body, p.influenced_dofs, pressure[:, q]))
            for q, p in enumerate(problems)]


def solve_problem(problem, formulation=None, direct=True, gf="Wu", greens_functions=None, ctx=None):
    return solve(problem, bem_formulation(formulation, direct, gf, greens_functions), ctx=ctx)


def problems_from_data(parameters: dict, body: FloatingBody) -> dict:
    """problems_from_data (problems_and_results.jl:242-283)."""
    oms = np.atleast_1d(np.asarray(parameters["wave_frequencies"], dtype=float))
    inf = list(parameters.get("influenced_dofs", list(body.dofs)))
    Us = list(parameters.get("forward_speeds", [0.0]))
    rad = []
    if "radiating_dofs" in parameters:
        betas = parameters.get("wave_directions", [0.0]) if "forward_speeds" in parameters else [0.0]
        for U in Us:
            for om in oms:
                for d in parameters["radiating_dofs"]:
                    for b in betas:
                        rad.append(RadiationProblem(body, om, d, inf, beta=b if U != 0 else None, forward_speed=U,
                                                    rho=parameters.get("rho"), g=parameters.get("g")))
    dif = []
    if "wave_directions" in parameters:
        for U in Us:
            for om in oms:
                for b in parameters["wave_directions"]:
                    dif.append(DiffractionProblem(body, om, b, inf, forward_speed=U, rho=parameters.get("rho"),
                                                  g=parameters.get("g")))
    return {"radiation": rad, "diffraction": dif}


def hydrodynamic_coefficients(body: FloatingBody, parameters: dict, formulation: BEMFormulation | None = None,
                              ctx=None, rho=None, g=None) -> dict:
    """hydrodynamic_coefficients (problems_and_results.jl:464-495).

    Returns numpy arrays with the reference's shapes.  Without a `forward_speeds` key:
      added_mass, radiation_damping: (n_inf, n_rad, n_omega, 1)
      diffraction_force, Froude_Krylov_force, excitation_force: (n_inf, n_omega, n_beta, 1)
    With `forward_speeds` (problems_and_results.jl:262-270, 346-363) the radiation arrays
    gain the heading axis, (n_inf, n_rad, n_omega, n_U, n_beta), and the diffraction arrays
    are (n_inf, n_omega, n_beta, n_U).
    Zero speed runs the device sweep (mh_hydrodynamic_coefficients): one assembly of S and
    D and one factorization per frequency serve every radiation and diffraction
    right-hand side.  A nonzero speed needs IndirectBEM (solve.jl:35-45); its problems are
    solved per (omega, beta) -- they share the encountered wavenumber -- with one
    assembly, one K matrix and one factorization for every dof and the diffraction.
    """
    f = formulation or DirectBEM()
    c = _ctx(ctx)
    oms = np.atleast_1d(np.asarray(parameters["wave_frequencies"], dtype=float))
    names = list(body.dofs)
    inf = list(parameters.get("influenced_dofs", names))
    rad = list(parameters.get("radiating_dofs", []))
    betas = list(parameters.get("wave_directions", []))
    rho = parameters.get("rho", SETTINGS["rho"]) if rho is None else rho
    g = parameters.get("g", SETTINGS["g"]) if g is None else g
    if "forward_speeds" not in parameters:
        A, B, Fd, Fk, Fe = _zero_speed_sweep(c, body, f, oms, rho, g, names, rad, inf, betas)
        out = {
            "added_mass": A[..., None] if rad else np.zeros(0),
            "radiation_damping": B[..., None] if rad else np.zeros(0),
            "diffraction_force": Fd[..., None] if betas else np.zeros(0),
            "Froude_Krylov_force": Fk[..., None] if betas else np.zeros(0),
            "excitation_force": Fe[..., None] if betas else np.zeros(0),
        }
        if _judged(c, f):
            est, rerun = surrogate_judge_report(oms.size, c)
            out["surrogate_judge"] = {"estimate": est, "rerun": rerun}
        return out
    Us = [float(u) for u in parameters["forward_speeds"]]
    if rad and "wave_directions" not in parameters:
        raise ValueError("radiation problems with forward_speeds need wave_directions "
                         "(problems_and_results.jl:268-270)")
    n_inf, n_rad, n_w, n_U, n_b = len(inf), len(rad), len(oms), len(Us), len(betas)
    A = np.zeros((n_inf, n_rad, n_w, n_U, n_b))
    B = np.zeros_like(A)
    Fd = np.zeros((n_inf, n_w, n_b, n_U), dtype=np.complex128)
    Fk = np.zeros_like(Fd)
    for iU, U in enumerate(Us):
        if U == 0:
            a, b, fd, fk, _ = _zero_speed_sweep(c, body, f, oms, rho, g, names, rad, inf, betas)
            if rad:
                A[:, :, :, iU, :] = a[..., None]
                B[:, :, :, iU, :] = b[..., None]
            if betas:
                Fd[..., iU] = fd
                Fk[..., iU] = fk
            continue
        for iw, om in enumerate(oms):
            for ib, beta in enumerate(betas):
                probs = [RadiationProblem(body, om, d, inf, beta=beta, forward_speed=U, rho=rho, g=g) for d in rad]
                probs.append(DiffractionProblem(body, om, beta, inf, forward_speed=U, rho=rho, g=g))
                res = _solve_group(probs, f, c)
                for ir in range(n_rad):
                    am, bd = added_mass(res[ir]), radiation_damping(res[ir])
                    A[:, ir, iw, iU, ib] = [am[d] for d in inf]
                    B[:, ir, iw, iU, ib] = [bd[d] for d in inf]
                fk = froude_krylov_force(res[-1])
                Fd[:, iw, ib, iU] = [res[-1].forces[d] for d in inf]
                Fk[:, iw, ib, iU] = [fk[d] for d in inf]
    return {
        "added_mass": A if rad else np.zeros(0),
        "radiation_damping": B if rad else np.zeros(0),
        "diffraction_force": Fd if betas else np.zeros(0),
        "Froude_Krylov_force": Fk if betas else np.zeros(0),
        "excitation_force": Fd + Fk if betas else np.zeros(0),
    }


def hydrodynamic_coefficients_derivative(body: FloatingBody, parameters: dict,
                                         formulation: BEMFormulation | None = None, ctx=None, rho=None,
                                         g=None) -> dict:
    """hydrodynamic_coefficients and its derivative with respect to the wave frequency,
    what the reference obtains with ForwardDiff.derivative over wave_frequencies
    (test/outputs_differentiation.jl:39-150, diffraction_differentiation.jl:63-78).

    Returns the keys of hydrodynamic_coefficients (zero forward speed, shapes with n_U = 1)
    plus "d_added_mass", "d_radiation_damping", "d_diffraction_force",
    "d_Froude_Krylov_force", "d_excitation_force" (d/d omega, same shapes).  FP64, the
    Rankine kinds with GFWu or ExactGuevelDelhommeau, direct or indirect, lids included
    (mh_hydro_frequency_derivative).
    """
    f = formulation or DirectBEM()
    if any(u != 0 for u in parameters.get("forward_speeds", [0.0])):
        raise ValueError("the frequency derivative covers zero forward speed")
    c = _ctx(ctx)
    oms = np.atleast_1d(np.asarray(parameters["wave_frequencies"], dtype=float))
    names = list(body.dofs)
    inf = list(parameters.get("influenced_dofs", names))
    rad = list(parameters.get("radiating_dofs", []))
    betas = list(parameters.get("wave_directions", []))
    rho = parameters.get("rho", SETTINGS["rho"]) if rho is None else rho
    g = parameters.get("g", SETTINGS["g"]) if g is None else g
    idx = {n: i for i, n in enumerate(names)}
    mesh, _ = body.mesh_including_lid()
    arrs = _device.hydro_frequency_derivative(c, mesh.device_mesh(c), oms, rho, g, gf_flags(f.greens), is_direct(f),
                                              body.padded_dof_array(names), [idx[d] for d in rad],
                                              [idx[d] for d in inf], betas)
    keys = ("added_mass", "radiation_damping", "diffraction_force", "Froude_Krylov_force", "excitation_force")
    out = {}
    for q, key in enumerate(keys + tuple("d_" + k for k in keys)):
        radiation = key.endswith(("added_mass", "radiation_damping"))
        out[key] = arrs[q][..., None] if (rad if radiation else betas) else np.zeros(0)
    return out


def _zero_speed_sweep(c, body, f, oms, rho, g, names, rad, inf, betas):
    """The zero-speed frequency sweep on the device (mh_hydrodynamic_coefficients)."""
    idx = {n: i for i, n in enumerate(names)}
    mesh, _ = body.mesh_including_lid()
    return _device.hydro_sweep(c, mesh.device_mesh(c), oms, rho, g, gf_flags(f.greens), is_direct(f),
                               body.padded_dof_array(names), [idx[d] for d in rad], [idx[d] for d in inf], betas,
                               f.precision_code)


def batch_hydrodynamic_coefficients(bodies, parameters_per_body, formulation: BEMFormulation | None = None,
                                    ctx=None, rho=None, g=None, n_streams=0) -> list:
    """hydrodynamic_coefficients for many bodies at once (one CUDA graph over several streams).

    Every body must have the same dof names; `parameters_per_body[b]` gives body b's
    wave_frequencies (radiating_dofs / influenced_dofs / wave_directions are taken
    from the first entry).  Returns one result dict per body, as hydrodynamic_coefficients.
    """
    f = formulation or DirectBEM()
    c = _ctx(ctx)
    p0 = parameters_per_body[0]
    names = list(bodies[0].dofs)
    for b in bodies:
        if list(b.dofs) != names:
            raise ValueError("every body of a batch must have the same dof names")
    inf = list(p0.get("influenced_dofs", names))
    rad = list(p0.get("radiating_dofs", []))
    betas = list(p0.get("wave_directions", []))
    idx = {n: i for i, n in enumerate(names)}
    rho = p0.get("rho", SETTINGS["rho"]) if rho is None else rho
    g = p0.get("g", SETTINGS["g"]) if g is None else g
    res = _device.batch_hydro(c, [b.mesh_including_lid()[0].device_mesh(c) for b in bodies],
                              [np.atleast_1d(np.asarray(p["wave_frequencies"], dtype=float)) for p in
                               parameters_per_body], rho, g, gf_flags(f.greens), is_direct(f),
                              [b.padded_dof_array(names) for b in bodies], [idx[d] for d in rad], [idx[d] for d in inf],
                              betas, f.precision_code, n_streams)
    out = []
    for A, B, Fd, Fk, Fe in res:
        out.append({"added_mass": A[..., None] if rad else np.zeros(0),
                    "radiation_damping": B[..., None] if rad else np.zeros(0),
                    "diffraction_force": Fd[..., None] if betas else np.zeros(0),
                    "Froude_Krylov_force": Fk[..., None] if betas else np.zeros(0),
                    "excitation_force": Fe[..., None] if betas else np.zeros(0)})
    if _judged(c, f):
        counts = [len(np.atleast_1d(p["wave_frequencies"])) for p in parameters_per_body]
        est, rerun = surrogate_judge_report(sum(counts), c)
        off = 0
        for o, m in zip(out, counts):
            o["surrogate_judge"] = {"estimate": est[off:off + m], "rerun": rerun[off:off + m]}
            off += m
    return out


def hydro_gradient(body: FloatingBody, wave_frequencies, objective_dofs, formulation: BEMFormulation | None = None,
                   ctx=None, rho=None, g=None, return_panel_terms=False):
    """Reverse-mode gradient of J = sum over wave_frequencies and objective_dofs h of
    added_mass[h, h] + radiation_damping[h, h], w.r.t. every mesh vertex.

    This is the quantity the reference obtains by differentiating
    hydrodynamic_coefficients with Zygote / Enzyme through the rules of
    ad_rules.jl:79-414 (Birk kernels, _mulvec, _linearsolve); here the adjoint is
    hand-written on the device (mh_hydro_gradient): one adjoint solve per frequency
    reusing the LU factors, pair derivatives recomputed instead of taped.

    The panel centres, normals and areas must be those meshes.face_fields derives from
    the vertices (they are differentiated through it); rigid rotation dofs follow the
    panel centres and are chained through them, other dof fields are held fixed.
    DirectBEM or IndirectBEM with the Birk Rankine family and GFWu or
    ExactGuevelDelhommeau, zero forward speed, FP64 arithmetic; formulation precision
    "mixed" factors in FP32 and refines both the forward and the adjoint solve to the
    FP64 backward-error test.

    Returns (J, dJ/dvertices as an (nvertices, 3) array); with return_panel_terms the
    raw per-panel terms of the C-ABI come back as a third item (a dict).
    """
    f = formulation or DirectBEM()
    if body.lid_mesh is not None:
        raise ValueError("hydro_gradient does not cover bodies with a lid")
    mesh = body.mesh
    _check_derived_fields(mesh)
    ctx_ = _ctx(ctx)
    names = list(body.dofs)
    idx = {n: i for i, n in enumerate(names)}
    obj = list(objective_dofs)
    rho = SETTINGS["rho"] if rho is None else rho
    g = SETTINGS["g"] if g is None else g
    oms = np.atleast_1d(np.asarray(wave_frequencies, dtype=float))
    J, gc, gn, ga, gv, gd = _device.hydro_gradient(ctx_, mesh.device_mesh(ctx_), oms, rho, g, gf_flags(f.greens),
                                                    body.dof_array(names), [idx[d] for d in obj], f.precision_code,
                                                    is_direct(f))
    grad = _vertex_gradient(body, gc, gn, ga, gv, {name: gd[h] for h, name in enumerate(obj)})
    if return_panel_terms:
        return J, grad, {"centers": gc, "normals": gn, "areas": ga, "corners": gv, "dofs": gd}
    return J, grad


def hydro_vjp(body: FloatingBody, wave_frequencies, radiating_dofs, influenced_dofs, added_mass_bar=None,
              radiation_damping_bar=None, formulation: BEMFormulation | None = None, ctx=None, rho=None, g=None,
              wave_directions=(), excitation_force_bar=None):
    """Pullback of hydrodynamic_coefficients with respect to the mesh vertices: for
    cotangents Abar, Bbar of shape (n_inf, n_rad, n_omega) and, with wave_directions, a
    complex Fbar of shape (n_inf, n_omega, n_beta) (the reference's trailing n_U = 1 axis
    may be present) returns (J, dJ/dvertices) with
    J = sum Abar * added_mass + Bbar * radiation_damping + Re Fbar * Re Fe + Im Fbar * Im Fe
    -- what Zygote / Enzyme reverse mode gives for the reference (ad_rules.jl:79-414).
    Hand-written on the device (mh_hydro_vjp): one adjoint solve per radiating dof, heading
    and frequency with the LU factors reused, pair derivatives recomputed.  Same scope as
    hydro_gradient (DirectBEM or IndirectBEM, Birk Rankine family with GFWu or
    ExactGuevelDelhommeau, zero forward speed, no lid)."""
    f = formulation or DirectBEM()
    if body.lid_mesh is not None:
        raise ValueError("hydro_vjp does not cover bodies with a lid")
    mesh = body.mesh
    _check_derived_fields(mesh)
    ctx_ = _ctx(ctx)
    names = list(body.dofs)
    idx = {n: i for i, n in enumerate(names)}
    rad, inf, betas = list(radiating_dofs), list(influenced_dofs), list(wave_directions)
    oms = np.atleast_1d(np.asarray(wave_frequencies, dtype=float))
    shape = (len(inf), len(rad), oms.size)
    ab = np.zeros(shape) if added_mass_bar is None else np.asarray(added_mass_bar, dtype=float).reshape(shape)
    bb = np.zeros(shape) if radiation_damping_bar is None else np.asarray(radiation_damping_bar,
                                                                          dtype=float).reshape(shape)
    fshape = (len(inf), oms.size, len(betas))
    fb = (np.zeros(fshape, complex) if excitation_force_bar is None
          else np.asarray(excitation_force_bar, dtype=complex).reshape(fshape))
    rho = SETTINGS["rho"] if rho is None else rho
    g = SETTINGS["g"] if g is None else g
    J, gc, gn, ga, gv, gd = _device.hydro_vjp(ctx_, mesh.device_mesh(ctx_), oms, rho, g, gf_flags(f.greens),
                                              body.dof_array(names), [idx[d] for d in rad], [idx[d] for d in inf],
                                              ab, bb, betas, fb, f.precision_code, is_direct(f))
    return J, _vertex_gradient(body, gc, gn, ga, gv, {name: gd[idx[name]] for name in set(rad) | set(inf)})


def _check_derived_fields(mesh):
    c, nrm, a, _ = face_fields(mesh.vertices, mesh.faces - 1)
    if not (np.allclose(c, mesh.centers, rtol=0, atol=1e-12) and np.allclose(nrm, mesh.normals, rtol=0, atol=1e-12)
            and np.allclose(a, mesh.areas, rtol=1e-12, atol=0)):
        raise ValueError("the vertex gradient needs panel fields derived from the vertices (meshes.face_fields)")


def _vertex_gradient(body, gc, gn, ga, gv, gd_by_name):
    """Chain the per-panel gradient terms to the mesh vertices: rigid rotation dof fields
    follow the panel centres, and centres, normals, areas and Birk corners are functions
    of each panel's corners (meshes.face_fields)."""
    mesh = body.mesh
    gc = gc.copy()
    # rotation dof field axis x (c - rc) on its panels: d/dc of gd . (axis x c) = gd x axis
    rot = getattr(body, "rotations", {})
    for name, gdn in gd_by_name.items():
        if name in rot:
            ax, _, p0, p1 = rot[name]
            e = np.zeros(3)
            e[ax] = 1.0
            gc[p0:p1] += np.cross(gdn[p0:p1], e)
    corner = face_fields_pullback(mesh.panel_vertices, gc, gn, ga) + gv.reshape(-1, 12)
    grad = np.zeros_like(mesh.vertices)
    faces0 = mesh.faces - 1
    for q in range(4):
        np.add.at(grad, faces0[:, q], corner[:, 3 * q:3 * q + 3])
    return grad


def train_surrogate(n_samples=10_000_000, seed=2026, epochs=8, batch=8192, lr=3e-3, ctx=None):
    """Train the learned Delhommeau wave-term surrogate on the device and install it on
    the context (mh_surrogate_train).  Returns (params, report)."""
    return _ctx(ctx).surrogate_train(n_samples, seed, epochs, batch, lr)


def set_surrogate(params, ctx=None):
    """Install surrogate parameters (as returned by train_surrogate) on the context."""
    _ctx(ctx).surrogate_set(params)


TILE_TABLE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "data", "tile_table_gb300.json")
_TILE_FIELDS = ("n_max", "ozaki_column_tiles", "bf16x3_column_tiles", "panel_cluster_fp64", "panel_cluster_fp32")


def autotune(sizes=(384, 768, 1536, 3072), batch=16, precisions=("fp64", "mixed", "fp64_tc"), reps=3, path=None,
             ctx=None) -> dict:
    """Pick the batched LU's launch shapes per matrix-order bucket by timing them on the
    device (mh_autotune) and install them on the context.  The table is keyed by order
    bucket (bounds at the geometric means of neighbouring `sizes`); `batch` is the number of
    matrices factored together (the frequencies of one body).  With `path` the table is
    written there as JSON (load it again with load_tile_table).  Returns the table and the
    tuned and default factorization times per precision and size."""
    c = _ctx(ctx)
    report = {"sizes": [int(n) for n in sizes], "batch": int(batch), "ms": {}}
    for p in precisions:
        best, dflt = c.autotune(_prec(p), sizes, batch, reps)
        report["ms"][p] = {"tuned": best.tolist(), "default": dflt.tolist()}
    table = [dict(zip(_TILE_FIELDS, e)) for e in c.tile_table()]
    for e in table:
        if e["n_max"] >= 2 ** 62:
            e["n_max"] = None  # the last bucket covers every larger order
    report["table"] = table
    if path is not None:
        import json

        with open(path, "w") as f:
            json.dump(report, f, indent=1)
    return report


def load_tile_table(path=None, ctx=None) -> list:
    """Install a tile table written by autotune (default: the shipped GB300 table,
    data/tile_table_gb300.json); returns its entries."""
    import json

    with open(path or TILE_TABLE) as f:
        table = json.load(f)["table"]
    entries = [((e["n_max"] if e["n_max"] is not None else 2 ** 63 - 1),) + tuple(int(e[k]) for k in _TILE_FIELDS[1:])
               for e in table]
    _ctx(ctx).set_tile_table(entries)
    return entries


SURROGATE_PARAMS = os.path.join(os.path.dirname(os.path.abspath(__file__)), "data", "surrogate_delhommeau.npy")


def set_surrogate_judge(n_samples=2048, tolerance=1e-3, seed=0x5EED, ctx=None):
    """Have the exact Guevel-Delhommeau term judge every surrogate result (mh_surrogate_set_judge):
    each frequency's surrogate-assembled S and D are checked on `n_samples` sampled panel pairs
    against the exact term, and a frequency whose sampled relative error exceeds `tolerance`
    is solved with the exact term instead.  n_samples = 0 turns the check off.  The
    per-frequency estimates and re-run flags come back with the results under
    "surrogate_judge"."""
    c = _ctx(ctx)
    c.check(c._L.mh_surrogate_set_judge(c.handle, int(n_samples), int(seed) & (2 ** 64 - 1), float(tolerance)),
            "surrogate judge")
    c._judge_on = n_samples > 0


def surrogate_judge_report(count, ctx=None):
    """(estimates, rerun flags) of the last judged surrogate sweep or batch (count frequency-solves)."""
    c = _ctx(ctx)
    est = np.empty(int(count))
    rerun = np.empty(int(count), dtype=np.int32)
    c.check(c._L.mh_surrogate_judge_read(c.handle, int(count), est.ctypes.data, rerun.ctypes.data),
            "surrogate judge report")
    return est, rerun.astype(bool)


def _judged(c, f):
    return getattr(c, "_judge_on", False) and any(isinstance(gf, SurrogateDelhommeau) for gf in f.greens)


def load_surrogate(path=None, ctx=None):
    """Install the shipped surrogate parameters (data/surrogate_delhommeau.npy, made by
    data/train_surrogate.py) or those in `path` on the context; returns them."""
    params = np.load(path or SURROGATE_PARAMS)
    set_surrogate(params, ctx)
    return params


def surrogate_wave_terms(r, z, ctx=None):
    """Surrogate (GF, dGF/dr, dGF/dz) at reduced coordinates (r, z): (m, 3) complex."""
    c = _ctx(ctx)
    r = np.ascontiguousarray(np.asarray(r, dtype=np.float64).ravel())
    z = np.ascontiguousarray(np.asarray(z, dtype=np.float64).ravel())
    if r.shape != z.shape:
        raise ValueError("r and z must have the same length")
    out = np.empty((r.size, 3), dtype=np.complex128)
    c.check(c._L.mh_surrogate_wave_terms(c.handle, r.size, r.ctypes.data, z.ctypes.data, out.ctypes.data,
                                         _lib.MH_MEM_HOST), "surrogate wave terms")
    return out


def compute_hydrodynamic_coefficients(parameters, body, formulation=None, direct=True, gf="Wu",
                                      greens_functions=None, ctx=None):
    return hydrodynamic_coefficients(body, parameters, bem_formulation(formulation, direct, gf, greens_functions),
                                     ctx=ctx)


def calculate_radiation_forces(mesh, dof, omega, rho=None, g=None, ctx=None):
    """calculate_radiation_forces (waves.jl:47-55): [A, B] for a uniform dof vector."""
    rho = SETTINGS["rho"] if rho is None else rho
    g = SETTINGS["g"] if g is None else g
    k = compute_wavenumber(omega, g)
    S, D = assemble_matrix_wu(mesh, k, ctx=ctx)
    bc = -1j * omega * (mesh.normals @ np.asarray(dof, dtype=float))
    phi, _ = solve_linear(D, S, bc, ctx=ctx)
    p = 1j * rho * omega * phi
    F = np.sum(p * -(mesh.normals @ np.asarray(dof, dtype=float)) * mesh.areas)
    return [F.real / omega ** 2, F.imag / omega]
