"""The calls this framework is measured by, over the sizes it is used at.

A case is a dict of plain values.  ``kind`` names the call:

  transport   Problem1D: new potentials, one batched transport solve, the densities and currents
  dropin      solve_transport_DG_2D: one call of the mode-space driver on a kept handle
  gummel      solve_rtd_self_consistent: self-consistent bias points
  transient   RTDSweep.transient: Crank-Nicolson steps after a drain-bias step
  subbands    SubbandSolver: the transverse eigensolve of one or of many gate points
  poisson     Poisson2D.solve: density projection and Newton update of one or of many bias points
  full2d      Full2DOperator.solve and its observables

Device parameters (barriers, doping, biases, gate voltages, states) are drawn from the seed around those of
the repository's own configurations.  Transport solves run to a residual of 1e-12, so that the results are those of
the linear system and not of the iteration that happened to reach a loose tolerance first.
"""
import ctypes as C
import math

import numpy as np
import torch

from real_space_dg_gb300 import Problem1D, devices
from real_space_dg_gb300.full2d import Full2DOperator
from real_space_dg_gb300.poisson2d import Poisson2D
from real_space_dg_gb300.rtd import RTDSweep, solve_rtd_self_consistent
from real_space_dg_gb300.subbands import SubbandSolver
from real_space_dg_gb300.transport import shape_from_mat, solve_transport_DG_2D

TOL = 1e-12
MAXIT = 60


def listed():
    return [
        # the smallest call of the drop-in: one short diode, where launches and latency count
        dict(name="dropin_small", kind="dropin", device="rtd", n_el=12, order=2, nk=32, modes=1, precision="fp64"),
        # one gate point of the multi-subband FET sweep: 2 valleys x 4 modes, transport only
        dict(name="dropin_fet", kind="dropin", device="fet", n_el=200, order=2, nk=256, modes=4, precision="mixed"),
        # the plain FP64 form (the default of the drop-in) at the size of the 80 nm diode
        dict(name="transport_fp64", kind="transport", n_el=240, order=3, nk=256, n_xi=256, batch=2, precision="fp64",
             fp64_tc=False),
        # the chosen form at the same size, a whole I-V sweep in one batch: the largest stationary solve
        dict(name="transport_mixed", kind="transport", n_el=240, order=3, nk=256, n_xi=256, batch=16,
             precision="mixed", fp64_tc=False),
        # ten iterations of the self-consistent loop of a short diode, plain FP64 as the reference's, odd Nk
        dict(name="gummel_fp64", kind="gummel", n_el=40, order=2, nk=65, batch=3, handles=1, precision="fp64",
             iterations=10),
        # the first iterations of the 80 nm diode's loop, 16 bias points over 8 concurrent handles
        dict(name="gummel_mixed", kind="gummel", n_el=240, order=3, nk=256, batch=16, handles=8, precision="mixed",
             iterations=4),
        # transients after a bias step, Nk = 512, the operator and the potential renewed every step
        dict(name="transient_mixed", kind="transient", n_el=240, order=2, nk=512, batch=4, steps=8, precision="mixed"),
        # the mode-space set-up of one gate point, host arrays in and out, ragged grid
        dict(name="subbands_one", kind="subbands", valleys=2, nx=117, ny=67, modes=4, batch=1, on_device=False),
        # the same for a whole gate sweep, on arrays that live on the device
        dict(name="subbands_sweep", kind="subbands", valleys=2, nx=401, ny=71, modes=8, batch=32, on_device=True),
        # one Poisson step of a self-consistent loop over one bias point, Neumann Y, ragged grid
        dict(name="poisson_one", kind="poisson", n_el_x=48, n_el_y=5, nk=3, nx=97, ny=11, batch=1, periodic=False),
        # the step of 16 bias points on the recorded run's material grid
        dict(name="poisson_sweep", kind="poisson", n_el_x=120, n_el_y=2, nk=3, nx=361, ny=13, batch=16,
             periodic=True),
        # the Full-2D solve of a contact-driven system, mixed form, at half the recorded run's length
        dict(name="full2d_mixed", kind="full2d", n_el_x=60, n_el_y=2, n_rho_x=121, n_rho_y=12, ybc="zero-inflow",
             mixed=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["transport", "transport", "dropin", "gummel", "transient", "subbands", "poisson", "full2d"])
    if kind in ("transport", "dropin", "gummel", "transient"):
        precision = rng.choice(["fp64", "mixed"])
        order = rng.choice([1, 2, 3])
        n_el = _log(rng, 12, 240)
        # any Nk in FP64 (odd ones too), multiples of 4 in the mixed form
        nk = _log(rng, 24, 256) if precision == "fp64" else 4 * _log(rng, 16, 64)
        if kind == "dropin":
            modes = rng.choice([1, 2, 4])
            return dict(kind=kind, device=rng.choice(["rtd", "fet"]), n_el=n_el, order=order, nk=nk, modes=modes,
                        precision=precision)
        if kind == "transport":
            tc = precision == "fp64" and rng.random() < 0.5
            if tc:
                nk = 4 * _log(rng, 16, 64)
            # more xi cells than wave numbers in a quarter of the draws
            n_xi = nk + (4 * rng.randint(1, nk // 8) if rng.random() < 0.25 else 0)
            return dict(kind=kind, n_el=n_el, order=order, nk=nk, n_xi=n_xi,
                        batch=_log(rng, 1, 2 if precision == "fp64" else 16), precision=precision, fp64_tc=tc)
        if kind == "gummel":
            batch = _log(rng, 1, 4 if precision == "fp64" else 16)
            return dict(kind=kind, n_el=n_el if precision == "mixed" else min(n_el, 40), order=order,
                        nk=nk if precision == "mixed" else min(nk, 65), batch=batch,
                        handles=rng.choice([h for h in (1, 2, 4, 8) if h <= batch]), precision=precision, iterations=4)
        return dict(kind=kind, n_el=n_el, order=min(order, 2), nk=nk, batch=_log(rng, 1, 4), steps=rng.randint(2, 6),
                    precision=precision)
    if kind == "subbands":
        return dict(kind=kind, valleys=rng.choice([1, 2]), nx=_log(rng, 24, 401), ny=_log(rng, 30, 160),
                    modes=rng.randint(1, 10), batch=_log(rng, 1, 16), on_device=rng.random() < 0.5)
    if kind == "poisson":
        nk, periodic = rng.choice([2, 3]), rng.random() < 0.5
        nex, ney = _log(rng, 10, 120), rng.randint(2, 6)
        return dict(kind=kind, n_el_x=nex, n_el_y=ney, nk=nk, nx=rng.randint(30, 361),
                    ny=rng.randint(4, 33 if periodic else 32), batch=_log(rng, 1, 16), periodic=periodic)
    return dict(kind=kind, n_el_x=rng.randint(5, 20), n_el_y=rng.choice([2, 3]), n_rho_x=2 * rng.randint(6, 20) + 1,
                n_rho_y=rng.choice([4, 5, 8]), ybc=rng.choice(["periodic", "zero-inflow", "specular"]),
                mixed=rng.random() < 0.7)


# ------------------------------------------------------------------------------------------------ devices

def _rtd_spec(case, r):
    """A diode of the case's shape, its length following the number of elements as in the repository's
    configurations (a third of a nm per element), 30 nm at least."""
    length = max(30.0, case["n_el"] / 3.0 if case["n_el"] > 120 else case["n_el"] / 2.0)
    return devices.RTDSpec(length_nm=length, contact_nm=length / 4, barrier_ev=r.uniform(0.24, 0.3),
                           barrier_nm=r.uniform(2.0, 3.5), well_nm=r.uniform(4.0, 6.0),
                           doping_m3=1e24 * r.uniform(0.8, 1.2), m_rel=0.067, order=case["order"], n_el=case["n_el"],
                           nk=case["nk"], n_xi=case.get("n_xi", 0))


def _dropin_inputs(case, r):
    if case["device"] == "fet":
        spec = devices.FETSpec(order=case["order"], n_el=case["n_el"], nk=case["nk"], n_modes=case["modes"],
                               width_nm=r.uniform(4.5, 5.5), barrier_ev=r.uniform(0.42, 0.48))
        return devices.make_fet(spec, r.uniform(0.0, 0.6), r.uniform(0.3, 0.4))
    spec = _rtd_spec(case, r)
    mat = devices.make_mat(spec)
    bias, nm = r.uniform(0.05, 0.2), case["modes"]
    mat["n_of_modes"] = nm
    esub = (devices.flatband_potential(mat, bias)[:, None] + 0.03 * np.arange(nm)[None, :])[None]
    vsub = np.ones((1, mat["Nx"], nm, 1))
    return (mat, esub, vsub) + devices.contact_fermi_levels(mat, bias)


def _transport_inputs(case, r):
    spec = _rtd_spec(case, r)
    mat = devices.make_mat(spec)
    biases = np.linspace(0.02, 0.3, case["batch"]) + r.uniform(0.0, 0.02)
    pots = []
    for v in biases:
        e = devices.flatband_potential(mat, v) + 0.01 * r.uniform(-1, 1) * np.sin(np.pi * mat["ramp"])
        pots.append((e,) + devices.contact_fermi_levels(mat, v))
    return mat, np.full(mat["Nx"], spec.m_rel * 9.109e-31), pots


def _gummel_options(case, **kw):
    return dict(dict(mixing=0.3, maxIterations=case.get("iterations", 4), precision=case["precision"],
                     transportTolerance=TOL, transportMaxCycles=MAXIT), **kw)


def _subband_inputs(case, r):
    """Cross-sections of gated thin bodies between oxides (devices.utb_cross_section) on the case's grid."""
    dy = 7.0 / (case["ny"] - 1)
    spec = devices.FETSpec(n_el=(case["nx"] - 1), order=1, width_nm=7.0 - 2 * 10 * dy, oxide_nm=10 * dy)
    me, V = None, []
    for vg in np.sort(r.uniform(0.0, 0.6, case["batch"])):
        _, _, me, v = devices.utb_cross_section(spec, vg, 0.4, dy_nm=dy, bend_ev=r.uniform(0.03, 0.08))
        V.append(v)
    me, V = me[:case["valleys"]], np.stack(V)
    return dy, np.ascontiguousarray(np.broadcast_to(me, (case["batch"],) + me.shape)), V


def _equilibrium(mat, case, drift):
    """An initial Wigner function (INIT.rho): in every DG node the contact's Fermi occupation, weighted so that
    the density follows the doping, a little shifted in k."""
    p, nl = mat["dg"]["params"], case["order"] + 1
    hb, m0, q, kt = 6.626e-34 / 2 / np.pi, 9.109e-31, 1.602e-19, 1.38e-23 * mat["Temp"]
    k = -2 * np.pi / p["Ly"] * (np.arange(1, p["N"] + 1) - 0.5 * (p["N"] + 1))
    kz = np.linspace(0.0, 2.5e9, 1001)
    e = hb ** 2 * (k * (1 + drift)) ** 2 / 2 / (mat["me_z_ch"] * m0) - 0.05 * q
    f = 2 / np.pi * kz[1] * np.sum(1 / (1 + np.exp(np.minimum(
        (e[:, None] + hb ** 2 * kz ** 2 / 2 / (mat["me_z_ch"] * m0)) / kt, 600.0))), 1)
    x, L = mat["x"], mat["L_x"]
    shape = 0.5 * (2 - np.tanh((x - L / 4) / 3) + np.tanh((x - 3 * L / 4) / 3))
    node = (np.arange(case["n_el"])[:, None] * (nl - 1) + np.arange(nl)).ravel()
    return np.ascontiguousarray((shape[node, None] * f[None, :] / np.sqrt(p["Ly"])).ravel() + 0j)


def _lobatto(n):
    """The n Gauss-Lobatto nodes and weights on [-1, 1]."""
    p = np.polynomial.legendre.Legendre.basis(n - 1)
    x = np.concatenate([[-1.0], np.sort(p.deriv().roots().real), [1.0]])
    return x, 2.0 / (n * (n - 1) * p(x) ** 2)


def _legendre(n, x):
    """Orthonormal Legendre polynomials 0..n-1 at x, and their derivatives, as columns."""
    v, d = [], []
    for j in range(n):
        p = np.polynomial.legendre.Legendre.basis(j) * math.sqrt(j + 0.5)
        v.append(p(x))
        d.append(p.deriv()(x) if j else np.zeros_like(x))
    return np.stack(v, 1), np.stack(d, 1)


def _axis(coord_m, nk, n_el):
    r, _ = _lobatto(nk)
    v, _ = _legendre(nk, r)
    vi = np.linalg.inv(v)
    verts = np.linspace(coord_m[0], coord_m[-1], n_el + 1)
    return dict(nl=nk, ne=n_el, nd=nk * n_el, r=r, M=vi.T @ vi, verts=verts, jac=np.diff(verts) / 2)


def _poisson_inputs(case, r):
    nx, ny = case["nx"], case["ny"]
    dx, dy = 90.0 / (nx - 1), 3.0 / (ny - 1)
    x, y = np.arange(nx) * dx, np.arange(ny) * dy
    well = ((x > 35) & (x < 40)) | ((x > 50) & (x < 55))
    eps = np.where(well, 11.6, 12.9)[:, None] * np.ones((1, ny))
    nd = np.where((x < 25) | (x > 65), 1e24 * r.uniform(0.8, 1.2), 1e21)[:, None] * np.ones((1, ny))
    mat = dict(Nx=nx, Ny=ny, dx=dx, dy=dy, x=x, y=y, eps=eps, Nd=nd, Temp=300.0,
               poisson=dict(yBoundary="periodic" if case["periodic"] else "neumann"))
    p = dict(X=_axis(x * 1e-9, case["nk"], case["n_el_x"]), Y=_axis(y * 1e-9, case["nk"], case["n_el_y"]))
    B = case["batch"]
    xd, yd = [np.add.outer((a["verts"][:-1] + a["verts"][1:]) / 2, a["jac"][0] * a["r"]).ravel() * 1e9
              for a in (p["X"], p["Y"])]
    n_dg = np.interp(xd, x, nd[:, 0])[None, :, None] * (
        1 + 0.1 * r.uniform(-1, 1, (B, 1, 1)) * np.cos(xd / 7)[None, :, None] * np.cos(2 * np.pi * yd / 3)[None, None])
    bias = np.linspace(0.0, 0.6, B) if B > 1 else np.array([r.uniform(0.0, 0.6)])
    ramp = np.clip((x - 30) / 30, 0, 1)
    phi0 = bias[:, None, None] * ramp[None, :, None] + 0.02 * r.uniform(-1, 1, (B, 1, 1)) * np.sin(
        np.pi * x / 90)[None, :, None] * np.ones((1, 1, ny))
    return mat, p, n_dg, phi0, bias


def _full2d_inputs(case, r):
    nex, ney = case["n_el_x"], case["n_el_y"]
    lx, ly = 0.75 * nex if nex >= 20 else 20.0, 3.0
    x, y = np.linspace(0, lx, 2 * nex + 1), np.linspace(0, ly, 2 * ney + 1)
    prm = dict(N_K_X=3, N_K_Y=3, N_el_X=nex, N_el_Y=ney, N_rho_x=case["n_rho_x"], N_rho_y=case["n_rho_y"],
               L_rho_x=0.8e-9 * case["n_rho_x"], full2D_X_flux="upwind", full2D_Y_flux="upwind",
               full2D_Y_boundary=case["ybc"], full2D_potentialQuadratureOrder=5,
               full2D_reservoirModel="material-default")
    if case["ybc"] != "periodic":
        prm["L_rho_y"] = ly * 1e-9
    mat = dict(x=x, y=y, Nx=len(x), Ny=len(y), me_x_ch=0.063, me_y_ch=0.063, me_z_ch=0.063, Temp=300.0, deg_factor=1,
               dg=dict(params=prm))
    c, X = lx / 2, x[:, None] + 0 * y[None, :]
    b = r.uniform(0.1, 0.2)
    V = 1.424 + b * (np.exp(-((X - c + 4) / 1.2) ** 2) + np.exp(-((X - c - 4) / 1.2) ** 2)) \
        - r.uniform(0.03, 0.08) * np.clip((X - 0.3 * lx) / (0.4 * lx), 0, 1) \
        + 0.005 * np.cos(2 * np.pi * y / ly)[None, :] * np.exp(-((X - c) / 4) ** 2)
    return mat, V, 1.474, 1.424


def prepare(case, seed):
    r = np.random.default_rng(seed)
    kind, s = case["kind"], dict(case=case)
    if kind == "dropin":
        s["args"] = _dropin_inputs(case, r)
        mat = s["args"][0]
        s["P"] = Problem1D(batch=mat["n_of_valleys"] * mat["n_of_modes"], precision=case["precision"],
                           **shape_from_mat(mat))
    elif kind == "transport":
        s["mat"], s["m"], s["pots"] = _transport_inputs(case, r)
        s["P"] = Problem1D(batch=case["batch"], precision=case["precision"], fp64_tc=case["fp64_tc"],
                           **shape_from_mat(s["mat"]))
    elif kind == "gummel":
        s["mat"] = devices.make_mat(_rtd_spec(case, r))
        s["mat"]["dy_norm_nm"] = devices.density_normalisation_nm(s["mat"])
        s["biases"] = np.linspace(0.02, 0.3, case["batch"]) + r.uniform(0.0, 0.02)
        s["options"] = _gummel_options(case)
    elif kind == "transient":
        mat = devices.make_mat(_rtd_spec(case, r))
        mat["dy_norm_nm"] = devices.density_normalisation_nm(mat)
        s["S"] = RTDSweep(mat, case["batch"], _gummel_options(case))
        s["bias"] = r.uniform(0.05, 0.3, case["batch"])
        s["rho"] = [_equilibrium(mat, case, r.uniform(-0.02, 0.02)) for _ in range(case["batch"])]
    elif kind == "subbands":
        s["dy"], me, V = _subband_inputs(case, r)
        s["solver"] = SubbandSolver(case["valleys"], case["nx"], case["ny"], case["modes"], batch=case["batch"])
        s["me"], s["V"] = me, V
        if case["on_device"]:
            s["me"], s["V"] = torch.from_numpy(me).cuda(), torch.from_numpy(V).cuda()
            shape = (case["batch"], case["valleys"], case["nx"], case["modes"])
            s["E"] = torch.empty(shape, dtype=torch.float64, device="cuda")
            s["Vsub"] = torch.empty(shape + (case["ny"],), dtype=torch.float64, device="cuda")
    elif kind == "poisson":
        mat, p, s["n_dg"], s["phi0"], s["bias"] = _poisson_inputs(case, r)
        s["op"] = Poisson2D(mat, batch=case["batch"])
        s["op"].set_projection(p, mat)
    else:
        mat, V, efl, efr = _full2d_inputs(case, r)
        s["op"] = Full2DOperator(mat, V)
        s["op"].set_preconditioner()
        s["rhs"], _ = s["op"].reservoir_rhs(efl, efr)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "dropin":
        DG = solve_transport_DG_2D(*s["args"], tol=TOL, maxit=MAXIT, problem=s["P"])
        return {"n": DG["n"], "j": DG["j"], "RHO": DG["RHO"]}
    if kind == "transport":
        P, mat = s["P"], s["mat"]
        for b, (e, efl, efr) in enumerate(s["pots"]):
            P.set_potential(b, mat["x"], e, s["m"], mat["me_z_ch"], mat["Temp"], efl, efr)
        P.solve(tol=TOL, maxit=MAXIT)
        nj = [P.observables(b) for b in range(case["batch"])]
        return {"n": np.stack([a for a, _ in nj]), "j": np.stack([b for _, b in nj])}
    if kind == "gummel":
        sw = solve_rtd_self_consistent(s["mat"], s["biases"], s["options"], handles=case["handles"])["sweep"]
        return {k: sw[k] for k in ("phi", "density", "current")}
    if kind == "transient":
        S = s["S"]
        for b, v in enumerate(s["bias"]):
            S.set(b, 0.0)
            S.P.set_rho(b, s["rho"][b])
            S.step_bias(b, v)
        _, _, n, j = S.transient(1e-15, case["steps"], "cn", refresh_every=1, refresh_first=1, tol=TOL, maxit=20)
        return {"n": n, "j": j, "phi": np.stack([S.get(b)[0] for b in range(case["batch"])])}
    if kind == "subbands":
        if not case["on_device"]:
            E, V = s["solver"].solve(s["me"], s["V"], s["dy"])
            return {"E": E, "V": V}
        ptr = [C.c_void_p(s[k].data_ptr()) for k in ("me", "V", "E", "Vsub")]
        s["solver"].solve_device(s["dy"], *ptr, stream=C.c_void_p(torch.cuda.current_stream().cuda_stream))
        return {"E": s["E"], "V": s["Vsub"]}
    if kind == "poisson":
        one = case["batch"] == 1
        phi, density, info = s["op"].solve(s["n_dg"], s["phi0"], s["bias"], method="newton-raphson", dg=True)
        keys = ("iter_err", "unmixed_step", "residual_scale", "source_integral", "target_integral")
        return {"phi": phi, "density": density,
                "info": np.array([[i[k] for k in keys] for i in ([info] if one else info)])}
    op = s["op"]
    _, _, rho = op.solve(s["rhs"], tol=1e-10, maxit=400, restart=40, mixed=case["mixed"])
    o = op.observables_all()
    return dict({k: o[k] for k in ("n", "jx", "jy", "j")}, rho=rho)


# ------------------------------------------------------------------------------------------------ work

# Krylov iterations of one solve of a kind (measured, nearly independent of the size)
ITERATIONS = dict(transport=200, dropin=200, gummel=200, transient=20, full2d=500)


def work(case):
    kind = case["kind"]
    if kind == "subbands":
        slices, ny, nm = case["batch"] * case["valleys"] * case["nx"], case["ny"], case["modes"]
        # per eigenpair: its location to half precision and one refinement, then the vector; about 10 sweeps
        return {"bytes": 8.0 * slices * (ny + ny / case["valleys"] + nm * (1 + ny)),
                "flops": slices * nm * 10 * 6.0 * ny}
    if kind == "poisson":
        nodes, nu = case["batch"] * case["nx"] * case["ny"], case["ny"] - int(case["periodic"])
        dofs = case["batch"] * case["n_el_x"] * case["n_el_y"] * case["nk"] ** 2
        # block elimination over x: one LU and two solves of each column's block
        return {"bytes": 8.0 * (3 * nodes + dofs), "flops": case["batch"] * case["nx"] * (2 / 3 * nu ** 3 + 4.0 * nu ** 2)}
    if kind == "full2d":
        nrel, npt = case["n_rho_x"] * case["n_rho_y"], 9 * case["n_el_x"] * case["n_el_y"]
        n, size = float(nrel * npt), 8 if case["mixed"] else 16
        its = ITERATIONS[kind]
        # per iteration: the operator and the preconditioner read and write a state each, the basis is read twice
        return {"bytes": its * n * size * (4 + 2 * 20), "flops": its * n * (8 * 3 * 9 + 16 * case["n_rho_x"] + 160)}
    nk, nl = case["nk"], case["order"] + 1
    n_xi = case.get("n_xi") or nk
    batch = case.get("batch") or case["modes"] * (2 if case["device"] == "fet" else 1)
    solves = {"gummel": min(case.get("iterations", 1), 20), "transient": case.get("steps", 1)}.get(kind, 1)
    nodes = float(batch * case["n_el"] * nl)
    n, size = nodes * nk, 8 if case["precision"] == "mixed" else 16
    its = ITERATIONS[kind] * solves
    # per iteration: the operator and the preconditioner read and write a state each and the operator its
    # potential weights; the basis (about 20 vectors, half as wide in the mixed form) is read twice
    basis = size if case["precision"] == "fp64" else size / 2
    by = n * (4 * size + 40 * basis) + nodes * (nl + 1) / 2 * (n_xi + 1) * size / 2
    # two transforms (by FFT), the flux, the xi stencil and 20 vectors' inner products and updates
    fl = nodes * (2 * 5 * n_xi * math.log2(2 * n_xi) + nk * (16 * nl + 20 * 16) + n_xi * 16 * nl)
    return {"bytes": its * by, "flops": its * fl}


# ------------------------------------------------------------------------------------------------ exact values

def exact(case, seed):
    r = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "transport":
        if case["batch"] * case["n_el"] * ((case["order"] + 1) * case["nk"]) ** 3 > 6e11:
            return None                                    # over about 20 seconds
        mat, m, pots = _transport_inputs(case, r)
        nj = [_transport_exact(mat, e, m, efl, efr)[:2] for e, efl, efr in pots]
        return {"n": np.stack([a for a, _ in nj]), "j": np.stack([b for _, b in nj])}
    if kind == "dropin":
        nv = 2 if case["device"] == "fet" else 1
        if nv * case["modes"] * case["n_el"] * ((case["order"] + 1) * case["nk"]) ** 3 > 8e11:
            return None
        mat, esub, vsub, efl, efr = _dropin_inputs(case, r)
        nl, ne = case["order"] + 1, case["n_el"]
        node = (np.arange(ne)[:, None] * (nl - 1) + np.arange(nl)).ravel()
        n, j, rho = 0.0, 0.0, []
        for iv in range(nv):
            for im in range(case["modes"]):
                nn, jj, ru = _transport_exact(mat, esub[iv, :, im], mat["me_x"][iv, :, 0] * 9.109e-31, efl, efr)
                n = n + nn[:, None] * np.abs(vsub[iv, node, im]) ** 2 / mat["dy"] / 1e-9
                j = j + jj
                rho.append(ru)
        return {"n": n, "j": j, "RHO": np.stack(rho).reshape(nv, case["modes"], *rho[0].shape)}
    if kind == "subbands":
        if case["batch"] * case["valleys"] * case["nx"] * case["ny"] ** 2 > 4e7:
            return None
        return _subbands_exact(case, *_subband_inputs(case, r))
    if kind == "poisson":
        return _poisson_exact(*_poisson_inputs(case, r))
    return None    # a loop over solves, or a four-dimensional system: too long to eliminate directly


def _transport_exact(mat, esub, m, efl, efr):
    """n, j and the Wigner function over xi of one subband: the transport system in the plane-wave basis,
    assembled per element and eliminated over x in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    prm = mat["dg"]["params"]
    nl, nk, nxi, lxi = prm["N_K_chi"], prm["N"], prm["N_xi"], prm["Ly"]
    nx, lx = mat["Nx"], mat["L_x"] * 1e-9
    ne = (nx - 1) // (nl - 1)
    hbar, qe, hb, kb, qv, m0 = 1.054571817e-34, 1.602176634e-19, 6.626e-34 / 2 / np.pi, 1.38e-23, 1.602e-19, 9.109e-31
    qdiff, qdrift = hbar / (0.041 * 9.1094e-31), qe / hbar
    dchi, dxi = lx / ne, lxi / (nxi - 1)
    xi = np.linspace(-(lxi - dxi) / 2, (lxi - dxi) / 2, nxi)
    k = -2 * np.pi / lxi * (np.arange(1, nk + 1) - 0.5 * (nk + 1))
    phi = np.exp(1j * np.outer(xi, k)) / np.sqrt(lxi)
    # contact occupation, cosine transformed and projected on the plane waves
    kz = np.linspace(0.0, np.sqrt(4 * m0 * mat["me_z_ch"] * qv * (esub.max() + 0.3)) / hb, 1001)
    ekz = hb ** 2 * kz ** 2 / 2 / m0 / mat["me_z_ch"] / qv
    occ = []
    for end, ef in ((0, efl), (-1, efr)):
        ek = esub[end] + hb ** 2 * k ** 2 / 2 / m[end] / qv
        with np.errstate(over="ignore"):
            f = 2 / np.pi * kz[1] * np.sum(1 / (1 + np.exp(qv * (ek[:, None] + ekz - ef) / (kb * mat["Temp"]))), 1)
        occ.append(np.cos(np.outer(xi, k)) @ f * abs(k[1] - k[0]) / 2 / np.pi)
    fnl, fnr = np.linalg.lstsq(phi, np.stack(occ, 1).astype(complex), rcond=None)[0].T
    # element matrices
    rn, _ = _lobatto(nl)
    v, dv = _legendre(nl, rn)
    vi = np.linalg.inv(v)
    mass = vi.T @ vi
    stiff = mass @ dv @ vi
    im = np.linalg.inv(dxi / 2 * mass)
    first, last = np.eye(nl)[0], np.eye(nl)[-1]
    pl, pr = np.outer(first, first), np.outer(last, last)
    k1 = im @ (stiff + 0.5 * pl - 0.5 * pr)
    k2 = im @ (0.5 * pl + 0.5 * pr)
    sc = 2 * qdiff / dchi
    # potential differences on the quadrature points and xi edges, absorbing layers, weights of the node pairs
    q, w = _lobatto(10)
    ye = np.linspace(-lxi / 2, lxi / 2, nxi + 1)
    xq = (np.arange(ne)[:, None] + (q + 1) / 2) * dchi

    def lookup(x):
        u = np.interp(x, mat["x"] * 1e-9, esub)
        return np.where(x >= lx, esub.min(), np.where(x < 0, esub[0], u))
    l0, wd = lxi / 2 - dxi, 0.4 * lxi
    cap = ((ye - l0 + wd) / wd) ** 2 * (ye >= l0 - wd) + ((ye + l0 - wd) / wd) ** 2 * (ye <= -l0 + wd)
    bq = lookup(xq[..., None] + ye / 2) - lookup(xq[..., None] - ye / 2) - 1j * cap
    wq = _legendre(nl, q)[0] @ vi
    beta = np.einsum("q,qa,qb,eqs->eabs", w, wq, wq, bq) * (qdrift * im)[None, :, :, None] * dxi / 4
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev, dtype=torch.complex128)  # noqa: E731
    ph, beta, n = t(phi), t(beta), nl * nk
    main, off = beta[..., :-1] + beta[..., 1:], beta[..., 1:-1]
    flux = torch.kron(t(k1), torch.diag(t(k))) + torch.kron(t(k2), torch.diag(t(np.abs(k))))
    low = sc * torch.kron(t(-0.5 * im[:, :1]), torch.diag(t(k + np.abs(k))))         # acts on the left neighbour's last node
    up = sc * torch.kron(t(0.5 * im[:, -1:]), torch.diag(t(k - np.abs(k))))          # on the right neighbour's first node
    rhs = np.zeros((ne, nl, nk), dtype=complex)
    rhs[0] += sc * im[:, :1] * ((k > 0) * np.abs(k) * fnl)
    rhs[-1] += sc * im[:, -1:] * ((k < 0) * np.abs(k) * fnr)
    rhs = t(rhs.reshape(ne, n, 1))
    elim, x = [], None
    for e in range(ne):
        cp = main[e][..., None] * ph
        cp[:, :, :-1] += off[e][..., None] * ph[1:]
        cp[:, :, 1:] += off[e][..., None] * ph[:-1]
        g = 1j * torch.einsum("sj,absm->ajbm", ph.conj(), cp).reshape(n, n)
        d, b = sc * flux + g, rhs[e].clone()
        if e:
            d[:, :nk] -= low @ elim[-1][-nk:, :nk]
            b -= low @ elim[-1][-nk:, nk:]
        elim.append(torch.linalg.solve(d, torch.cat([up, b], 1)))
    rho = [None] * ne
    for e in range(ne - 1, -1, -1):
        rho[e] = elim[e][:, nk:] if e == ne - 1 else elim[e][:, nk:] - elim[e][:, :nk] @ rho[e + 1][:nk]
    ru = (torch.stack(rho).reshape(ne * nl, nk) @ ph.T).cpu().numpy()
    mm = m[(np.arange(ne)[:, None] * (nl - 1) + np.arange(nl)).ravel()]
    c = nxi // 2
    if nxi % 2:
        return ru[:, c].real, qe * hb / mm * (ru[:, c + 1] - ru[:, c - 1]).imag / 2 / dxi, ru
    return (ru[:, c - 1] + ru[:, c]).real / 2, qe * hb / mm * (ru[:, c] - ru[:, c - 1]).imag / dxi, ru


def _subbands_exact(case, dy, me, V):
    """The eigenpairs of smallest magnitude of every slice's transverse Hamiltonian, from a dense symmetric
    eigensolve of the similar symmetric matrix."""
    ny, nm = case["ny"], case["modes"]
    t0 = (6.626e-34 / 2 / np.pi) ** 2 / 2 / (9.109e-31 * dy ** 2 * 1.602e-19 * 1e-18)
    V = np.broadcast_to(V[:, None], me.shape)
    hop = -2 * t0 / (me[..., 1:] + me[..., :-1])
    up, lo = hop.copy(), hop.copy()                    # entries (i, i+1) and (i+1, i)
    d = V.copy()
    d[..., 1:-1] -= hop[..., :-1] + hop[..., 1:]
    d[..., 0], d[..., -1] = d[..., 1], d[..., -2]
    up[..., 0], lo[..., -1] = up[..., 1], lo[..., -2]
    scale = np.cumprod(np.concatenate([np.ones(me.shape[:-1] + (1,)), np.sqrt(lo / up)], -1), -1)
    H = np.zeros(me.shape + (ny,))
    i = np.arange(ny - 1)
    H[..., np.arange(ny), np.arange(ny)] = d
    H[..., i, i + 1] = H[..., i + 1, i] = -np.sqrt(lo * up)
    E, U = np.linalg.eigh(H)
    pick = np.sort(np.argsort(np.abs(E), -1, kind="stable")[..., :nm], -1)
    E = np.take_along_axis(E, pick, -1)
    U = np.swapaxes(np.take_along_axis(U, pick[..., None, :], -1), -1, -2) * scale[..., None, :]
    U /= np.linalg.norm(U, axis=-1, keepdims=True)
    U *= np.sign(U[..., -1:])
    flip = np.einsum("bmy,bxmy->bxm", U[:, 0, 0], U[:, 0]) < -0.5
    flip[:, 0] = False
    U[:, 0] *= np.where(flip, -1.0, 1.0)[..., None]
    return {"E": E[0], "V": U[0]} if case["batch"] == 1 and not case["on_device"] else {"E": E, "V": U}


def _poisson_exact(mat, p, n_dg, phi0, bias):
    """The projected density and one Newton update, eliminated column by column over x."""
    q, kb, eps0 = 1.602176634e-19, 1.380649e-23, 8.8541878128e-12
    nx, ny = mat["Nx"], mat["Ny"]
    per = mat["poisson"]["yBoundary"] == "periodic"
    nu, B = ny - int(per), len(bias)
    maps, widths = [], []
    for a, nodes in ((p["X"], mat["x"] * 1e-9), (p["Y"], mat["y"] * 1e-9)):
        edges = np.concatenate([nodes[:1], (nodes[1:] + nodes[:-1]) / 2, nodes[-1:]])
        T = np.zeros((len(nodes), a["nd"]))
        g, wg = np.polynomial.legendre.leggauss(a["nl"])
        c = np.linalg.inv(np.vander(a["r"], increasing=True))
        for e in range(a["ne"]):
            for i in np.flatnonzero((edges[:-1] < a["verts"][e + 1]) & (edges[1:] > a["verts"][e])):
                lo, hi = max(edges[i], a["verts"][e]), min(edges[i + 1], a["verts"][e + 1])
                z = ((lo + hi) / 2 + (hi - lo) / 2 * g - (a["verts"][e] + a["verts"][e + 1]) / 2) / a["jac"][e]
                T[i, e * a["nl"]:(e + 1) * a["nl"]] = (hi - lo) / 2 * wg @ np.vander(z, a["nl"], increasing=True) @ c
        maps.append(T)
        widths.append(np.diff(edges))
    Tx, Ty, wx, wy = *maps, *widths
    if per:
        Ty[0] += Ty[-1]
        wy[0] += wy[-1]
        Ty, wy = Ty[:-1], wy[:-1]
    charge_n = Tx @ n_dg @ Ty.T                                          # [B, nx, nu] integrals
    dens = charge_n / np.outer(wx, wy)
    src = [np.concatenate([a["M"].sum(0) * j for j in a["jac"]]) for a in (p["X"], p["Y"])]
    source = np.einsum("x,bxy,y->b", src[0], n_dg, src[1])
    er, net = mat["eps"][:, :nu], mat["Nd"][:, :nu]
    cx, cy = eps0 * 1e18 / mat["dx"] ** 2, eps0 * 1e18 / mat["dy"] ** 2
    har = lambda a, b: 2 * a * b / (a + b)  # noqa: E731
    fx = cx * har(er[1:], er[:-1])
    A = np.zeros((nx, nu, nu))                                           # the Y couplings and the diagonal
    for i in range(nu if per else nu - 1):
        j = (i + 1) % nu
        f = cy * har(er[:, i], er[:, j])
        for a, b in ((i, j), (j, i)):
            ff = f * (2 if not per and a in (0, nu - 1) else 1)
            A[:, a, b] += ff
            A[:, a, a] -= ff
    A[1:, np.arange(nu), np.arange(nu)] -= fx
    A[:-1, np.arange(nu), np.arange(nu)] -= fx
    old = phi0[:, :, :nu]
    v = old.copy()
    v[:, 0], v[:, -1] = 0.0, bias[:, None]
    Av = np.einsum("xij,bxj->bxi", A, v)
    Av[:, 1:-1] += fx[:-1] * v[:, :-2] + fx[1:] * v[:, 2:]
    F = (Av - q * (dens - net))[:, 1:-1]
    scale = np.maximum.reduce([np.abs(q * dens[:, 1:-1]).max((1, 2)), np.full(B, np.abs(q * net[1:-1]).max()),
                               np.abs(Av[:, 1:-1]).max((1, 2)), np.full(B, q)])
    D = np.broadcast_to(A[1:-1], (B, nx - 2, nu, nu)).copy()
    D[..., np.arange(nu), np.arange(nu)] -= q * q * dens[:, 1:-1] / (kb * mat["Temp"])
    G, h = [], []
    for i in range(nx - 2):
        S, b = D[:, i], -F[:, i]
        if i:
            S = S - fx[i][None, :, None] * G[-1]
            b = b - fx[i] * h[-1]
        sol = np.linalg.solve(S, np.concatenate([np.broadcast_to(np.diag(fx[i + 1]), S.shape), b[..., None]], -1))
        G.append(sol[..., :-1])
        h.append(sol[..., -1])
    d = np.zeros((B, nx, nu))
    for i in range(nx - 3, -1, -1):
        d[:, i + 1] = h[i] - (np.einsum("bij,bj->bi", G[i], d[:, i + 2]) if i < nx - 3 else 0)
    new = v + d
    info = np.stack([np.sqrt(((new - old)[:, 1:-1] ** 2).sum((1, 2))), np.abs(d).max((1, 2)), scale, source,
                     charge_n.sum((1, 2))], 1)
    if per:
        new, dens = [np.concatenate([a, a[:, :, :1]], 2) for a in (new, dens)]
    return {"phi": new[0] if B == 1 else new, "density": dens[0] if B == 1 else dens, "info": info}
