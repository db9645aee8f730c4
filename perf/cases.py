"""Performance cases of the explicit SMA solid: what its users run, at the
sizes they run it, through the package's public entry points.

A case is a dict of plain values whose ``kind`` says which entry point it
goes through:

* ``steps``       -- ``ExplicitSolid.step``: a chunk of explicit steps up to the
  next output, then the fields the output needs;
* ``assemble``    -- ``ExplicitSolid.assemble``: one element loop on host arrays,
  the call a host code that keeps the time loop makes every step;
* ``postprocess`` -- ``ExplicitSolid.postprocess``: nodal stress and strain output;
* ``law``, ``tangent`` -- ``eval_sld_stress_model_160``: the material plugin on a
  batch of Gauss points, without and with the algorithmic tangent;
* ``gradient``    -- ``surrogate.Surrogate.gradient``: loss and gradient of the
  learned surrogate on one batch.

``exact`` restates the path in plain torch and numpy in 64 bits: law 160 from
an eigen-decomposition, trilinear hexahedra, and the two explicit schemes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import alya_sma_b200 as sma
from alya_sma_b200 import problem as P
from alya_sma_b200 import surrogate as S

MILLION = 1_000_000


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # a host code's material routine asks for the Gauss points of a few
        # elements at a time: nothing but latency and launches
        {"name": "law_few_points_fp64", "kind": "law", "n": 64, "precision": "fp64", "e_mart": 0.0},
        # the plugin on a whole mesh's Gauss points, two moduli
        {"name": "law_3m_points_fp32", "kind": "law", "n": 3 * MILLION + 1, "precision": "fp32", "e_mart": 40000.0},
        # an implicit host code's stress and consistent tangent
        {"name": "tangent_131k_points", "kind": "tangent", "n": 131_071, "precision": "fp64", "e_mart": 0.0},
        # the 40x4x4 uniaxial bar (material calibration): thousands of steps
        # of a mesh far smaller than the GPU, so the time of a step is latency
        {"name": "bar_640_fp64", "kind": "steps", "mesh": "bar", "nx": 40, "ny": 4, "nz": 4, "precision": "fp64",
         "scheme": "cd", "damp": 0.0, "energy": False, "steps": 500},
        # the 640 k-element traction-loaded cantilever, one material
        {"name": "cantilever_640k_fp32", "kind": "steps", "mesh": "cantilever", "nx": 400, "ny": 40, "nz": 40,
         "precision": "fp32", "scheme": "cd", "damp": 0.0, "energy": False, "steps": 100},
        # a damped run with the energy balance on, as the decks that set
        # Rayleigh alpha run it
        {"name": "cantilever_80k_fp64_damped", "kind": "steps", "mesh": "cantilever", "nx": 200, "ny": 20, "nz": 20,
         "precision": "fp64", "scheme": "cd", "damp": 1.0e4, "energy": True, "steps": 100},
        # the 2.0 M-element cylinder, a material per element and a
        # temperature field: the benchmark's workload and the largest case
        {"name": "cylinder_2m_fp32", "kind": "steps", "mesh": "cylinder", "div": 1, "layers": 488, "precision": "fp32",
         "scheme": "cd", "damp": 0.0, "energy": False, "steps": 100},
        # an eighth of it in the reference's own precision
        {"name": "cylinder_250k_fp64", "kind": "steps", "mesh": "cylinder", "div": 1, "layers": 61, "precision": "fp64",
         "scheme": "cd", "damp": 0.0, "energy": False, "steps": 100},
        # a parameter study: specimens of 1,250 to 49,130 elements with a
        # material each, concatenated into one run
        {"name": "ensemble_24_fp32", "kind": "steps", "mesh": "ensemble", "nspec": 24, "precision": "fp32",
         "scheme": "cd", "damp": 0.0, "energy": False, "steps": 64},
        # a host code that keeps the time loop: displacement in, residual
        # out, page-locked host arrays
        {"name": "assemble_250k_fp32", "kind": "assemble", "mesh": "cylinder", "div": 1, "layers": 61,
         "precision": "fp32", "all": False},
        # nodal output of a run
        {"name": "postprocess_80k_fp64", "kind": "postprocess", "mesh": "cantilever", "nx": 200, "ny": 20, "nz": 20,
         "precision": "fp64"},
        # one large batch of the surrogate's training
        {"name": "surrogate_gradient_262k", "kind": "gradient", "n": 262_144},
    ]


def _between(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_mesh(rng):
    mesh = rng.choice(["bar", "cantilever", "cylinder", "cylinder", "ensemble"])
    if mesh == "ensemble":
        return {"mesh": mesh, "nspec": _between(rng, 2, 24)}
    if mesh == "cylinder":
        div = rng.choice([1, 1, 2, 4, 8])
        return {"mesh": mesh, "div": div, "layers": _between(rng, 5, 122)}
    ny, nz = _between(rng, 2, 30), _between(rng, 2, 30)
    return {"mesh": mesh, "nx": _between(rng, 20, 300), "ny": ny, "nz": nz}


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "assemble", "postprocess", "law", "law", "tangent",
                       "gradient"])
    precision = rng.choice(["fp32", "fp64"])
    if kind == "law":
        return {"kind": kind, "n": _between(rng, 64, 3 * MILLION), "precision": precision,
                "e_mart": rng.choice([0.0, 40000.0])}
    if kind == "tangent":
        return {"kind": kind, "n": _between(rng, 64, 200_000), "precision": "fp64",
                "e_mart": rng.choice([0.0, 40000.0])}
    if kind == "gradient":
        return {"kind": kind, "n": _between(rng, 4_096, 500_000)}
    case = {"kind": kind, **_draw_mesh(rng), "precision": precision}
    if kind == "assemble":
        case["all"] = rng.random() < 0.5
    if kind == "steps":
        # the energy balance is an audit of FP64 runs: its work terms cancel
        case.update(scheme=rng.choice(["cd", "cd", "tw"]), damp=rng.choice([0.0, 0.0, 1.0e4]),
                    energy=precision == "fp64" and rng.random() < 0.5, steps=_between(rng, 2, 64))
    return case


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _box_problem(case, seed):
    """The bar (pushed end) or the cantilever (tip traction) at the case's
    resolution, elements of the named workloads' size (1 mm)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    coord, lnods = P.structured_box(nx, ny, nz, float(nx), float(ny), float(nz), 0.05, seed)
    props = P.nitinol_props(**P.NITI)[None, :]
    e_mart, densi = np.array([P.NITI_E_MART]), np.array([P.NITI_DENSITY])
    npoin = coord.shape[0]
    fixno = np.zeros((npoin, 3), np.int32)
    bcfun = np.full(npoin, -1, np.int32)
    fixno[P.face_nodes(coord, 0, 0.0)] = 1
    dt = 0.5 * P.critical_dt(coord, lnods, props, densi)
    push = case["mesh"] == "bar"
    if push:
        tip = P.face_nodes(coord, 0, float(nx))
        fixno[tip, 0] = 1
        bcfun[tip] = 0
    tab = P.smooth_cycle_table(20000 * dt, 0.06 * nx if push else 1.5 * P.NITI["Sf_AS"])
    return P.Problem(coord=coord, lnods=lnods, props=props, e_mart=e_mart, densi=densi, fixno=fixno, bcfun=bcfun,
                     fun_npts=np.array([3], np.int32), fun_smooth=np.array([1], np.int32), fun_tab=tab,
                     fext=None if push else P.face_load(coord, lnods, 0, float(nx), (1.0, 0.0, 0.0)),
                     load_fun=-1 if push else 0, dtime=dt, nsteps=20000, name=case["mesh"])


def _problem(case, seed):
    """The case's mesh, materials and loads, and the displacement it starts
    from: an axial prestrain near 1 %, where the return map is active."""
    mesh = case["mesh"]
    if mesh == "cylinder":
        prob = P.cylinder_2m(seed=seed, div=case["div"], layers=case["layers"])
    elif mesh == "ensemble":
        # the specimens' sizes belong to the case, their materials to the seed
        prob = P.ensemble(nspec=case["nspec"], seed=0)
        f = np.random.default_rng(seed + 3).uniform(0.95, 1.0, size=(case["nspec"], 3))
        prob.props[:, 0] *= f[:, 0]
        prob.props[:, 2:5] *= f[:, 1:2]
        prob.props[:, 9:11] *= f[:, 2:3]
    else:
        prob = _box_problem(case, seed)
    if case.get("damp"):
        prob.dampi = np.tile([case["damp"], 0.0], (prob.props.shape[0], 1))
    eps = float(np.random.default_rng(seed + 7).uniform(0.009, 0.011))
    return prob, np.ascontiguousarray(P.prestrain(prob, eps))


def _solid(case, prob, u):
    solid = sma.ExplicitSolid(prob, precision=case["precision"], scheme=case.get("scheme", "cd"))
    solid.set("displ", u)
    if case.get("energy"):
        solid.set_energy(True)
    return solid


def _gauss_points(n, seed):
    """Gauss points with consistent histories: austenite below the forward
    start, mixtures between the finish lines (away from the corners where the
    flow rule's pivot vanishes), martensite above the reverse start and small
    strains, a quarter each; F = R U whose deviatoric log
    strain is within 5 % of the previous one, rotations up to 0.2 rad.
    (F (n, 3, 3), state (n, 3)) on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def uni(lo, hi, *shape):
        return torch.rand(*(shape or (n,)), generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    pr = P.nitinol_props(**P.NITI)
    shear2 = pr[0] / (1.0 + pr[1])
    rs_as, rf_as, rs_sa, rf_sa = (pr[k] * math.sqrt(2.0 / 3.0) for k in (3, 4, 9, 10))
    kind = torch.arange(n, device="cuda") % 4
    zero = torch.zeros(n, device="cuda", dtype=torch.float64)
    x0 = torch.where(kind == 1, uni(0.05, 0.95), torch.where(kind == 2, zero + 1.0, zero))
    f0 = torch.where(kind == 0, uni(0.0, rs_as), torch.where(kind == 1, uni(rf_sa, rf_as), torch.where(
        kind == 2, uni(rs_sa, 1.5 * rf_as), uni(0.0, 0.05 * rs_as))))
    en = ((f0 / shear2 + pr[2] * x0) * (1.0 + uni(-0.05, 0.05))).clamp_min(1e-7)
    # the activation tests are strict inequalities: the few points within FP32
    # rounding of one, with either modulus, are moved off it
    near = torch.zeros(n, device="cuda", dtype=torch.bool)
    for young in (pr[0], 1.0 / ((1.0 - x0) / pr[0] + x0 / P.NITI_E_MART)):
        load = young / (1.0 + pr[1]) * (en - pr[2] * x0)
        for at in (f0, rs_as, rs_sa):
            near |= (load - at).abs() < 1e-4 * rs_sa
    en = torch.where(near, en * 1.003, en)
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    d = d - d.mean(1, keepdim=True)
    d = d / d.norm(dim=1, keepdim=True)
    lam = torch.exp(en[:, None] * d + uni(-0.005, 0.005)[:, None] / 3.0)

    def turn(angle):                                      # rotations by `angle` about random axes (Rodrigues)
        w = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
        w = w / w.norm(dim=1, keepdim=True)
        k = torch.zeros(n, 3, 3, device="cuda", dtype=torch.float64)
        k[:, 0, 1], k[:, 0, 2], k[:, 1, 2] = -w[:, 2], w[:, 1], -w[:, 0]
        k = k - k.transpose(1, 2)
        eye = torch.eye(3, device="cuda", dtype=torch.float64)
        return eye + torch.sin(angle)[:, None, None] * k + (1.0 - torch.cos(angle))[:, None, None] * (k @ k)

    q = turn(uni(0.0, math.pi))
    f = turn(uni(0.0, 0.2)) @ (q * lam[:, None, :]) @ q.transpose(1, 2)
    return f.contiguous(), torch.stack([x0, f0, f0], 1).contiguous()


def _surrogate_batch(n, seed):
    """Plain-law samples around the cylinder's materials, and a network with
    its normalisation fitted to them: (network, inputs, outputs)."""
    base = P.nitinol_props(**P.NITI, C_AS=6.5 * P.SQRT_2_3, C_SA=6.5 * P.SQRT_2_3, T_ref=300.0)
    x, y = S.generate(base, P.NITI_E_MART, -(-2 * n // 256) + 1, nstep=256, seed=seed, inactive_only=True)
    net = S.Surrogate(seed=seed + 1)
    net.fit_stats(x, y)
    return net, x[:n].contiguous(), y[:n].contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("law", "tangent"):
        f, s0 = _gauss_points(case["n"], seed)
        return {"case": case, "props": P.nitinol_props(**P.NITI), "F": f, "state": s0}
    if kind == "gradient":
        net, x, y = _surrogate_batch(case["n"], seed)
        return {"case": case, "net": net, "x": x, "y": y}
    prob, u = _problem(case, seed)
    st = {"case": case, "solid": _solid(case, prob, u)}
    if kind == "assemble":
        st["u"] = torch.from_numpy(u).pin_memory().numpy()
        st["rhsid"] = torch.empty(u.shape, dtype=torch.float64, pin_memory=True).numpy()
    return st


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
SMALL = 20_000          # meshes of at most this many elements also read the Gauss-point state back


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("law", "tangent"):
        return sma.eval_sld_stress_model_160(st["props"], st["F"], st["state"], flagt=int(kind == "tangent"),
                                             e_mart=case["e_mart"], precision=case["precision"])
    if kind == "gradient":
        return st["net"].gradient(st["x"], st["y"])
    solid = st["solid"]
    if kind == "assemble":
        out = solid.assemble(st["u"], fext_scale=1.0, want_all=case["all"], rhsid=st["rhsid"])
        return {k: v for k, v in out.items() if v is not None}
    if kind == "postprocess":
        return solid.postprocess()
    solid.step(case["steps"])
    out = {"displ": solid.get("displ")}
    if case["energy"]:
        out["energy"] = solid.energy()[0]
    if solid.nelem <= SMALL:
        out["veloc"] = solid.get("veloc")
        out["state"] = solid.state[:, 1]             # slot TIME_N: after the last step
    return out


# --------------------------------------------------------------------------
# work: what the path cannot do without
# --------------------------------------------------------------------------
# flops of one Gauss-point update of the explicit element loop: the reference
# path counted on an instrumented restatement (law included), and the law alone
GP_FLOPS, LAW_FLOPS = 1937.0, 580.0


def _sizes(case):
    """(elements, nodes, materials) of a mesh case."""
    if case["mesh"] == "ensemble":
        k = [int(round((n / 10) ** (1.0 / 3.0))) for n in P.ensemble_sizes(case["nspec"], 0)]
        return sum(10 * v ** 3 for v in k), sum((10 * v + 1) * (v + 1) ** 2 for v in k), case["nspec"]
    if case["mesh"] == "cylinder":
        nc, nr = max(2, 32 // case["div"]), max(1, 24 // case["div"])
        quads, pts = nc * nc + 4 * nc * nr, (nc + 1) ** 2 + 4 * nc * nr
        return quads * case["layers"], pts * (case["layers"] + 1), quads * case["layers"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1), 1


def work(case):
    kind = case["kind"]
    if kind in ("law", "tangent"):
        out = 9 + 3 + (81 if kind == "tangent" else 0)
        return {"bytes": case["n"] * (8.0 * (12 + out) + 4), "flops": case["n"] * LAW_FLOPS * (7 if kind == "tangent" else 1)}
    if kind == "gradient":
        # 14 -> 64 x 4 -> 13: forward, backward and weight gradients
        return {"bytes": case["n"] * 4.0 * 27, "flops": case["n"] * 6.0 * (14 * 64 + 3 * 64 * 64 + 64 * 13)}
    ne, npo, nm = _sizes(case)
    s = 4 if case["precision"] == "fp32" else 8
    # an element loop: connectivity, the state, materials of their own, and
    # the nodes' coordinates and displacement in, the residual out
    loop = ne * (32.0 + (8 * s if nm == ne else 0)) + npo * 72.0
    if kind == "postprocess":
        return {"bytes": loop + ne * 24.0 * s + npo * 8.0 * 19, "flops": 8.0 * ne * GP_FLOPS}
    loop += ne * 2.0 * 24 * s
    if kind == "assemble":
        return {"bytes": loop + (npo * 8.0 * 10 if case["all"] else 0.0), "flops": 8.0 * ne * GP_FLOPS}
    # a step adds the nodal update: residual, half-step velocity and
    # displacement read and the last two written, the inverse mass
    step = loop + npo * 8.0 * (3 * 5 + 1)
    return {"bytes": case["steps"] * step, "flops": case["steps"] * (8.0 * ne * GP_FLOPS + npo * 12.0)}


def tolerance(case):
    """About four times what `exact` and the path were seen to differ by over
    these ranges.  A chunk of steps feeds every rounding back through the
    law's activation tests (strict inequalities), so a Gauss point may start
    transforming a step apart: that, and no single step's rounding, sets the
    FP32 figures, after three chunks in a row."""
    kind, fp64 = case["kind"], case.get("precision") == "fp64"
    if kind == "gradient":                      # BF16 products
        return {"rel": 2e-3, "max": 2e-2}
    if kind == "tangent":                       # forward differences, eps = 1e-5
        return {"rel": 1e-10, "max": 1e-9, "differ": 1e-4}
    if kind == "steps":
        if fp64:
            return {"rel": 1e-9, "max": 1e-6}
        return {"rel": 1e-4, "max": 1e-2} if _sizes(case)[0] > SMALL else {"rel": 1e-3, "max": 0.2}
    return {"rel": 1e-12, "max": 1e-10, "differ": 1e-4} if fp64 else {"rel": 6e-6, "max": 1e-4, "differ": 1e-3}


# --------------------------------------------------------------------------
# the path in 64 bits, in plain torch
# --------------------------------------------------------------------------
GAUSS = 0.577350269189626


def _material(props, e_mart):
    """Law-160 constants of parameter rows (m, 18) and martensite moduli (m,), as columns on the GPU."""
    pr = torch.as_tensor(np.atleast_2d(props), dtype=torch.float64, device="cuda")
    em = torch.as_tensor(np.atleast_1d(e_mart), dtype=torch.float64, device="cuda").expand(pr.shape[0])
    aux = math.sqrt(2.0 / 3.0) + pr[:, 14]
    return {"EA": pr[:, 0], "EM": torch.where(em > 0.0, em, pr[:, 0]), "nu": pr[:, 1], "eL": pr[:, 2], "alfa": pr[:, 14],
            "C_AS": pr[:, 5], "C_SA": pr[:, 11],
            "Rs_AS": pr[:, 3] * aux + pr[:, 5] * pr[:, 7], "Rf_AS": pr[:, 4] * aux + pr[:, 5] * pr[:, 6],
            "Rs_SA": pr[:, 9] * aux + pr[:, 11] * pr[:, 13], "Rf_SA": pr[:, 10] * aux + pr[:, 11] * pr[:, 12]}


def _eigen(a, b, c, d, e, f):
    """Eigenvalues and eigenvectors of symmetric 3x3 matrices (xx, yy, zz, xy,
    yz, xz) by cyclic Jacobi rotations: ([w0, w1, w2], v[row][column])."""
    m = [[a, d, f], [d, b, e], [f, e, c]]
    one, zero = torch.ones_like(a), torch.zeros_like(a)
    v = [[one if i == j else zero for j in range(3)] for i in range(3)]
    for _ in range(5):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            apq = m[p][q]
            th = (m[q][q] - m[p][p]) / (2.0 * torch.where(apq == 0.0, one, apq))
            t = torch.where(th >= 0.0, one, -one) / (th.abs() + torch.sqrt(th * th + 1.0))
            t = torch.where(apq == 0.0, zero, t)
            cs = torch.rsqrt(t * t + 1.0)
            sn = t * cs
            m[p][p], m[q][q] = m[p][p] - t * apq, m[q][q] + t * apq
            arp, arq = m[r][p], m[r][q]
            m[p][q] = m[q][p] = zero
            m[r][p] = m[p][r] = cs * arp - sn * arq
            m[r][q] = m[q][r] = sn * arp + cs * arq
            for i in range(3):
                v[i][p], v[i][q] = cs * v[i][p] - sn * v[i][q], sn * v[i][p] + cs * v[i][q]
    return [m[0][0], m[1][1], m[2][2]], v


PAIRS = ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2))


def _law(mat, h, tmp, state):
    """Kirchhoff stress [6 components], new state [xS, F_AS, F_SA], the flag
    and ln V [6] of F = I + h (h[3 i + j]).  Both transformations cannot be
    active at once here: their slopes and previous loading values are equal."""
    a = [h[3 * i + j] + h[3 * j + i] + sum(h[3 * i + k] * h[3 * j + k] for k in range(3)) for i, j in PAIRS]
    w, v = _eigen(*a)
    lg = [0.5 * torch.log1p(x) for x in w]
    lnv = [sum(lg[k] * v[i][k] * v[j][k] for k in range(3)) for i, j in PAIRS]
    del v
    theta = lg[0] + lg[1] + lg[2]
    en = torch.sqrt(sum((x - theta / 3.0) ** 2 for x in lg))
    x0, fas0, fsa0 = state
    young = 1.0 / ((1.0 - x0) / mat["EA"] + x0 / mat["EM"])
    bulk, shear = young / (3.0 - 6.0 * mat["nu"]), young / (2.0 + 2.0 * mat["nu"])
    el, alfa = mat["eL"], mat["alfa"]
    g1 = (2.0 * shear + 9.0 * alfa * alfa * bulk) * el

    def load(c, x):
        return 2.0 * shear * (en - el * x) + 3.0 * alfa * bulk * (theta - 3.0 * alfa * el * x) - c * tmp

    fas, fsa = load(mat["C_AS"], x0), load(mat["C_SA"], x0)
    k_as = (fas > fas0) & (fas - mat["Rs_AS"] > 0.0) & (x0 < 1.0)
    k_sa = (fsa < fsa0) & (fsa - mat["Rs_SA"] < 0.0) & (x0 > 0.0)
    rhs = torch.where(k_as, (fas - fas0) * (1.0 - x0), -(fsa - fsa0) * x0)
    piv = torch.where(k_as, (fas - mat["Rf_AS"]) - (fas - fas0) - (1.0 - x0) * g1,
                      (fsa - mat["Rf_SA"]) - (fsa - fsa0) + x0 * g1)
    go = (k_as | k_sa) & (rhs * rhs > 1.0e-8)
    x = torch.where(go, x0 - rhs / torch.where(go, piv, torch.ones_like(piv)), x0)
    fas, fsa = load(mat["C_AS"], x), load(mat["C_SA"], x)
    x = x.clamp(0.0, 1.0)
    pv = bulk * (theta - 3.0 * alfa * el * x)
    tiny = torch.finfo(torch.float64).eps
    kp = 2.0 * shear * torch.where(en > tiny, 1.0 - el * x / en.clamp_min(tiny), torch.ones_like(en))
    tau = [kp * lnv[k] + (pv - kp * theta / 3.0 if k < 3 else 0.0) for k in range(6)]
    return tau, [x, fas, fsa], (k_as | k_sa).to(torch.int32), lnv


def _inverse(m):
    """Inverse and determinant of (..., 3, 3)."""
    r = [m[..., k, :] for k in range(3)]
    cof = torch.stack([torch.linalg.cross(r[1], r[2]), torch.linalg.cross(r[2], r[0]), torch.linalg.cross(r[0], r[1])], -1)
    det = (r[0] * cof[..., :, 0]).sum(-1)
    return cof / det[..., None, None], det


def _from6(t):
    return torch.stack([t[0], t[3], t[5], t[3], t[1], t[4], t[5], t[4], t[2]], -1).reshape(*t[0].shape, 3, 3)


class _Mesh:
    """Trilinear hexahedra with 2x2x2 Gauss points: kinematics, forces, masses and the two explicit schemes."""

    def __init__(self, case, prob):
        dev = dict(dtype=torch.float64, device="cuda")
        s = np.array([[-1, 1, 1, -1, -1, 1, 1, -1], [-1, -1, 1, 1, -1, -1, 1, 1], [-1, -1, -1, -1, 1, 1, 1, 1]], float)
        g = GAUSS * np.array([[(k >> 2 & 1) * 2 - 1, (k >> 1 & 1) * 2 - 1, (k & 1) * 2 - 1] for k in range(8)], float)
        f = 0.5 * (1.0 + g[:, :, None] * s[None])                   # (gauss, direction, node)
        dn = np.stack([0.5 * s[0] * f[:, 1] * f[:, 2], 0.5 * s[1] * f[:, 0] * f[:, 2], 0.5 * s[2] * f[:, 0] * f[:, 1]], -1)
        self.N = torch.as_tensor(f.prod(1), **dev)                  # (gauss, node)
        dn = torch.as_tensor(dn, **dev)                             # (gauss, node, direction)
        self.case, self.prob = case, prob
        self.ln = torch.as_tensor(prob.lnods, dtype=torch.int64, device="cuda")
        self.npoin, self.ne = prob.npoin, prob.nelem
        x = torch.as_tensor(prob.coord, **dev)[self.ln]             # (element, node, 3)
        ji, det = _inverse(torch.einsum("eai,gaj->egij", x, dn))
        self.dv = det                                               # (element, gauss)
        d = torch.einsum("gaj,egjk->eagk", dn, ji)
        self.d = d.reshape(self.ne, 8, 24).contiguous()             # dN_a/dX_k at (gauss, k)
        lm = None if prob.lmate is None else torch.as_tensor(prob.lmate, dtype=torch.int64, device="cuda")
        mat = _material(prob.props, prob.e_mart)
        self.mat = {k: (v if lm is None else v[lm][:, None]) for k, v in mat.items()}
        self.tmp = 0.0 if prob.tempe is None else torch.as_tensor(prob.tempe, **dev)[:, None]
        rho = torch.as_tensor(prob.densi, **dev)
        self.rho = rho if lm is None else rho[lm][:, None]
        m = ((self.rho * self.dv) @ self.N).reshape(-1)             # the rows of the consistent mass add up to N
        self.mass = torch.zeros(self.npoin, **dev).index_add_(0, self.ln.reshape(-1), m)
        self.state = [torch.zeros(self.ne, 8, **dev) for _ in range(3)]

    def grad(self, u):
        h = torch.bmm(u[self.ln].transpose(1, 2), self.d).reshape(self.ne, 3, 8, 3)
        return [h[:, i, :, j].contiguous() for i in range(3) for j in range(3)]

    def nodal(self, fe):
        return torch.zeros(self.npoin, 3, dtype=torch.float64, device="cuda").index_add_(0, self.ln.reshape(-1), fe.reshape(-1, 3))

    def forces(self, u):
        """Internal force and the new state at displacement u."""
        h = self.grad(u)
        tau, new, _, _ = _law(self.mat, h, self.tmp, self.state)
        fm = torch.stack(h, -1).reshape(self.ne, 8, 3, 3) + torch.eye(3, dtype=torch.float64, device="cuda")
        fi, _ = _inverse(fm)
        del h, fm
        p = torch.einsum("egik,egjk->egij", _from6(tau), fi) * self.dv[..., None, None]     # dV tau F^-T
        return self.nodal(torch.bmm(self.d, p.transpose(2, 3).reshape(self.ne, 24, 3))), new

    def damping(self, v):
        w = (self.case["damp"] * self.rho * self.dv)[..., None] * torch.einsum("ga,eai->egi", self.N, v[self.ln])
        return self.nodal(torch.einsum("ga,egi->eai", self.N, w))

    def table(self, col, t):
        """The one smooth cycle table 0 -> peak -> 0 at time t."""
        rows = self.prob.fun_table(0)
        for r0, r1 in zip(rows[:-1], rows[1:]):
            if r0[0] <= t <= r1[0]:
                m = (t - r0[0]) / (r1[0] - r0[0])
                return float(r0[1 + col] + (r1[1 + col] - r0[1 + col]) * m ** 3 * (10.0 - 15.0 * m + 6.0 * m * m))
        return float(rows[-1][1 + col] * t / rows[-1][0])

    def steps(self, u):
        case, prob, dt = self.case, self.prob, self.prob.dtime
        dev = dict(dtype=torch.float64, device="cuda")
        tw = case["scheme"] == "tw"
        fixed = torch.as_tensor(prob.fixno == 1, device="cuda")
        timed = torch.as_tensor(prob.bcfun >= 0, device="cuda")
        fext = None if prob.fext is None else torch.as_tensor(prob.fext, **dev)
        v, a = torch.zeros_like(u), torch.zeros_like(u)
        uprev, fint0, fext0 = u.clone(), torch.zeros_like(u), torch.zeros_like(u)
        en, t = {"allie": 0.0, "allwk": 0.0, "allke": 0.0, "eener": 0.0}, 0.0
        for k in range(case["steps"]):
            t += dt
            if tw:
                vt, u = v + dt * a, u + dt * v + 1.033 * dt * dt * a
            else:
                vt = v + 0.5 * dt * a
                u = u + dt * vt
            bc = torch.tensor([self.table(c, t) for c in range(3)], **dev)
            u = torch.where(fixed, torch.where(timed[:, None], bc, torch.zeros_like(bc)), u)
            fx = torch.zeros_like(u) if fext is None else fext * self.table(0, t)
            fi, self.state = self.forces(u)
            r = fx - fi - (self.damping(vt if tw else v) if case["damp"] else 0.0)
            a = r / self.mass[:, None]
            if tw:
                v, a = (torch.where(fixed, torch.zeros_like(x), x) for x in (vt, a))
            else:
                v = vt + 0.5 * dt * a
            if case["energy"]:
                du, w = u - uprev, 1.0 if k == 0 else 0.5
                en["allie"] += w * abs(float(((fi + fint0) * du).sum()))
                en["allwk"] += w * abs(float(((fx + fext0) * du).sum()))
                en["allke"] = 0.5 * float((v * v * self.mass[:, None]).sum())
                en["eener"] = abs(float((r * du).sum()))
                uprev, fint0, fext0 = u, fi, fx
        out = {"displ": u.cpu().numpy()}
        if case["energy"]:
            en["etota"] = en["allie"] + en["allke"] - en["allwk"]
            out["energy"] = en
        if self.ne <= SMALL:
            out["veloc"] = v.cpu().numpy()
            out["state"] = torch.stack(self.state, -1).cpu().numpy()
        return out

    def assemble(self, u):
        prob = self.prob
        fi, _ = self.forces(u)
        fx = torch.zeros_like(u) if prob.fext is None else torch.as_tensor(prob.fext, dtype=torch.float64, device="cuda")
        out = {"rhsid": fx - fi}
        if self.case["all"]:
            fixed = torch.as_tensor(prob.fixno == 1, device="cuda")
            out.update(finte=fi, fexte=fx, frxid=torch.where(fixed, -fi, torch.zeros_like(fi)), vmass=self.mass)
        return {k: x.cpu().numpy() for k, x in out.items()}

    def postprocess(self, u):
        h = self.grad(u)
        tau, _, _, lnv = _law(self.mat, h, self.tmp, self.state)
        fm = torch.stack(h, -1).reshape(self.ne, 8, 3, 3) + torch.eye(3, dtype=torch.float64, device="cuda")
        det = _inverse(fm)[1]
        order = ((0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1))    # Voigt order of the output
        at = [PAIRS.index(p) for p in order]
        gre = [0.5 * (h[3 * i + j] + h[3 * j + i] + sum(h[3 * k + i] * h[3 * k + j] for k in range(3))) for i, j in order]
        rows = torch.stack([tau[k] / det for k in at] + gre + [lnv[k] for k in at] + [torch.ones_like(det)], -1)
        fe = torch.einsum("ga,egq->eaq", self.N, rows * self.dv[..., None])
        acc = torch.zeros(self.npoin, 19, dtype=torch.float64, device="cuda").index_add_(0, self.ln.reshape(-1), fe.reshape(-1, 19))
        acc = acc[:, :18] / acc[:, 18:]
        c = acc[:, :6]
        vm = torch.sqrt(0.5 * ((c[:, 0] - c[:, 1]) ** 2 + (c[:, 1] - c[:, 2]) ** 2 + (c[:, 2] - c[:, 0]) ** 2
                               + 6.0 * (c[:, 3:] ** 2).sum(1)))
        out = {"caust": acc[:, :6], "green": acc[:, 6:12], "lepsi": acc[:, 12:18], "seqvm": vm}
        return {k: x.contiguous().cpu().numpy() for k, x in out.items()}


def _law_batch(mat, f, state):
    """(second Piola stress, Kirchhoff stress, new state, flag) of points F (n, 3, 3)."""
    h = f - torch.eye(3, dtype=torch.float64, device="cuda")
    tau, new, flag, _ = _law(mat, [h[:, i, j].contiguous() for i in range(3) for j in range(3)], 0.0, state)
    fi, _ = _inverse(f)
    tau = _from6(tau)
    return fi @ tau @ fi.transpose(1, 2), tau, torch.stack(new, 1), flag


def _tangent(mat, f, state, tau):
    """The algorithmic tangent by forward differences of the Kirchhoff stress
    at F + eps/2 (e_i e_j + e_j e_i) F, eps = 1e-5, the correction of the
    stress's frame change and the pull-back."""
    eps, n = 1.0e-5, f.shape[0]
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    d = torch.zeros(n, 3, 3, 3, 3, dtype=torch.float64, device="cuda")
    for i in range(3):
        for j in range(3):
            sym = torch.outer(eye[i], eye[j]) + torch.outer(eye[j], eye[i])
            tp = _law_batch(mat, f + 0.5 * eps * (sym @ f), state)[1]
            corr = (torch.einsum("c,nd->ncd", eye[i], tau[:, :, j]) + torch.einsum("c,nd->ncd", eye[j], tau[:, i, :])
                    + torch.einsum("d,nc->ncd", eye[i], tau[:, :, j]) + torch.einsum("d,nc->ncd", eye[j], tau[:, i, :]))
            d[:, i, j] = (tp - tau) / eps - 0.5 * corr
    fi, _ = _inverse(f)
    for _ in range(4):                                              # one index after the other
        d = torch.einsum("npqrs,nip->nqrsi", d, fi)
    return d


def exact(case, seed):
    kind = case["kind"]
    if kind in ("law", "tangent"):
        f, s0 = _gauss_points(case["n"], seed)
        mat, state = _material(P.nitinol_props(**P.NITI), case["e_mart"]), list(s0.T.contiguous())
        pk2, tau, new, flag = _law_batch(mat, f, state)
        return (pk2, new, None) + ((_tangent(mat, f, state, tau),) if kind == "tangent" else ())
    if kind == "gradient":
        net, x, y = _surrogate_batch(case["n"], seed)
        return _mlp_gradient(net, x.double(), y.double())
    prob, u = _problem(case, seed)
    mesh = _Mesh(case, prob)
    return getattr(mesh, kind)(torch.as_tensor(u, dtype=torch.float64, device="cuda"))


def _mlp_gradient(net, x, y):
    """Mean squared error of the normalised outputs and its gradient, laid out
    as the network's parameters, on its BF16 weights."""
    w = torch.as_tensor(net.params_bf16(), dtype=torch.float64, device="cuda").requires_grad_()
    st = torch.as_tensor(net.stats_array(), device="cuda")
    mx, sx, my, sy = st[:14], st[14:28], st[28:41], st[41:54]
    z = torch.nn.functional.pad((x - mx) / sx, (0, 2))
    for k, (n_in, n_out) in enumerate(((16, 64), (64, 64), (64, 64), (64, 64), (64, 16)), 1):
        at, b = S.OFF["W%d" % k], S.OFF["b%d" % k]
        z = z @ w[at:at + n_in * n_out].reshape(n_out, n_in).T + w[b:b + n_out]
        if k < 5:
            z = z * torch.sigmoid(z)
    loss = (((z[:, :13] - (y - my) / sy)) ** 2).mean()
    loss.backward()
    return float(loss.detach()), w.grad.cpu().numpy()
