"""The thread-per-element kernel against the 8-lane one: meshes large enough
to take it by default, element counts that are no multiple of its warps or
state tiles, every material layout, and Gauss points that leave its short
forms (large strains, inverted elements)."""
import dataclasses

import numpy as np
import pytest

import alya_sma_b200 as sma
from alya_sma_b200 import problem as P

pytestmark = pytest.mark.gpu


def _mesh(kind):
    """20,060 elements (not a multiple of 32), above the kernel's threshold of
    one warp per scheduler."""
    nx, ny, nz = 59, 17, 20
    coord, lnods = P.structured_box(nx, ny, nz, float(nx), float(ny), float(nz), 0.1, 5)
    ne, npo = len(lnods), len(coord)
    rng = np.random.default_rng(6)
    props, em = P.nitinol_props(**P.NITI)[None, :], np.array([P.NITI_E_MART])
    lmate = None
    if kind == "one_modulus":
        em = np.zeros(1)
    if kind in ("compact", "table"):
        nm = ne if kind == "compact" else 7
        props = np.tile(P.nitinol_props(**P.NITI, C_AS=5.0, C_SA=5.0, T_ref=300.0), (nm, 1))
        f = rng.uniform(0.9, 1.1, size=(nm, 3))
        props[:, 0] *= f[:, 0]
        props[:, 2] *= f[:, 1]
        props[:, 3:5] *= f[:, 2:]
        em = P.NITI_E_MART * f[:, 1]
        lmate = rng.integers(0, nm, ne).astype(np.int32) if kind == "table" else np.arange(ne, dtype=np.int32)
        if kind == "table":
            props[:, 1] = rng.uniform(0.3, 0.35, nm)       # Poisson's ratio: no compact record
            props[:, 14] = 0.02                             # pressure sensitivity
    fixno = np.zeros((npo, 3), np.int32)
    fixno[P.face_nodes(coord, 0, 0.0)] = 1
    densi = np.full(len(props), P.NITI_DENSITY)
    dt = 0.5 * P.critical_dt(coord, lnods, props, densi, lmate)
    return P.Problem(coord=coord, lnods=lnods, props=props, e_mart=em, densi=densi, fixno=fixno,
                     bcfun=np.full(npo, -1, np.int32), fun_npts=np.array([3], np.int32),
                     fun_smooth=np.array([1], np.int32), fun_tab=P.smooth_cycle_table(1000 * dt, 700.0), lmate=lmate,
                     tempe=None if lmate is None else rng.uniform(300.0, 310.0, ne),
                     fext=P.face_load(coord, lnods, 0, float(nx), (1.0, 0.0, 0.0)), load_fun=0, dtime=dt, nsteps=1000)


def _pair(prob, precision):
    return sma.ExplicitSolid(prob, precision=precision), sma.ExplicitSolid(prob, precision=precision, variant="plain")


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["one", "one_modulus", "compact", "table"])
def test_steps_equal_the_8_lane_kernel(kind, precision):
    prob = _mesh(kind)
    u = P.prestrain(prob, 0.01)
    a, b = _pair(prob, precision)
    assert a.launch_info()["block"] == 64
    for s in (a, b):
        s.set("displ", u)
        s.step(12)
    # rounding in another order through 12 steps; a Gauss point within
    # rounding of an activation test may start a step apart
    tol = 1e-11 if precision == "fp64" else 2e-5
    for f in ("displ", "veloc", "rhsid"):
        x, y = a.get(f), b.get(f)
        assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y), f
    x, y = a.state, b.state
    assert np.linalg.norm(x - y) <= 10 * tol * np.linalg.norm(y)
    ca, cb = a.counters(), b.counters()
    # where the uniform prestrain is still at rest a point's loading function
    # equals the previous step's to rounding, and rounding decides its test
    assert cb["nr_active"] > 0 and abs(ca["nr_active"] - cb["nr_active"]) <= 0.1 * cb["nr_active"]
    assert ca["neg_det"] == cb["neg_det"] == 0
    # the state comes back through the reference's layout, also from a file
    a.state = y
    assert np.array_equal(a.state, y if precision == "fp64" else y.astype(np.float32))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["one", "compact", "table"])
def test_points_outside_the_short_forms(kind, precision):
    """Strains beyond the logarithm polynomial, an inverted element and a NaN
    displacement: the same forces and counters as the 8-lane kernel."""
    prob = _mesh(kind)
    rng = np.random.default_rng(3)
    u = 0.01 * prob.coord @ rng.normal(size=(3, 3))
    big = rng.choice(prob.npoin, 300, replace=False)
    u[big] += 0.3 * rng.normal(size=(300, 3))               # strains of order one, some elements inverted
    a, b = _pair(prob, precision)
    ra, rb = a.assemble(u)["rhsid"], b.assemble(u)["rhsid"]
    fin = np.isfinite(rb).all(axis=1)
    assert np.array_equal(fin, np.isfinite(ra).all(axis=1))
    # per node, relative to one element's force (E strain h^2 / 8, about 100)
    # or what the node holds: strains of order one magnify FP32 rounding most
    # where an element is nearly flat (1 / det F), so the bulk is compared
    err = np.linalg.norm(ra[fin] - rb[fin], axis=1) / np.linalg.norm(rb[fin], axis=1).clip(100.0)
    assert np.quantile(err, 0.99) < (1e-9 if precision == "fp64" else 1e-2)
    assert np.median(err) < (1e-13 if precision == "fp64" else 1e-5)
    ca, cb = a.counters(), b.counters()
    assert cb["neg_det"] > 0 and abs(ca["neg_det"] - cb["neg_det"]) <= (0 if precision == "fp64" else 2)
    assert ca["ielem_min"] == cb["ielem_min"]
    assert abs(ca["gpdet_min"] - cb["gpdet_min"]) <= 1e-5 * abs(cb["gpdet_min"])
    assert abs(ca["nr_active"] - cb["nr_active"]) <= 1e-3 * cb["nr_active"]
    v = np.zeros_like(u)
    v[7] = np.nan
    assert np.array_equal(np.isnan(a.assemble(v)["rhsid"]), np.isnan(b.assemble(v)["rhsid"]))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,slabs", [(57, 1), (97, 2), (113, 2), (146, 2), (176, 3), (500, 8)])
def test_element_loop_on_host_arrays_in_slabs(nx, slabs, precision):
    """The pipelined element loop on host arrays: slabs of the thread-per-element
    kernel, except the two that overlap the copies of a mesh too small for two
    of them; the same residual as one serial call of the 8-lane kernel."""
    base = _mesh("one")
    coord, lnods = P.structured_box(nx, 17, 20, float(nx), 17.0, 20.0, 0.1, 5)
    npo = len(coord)
    prob = dataclasses.replace(base, coord=coord, lnods=lnods, fixno=np.zeros((npo, 3), np.int32),
                               bcfun=np.full(npo, -1, np.int32),
                               fext=P.face_load(coord, lnods, 0, float(nx), (1.0, 0.0, 0.0)))
    u = P.prestrain(prob, 0.01) + 1e-3 * np.random.default_rng(2).normal(size=coord.shape)
    a, b = _pair(prob, precision)
    n0 = a.kernel_launches
    ra = a.assemble(u, fext_scale=0.5, want_all=False)["rhsid"]
    # per slab: displacement in, elements, finished residual rows out (one: displacement, load, elements, residual)
    assert a.kernel_launches - n0 == (3 * slabs if slabs > 1 else 4)
    rb = b.assemble(u, fext_scale=0.5)["rhsid"]
    assert np.linalg.norm(ra - rb) <= (1e-12 if precision == "fp64" else 2e-6) * np.linalg.norm(rb)
    assert np.linalg.norm(a.state - b.state) <= (1e-12 if precision == "fp64" else 1e-5) * np.linalg.norm(b.state)


def _close(a, b, tol):
    for f in ("displ", "veloc"):
        x, y = a.get(f), b.get(f)
        assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y), f
    x, y = a.state, b.state
    assert np.linalg.norm(x - y) <= 10 * tol * np.linalg.norm(y)
    ca, cb = a.counters(reset=True), b.counters(reset=True)
    # as in test_steps_equal_the_8_lane_kernel
    assert cb["nr_active"] > 0 and abs(ca["nr_active"] - cb["nr_active"]) <= 0.1 * cb["nr_active"]
    assert ca["neg_det"] == cb["neg_det"] == 0


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["one", "compact", "table"])
def test_ranges_checkpoints_and_plans_share_the_state(tmp_path, kind, precision):
    """One context's element ranges go to either kernel (a launch plan with
    narrow and wide blocks, element ranges below and above the threshold that
    start inside a state tile), and a checkpoint moves between state layouts."""
    prob = _mesh(kind)
    u = P.prestrain(prob, 0.01)
    a, b = _pair(prob, precision)
    lib, n = sma.lib(), prob.nelem
    tol = 1e-11 if precision == "fp64" else 2e-5
    for s in (a, b):
        s.set("displ", u)
    for ends, blocks in (([19_001, n], [32, 128]), ([1_003, n], [256, 64])):
        a.set_launch_plan(ends, blocks)
        for s in (a, b):
            s.step(5)
        _close(a, b, tol)
    a.set_launch_plan([], [])
    for s in (a, b):
        assert lib.sma_step_prologue(s._ctx) == 0
        for k in range(5):
            for beg, end in ((0, 1_003), (1_003, n)):
                assert lib.sma_step_elements_range(s._ctx, beg, end, int(beg == 0), int(end == n)) == 0
            assert lib.sma_step_nodes(s._ctx, int(k == 4)) == 0
    _close(a, b, tol)
    a.save(str(tmp_path / "c"))
    b.load(str(tmp_path / "c"))
    assert np.array_equal(a.state, b.state)
    a.counters(reset=True), b.counters(reset=True)
    for s in (a, b):
        s.step(5)
    _close(a, b, tol)


def test_surrogate_and_postprocessing_read_the_tiled_state():
    from alya_sma_b200 import surrogate as S
    prob = _mesh("compact")
    u = P.prestrain(prob, 0.01)
    a, b = _pair(prob, "fp32")
    base, em, spread, t = S.training_setup(prob)
    x, y = S.generate(base, em, 512, nstep=256, seed=3, spread=spread, t_range=t, inactive_only=True)
    net = S.Surrogate(seed=4)
    net.fit_stats(x, y)
    out = []
    for s in (b, a):
        s.set("displ", u)
        s.step(4)
        pp = s.postprocess()
        s.state = b.state                                   # the same state, displacement and network
        s.set("displ", u)
        s.set_surrogate(net)
        out.append((pp["caust"], s.assemble(u)["rhsid"]))
    (p0, r0), (p1, r1) = out
    assert np.linalg.norm(p0 - p1) <= 1e-4 * np.linalg.norm(p0)
    assert np.abs(r0 - r1).max() <= 1e-6 * np.abs(r0).max()


def _damped_mesh():
    """39,884 elements, above two warps per scheduler: the damping force comes
    from the pass beside the element loop."""
    coord, lnods = P.structured_box(59, 26, 26, 59.0, 26.0, 26.0, 0.05, 5)
    npo = len(coord)
    fixno = np.zeros((npo, 3), np.int32)
    fixno[P.face_nodes(coord, 0, 0.0)] = 1
    return dataclasses.replace(_mesh("one"), coord=coord, lnods=lnods, fixno=fixno, bcfun=np.full(npo, -1, np.int32),
                               fext=P.face_load(coord, lnods, 0, 59.0, (1.0, 0.0, 0.0)),
                               dampi=np.array([[2.0e5, 0.0]]))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("scheme,energy", [("cd", True), ("cd", False), ("tw", True)])
def test_damped_steps_equal_the_8_lane_kernel(precision, scheme, energy):
    prob = _damped_mesh()
    u = P.prestrain(prob, 0.01)
    v = 1.0e3 * np.random.default_rng(1).normal(size=u.shape)
    a = sma.ExplicitSolid(prob, precision=precision, scheme=scheme)
    b = sma.ExplicitSolid(prob, precision=precision, scheme=scheme, variant="plain")
    for s in (a, b):
        s.set("displ", u)
        s.set("veloc", v)
        if energy:
            s.set_energy(True, 32)
        s.step(3)
        s.step(20)                                          # eager steps and graphs
    tol = 1e-10 if precision == "fp64" else 1e-4
    for f in ("displ", "veloc"):
        x, y = a.get(f), b.get(f)
        assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y), f
    ra, rb = (s.assemble(u, fext_scale=0.5) for s in (a, b))
    for k in ("rhsid", "finte", "frxid"):
        assert np.linalg.norm(ra[k] - rb[k]) <= tol * np.linalg.norm(rb[k]), k
    if energy:
        (ta, ha), (tb, hb) = a.energy(), b.energy()
        assert len(ha) == len(hb) == 23
        for k in ("allie", "allke", "eener"):
            assert abs(ta[k] - tb[k]) <= 10 * tol * abs(tb[k]), k


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_one_damping_force_under_plans_and_host_driven_steps(precision):
    """The damping force is added once, whether the pass beside the loop or
    the 8-lane kernel adds it: launch plans, element ranges and whole steps of
    one context."""
    prob = _damped_mesh()
    u = P.prestrain(prob, 0.01)
    v = 1.0e3 * np.random.default_rng(1).normal(size=u.shape)
    a, b = _pair(prob, precision)
    lib, n = sma.lib(), prob.nelem
    for s in (a, b):
        s.set("displ", u)
        s.set("veloc", v)
    a.set_launch_plan([20_011, n], [64, 128])
    for s in (a, b):
        s.step(4)
    a.set_launch_plan([], [])
    for s in (a, b):
        s.step(4)
        assert lib.sma_step_prologue(s._ctx) == 0
        for cut in (0, 19_999, n):                          # whole, and in two ranges
            for beg, end in zip((0, cut), (cut, n)):
                if end > beg:
                    assert lib.sma_step_elements_range(s._ctx, beg, end, int(beg == 0), int(end == n)) == 0
            assert lib.sma_step_nodes(s._ctx, int(cut == n)) == 0
    tol = 1e-10 if precision == "fp64" else 1e-4
    for f in ("displ", "veloc"):
        x, y = a.get(f), b.get(f)
        assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y), f


@pytest.mark.parametrize("timed", [False, True])
@pytest.mark.parametrize("scheme,energy", [("cd", False), ("cd", True), ("tw", False)])
def test_residual_witnesses_hold_the_damping_force(scheme, energy, timed):
    """Residual witnesses of a damped run record the whole residual of every
    step, eager, captured or timed, with the force of the pass beside the
    element loop in it."""
    prob = _damped_mesh()
    u = P.prestrain(prob, 0.01)
    v = 1.0e3 * np.random.default_rng(1).normal(size=u.shape)
    rng = np.random.default_rng(2)
    free = 3 * prob.npoin + rng.choice(3 * prob.npoin, 2000, replace=False)
    root = P.face_nodes(prob.coord, 0, 0.0)
    wit = np.concatenate([free, 3 * prob.npoin + 3 * root, 3 * rng.choice(prob.npoin, 50, replace=False)])
    h = []
    for variant, damped in (("auto", True), ("plain", True), ("plain", False)):
        s = sma.ExplicitSolid(prob if damped else dataclasses.replace(prob, dampi=None), precision="fp64",
                              scheme=scheme, variant=variant)
        s.set("displ", u)
        s.set("veloc", v)
        s.set_energy(energy, 32)
        s.set_witness(wit, 32)
        s.set_timing(timed)
        rows = []
        for n in (3, 20):                                   # eager steps, then graphs; a call's rows
            s.step(n)
            rows.append(s.witness())
        h.append(np.concatenate(rows))
    a, b, und = h
    assert a.shape == b.shape == (23, len(wit))
    nf = len(wit) - 50                                      # residuals, then displacements
    for x, y in zip(a, b):
        scale = np.linalg.norm(y[:nf])
        assert np.linalg.norm(x[:nf] - y[:nf]) <= 1e-9 * scale
        assert np.linalg.norm(x[nf:] - y[nf:]) <= 1e-10 * np.linalg.norm(y[nf:])
    # the damping force is a part of the first residual that a miss would show
    assert np.linalg.norm(b[0][:nf] - und[0][:nf]) > 1e-3 * np.linalg.norm(b[0][:nf])


def _two_materials(kind):
    """(18-parameter rows, martensite moduli, temperatures or None) of a mesh
    of a few materials that share what compact records do not hold."""
    base = P.nitinol_props(**P.NITI, C_AS=5.0, C_SA=5.0, T_ref=300.0)
    pr, em, t = np.stack([base, base]), np.array([P.NITI_E_MART, P.NITI_E_MART]), (300.0, 310.0)
    if kind == "similar":
        pr[1, [0, 2, 3, 4, 9, 10]] *= 1.08
    if kind == "elastic":                                   # material 0: thresholds out of reach
        pr[0, 3:5], pr[0, 9:11] = (1e9, 2e9), (-1e9, -2e9)
    if kind == "soft":
        pr[0, 0] = em[0] = 1.0
    if kind == "celsius":
        pr[:, [6, 7, 12, 13]] = -26.85
        t = (10.0, 90.0)
    return pr, em, t


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("kind,records", [("similar", True), ("celsius", True), ("elastic", False), ("soft", False)])
def test_fp32_records_only_where_they_hold_the_constants(kind, records, many):
    """A few (or many) materials in the FP32 form: records of offsets from
    material 0 where those hold every constant, else the FP64 table; the
    forces agree with the table's either way."""
    pr, em, t = _two_materials(kind)
    base = _mesh("one")
    ne = base.nelem
    lmate = np.repeat([0, 1], [ne // 3, ne - ne // 3]).astype(np.int32)
    if many:                                                # the same two, one row per element
        pr, em, lmate = pr[lmate], em[lmate], np.arange(ne, dtype=np.int32)
    prob = dataclasses.replace(base, props=pr, e_mart=em, densi=np.full(len(pr), P.NITI_DENSITY), lmate=lmate,
                               tempe=np.random.default_rng(5).uniform(*t, ne))
    u = P.prestrain(prob, 0.012)
    a = sma.ExplicitSolid(prob, precision="fp32")
    b = sma.ExplicitSolid(prob, precision="fp32", variant="table")
    d = sma.ExplicitSolid(prob, precision="fp64", variant="table")
    assert a.launch_info()["compact_records"] == records and not b.launch_info()["compact_records"]
    ra, rb, rd = (s.assemble(u)["rhsid"] for s in (a, b, d))
    # the kernels round in another order (an element's FP32 forces, 2^-24 a
    # rounding, about 20 of them); the records no more than a rounding on top
    scale = np.linalg.norm(rd)
    eb = np.linalg.norm(rb - rd) / scale
    assert eb <= 2e-6 and np.linalg.norm(ra - rd) <= (2 * eb + 1e-7) * scale
    ca, cb = a.counters(), b.counters()
    assert cb["nr_active"] > 0 and abs(ca["nr_active"] - cb["nr_active"]) <= 1e-3 * cb["nr_active"]
    # the surrogate takes a row per element and refuses a few rows, as before
    import torch
    from alya_sma_b200 import surrogate as S
    net = S.Surrogate(seed=4)
    net.fit_stats(torch.randn(256, S.NIN, device="cuda"), torch.randn(256, S.NOUT, device="cuda"))
    if many:
        a.set_surrogate(net)
    else:
        with pytest.raises(sma.SmaError, match="compact records"):
            a.set_surrogate(net)


@pytest.mark.parametrize("unit,solo", [(1.0, True), (1.0e3, False), (1.0e6, False)])
def test_fp64_return_map_is_the_references_in_any_unit(unit, solo):
    """The reference's iteration ends on an absolute residual: with stresses in
    Pa it uses up its steps on most transforming points and restores them.
    The FP64 form does the same at any mesh size."""
    prob = _mesh("one")
    props = prob.props.copy()
    props[:, [0, 3, 4, 9, 10]] *= unit
    prob = dataclasses.replace(prob, props=props, e_mart=prob.e_mart * unit)
    u = P.prestrain(prob, 0.012)
    a, b = _pair(prob, "fp64")
    assert a.launch_info()["block"] == (64 if solo else 32)
    ra, rb = a.assemble(u)["rhsid"], b.assemble(u)["rhsid"]
    assert np.linalg.norm(ra - rb) <= 1e-11 * np.linalg.norm(rb)
    ca, cb = a.counters(), b.counters()
    assert cb["nr_active"] == ca["nr_active"] == 8 * prob.nelem
    assert ca["nr_failed"] == cb["nr_failed"] and (cb["nr_failed"] > 0) == (unit == 1.0e6)
    assert np.abs(a.state - b.state).max() <= 1e-11 * np.abs(b.state).max()


def test_fp64_steps_the_reference_goes_on_from():
    """In MPa too the reference's loop goes on where the pivot is near zero:
    those points leave the closed form, and as many fail as with 8 lanes."""
    prob = _mesh("one_modulus")
    m = prob.props[0]
    two_g, eL, rf = m[0] / (1.0 + m[1]), m[2], m[4] * np.sqrt(2.0 / 3.0)
    # isochoric stretch at xS = 1/2 with F_AS 50 above its previous value,
    # which makes the pivot (F_AS0 - Rf) - (1 - xS) 2G eL that far from zero
    f0 = rf + 0.5 * two_g * eL
    en = (f0 + 50.0) / two_g + 0.5 * eL
    lam = np.exp(en * np.sqrt(2.0 / 3.0) * np.array([1.0, -0.5, -0.5]))
    u = prob.coord * (lam - 1.0)
    rng = np.random.default_rng(4)
    st = np.zeros((prob.nelem, 2, 8, 3))
    st[..., 0] = 0.5
    st[..., 1] = f0 + 10.0 ** rng.uniform(-5.0, -3.0, st.shape[:3]) * rng.choice([-1.0, 1.0], st.shape[:3])
    fails = []
    for s in _pair(prob, "fp64"):
        s.state = st
        s.assemble(u)
        c = s.counters()
        assert c["nr_active"] == 8 * prob.nelem
        fails.append(c["nr_failed"])
    # rounding decides each point (the two kernels round differently): counts
    # of a few ten thousand, compared to five standard deviations and 1 %
    assert fails[1] > 1000 and abs(fails[0] - fails[1]) <= 5.0 * np.sqrt(2.0 * fails[1]) + 0.01 * fails[1], fails
