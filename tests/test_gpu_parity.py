"""Parity of the CUDA timestep (libeu3d.so) with the reference, on a B200.

The reference's outputs come from the committed golden fixtures (produced by
the reference's own CPU code, tests/golden/make_golden.py) and, at sizes the
fixtures do not cover, from the CPU restatement oracle/eu3d_oracle.c, which is
pinned value-for-value to the reference (tests/test_oracle_pin.py).

Tolerances:
  strict arithmetic (no FMA): relative L-inf per field <= 1e-11 after 3 steps
    (conserved variables <= 1e-12; primitives such as a near-zero transverse
    velocity carry the cancellation of their division),
    <= 1e-9 per conserved variable after 100 steps (the required bound), Nchem exact;
  fast arithmetic (FMA): <= 1e-9 per conserved variable after 100 steps;
  mixed precision (FP32 MUSCL/AUSM): species mass-fraction L1 error <= 1e-3 of
    the FP64 run, stated, not exact.
"""
import numpy as np
import pytest

import eu3d_cases as cases
from helpers import golden, golden_mechanism, init_state, interior, n_unequal, rel_linf

pytestmark = pytest.mark.gpu

FIELDS = ["CS", "T", "E", "P", "D", "U", "V", "W", "H", "Gamma", "Yi", "Nchem", "CMS", "Mc", "Di", "Wav", "Rgas",
          "Cp", "C", "Ma"]


def solver_from_golden(eu3d, z, arith="strict", precision="fp64", chemistry="stiff"):
    ext = tuple(float(v) for v in z["extent"])
    s = eu3d.Solver(int(z["ni"]), int(z["nj"]), int(z["nk"]), ext, arith=arith, precision=precision,
                    chemistry=chemistry, record_sources=True)
    s.load_mechanism(cases.MECH_JA919, cases.THERMO)
    if "init_CS" in z:
        s.set_state(init_state(z))
    else:
        s.set_primitive(*[z[f"prim_{k}"] for k in "PTUVWY"])
    return s


def test_nodes_match_reference(gpu):
    z = golden("rsbi_17x13x4_s3.npz")
    s = solver_from_golden(gpu, z)
    for got, want in zip(s.nodes(), (z["x"], z["y"], z["z"])):
        assert np.array_equal(got, want)


def test_strict_three_steps_every_field(gpu):
    z = golden("rsbi_17x13x4_s3.npz")
    s = solver_from_golden(gpu, z)
    st = s.step(int(z["steps"]), float(z["dt"]))
    assert st["nonfinite"] == 0
    for f in FIELDS:
        got = interior(s.get(f))
        want = z[f"out_{f}"]
        if f == "Nchem":
            assert n_unequal(got, want) == 0
        else:
            tol = 1e-12 if f in ("CS", "Di") else 1e-11
            assert rel_linf(got, want).max() <= tol, (f, rel_linf(got, want).max())


@pytest.mark.parametrize("arith", ["strict", "fast"])
def test_hundred_steps_conserved_variables(gpu, arith):
    """The required bound: relative L-inf <= 1e-9 per conserved variable after 100 steps."""
    z = golden("rsbi_36x18x3_s100.npz")
    s = solver_from_golden(gpu, z, arith=arith)
    st = s.step(int(z["steps"]), float(z["dt"]))
    assert st["max_nchem"] == int(z["out_Nchem"].max())
    err = rel_linf(interior(s.get("CS")), z["out_CS"])
    assert err.max() <= 1e-9, err
    assert n_unequal(interior(s.get("Nchem")), z["out_Nchem"]) == 0
    assert rel_linf(interior(s.get("T")), z["out_T"]).max() <= 1e-9


@pytest.mark.parametrize("arith", ["strict", "fast"])
def test_shock_bubble_twenty_steps(gpu, arith):
    z = golden("bubble_25x13x13_s20.npz")
    s = solver_from_golden(gpu, z, arith=arith)
    s.step(int(z["steps"]), float(z["dt"]))
    err = rel_linf(interior(s.get("CS")), z["out_CS"])
    assert err.max() <= (1e-11 if arith == "strict" else 1e-9), err
    assert rel_linf(interior(s.get("CMS")), z["out_CMS"]).max() <= 1e-8
    assert n_unequal(interior(s.get("Nchem")), z["out_Nchem"]) == 0


@pytest.mark.parametrize("arith", ["strict", "fast"])
def test_shock_bubble_hundred_steps(gpu, arith):
    """The required bound on the 3-D case: 100 steps of the shock-bubble (the
    shock runs through the whole perturbed sphere) against the reference's
    own CPU run, relative L-inf <= 1e-9 per conserved variable, Nchem exact."""
    z = golden("bubble_33x17x17_s100.npz")
    s = solver_from_golden(gpu, z, arith=arith)
    st = s.step(int(z["steps"]), float(z["dt"]))
    assert st["nonfinite"] == 0
    err = rel_linf(interior(s.get("CS")), z["out_CS"])
    assert err.max() <= 1e-9, err
    assert rel_linf(interior(s.get("T")), z["out_T"]).max() <= 1e-9
    assert n_unequal(interior(s.get("Nchem")), z["out_Nchem"]) == 0


def test_larger_grid_against_restatement(gpu, port_lib):
    """A grid the fixtures do not cover, against the pinned C restatement."""
    ni, nj, nk = 49, 25, 25
    ext = (0.0, 0.024, 0.0, 0.012, 0.0, 0.012)
    mech = golden_mechanism()
    x, y, zc = (cases.node_coordinates(n, a, b) for n, a, b in ((ni, 0, 0.024), (nj, 0, 0.012), (nk, 0, 0.012)))
    prim = cases.shock_bubble(x, y, zc, mech.mw, 9, radius=4e-3, shock_x=3e-3, standoff=5e-3, seed=3)
    port = port_lib(ni, nj, nk, x, y, zc, mech)
    port.set_primitive(*prim)
    s = gpu.Solver(ni, nj, nk, ext, record_sources=True)
    s.set_mechanism(mech)
    s.set_primitive(*prim)
    port.step(30, 5e-8)
    s.step(30, 5e-8)
    assert rel_linf(interior(s.get("CS")), interior(port.get("CS"))).max() <= 1e-10
    assert n_unequal(interior(s.get("Nchem")), interior(port.get("Nchem"))) == 0


def test_mixed_precision_error_is_bounded(gpu):
    """FP32 reconstruction + AUSM, FP64 update/recovery/kinetics: the species
    mass fractions stay within L1 1e-3 of the all-FP64 run (error stated)."""
    z = golden("bubble_25x13x13_s20.npz")
    a = solver_from_golden(gpu, z)
    b = solver_from_golden(gpu, z, precision="mixed")
    a.step(20, float(z["dt"]))
    b.step(20, float(z["dt"]))
    ya, yb = interior(a.get("Yi")), interior(b.get("Yi"))
    l1 = np.abs(ya - yb).sum(axis=0).mean()
    assert l1 <= 1e-3, l1
    assert rel_linf(interior(b.get("CS")), interior(a.get("CS"))).max() <= 1e-3


@pytest.mark.parametrize("dims", [(40, 20, 45), (17, 7, 32), (17, 8, 32), (33, 9, 5), (270, 62, 62)])
def test_mixed_precision_tiles_match_fp64_closely(gpu, dims):
    """FP32 fluxes against FP64 ones: on grids that the face kernel takes (ragged
    against its tiles, 7 x 32 cells, one row more, thin in z) and on one that the
    plane-tiled kernel takes (a million cells, its last tiles partly filled). After
    two steps the conserved state stays within 2e-6 of the all-FP64 run, each
    error measured against the scale of its quantity (species partial
    densities against the largest density, momentum components against the
    largest momentum component, energy against its largest value). FP32 face
    fluxes perturb each update by ~1e-7 of that scale; a wrong face or stencil
    index shows up as an O(1e-2) error. (Per plane, relative errors are
    meaningless here: trace radicals sit at 1e-49 and the transverse momenta
    at 1e-6 of the streamwise one.)"""
    ni, nj, nk = dims
    ext = (0.0, 0.02, 0.0, 0.01, 0.0, 0.012)
    x = cases.node_coordinates(ni, ext[0], ext[1])
    y = cases.node_coordinates(nj, ext[2], ext[3])
    z = cases.node_coordinates(nk, ext[4], ext[5])
    mech = gpu.parse_mechanism(cases.MECH_JA919, cases.THERMO)
    prim = cases.shock_bubble(x, y, z, mech["mw"], mech["ns"], radius=3e-3, shock_x=3e-3, standoff=5e-3, seed=5)
    p, cs, T, E = gpu.initial_state(mech, ni, nj, nk, *prim)
    dt = cases.cfl_dt(x, y, p[0], p[1], p[2], p[3], p[6], 0.5)
    out = {}
    for precision in ("fp64", "mixed"):
        s = gpu.Solver(ni, nj, nk, ext, precision=precision, arith="fast")
        s.set_mechanism(mech)
        s.set_primitive(*prim)
        s.step(2, dt)
        out[precision] = interior(s.get("CS"))
        s.close()
    a, b = out["mixed"].reshape(13, -1), out["fp64"].reshape(13, -1)
    assert np.all(np.isfinite(a))
    d = np.abs(a - b).max(axis=1)
    err = np.concatenate([d[:9] / b[:9].sum(axis=0).max(), d[9:12] / np.abs(b[9:12]).max(), d[12:] / np.abs(b[12]).max()])
    assert err.max() <= 2e-6, err


@pytest.mark.parametrize("dims", [(2, 2, 2), (5, 3, 9), (67, 2, 2), (9, 33, 3), (3, 5, 17), (18, 9, 13)])
def test_face_kernel_tiles_match_restatement(gpu, port_lib, dims):
    """k_flux_update_faces (strict FP64) on grids smaller than a tile, thin in
    one or two directions and ragged against its tiles, against the pinned C
    restatement: the fluxes round as the reference's, so after three steps the
    conserved state differs by what the kinetics' exp, log and pow leave (the
    bound of the golden three-step test, momentum planes against the largest
    momentum)."""
    from helpers import cs_rel_linf
    ni, nj, nk = dims
    h = 5e-4
    ext = (0.0, h * (ni - 1), 0.0, h * (nj - 1), 0.0, h * (nk - 1))
    mech = golden_mechanism()
    x, y, z = (cases.node_coordinates(n, 0.0, h * (n - 1)) for n in dims)
    rng = np.random.default_rng(sum(dims))
    shape = (ni + 4, nj + 4, nk + 4)
    P, T = 1e5 * rng.uniform(0.7, 1.4, shape), rng.uniform(400.0, 1300.0, shape)
    U, V, W = (rng.uniform(-900.0, 900.0, shape) for _ in range(3))
    f = rng.uniform(0.0, 1.0, shape)
    Y = np.zeros((9,) + shape)
    Y[5], Y[4], Y[8] = 0.1 * f, 0.8 * f, 1 - 0.9 * f
    port = port_lib(ni, nj, nk, x, y, z, mech)
    port.set_primitive(P, T, U, V, W, Y)
    s = gpu.Solver(ni, nj, nk, ext)
    s.set_mechanism(mech)
    s.set_primitive(P, T, U, V, W, Y)
    port.step(3, 2e-8)
    s.step(3, 2e-8)
    assert cs_rel_linf(interior(s.get("CS")), interior(port.get("CS"))).max() <= 1e-12


@pytest.mark.parametrize("precision,nk", [("fp64", 4), ("mixed", 17)])
def test_face_kernel_beyond_65535_tiles_along_y(gpu, precision, nk):
    """Grids with more tiles of four rows along y than a launch has blocks in y: the
    rows repeat with period 20, so a step gives them, away from the ends, the bits
    of a grid of 60 rows."""
    ni, long = 2, 262200
    mech = golden_mechanism()
    rng = np.random.default_rng(2)
    shape = (ni + 4, 24, nk + 4)
    f = rng.uniform(0.0, 1.0, shape)
    Y = np.zeros((9,) + shape)
    Y[5], Y[4], Y[8] = 0.1 * f, 0.8 * f, 1 - 0.9 * f
    _, cs, T, E = gpu.initial_state(mech, ni, 20, nk, 1e5 * rng.uniform(0.7, 1.4, shape), rng.uniform(400.0, 1300.0, shape),
                                    *(rng.uniform(-900.0, 900.0, shape) for _ in range(3)), Y)
    h = 2.0**-11  # every spacing exact
    got = {}
    for nj in (60, long):
        rows = 2 + np.arange(nj + 4) % 20  # (the ghost rows of the state are not formed)
        s = gpu.Solver(ni, nj, nk, (0.0, h * (ni - 1), 0.0, h * (nj - 1), 0.0, h * (nk - 1)), chemistry="frozen", precision=precision,
                       arith="fast")
        s.set_mechanism(mech)
        s.set_conserved(cs[:, :, rows], T[:, :, rows], E[:, :, rows])
        s.step(1, 2e-8)
        got[nj] = interior(s.get("T"))[0]
        s.close()
    want = got[60][:, 20:40]
    assert np.array_equal(got[long][:, 20:long - 20].reshape(ni, -1, 20, nk), np.broadcast_to(want[:, None], (ni, long // 20 - 2, 20, nk)))


def test_strict_warp_kinetics_match_restatement(gpu, port_lib):
    """Strict FP64 on igniting gas whose long substep chains run a warp each
    (k_react_heavy), against the pinned C restatement, eight steps: Nchem exact,
    and the conserved state within the 1e-14 of CUDA's exp, log and pow carried
    through some hundred substeps of chain branching (bound 1e-9). The fast
    FP64 forms stay within 1e-9 of it too."""
    from helpers import cs_rel_linf
    ni, nj, nk = 11, 5, 6
    ext = (0.0, ni * 2.5e-4, 0.0, nj * 2.5e-4, 0.0, nk * 2.5e-4)
    mech = golden_mechanism()
    x, y, z = (cases.node_coordinates(n, ext[2 * a], ext[2 * a + 1]) for a, n in enumerate((ni, nj, nk)))
    prim = cases.hot_reacting_block(ni + 4, nj + 4, nk + 4, mech.mw, 9)
    port = port_lib(ni, nj, nk, x, y, z, mech)
    port.set_primitive(*prim)
    port.step(8, 2e-8)
    out = {}
    for arith in ("strict", "fast"):
        s = gpu.Solver(ni, nj, nk, ext, arith=arith)
        s.set_mechanism(mech)
        s.set_primitive(*prim)
        assert max(s.step(1, 2e-8)["max_nchem"] for _ in range(8)) > 4
        out[arith] = interior(s.get("CS"))
        if arith == "strict":
            assert n_unequal(interior(s.get("Nchem")), interior(port.get("Nchem"))) == 0
        s.close()
    assert cs_rel_linf(out["strict"], interior(port.get("CS"))).max() <= 1e-9
    assert cs_rel_linf(out["fast"], out["strict"]).max() <= 1e-9


def igniting_samples(n, seed=3):
    """Chemistry samples, more than one in ten beyond four substeps: T, p, Y, dt on the device."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = lambda a, b: a + (b - a) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    Y = torch.zeros(9, n, device="cuda", dtype=torch.float64)
    Y[5], Y[4], Y[3], Y[0], Y[8] = 0.03, 0.23, 0.005, 0.001, 0.734
    return u(1200, 2600), u(1e5, 8e5), Y, 10 ** u(-8.5, -6.5)


def test_samples_on_a_warp_match_the_thread_form(gpu):
    """eu_chem_advance's samples beyond four substeps, a warp each, against a thread
    each, bit for bit in every state, temperature, energy and Nchem: the mechanism's
    last reaction at rate 0, as it is and with sides of four and three molecules,
    which the warp form does not take (its terms are exact zeros in either). Calls
    of one sample, of less and of more than a block, a larger one after a smaller."""
    import torch
    OH, H2O, H2 = 3, 2, 5
    s = gpu.Solver(5, 5, 5, (0, 1, 0, 1, 0, 1))
    T0, p0, Y0, dt0 = igniting_samples(1000, seed=7)
    deferred = 0
    for n in (1, 100, 1000):
        got = []
        for warp in (True, False):
            mech = gpu.parse_mechanism(cases.MECH_JA919, cases.THERMO)
            mech["af"][18] = 0
            if not warp:
                for key, side in (("stoi_f", {OH: 2, H2: 2}), ("stoi_b", {H2O: 2, H2: 1})):
                    mech[key][:, 18] = [side.get(q, 0) for q in range(9)]
            s.set_mechanism(mech)
            T, p, Y, dt = T0[:n].clone(), p0[:n].clone(), Y0[:, :n].contiguous(), dt0[:n].clone()
            cs, E = torch.zeros(13, n, device="cuda", dtype=torch.float64), torch.zeros(n, device="cuda", dtype=torch.float64)
            nchem = torch.zeros(n, device="cuda", dtype=torch.int32)
            torch.cuda.synchronize()
            s.chem_states(T, p, Y, cs, E)
            s.chem_advance(cs, T, E, dt, nchem)
            got.append((cs, T, E, nchem))
        for a, b in zip(*got):
            assert torch.isfinite(a).all() and torch.equal(a, b), n
        deferred = int((got[0][3] > 4).sum())
    assert deferred > 50


def test_samples_without_memory_for_the_queue(gpu):
    """eu_chem_advance where the queue of the samples left to a warp each (256 MB)
    does not fit the device any more: it runs every sample on a thread, to the same
    bits in every state and Nchem. (The samples compared lie at both ends of a call
    whose other samples take one substep.)"""
    import torch
    n, part = 1 << 26, 1 << 12
    s = gpu.Solver(5, 5, 5, (0, 1, 0, 1, 0, 1))
    s.set_mechanism(golden_mechanism())
    T0, p0, Y0, dt0 = igniting_samples(part)
    cs0, E0 = torch.zeros(13, part, device="cuda", dtype=torch.float64), torch.zeros(part, device="cuda", dtype=torch.float64)
    s.chem_states(T0, p0, Y0, cs0, E0)
    want = [cs0.clone(), T0.clone(), E0.clone(), torch.zeros(part, device="cuda", dtype=torch.int32)]
    torch.cuda.synchronize()
    s.chem_advance(*want[:3], dt0, want[3])
    assert int((want[3] > 4).sum()) > part // 10 and all(torch.isfinite(t).all() for t in want)
    cs = cs0[:, :1].repeat(1, n)
    E, nchem = E0[:1].repeat(n), torch.zeros(n, device="cuda", dtype=torch.int32)
    dt = torch.full((n,), 1e-12, device="cuda", dtype=torch.float64)
    T = T0[:1].repeat(n)
    for at in (slice(0, part), slice(n - part, n)):
        cs[:, at], T[at], E[at], dt[at] = cs0, T0, E0, dt0
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    room = torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), device="cuda", dtype=torch.uint8)
    s.chem_advance(cs, T, E, dt, nchem)
    del room
    torch.cuda.empty_cache()
    for at in (slice(0, part), slice(n - part, n)):
        for a, b in zip((cs[:, at], T[at], E[at], nchem[at]), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("precision,bound", [("fp64", 1e-9), ("mixed", 1e-5)])
def test_reactions_that_change_the_mole_number_by_two(gpu, precision, bound):
    """A mechanism with 2 H + O -> H2O and H2O -> 2 H + O (the sides differ by two
    moles, so Kc carries (RT/p0)^-2 and ^2): the fast forms of the rates against
    the strict ones on gas near equilibrium, where the backward rates count. FP64:
    rounding only; mixed: FP32 fluxes of a gas nearly at rest."""
    mech = gpu.parse_mechanism(cases.MECH_JA919, cases.THERMO)
    H, O, H2O = 0, 1, 2
    for r, (f, b), (A, Bf, E) in ((5, ({H: 2, O: 1}, {H2O: 1}), (1e18, -1.0, 0.0)), (18, ({H2O: 1}, {H: 2, O: 1}), (1e19, 0.0, 2.2e5))):
        for key, side in (("stoi_f", f), ("stoi_b", b)):
            mech[key][:, r] = [side.get(s, 0) for s in range(9)]
        mech["tb"][:, r] = 0
        mech["af"][r], mech["bf"][r], mech["eaf"][r] = A, Bf, E
    shape = (10, 9, 8)
    rng = np.random.default_rng(8)
    Y = np.zeros((9,) + shape)
    Y[H], Y[O], Y[H2O], Y[3], Y[4], Y[5] = 0.002, 0.02, 0.2, 0.03, 0.03, 0.004
    Y[8] = 1 - Y.sum(axis=0)
    T = rng.uniform(2800.0, 3200.0, shape)
    got = {}
    for prec, arith in (("fp64", "strict"), (precision, "fast")):
        s = gpu.Solver(6, 5, 4, (0.0, 5e-3, 0.0, 4e-3, 0.0, 3e-3), precision=prec, arith=arith)
        s.set_mechanism(mech)
        s.set_primitive(np.full(shape, 1e5), T, *(np.zeros(shape) for _ in range(3)), Y)
        s.step(3, 2e-8)
        got[arith] = interior(s.get("T")), interior(s.get("CS"))
    for a, b in zip(got["fast"], got["strict"]):
        for q in (range(len(b)) if len(b) == 1 else (H, O, H2O, 12)):
            assert np.abs(a[q] - b[q]).max() <= bound * np.abs(b[q]).max(), q


@pytest.mark.parametrize("precision,bound,deferred", [("fp64", 1e-9, False), ("fp64", 1e-9, True), ("mixed", 1e-5, False)])
def test_rates_of_very_cold_gas(gpu, precision, bound, deferred):
    """The fast forms of the rates at 41 to 42 K, where the exponential of water
    vapour's G/(R T) has left the range of doubles (43 K), on a thread per cell
    and, with radicals, a warp per cell, against the strict ones: far below the
    thermo fit, but a step that the reference's forms take. FP64: rounding, of
    exponents up to 1,000; mixed: FP32 fluxes of a gas nearly at rest."""
    shape = (10, 9, 8)
    rng = np.random.default_rng(8)
    Y = np.zeros((9,) + shape)
    Y[4], Y[5] = 0.2, 0.02
    if deferred:
        Y[0] = 1e-6
    else:
        Y[2], Y[6], Y[7] = 1e-3, 1e-5, 1e-5
    Y[8] = 1 - Y.sum(axis=0)
    T, dt = rng.uniform(41.0, 42.0, shape), 1e-9
    got = {}
    for prec, arith in (("fp64", "strict"), (precision, "fast")):
        s = gpu.Solver(6, 5, 4, (0.0, 5e-3, 0.0, 4e-3, 0.0, 3e-3), precision=prec, arith=arith)
        s.set_mechanism(gpu.parse_mechanism(cases.MECH_JA919, cases.THERMO))
        s.set_primitive(np.full(shape, 1e4), T, *(np.zeros(shape) for _ in range(3)), Y)
        stats = s.step(1, dt)
        assert (stats["max_nchem"] > 4) == deferred, stats
        got[arith] = interior(s.get("T")), interior(s.get("CS"))
    for a, b in zip(got["fast"], got["strict"]):
        assert np.isfinite(a).all()
        for q in (range(len(b)) if len(b) == 1 else (0, 1, 2, 3, 12)):
            assert np.abs(a[q] - b[q]).max() <= bound * np.abs(b[q]).max(), q


def mixed_block(gpu, dims, **kw):
    """A mixed-precision solver on random reacting gas with O(1) changes between nodes."""
    h = 5e-4
    s = gpu.Solver(*dims, tuple(v for n in dims for v in (0.0, h * (n - 1))), precision="mixed", arith="fast", **kw)
    s.set_mechanism(golden_mechanism())
    rng = np.random.default_rng(sum(dims))
    shape = tuple(n + 4 for n in dims)
    f = rng.uniform(0.0, 1.0, shape)
    Y = np.zeros((9,) + shape)
    Y[5], Y[4], Y[8] = 0.1 * f, 0.8 * f, 1 - 0.9 * f
    s.set_primitive(1e5 * rng.uniform(0.7, 1.4, shape), rng.uniform(400.0, 1300.0, shape),
                    *(rng.uniform(-900.0, 900.0, shape) for _ in range(3)), Y)
    return s


def flux_launches(fn):
    """The flux kernels that fn launches: {(name, grid)}."""
    import json
    import os
    import tempfile
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
        fn()
        torch.cuda.synchronize()
    with tempfile.TemporaryDirectory() as d:
        p.export_chrome_trace(os.path.join(d, "trace.json"))
        with open(os.path.join(d, "trace.json")) as f:
            events = json.load(f)["traceEvents"]
    return {(k, tuple(e["args"]["grid"])) for e in events if e.get("cat") == "kernel"
            for k in ("k_flux_update_faces", "k_flux_update_tiled") if k in e["name"]}


def flux_kernels(fn):
    return {k for k, _ in flux_launches(fn)}


@pytest.mark.parametrize("dims,chemistry", [((50, 7, 32), "frozen"), ((25, 36, 64), "frozen"), ((24, 14, 161), "frozen"),
                                            ((2, 7, 26), "frozen"), ((49, 35, 32), "stiff"), ((26, 13, 31), "stiff")])
def test_tiled_flux_gives_the_face_kernels_bits(gpu, dims, chemistry):
    """A mixed instance alone takes the face kernel at these sizes, in a batch of a
    million cells the plane-tiled one: the same bits, on which a batch's equality
    with its instances alone rests. Exactly one 7 x 32 tile, a last row and a last
    column of one cell, partly filled tiles, and x extents that the march of 24
    planes divides, leaves one plane of, or exceeds."""
    alone, together = (mixed_block(gpu, dims, chemistry=chemistry) for _ in range(2))
    assert flux_kernels(lambda: alone.step(3, 2e-8)) == {"k_flux_update_faces"}
    b = gpu.Batch([together, mixed_block(gpu, (128, 98, 96), chemistry="frozen")])
    assert flux_kernels(lambda: b.step(3, 2e-8)) == {"k_flux_update_tiled"}
    assert np.array_equal(alone.get("CS"), together.get("CS")) and np.array_equal(alone.get("T"), together.get("T"))


def test_flux_kernel_follows_the_call(gpu):
    """Which FP32 flux kernel a handle runs depends on the cells that run together:
    its own alone (too few here for the tiled kernel), all instances' in a batch.
    The captured step follows each call, whatever the calls before it were, also
    where the kinetics leave nothing to a batch's shared stage (frozen)."""
    a, b = (mixed_block(gpu, (50, 7, 32), chemistry="frozen") for _ in range(2))
    big = mixed_block(gpu, (128, 98, 96), chemistry="frozen")  # 1.2 M cells
    small = mixed_block(gpu, (10, 7, 32), chemistry="frozen")
    large, little = gpu.Batch([b, big]), gpu.Batch([b, small])
    calls = [(lambda: a.step(2, 2e-8), "k_flux_update_faces"), (lambda: large.step(2, 2e-8), "k_flux_update_tiled"),
             (lambda: b.step(2, 2e-8), "k_flux_update_faces"), (lambda: large.step(2, 2e-8), "k_flux_update_tiled"),
             (lambda: little.step(2, 2e-8), "k_flux_update_faces"), (lambda: large.step(2, 2e-8), "k_flux_update_tiled")]
    for k, (call, kernel) in enumerate(calls):
        assert flux_kernels(call) == {kernel}, k
    a.step(8, 2e-8)  # b's steps one by one
    assert np.array_equal(a.get("CS"), b.get("CS"))


def test_deterministic(gpu):
    z = golden("bubble_25x13x13_s20.npz")
    a = solver_from_golden(gpu, z, arith="fast")
    b = solver_from_golden(gpu, z, arith="fast")
    a.step(10, float(z["dt"]))
    b.step(10, float(z["dt"]))
    assert n_unequal(a.get("CS"), b.get("CS")) == 0


def test_mixed_stiff_heavy_cells_match_fp64(gpu):
    """Igniting gas in mixed precision: cells whose predicted Nchem exceeds 4
    are advanced one warp per cell (k_react_heavy). Over 8 steps of a hot
    2H2+O2/N2 block (1300-2600 K, dt 2e-8 s) the run must reach such cells and
    stay within a species L1 (mean over cells of sum_s |dY_s|) of 1e-4 and a
    relative temperature error of 1e-4 of the FP64 stiff run."""
    ni, nj, nk = 24, 8, 8
    ext = (0.0, 0.006, 0.0, 0.002, 0.0, 0.002)
    mech = gpu.parse_mechanism(cases.MECH_JA919, cases.THERMO)
    prim = cases.hot_reacting_block(ni + 4, nj + 4, nk + 4, mech["mw"], mech["ns"])
    out, peak = {}, {}
    for precision in ("fp64", "mixed"):
        s = gpu.Solver(ni, nj, nk, ext, precision=precision, arith="fast")
        s.set_mechanism(mech)
        s.set_primitive(*prim)
        peak[precision] = 0
        for _ in range(8):
            peak[precision] = max(peak[precision], s.step(1, 2e-8)["max_nchem"])
        out[precision] = (interior(s.get("Yi")), interior(s.get("T")))
        s.close()
    assert peak["mixed"] > 4, peak
    l1 = np.abs(out["mixed"][0] - out["fp64"][0]).sum(axis=0)
    terr = np.abs(out["mixed"][1] - out["fp64"][1]) / out["fp64"][1]
    assert l1.mean() <= 1e-4 and terr.max() <= 1e-4, (l1.mean(), l1.max(), terr.max(), peak)


@pytest.mark.parametrize("precision,arith,chemistry", [("mixed", "fast", "stiff"), ("fp64", "strict", "stiff"),
                                                        ("mixed", "fast", "learned")])
def test_autotuned_launch_shapes_change_no_bits(gpu, precision, arith, chemistry):
    """Every launch shape the autotuner may pick gives bitwise the same state:
    steps after tuning equal steps with the default shapes, and tuning leaves
    the state it timed on unchanged (ragged grid: 40 x 21 x 45 nodes, which the
    face kernel takes in either precision). In learned mode the tuner also picks the recovery's register target."""
    ni, nj, nk = 40, 21, 45
    ext = (0.0, 0.02, 0.0, 0.01, 0.0, 0.012)
    x, y, z = (cases.node_coordinates(n, a, b) for n, a, b in ((ni, 0, 0.02), (nj, 0, 0.01), (nk, 0, 0.012)))
    mech = gpu.parse_mechanism(cases.MECH_JA919, cases.THERMO)
    prim = cases.shock_bubble(x, y, z, mech["mw"], mech["ns"], radius=3e-3, shock_x=3e-3, standoff=5e-3, seed=5)
    out = []
    for tune in (False, True):
        s = gpu.Solver(ni, nj, nk, ext, precision=precision, arith=arith, chemistry=chemistry)
        s.set_mechanism(mech)
        s.set_primitive(*prim)
        if chemistry == "learned":
            import learned
            model, gate = learned.load()
            learned.attach(s, model, gate)
        s.step(1, 2e-8)
        before = s.get("CS")
        if tune:
            rep = s.autotune(reps=2)
            assert len(rep["flux_ms"]) >= 5 and rep["flux_ci"] in rep["flux_ms"], rep
            # learned: 3 block sizes x 4 register targets; stiff: 3 x 3 (the
            # kinetics kernel's); frozen: 3 block sizes
            assert len(rep["recover_ms"]) == {"learned": 12, "stiff": 9}.get(chemistry, 3), rep
            assert n_unequal(s.get("CS"), before) == 0
        s.step(4, 2e-8)
        out.append((s.get("CS"), s.get("T")))
        s.close()
    for a, b in zip(*out):
        assert n_unequal(a, b) == 0


@pytest.mark.parametrize("precision,arith", [("fp64", "strict"), ("fp64", "fast"), ("mixed", "fast")])
def test_face_tiles_follow_the_batch(gpu, precision, arith):
    """A small instance's faces come in the small grids' tiles alone and in the large
    grids' in a batch of many cells (other blocks), with the same bits, whatever the
    calls before; a batch of one is the instance alone."""
    mech = golden_mechanism()

    def make(dims):
        h = 5e-4
        s = gpu.Solver(*dims, tuple(v for n in dims for v in (0.0, h * (n - 1))), precision=precision, arith=arith, chemistry="frozen")
        s.set_mechanism(mech)
        ax = [cases.node_coordinates(n, 0.0, h * (n - 1)) for n in dims]
        s.set_primitive(*cases.shock_bubble(*ax, mech.mw, 9, radius=2e-3, shock_x=2e-3, standoff=3e-3, seed=4))
        return s

    a, b, big = make((21, 14, 11)), make((21, 14, 11)), make((64, 60, 41))
    both, one = gpu.Batch([b, big]), gpu.Batch([b])
    alone = flux_launches(lambda: a.step(2, 2e-8))
    together = flux_launches(lambda: both.step(2, 2e-8))
    assert len(alone) == 1 and {k for k, _ in together} == {"k_flux_update_faces"} and not alone <= together
    assert flux_launches(lambda: one.step(2, 2e-8)) == alone and flux_launches(lambda: b.step(2, 2e-8)) == alone
    a.step(4, 2e-8)
    assert np.array_equal(a.get("CS"), b.get("CS")) and np.array_equal(a.get("T"), b.get("T"))


def test_tiled_marches_change_no_bits(gpu):
    """The marches that the tuner may give the tiled kernel (a grid that takes it
    alone, 130 planes: last marches of 1, 2, 10, 14 ... planes) against its default
    one, bitwise: each candidate is timed, one is kept, and steps go on with it."""
    out = []
    for tune in (False, True):
        s = mixed_block(gpu, (130, 84, 96), chemistry="frozen")
        assert flux_kernels(lambda: s.step(1, 2e-8)) == {"k_flux_update_tiled"}
        if tune:
            before = s.get("CS")
            rep = s.autotune(reps=2)
            assert len(rep["flux_ms"]) >= 9 and 1 not in rep["flux_ms"] and rep["flux_ci"] in rep["flux_ms"], rep
            assert np.array_equal(s.get("CS"), before)
        s.step(3, 2e-8)
        out.append(s.get("CS"))
        s.close()
    assert np.array_equal(*out)


def test_tuned_march_belongs_to_its_kernel(gpu):
    """A march tuned on the face kernel, which a small grid takes alone, is not the
    tiled kernel's in a batch: that one keeps its default there (blocks of 24
    planes: 3 for the 50 of the small instance, 6 for the large one's 128)."""
    a = mixed_block(gpu, (50, 7, 32), chemistry="frozen")
    assert 1 in a.autotune(reps=1)["flux_ms"]
    big = mixed_block(gpu, (128, 98, 96), chemistry="frozen")
    b = gpu.Batch([a, big])
    assert flux_launches(lambda: b.step(1, 2e-8)) == {("k_flux_update_tiled", (1, 1, 3)), ("k_flux_update_tiled", (3, 14, 6))}


def test_autotune_beyond_65535_planes(gpu):
    """A mixed grid that takes the tiled flux kernel with more planes along x than
    a launch has blocks in z: the tuner offers no march that needs more (nor a
    single plane, which only the face kernel has), and the tuned steps' bits are
    the untuned ones' (a state of 20 different planes repeated along x)."""
    ni, nj, nk = 65560, 7, 26
    mech = golden_mechanism()
    rng = np.random.default_rng(1)
    shape = (24, nj + 4, nk + 4)
    f = rng.uniform(0.0, 1.0, shape)
    Y = np.zeros((9,) + shape)
    Y[5], Y[4], Y[8] = 0.1 * f, 0.8 * f, 1 - 0.9 * f
    prim = (1e5 * rng.uniform(0.7, 1.4, shape), rng.uniform(400.0, 1300.0, shape), *(rng.uniform(-900.0, 900.0, shape) for _ in range(3)), Y)
    _, cs, T, E = gpu.initial_state(mech, 20, nj, nk, *prim)
    planes = 2 + np.arange(ni + 4) % 20  # (the ghost planes of the state are not formed)
    h = 5e-4
    s = gpu.Solver(ni, nj, nk, (0.0, h * (ni - 1), 0.0, h * (nj - 1), 0.0, h * (nk - 1)), chemistry="frozen", precision="mixed", arith="fast")
    s.set_mechanism(mech)
    got = []
    for tune in (False, True):
        s.set_conserved(cs[:, planes], T[:, planes], E[:, planes])
        if tune:
            assert min(s.autotune(reps=1)["flux_ms"]) >= 8
        s.step(1, 2e-8)
        got.append(s.get("T"))
    assert np.array_equal(*got) and np.isfinite(got[0]).all()


@pytest.mark.parametrize("width,steps,tol", [(2.0, 40, 1e-11), (6.0, 100, 1e-10)])
def test_znd_against_restatement(gpu, port_lib, width, steps, tol):
    """The 1-D ZND initiation (2H2+O2+7Ar on the Ar variant of the mechanism,
    1 MPa / 3000 K driver at a reflecting wall, 6.67 kPa / 298 K gas ahead,
    parameters from data/input-1dZND.txt, driver edge a tanh profile `width`
    cells wide) with the ZND ghost fill, on a 401 x 2 x 2 node grid at 25 um
    spacing, against the pinned C restatement with the same ghost fill
    (strict arithmetic), Nchem exact. Each step's dt comes from the
    device-side CFL reduction at 0.5 (eu_step_cfl) and the restatement takes
    the same dt.

    The two builds start 1e-14 apart (CUDA's exp/log/pow against glibc's, in
    the last bit); the rarefaction running into the wall amplifies that. With
    the 2-cell edge the difference stays below 1e-13 for 20 steps, reaches
    1e-12 at 40 and 2e-9 by step 100 (a limiter switching branch on values
    that differ in the last bit); with a 6-cell edge it is 3e-12 at step 100.
    So the bounds: 1e-11 after 40 steps at the 2-cell edge, 1e-10 after 100 at
    the 6-cell one."""
    from oracle import Mechanism
    ni, nj, nk = 401, 2, 2
    dx = 25e-6
    ext = (0.0, (ni - 1) * dx, 0.0, dx, 0.0, dx)
    x = cases.node_coordinates(ni, ext[0], ext[1])
    y = cases.node_coordinates(nj, ext[2], ext[3])
    mech = gpu.parse_mechanism(cases.MECH_JA919_AR, cases.THERMO_AR)
    prim = cases.znd(x, y, y, mech["mw"], mech["ns"], interface_cells=width)
    port = port_lib(ni, nj, nk, x, y, y, Mechanism.from_dict(mech), boundary="znd")
    port.set_primitive(*prim)
    s = gpu.Solver(ni, nj, nk, ext, record_sources=True, boundary="znd")
    s.set_mechanism(mech)
    s.set_primitive(*prim)
    # the first dt against the host rule on the initial state (interior
    # spacings: the reference's rule takes dy from its ghost nodes, which a
    # two-node direction makes negative)
    p, cs, T, E = gpu.initial_state(mech, ni, nj, nk, *prim)
    dt0 = cases.cfl_dt(x, x, p[0], p[1], p[2], p[3], p[6], 0.5)
    peak = 0
    for n in range(steps):
        st, dt = s.step_cfl(1, 0.5)
        if n == 0:
            assert abs(dt - dt0) <= 1e-12 * dt0, (dt, dt0)
        port.step(1, dt)
        peak = max(peak, st["max_nchem"])
    assert peak >= 1
    assert rel_linf(interior(s.get("CS")), interior(port.get("CS"))).max() <= tol
    assert n_unequal(interior(s.get("Nchem")), interior(port.get("Nchem"))) == 0


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("mixed", 1e-6)])
def test_set_conserved_matches_set_state(gpu, precision, tol):
    """eu_set_conserved (CS, T, E up; the primitives formed on the device by
    the recovery) steps like eu_set_state with the full state: the recovered
    temperature is within 1e-12 of the uploaded one, and after three steps each
    conserved plane agrees to its relative tolerance (the transverse momenta,
    whose planes peak at ~1e-6 of the streamwise one, carry the primitives'
    initial rounding difference at a few 1e-10 of their own maxima)."""
    ni, nj, nk = 33, 17, 17
    ext = (0.0, 0.016, 0.0, 0.008, 0.0, 0.008)
    mech = gpu.parse_mechanism(cases.MECH_JA919, cases.THERMO)
    x, y, z = (cases.node_coordinates(n, a, b) for n, a, b in ((ni, 0, 0.016), (nj, 0, 0.008), (nk, 0, 0.008)))
    prim = cases.shock_bubble(x, y, z, mech["mw"], mech["ns"], radius=3e-3, shock_x=3e-3, standoff=5e-3, seed=5)
    p, cs, T, E = gpu.initial_state(mech, ni, nj, nk, *prim)
    st = {"CS": cs, "T": T, "E": E, "P": p[0], "D": p[1], "U": p[2], "V": p[3], "W": p[4], "H": p[5],
          "Gamma": p[6], "Yi": p[7:]}
    out = []
    for full in (True, False):
        s = gpu.Solver(ni, nj, nk, ext, precision=precision, arith="fast")
        s.set_mechanism(mech)
        if full:
            s.set_state(st)
        else:
            s.set_conserved(cs, T, E)
            t0 = np.asarray(T).reshape((1,) + s.shape)
            assert rel_linf(interior(s.get("T")), interior(t0)).max() <= 1e-12
        s.step(3, 4e-8)
        out.append((s.get("CS"), s.get("T")))
        s.close()
    for a, b in zip(out[0], out[1]):
        assert rel_linf(interior(b), interior(a)).max() <= tol


@pytest.mark.parametrize("arith", ["strict", "fast"])
def test_rk3_against_restatement(gpu, port_lib, arith):
    """The three-stage TVD Runge-Kutta advection (eu_set_time_scheme) against
    the C restatement's: 10 steps of the shock-bubble fixture's initial state,
    conserved state within 1e-10 (strict) or 1e-9 (fast) per variable, Nchem
    exact; and the scheme changes the result (it is not the Euler step)."""
    z = golden("bubble_25x13x13_s20.npz")
    mech = golden_mechanism()
    port = port_lib(int(z["ni"]), int(z["nj"]), int(z["nk"]), z["x"], z["y"], z["z"], mech)
    port.set_primitive(*[z[f"prim_{k}"] for k in "PTUVWY"])
    port.set_scheme("rk3")
    port.step(10, float(z["dt"]))
    s = solver_from_golden(gpu, z, arith=arith)
    s.set_time_scheme("rk3")
    st = s.step(10, float(z["dt"]))
    assert st["nonfinite"] == 0
    want = interior(port.get("CS"))
    assert rel_linf(interior(s.get("CS")), want).max() <= (1e-10 if arith == "strict" else 1e-9)
    assert n_unequal(interior(s.get("Nchem")), interior(port.get("Nchem"))) == 0
    ee = solver_from_golden(gpu, z, arith=arith)
    ee.step(10, float(z["dt"]))
    assert rel_linf(interior(ee.get("CS")), want).max() > 1e-6


def test_rk3_learned_mixed_stays_close(gpu):
    """RK3 with the benchmark's learned + mixed step: finite, and its species
    within L1 1e-3 of the FP64 RK3 run."""
    import learned
    z = golden("bubble_25x13x13_s20.npz")
    a = solver_from_golden(gpu, z)
    a.set_time_scheme("rk3")
    b = solver_from_golden(gpu, z, precision="mixed", chemistry="learned", arith="fast")
    model, gate = learned.load(device=0)
    learned.attach(b, model, gate)
    b.set_time_scheme("rk3")
    a.step(10, float(z["dt"]))
    st = b.step(10, float(z["dt"]))
    assert st["nonfinite"] == 0
    l1 = np.abs(interior(a.get("Yi")) - interior(b.get("Yi"))).sum(axis=0).mean()
    assert l1 <= 1e-3, l1
