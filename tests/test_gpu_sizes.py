"""One whole step at sizes where the tiles of the stage kernels end unevenly
(the smallest meshes, odd extents, a last tile of one zone, more layers than
a thread's column segment; with one radial zone and four ghost layers the
padding runs through r = 0, where the ADP matrices are too ill conditioned for
their inverses and the mesh keeps the factors) against the CPU oracle, and batches of FP64 members
run side by side, which must give each member's own result to the bit.

Tolerances: those of test_gpu_parity (1e-12 of the largest value for the
state, FP64); the precision form's bounds of test_gpu_precision scaled to one
step (rounding of FP32 storage, 6e-8, times the two or three stages' few
operations on it: 5e-6 of the largest value; momentum at rest: of the largest
sound-speed momentum).
"""
import numpy as np
import pytest

import cubesphere_b200 as cs
from conftest import has_gpu
from test_gpu_parity import check_state, face_b_errors, zones

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

SIZES = [(5, 2, 3), (6, 1, 4), (7, 5, 3), (13, 3, 4), (19, 9, 4), (9, 6, 5)]


@pytest.mark.parametrize("ntp,nr,ghosts", SIZES)
@pytest.mark.parametrize("rk", [cs.CS_RK2, cs.CS_SSPRK3, cs.CS_IMEX_RK2])
def test_one_step_at_uneven_sizes_matches_the_oracle(ntp, nr, ghosts, rk):
    from oracle import Oracle
    pr = cs.preset("shell16")
    pr["params"].update(ntp=ntp, nr=nr, nghost=ghosts, rk_scheme=rk)
    s = cs.Solve(**pr["params"])
    s.mesh_build()
    s.init_problem(**pr["init"])
    st = s.get_state()
    o = Oracle(s)
    o.put_state(st)
    dt, dto = s.evaluate_timestep(1e30), o.evaluate_timestep(1e30)
    assert abs(dt - dto) <= 1e-12 * dto
    dt, dto = s.steps(1, dt), o.step(dto)
    assert abs(dt - dto) <= 1e-12 * dto
    check_state(s, s.get_state(), o.get_state())


@pytest.mark.parametrize("ntp,nr,ghosts", SIZES[::2])
@pytest.mark.parametrize("p2", [0, cs.CS_FLAG_P2])
def test_precision_form_at_uneven_sizes(ntp, nr, ghosts, p2):
    pr = cs.preset("shell16")
    pr["params"].update(ntp=ntp, nr=nr, nghost=ghosts)
    out = []
    for form in (0, cs.CS_FLAG_FP32):
        s = cs.Solve(**pr["params"], flags=form | p2)
        s.mesh_build()
        s.init_problem(**pr["init"])
        s.steps(1, s.evaluate_timestep(1e30))
        out.append((s, s.get_state()))
    (s, want), (_, got) = out
    for q in (0, 4):
        den = np.abs(zones(s, want["U"][q])).max()
        assert np.abs(zones(s, got["U"][q]) - zones(s, want["U"][q])).max() <= 5e-6 * den, q
    mom = np.sqrt(np.abs(zones(s, want["U"][0])).max() * np.abs(zones(s, want["U"][4])).max())
    for q in (1, 2, 3):
        assert np.abs(zones(s, got["U"][q]) - zones(s, want["U"][q])).max() <= 5e-6 * mom, q
    assert max(face_b_errors(s, got, want).values()) <= 5e-6


@pytest.mark.parametrize("name,ntp,nr,ghosts,kernel", [("shell16", 6, 1, 4, "k_adp_solve"), ("surface32", 12, 3, 4, "k_adp6")])
def test_precision_form_on_ill_conditioned_meshes(name, ntp, nr, ghosts, kernel):
    """The meshes at both sides of the choice between inverse and factors (max
    |K| max |K^-1| of 1.4e9 and 2200), at the bound of the test above; measured
    3e-7."""
    pr = cs.preset(name)
    pr["params"].update(ntp=ntp, nr=nr, nghost=ghosts)
    out = []
    for form in (0, cs.CS_FLAG_FP32):
        s = cs.Solve(**pr["params"], flags=form)
        s.mesh_build()
        s.init_problem(**pr["init"])
        s.profile_begin()
        s.step(s.evaluate_timestep(1e30))
        assert kernel in s.profile_end()
        out.append(s.get_state())
    want, got = out
    for q in (0, 4, 5, 6, 7):
        assert np.abs(zones(s, got["U"][q]) - zones(s, want["U"][q])).max() <= 5e-6 * np.abs(zones(s, want["U"][q])).max(), q
    assert max(face_b_errors(s, got, want).values()) <= 5e-6


def test_fp64_batches_give_each_members_own_result():
    """Members of different sizes side by side, many times: every state equals
    the member's run alone to the bit (an earlier pair of ADP kernels
    left a few wrong zones in one member run of thirty)."""
    members = []
    for name, over in (("shell32", {}), ("surface32", dict(ntp=48)), ("shell32", dict(ntp=48, nr=24)),
                       ("shell16", dict(ntp=24, nr=16))):
        pr = cs.preset(name)
        pr["params"].update(over)
        s = cs.Solve(**pr["params"])
        s.mesh_build()
        s.init_problem(**pr["init"])
        st = s.get_state()
        s.steps(1, s.evaluate_timestep(1e30))
        members.append((s, st, s.get_state()))
    b = cs.Batch([m[0] for m in members])
    for rep in range(40):
        for s, st, _ in members:
            s.put_state(st)
        b.steps(1, [s.evaluate_timestep(1e30) for s, _, _ in members])
        for n, (s, _, want) in enumerate(members):
            got = s.get_state()
            for k in want:
                assert np.array_equal(got[k], want[k]), (rep, n, k)
    b.close()


@pytest.mark.parametrize("codes,flags", [((0, 0), 0), ((2, 0), cs.CS_FLAG_FP32), ((0, 2), cs.CS_FLAG_ADP_PER_PANEL)])
def test_callers_ghosts_take_their_zone_b(codes, flags):
    """A radial boundary code other than outflow leaves the radial ghosts to the
    caller, so the zone B that STEP 8.d sets in all but the last layer has to
    reach the next stage."""
    pr = cs.preset("shell16")
    pr["params"].update(ntp=10, nr=5, bc_lower=codes[0], bc_upper=codes[1])
    s = cs.Solve(**pr["params"], flags=flags)
    s.mesh_build()
    s.init_problem(**pr["init"])
    G, N, nr = s.G, s.N, s.nr
    s.fill_ghosts()
    before = s.get_state()["U"][5:8].copy()
    s.limit_all_slopes_p12()
    after = s.get_state()["U"][5:8]
    for layer, code in ((2 - G, codes[0]), (nr + G - 1, codes[1])):
        b, a = (x[:, :, G + layer, G + 1:G + N + 1, G + 1:G + N + 1] for x in (before, after))
        if code == 0:
            assert np.abs(a - b).max() > 0.0


def own_columns(s, a, face=None):
    """Zones (or faces of direction `face`) of the panels' own columns, through all radial layers."""
    G, N = s.G, s.N
    return a[..., 1 - (face == 2):, G + 1 - (face == 1):G + N + 1, G + 1 - (face == 0):G + N + 1]


def check_columns(s, got, want, tol=1e-12):
    """check_state through the radial ghosts."""
    for q in range(8):
        a, b = own_columns(s, got["U"][q]), own_columns(s, want["U"][q])
        assert np.abs(a - b).max() <= tol * np.abs(b).max(), ("U", q, np.abs(a - b).max() / np.abs(b).max())
    a, b = own_columns(s, got["ent"]), own_columns(s, want["ent"])
    assert np.abs(a - b).max() <= tol * np.abs(b).max(), ("ent", np.abs(a - b).max() / np.abs(b).max())
    den = max(np.abs(own_columns(s, want[k], d)).max() for d, k in enumerate(("bxf", "byf", "bzf")))
    for d, k in enumerate(("bxf", "byf", "bzf")):
        e = np.abs(own_columns(s, got[k], d) - own_columns(s, want[k], d)).max()
        assert e <= tol * den, (k, e / den)


@pytest.mark.parametrize("codes", [(0, 0), (2, 0), (0, 2)])
@pytest.mark.parametrize("rk", [cs.CS_RK2, cs.CS_SSPRK3, cs.CS_IMEX_RK2])
def test_callers_ghosts_match_the_oracle_over_whole_steps(codes, rk):
    """Radial ghosts of the caller's, which the stages advance like the
    reference's: three steps, ghosts compared too."""
    from oracle import Oracle
    pr = cs.preset("shell16")
    pr["params"].update(ntp=10, nr=5, rk_scheme=rk)
    filled = cs.Solve(**pr["params"])
    filled.mesh_build(device=False)
    o = Oracle(filled)
    o.put_state(filled.init_problem_host(**pr["init"]))
    o.fill_ghosts()
    st = o.get_state()
    noise = 1.0 + 0.02 * np.random.default_rng(11).uniform(-1.0, 1.0, st["U"].shape[1:])
    noise[:, filled.G + 1:filled.G + filled.nr + 1] = 1.0
    st["U"] = st["U"] * noise
    s = cs.Solve(**{**pr["params"], "bc_lower": codes[0], "bc_upper": codes[1]})
    s.mesh_build()
    o = Oracle(s)
    s.put_state(st)
    o.put_state(st)
    dt, dto = s.evaluate_timestep(1e30), o.evaluate_timestep(1e30)
    for n in range(3):
        dt, dto = s.step(dt), o.step(dto)
        assert abs(dt - dto) <= 1e-12 * dto, (n, dt, dto)
        check_columns(s, s.get_state(), o.get_state())


@pytest.mark.parametrize("ghosts", [3, 4])
@pytest.mark.parametrize("rk", [cs.CS_RK2, cs.CS_SSPRK3, cs.CS_IMEX_RK2])
def test_radial_ghosts_at_the_pressure_floor_match_the_oracle(rk, ghosts):
    """A shell whose first and last radial layers start 2 % above the pressure
    floor (not on it, where rounding decides): the outer ghosts, copied with the
    ratio of the volumes, fall below it and take their pressure from the entropy
    that the last stage left in them (kept from before that stage instead, it
    moves the state by 1e-2).  The ghosts' own state is compared too."""
    from oracle import Oracle
    pr = cs.preset("shell16")
    pr["params"].update(ntp=10, nr=6, nghost=ghosts, rk_scheme=rk, prsfloor=0.05)
    s = cs.Solve(**pr["params"])
    s.mesh_build()
    st = s.init_problem_host(**pr["init"])
    U, p, g = st["U"], 0.051, s.params.gamma
    for layer in (s.G + 1, s.G + s.nr):
        on = U[0][:, layer] > 0.0
        rho = np.where(on, U[0][:, layer], 1.0)
        e = p / (g - 1) + 0.5 * (U[1:4, :, layer] ** 2).sum(0) / rho + (U[5:8, :, layer] ** 2).sum(0) / (8 * np.pi)
        U[4][:, layer] = np.where(on, e, U[4][:, layer])
        st["ent"][0][:, layer] = np.where(on, p / rho ** (g - 1), st["ent"][0][:, layer])
    o = Oracle(s)
    s.put_state(st)
    o.put_state(st)
    dt, dto = s.evaluate_timestep(1e30), o.evaluate_timestep(1e30)
    for n in range(3):
        dt, dto = s.step(dt), o.step(dto)
        assert abs(dt - dto) <= 1e-12 * dto, (n, dt, dto)
        check_columns(s, s.get_state(), o.get_state())


@pytest.mark.parametrize("p2,out_to", [(0, 3), (cs.CS_FLAG_P2, 2)])
def test_ghosts_that_give_up_zero_their_entropy_like_the_oracle(p2, out_to):
    """STEP 7.c in ghosts of the caller's that are rough enough to exhaust its
    shrink passes in every layer that has modes."""
    from oracle import Oracle
    pr = cs.preset("shell16")
    pr["params"].update(ntp=10, nr=5)
    filled = cs.Solve(**pr["params"])
    filled.mesh_build(device=False)
    o = Oracle(filled)
    o.put_state(filled.init_problem_host(**pr["init"]))
    o.fill_ghosts()
    st = o.get_state()
    s = cs.Solve(**pr["params"], bc_lower=0, bc_upper=0, flags=p2)
    rough = 1.0 - 0.97 * np.random.default_rng(1).uniform(0.0, 1.0, st["U"].shape[1:])
    rough[:, s.params.nghost:s.params.nghost + s.params.nr + 2] = 1.0  # the interior and the first ghosts
    st["U"] = st["U"] * rough
    s.mesh_build()
    o = Oracle(s)
    out = []
    for x in (s, o):
        x.put_state(st)
        x.fill_ghosts()
        x.limit_all_slopes_p12()
        out.append(own_columns(s, x.get_state()["ent"])[0])
    got, want = out
    for layer in (s.G - out_to, s.G + s.nr + out_to - 1):  # the columns start with ghost layer G
        assert (want[:, layer] == 0.0).any()
    assert np.array_equal(got == 0.0, want == 0.0)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


def test_a_shared_mesh_serves_solves_of_other_boundary_codes():
    """Solves that share a mesh may differ in their boundary codes; each gives
    what it gives on its own mesh (up to the ADP operators' rounding, 1e-12)."""
    pr = cs.preset("shell16")
    pr["params"].update(ntp=10, nr=5)
    for first, second in (((2, 2), (0, 0)), ((0, 0), (2, 2))):
        a = cs.Solve(**{**pr["params"], "bc_lower": first[0], "bc_upper": first[1]})
        a.mesh_build()
        out = []
        for share in (False, True):
            s = cs.Solve(**{**pr["params"], "bc_lower": second[0], "bc_upper": second[1]})
            s.mesh_share(a) if share else s.mesh_build()
            s.init_problem(**pr["init"])
            s.steps(2, s.evaluate_timestep(1e30))
            out.append(s.get_state())
        check_state(s, out[1], out[0])


@pytest.mark.parametrize("first,second", [((2, 2), (0, 0)), ((0, 0), (2, 2)), ((2, 2), (0, 2))])
def test_a_shared_mesh_serves_its_adp_operators_whatever_the_boundary_codes(first, second):
    """Solves on one mesh use its ADP inverses in every stage, whichever
    boundary codes the mesh was built with."""
    pr = cs.preset("shell16")
    pr["params"].update(ntp=10, nr=5)
    a = cs.Solve(**{**pr["params"], "bc_lower": first[0], "bc_upper": first[1]})
    a.mesh_build()
    s = cs.Solve(**{**pr["params"], "bc_lower": second[0], "bc_upper": second[1]})
    s.mesh_share(a)
    s.init_problem(**pr["init"])
    s.profile_begin()
    s.step(s.evaluate_timestep(1e30))
    kernels = s.profile_end()
    assert kernels["k_adp6"][1] == 2 and "k_adp" not in kernels, sorted(kernels)


@pytest.mark.parametrize("name,ntp,nr,ghosts", [("surface32", 12, 3, 4), ("shell16", 13, 3, 4), ("shell16", 12, 3, 4)])
def test_adp_inverses_are_as_accurate_as_the_factors(name, ntp, nr, ghosts):
    """B modes by the packed inverse against the per-panel factors on meshes whose
    matrices are the worst conditioned that keep the inverse (max |K| max
    |K^-1| of 2200, 880 and 640).  Against 80-bit elimination the factors err by
    up to 5e-14 of a zone's largest mode and a rounded inverse by 1e-14, and the
    right-hand sides' roundings add 2e-14: 2e-13 leaves them twice that and is
    below an inverse that keeps the elimination's own errors (2e-13 to 6e-13)."""
    pr = cs.preset(name)
    pr["params"].update(ntp=ntp, nr=nr, nghost=ghosts)
    out = []
    for flags, kernel in ((0, "k_adp6"), (cs.CS_FLAG_ADP_PER_PANEL, "k_adp_solve")):
        s = cs.Solve(**pr["params"], flags=flags)
        s.mesh_build()
        s.init_problem(**pr["init"])
        s.fill_ghosts()
        s.limit_all_slopes_p12()
        V = s.debug("V")
        s.profile_begin()
        s.step(s.evaluate_timestep(1e30))
        assert kernel in s.profile_end()
        out.append(np.stack([V[8 * m + c] for m in range(10) for c in (5, 6, 7)]))
    lay = slice(s.G + 1 - (s.G - 1), s.G + s.nr + s.G)  # layers 2 - G .. nr + G - 1
    side = slice(s.G - 1, s.G + s.N + 3)                # two beside the panel
    a, b = (x[:, :, lay, side, side] for x in out)
    on = (s.mask()[:, lay, side, side] == 1) & (np.abs(b).max(0) > 0.0)
    err = (np.abs(a - b).max(0)[on] / np.abs(b).max(0)[on]).max()
    assert err <= 2e-13, err


def test_reciprocals_by_newton_steps_are_within_two_units():
    """The stage kernels form 1 / rho by Newton steps.  Two gases at rest without
    field, rho over 22 decades: the fast speed is sqrt(gamma p / rho), where two
    units of the reciprocal, the two products' roundings and the two roots' add
    up to less than 4 units (eps each) of the speed."""
    rng = np.random.default_rng(7)
    rho = 10.0 ** rng.uniform(-11.0, 11.0, 4096)
    prs = rng.uniform(0.5, 2.0, rho.size)
    c = np.zeros((rho.size, 18))
    for side in (0, 8):
        c[:, side] = rho
        c[:, side + 4] = prs
    c[:, 16:] = 1.0
    gamma = 5.0 / 3.0
    out = cs.pointwise(2, c, ntp=8, nr=4, gamma=gamma)
    want = np.sqrt(np.longdouble(gamma) * prs.astype(np.longdouble) / rho.astype(np.longdouble))
    for sign, got in ((-1.0, out[:, 32]), (1.0, out[:, 33])):
        err = np.abs(sign * got - want) / want
        assert err.max() <= 4 * np.finfo(float).eps, float(err.max())


def test_a_star_density_of_zero_matches_the_oracle():
    """Two gases that leave each other at 2^60 with a jump in the transverse field:
    the star density is exactly 0 and the star momentum is not, so the pressure
    is -infinity and the entropy repair makes the energy infinite."""
    from oracle import Oracle
    c = np.zeros((1, 18))
    c[0, [0, 8, 4, 12, 16, 17]] = 1.0
    c[0, 1], c[0, 9] = -2.0 ** 60, 2.0 ** 60
    c[0, [5, 13, 14]] = 1.0
    got = cs.pointwise(2, c, ntp=8, nr=4)[0]
    want = Oracle(params=cs.make_params(ntp=8, nr=4), mesh=False).pointwise(2, c)[0]
    assert want[4] == want[12] == -np.inf
    assert np.array_equal(np.isinf(got), np.isinf(want)) and np.array_equal(got[[4, 12]], want[[4, 12]])
    on = np.isfinite(want)
    assert np.abs(got[on] - want[on]).max() <= 1e-14 * np.abs(want[on]).max()


@pytest.mark.parametrize("form", [0, cs.CS_FLAG_FP32])
def test_smoothness_indicators_that_overflow_weigh_nothing(form):
    """One zone so fast that the indicators of the stencils through it overflow:
    its neighbours take their modes from the other stencils, finite where the
    oracle's are (P2, whose modes are the weighted stencils' own)."""
    from oracle import Oracle
    from seeded_states import uniform_state
    pr = cs.preset("shell16")
    pr["params"].update(ntp=8, nr=6, gm=0.0)
    s = cs.Solve(**pr["params"], flags=cs.CS_FLAG_P2 | form)
    s.mesh_build()
    st = uniform_state(s)
    z = (2, s.G + 3, s.G + 4, s.G + 4)
    v = 8e153 if not form else 1e18  # squares near the largest value of the state's type
    st["U"][(1,) + z], st["U"][(4,) + z] = v, 0.5 * v * v + 1.5
    o = Oracle(s)
    V = []
    for x in (s, o):
        x.put_state(st)
        x.fill_ghosts()
        x.limit_all_slopes_p12()
        V.append(zones(s, x.debug("V")))
    if not form:
        assert not np.isfinite(V[1]).all()
    assert np.array_equal(np.isfinite(V[0]), np.isfinite(V[1]))
