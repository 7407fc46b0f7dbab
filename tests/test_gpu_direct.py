"""The direct form of long ADMM solves (nested-dissection factors applied with
refinement) against the CG it replaces."""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from silk_physics_b200 import native as N
from silk_physics_b200 import scenes as S

DIRECT_FROM = 16  # ADMM iteration from which the systems go to the direct form


def _strip(nx, ny):
    V, F = S.grid_sheet(max(nx, ny), side=1.0, jitter=1e-4, seed=1)
    s = max(nx, ny)
    keep = [j * s + i for j in range(ny) for i in range(nx)]
    new = -np.ones(s * s, int)
    new[keep] = np.arange(len(keep))
    F = new[F]
    return V[keep], F[(F >= 0).all(1)].astype(np.int32)


def _mesh(kind):
    if kind == "triangle":
        return (np.array([[0, 0, 1], [0.02, 0, 1], [0, 0.02, 1]], np.float32),
                np.array([[0, 1, 2]], np.int32))
    if kind.startswith("sphere"):
        return S.icosphere(int(kind[6:]), 0.3)
    nx, ny = (int(k) for k in kind.split("x"))
    return _strip(nx, ny)


# One front (3 to 256 vertices, both sides of a 64 tile and a 32 panel), two
# and more levels, leaf sizes of both ranges, a long strip and closed surfaces
# (no boundary to the separators' advantage).
@pytest.mark.parametrize("kind", ["triangle", "4x8", "5x13", "16x16", "16x17", "40x40", "7x200",
                                  "sphere3", "sphere4", "150x150"])
def test_direct_form_matches_cg(kind):
    """Forty ADMM iterations per step, three steps: the default form solves
    the systems from DIRECT_FROM on directly, form 1 by CG throughout, both to
    a relative residual of 1e-6.  Forty unconverged iterations amplify what
    either leaves, so the yardstick is the CG itself: the direct form must be
    within three times the CG's own distance (at least 5e-6 m, the FP32 bound
    of the well-conditioned parity test) of the CG solved to 1e-8."""
    V, F = _mesh(kind)
    out = []
    for form, tol in ((0, 1e-6), (1, 1e-6), (1, 1e-8)):
        w = N.World()
        assert w.init()
        assert w.set_global_config(N.GlobalConfig(max_inner_iteration=40, admm_abs_tol=0.0,
                                                  admm_rel_tol=0.0))
        assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=tol, cg_form=form))
        r, h = w.add_cloth(N.ClothConfig(elastic_stiffness=10.0, bending_stiffness=1e-4,
                                         density=5.0, damping=0.01),
                           N.CollisionConfig(is_collision_on=False, is_self_collision_on=False),
                           V, F, [0])
        assert r, r.to_string()
        for _ in range(3):
            r = w.solver_step()
            assert r, r.to_string()
            st = w.step_stats()
            assert st.admm_iterations == 40
            assert st.cg_solves == (DIRECT_FROM - 1 if form == 0 else 39)
        x = np.zeros(V.size, np.float32)
        assert w.get_cloth_position(h, x)
        out.append(x.astype(np.float64))
    err, own = np.abs(out[0] - out[2]).max(), np.abs(out[1] - out[2]).max()
    print(f"{kind}: direct {err:.2e}, CG {own:.2e} from the CG at 1e-8")
    assert np.isfinite(out[0]).all()
    assert err <= max(3.0 * own, 5e-6)


def test_direct_form_leaves_what_it_cannot_meet_to_the_cg():
    """A tolerance that no refinement reaches (1e-30): no direct solve
    may be taken, every system is solved by the CG from its own start, and
    the step gives the CG form's bits."""
    V, F = S.grid_sheet(24, jitter=1e-4, seed=3)
    out = []
    for form in (0, 3):
        w = N.World()
        assert w.init()
        assert w.set_global_config(N.GlobalConfig(max_inner_iteration=24, admm_abs_tol=0.0,
                                                  admm_rel_tol=0.0, linear_solver_abs_tol=0.0))
        assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-30, cg_form=form,
                                                    cg_max_iter=40))
        r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(
            is_collision_on=False, is_self_collision_on=False), V, F, S.top_corner_pins(24))
        assert r
        assert w.solver_step()
        assert w.step_stats().cg_solves == 23
        x = np.zeros(V.size, np.float32)
        assert w.get_cloth_position(h, x)
        out.append(x)
    np.testing.assert_array_equal(out[0], out[1])


def test_direct_form_on_every_device():
    """Resident-block limits and shared-memory opt-ins belong to a device: the
    same scene on device 1 is solved directly as on device 0, to the bit."""
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("one device")
    V, F = S.grid_sheet(60, jitter=1e-4, seed=3)
    out = []
    for dev in range(2):
        with torch.cuda.device(dev):
            w = N.World()
            assert w.init()
            assert w.set_global_config(N.GlobalConfig(max_inner_iteration=24, admm_abs_tol=0.0,
                                                      admm_rel_tol=0.0))
            assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-5))
            r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(
                is_collision_on=False, is_self_collision_on=False), V, F, S.top_corner_pins(60))
            assert r
            assert w.solver_step()
            assert w.step_stats().cg_solves == DIRECT_FROM - 1
            x = np.zeros(V.size, np.float32)
            assert w.get_cloth_position(h, x)
            out.append(x)
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("block", [1, 2])
def test_direct_barrier_wait_runs_out(block):
    """A direct solve in which one block never arrives at its barriers (test
    switch debug_withhold_block; the CG before it runs as one cluster, whose
    barrier the switch does not reach): the bounded waits end, the step
    reports IterativeSolveFail, and the world steps normally afterwards."""
    V, F = S.grid_sheet(60, jitter=1e-4, seed=3)
    w = N.World()
    assert w.init()
    assert w.set_global_config(N.GlobalConfig(max_inner_iteration=24, admm_abs_tol=0.0,
                                              admm_rel_tol=0.0))
    r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(
        is_collision_on=False, is_self_collision_on=False), V, F, S.top_corner_pins(60))
    assert r
    assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-5,
                                                barrier_spin_limit=1 << 16,
                                                debug_withhold_block=block))
    r = w.solver_step()
    assert r.code == N.ErrorCode.IterativeSolveFail, r.to_string()
    assert "barrier" in r.detail, r.detail
    assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-5))
    assert w.set_cloth_state(h, V)
    r = w.solver_step()
    assert r, r.to_string()
    st = w.step_stats()
    assert st.admm_iterations == 24 and st.cg_solves == DIRECT_FROM - 1


def test_direct_form_is_counted():
    """What the direct form did in a step: every system from the threshold on
    is counted as solved or missed, with its factorisations, applications and
    event times; a step without it counts nothing."""
    V, F = S.grid_sheet(40, jitter=1e-4, seed=3)
    w = N.World()
    assert w.init()
    r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(
        is_collision_on=False, is_self_collision_on=False), V, F, S.top_corner_pins(40))
    assert r
    for inner, form in ((24, 0), (DIRECT_FROM, 0), (24, 3), (24, 0)):
        assert w.set_global_config(N.GlobalConfig(max_inner_iteration=inner, admm_abs_tol=0.0,
                                                  admm_rel_tol=0.0))
        assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-5, cg_form=form,
                                                    profile=1))
        assert w.solver_step()
        st, d = w.step_stats(), w.direct_stats()
        direct = inner - DIRECT_FROM if form == 0 else 0
        assert d["first_iteration"] == DIRECT_FROM
        assert d["solves"] == direct and d["misses"] == 0
        assert st.cg_solves == inner - 1 - direct
        assert d["factorisations"] == (1 if direct else 0)
        assert direct <= d["applications"] <= 4 * direct
        for key in ("application_bytes", "factor_ms", "solve_ms"):
            assert (d[key] > 0) == (direct > 0)


def test_direct_form_gives_up_on_a_tolerance_out_of_reach():
    """A sheet landing on a ball at a tolerance that no refinement reaches:
    one miss ends the tries of its ADMM solve and of the step's later ones,
    which do not factorise either; the CG form's bits."""
    V, F = S.grid_sheet(24, side=0.5, z=0.31, jitter=1e-4, seed=3)
    SV, SF = S.icosphere(2, radius=0.3)
    out = []
    for form in (0, 3):
        w = N.World()
        assert w.init()
        assert w.set_global_config(N.GlobalConfig(max_inner_iteration=24, admm_abs_tol=0.0,
                                                  admm_rel_tol=0.0, linear_solver_abs_tol=0.0))
        assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-30, cg_form=form,
                                                    cg_max_iter=40))
        r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(), V, F, [])
        assert r
        r, _ = w.add_obstacle(N.CollisionConfig(), SV, SF)
        assert r
        got = []
        for _ in range(3):
            r = w.solver_step()
            assert r, r.to_string()
            st, d = w.step_stats(), w.direct_stats()
            got.append((st.outer_iterations, st.cg_solves))
            assert st.cg_solves == 23 * st.outer_iterations
            assert (d["factorisations"], d["misses"], d["solves"]) == \
                ((1, 1, 0) if form == 0 else (0, 0, 0))
        x = np.zeros(V.size, np.float32)
        assert w.get_cloth_position(h, x)
        out.append((got, x))
    assert max(o for o, _ in out[0][0]) > 1
    assert out[0][0] == out[1][0]
    np.testing.assert_array_equal(out[0][1], out[1][1])


def _two_cloths(form, tol, sizes, over):
    """Cloths of the given sides, each flat within contact distance of its own
    plate (over) or free, one ADMM solve of 40 iterations in one world."""
    w = N.World()
    assert w.init()
    assert w.set_global_config(N.GlobalConfig(max_inner_iteration=40, max_outer_iteration=1,
                                              admm_abs_tol=0.0, admm_rel_tol=0.0,
                                              linear_solver_abs_tol=0.0))
    assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=tol, cg_form=form))
    handles = []
    for k, s in sizes:
        V, F = S.grid_sheet(s, side=(s - 1) / 79, z=1.0, jitter=1e-5, seed=k)
        V[:, 0] += 3.0 * k
        r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(
            is_collision_on=over, is_self_collision_on=False), V, F, [])
        assert r, r.to_string()
        handles.append((h, V.size))
        if over:
            n = s // 4
            OV, OF = S.grid_sheet(n, side=1.1 * (s - 1) / 79, z=0.0)
            OV[:, 0] += 3.0 * k + 0.5 * (V[:, 0].min() + V[:, 0].max() - 6.0 * k) \
                - 0.5 * (OV[:, 0].min() + OV[:, 0].max())
            OV[:, 1] += 0.5 * (V[:, 1].min() + V[:, 1].max() - OV[:, 1].min() - OV[:, 1].max())
            OV[:, 2] = V[:, 2].min() - 2e-4
            r, _ = w.add_obstacle(N.CollisionConfig(), OV, OF)
            assert r, r.to_string()
    r = w.solver_step()
    assert r, r.to_string()
    out = []
    for h, n in handles:
        x = np.zeros(n, np.float32)
        assert w.get_cloth_position(h, x)
        out.append(x.astype(np.float64))
    return out, w.step_stats(), w.direct_stats()


# A CG in one cluster (its own stream) beside a cooperative grid (the world's
# stream), in both orders, and two clusters side by side.
TWO = [((0, 24), (1, 136)), ((0, 136), (1, 24)), ((0, 40), (1, 33))]


@pytest.mark.parametrize("sizes", TWO)
def test_two_cloths_are_solved_as_alone(sizes):
    """Cloths without contact are independent systems: stepped in one world
    and each in a world of its own they end in the same bits."""
    both, st, d = _two_cloths(0, 1e-5, sizes, False)
    assert d["solves"] == 2 * (40 - DIRECT_FROM) and d["misses"] == 0
    assert st.cg_solves == 2 * (DIRECT_FROM - 1)
    for x, size in zip(both, sizes):
        alone, _, _ = _two_cloths(0, 1e-5, [size], False)
        np.testing.assert_array_equal(x, alone[0])


@pytest.mark.parametrize("sizes", TWO)
def test_two_cloths_in_contact_match_cg(sizes):
    """Two cloths in contact, the direct form against CG throughout.  Contacts
    that open or close amplify what a solve leaves and how it is rounded, so
    the yardstick is the larger distance of two CG forms (solved to 1e-6, sums
    in other orders) from the CG solved to 1e-8; no absolute tolerance, which
    would stop all of them alike."""
    out = [_two_cloths(form, tol, sizes, True) for form, tol in
           ((0, 1e-6), (3, 1e-6), (1, 1e-6), (3, 1e-8))]
    assert out[0][2]["solves"] > 0 and out[0][1].contacts > 0
    assert all(o[1].contacts == out[0][1].contacts for o in out)
    for k in range(2):
        err = np.abs(out[0][0][k] - out[3][0][k]).max()
        own = max(np.abs(o[0][k] - out[3][0][k]).max() for o in out[1:3])
        print(f"{sizes[k]}: {out[0][1].contacts} contacts, direct {err:.2e}, CG {own:.2e}")
        assert err <= max(3.0 * own, 5e-6)


@pytest.mark.parametrize("learned, extrapolated", [(True, False), (False, True), (True, True)])
def test_no_starts_for_systems_solved_directly(learned, extrapolated):
    """The learned and extrapolated starts are offered to the CG alone: an
    iteration whose systems are solved directly launches what the plain one
    does, and the steps before the threshold start as before."""
    V, F = S.grid_sheet(24, jitter=1e-4, seed=3)

    def run(inner, **opts):
        w = N.World()
        assert w.init()
        assert w.set_global_config(N.GlobalConfig(max_inner_iteration=inner, admm_abs_tol=0.0,
                                                  admm_rel_tol=0.0))
        assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-6, **opts))
        r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(
            is_collision_on=False, is_self_collision_on=False), V, F, S.top_corner_pins(24))
        assert r
        if opts.get("learned_warm_start"):
            assert w.set_warm_start_model(learned_model)
        for _ in range(2):  # the second step has the direct system from the start
            r = w.solver_step()
            assert r, r.to_string()
        st = w.step_stats()
        assert st.cg_solves == DIRECT_FROM - 1
        return st.kernel_launches, st.learned_iterate_starts + st.extrapolated_starts

    from silk_physics_b200 import learned as L
    learned_model = L.load(str(Path(N.__file__).resolve().parent / "models" / "warm_start.npy"))
    opts = dict(learned_warm_start=learned, admm_extrapolated_start=extrapolated)
    plain = [run(k)[0] for k in (24, 40)]
    other = [run(k, **opts) for k in (24, 40)]
    assert other[1][0] - other[0][0] == plain[1] - plain[0]
    assert other[0][0] > plain[0] and other[0][1] > 0
