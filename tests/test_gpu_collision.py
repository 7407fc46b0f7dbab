"""GPU collision pipeline against the oracle: broadphase candidate sets, DCD
contact sets and CCD decisions are compared bit for bit; colourings are
valid and identical; full steps with contacts stay within tolerance."""
import numpy as np
import pytest

import ccd_cases as CC
from silk_physics_b200 import native as N
from silk_physics_b200 import scenes as S

pytestmark = pytest.mark.gpu


def _scene(oracle, jitter=1e-3, self_on=True, seed=1):
    """Two 12x12 sheets 1.5 cm apart over a small icosphere."""
    col = N.CollisionConfig(is_self_collision_on=self_on)
    ocol = (1, int(self_on), 0, 0.3, 0.3)
    w = N.World()
    assert w.init()
    ow = oracle.OracleWorld()
    sheets = []
    for k, z in enumerate((0.35, 0.365)):
        V, F = S.grid_sheet(12, side=0.6, z=z, jitter=jitter, seed=seed + k)
        r, h = w.add_cloth(N.ClothConfig(), col, V, F, [])
        assert r
        perm, offs = w.cloth_partition(h, len(V))
        oh = ow.add_cloth(V, F, [], perm, offs, collision=ocol)
        assert oh == h
        sheets.append((h, V, F, perm))
    SV, SF = S.icosphere(2, radius=0.3)
    r, hs = w.add_obstacle(N.CollisionConfig(), SV, SF)
    assert r
    assert ow.add_obstacle(SV, SF) == hs
    return w, ow, sheets


def _disp(sheets, scale, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _, V, _, _ in sheets:
        d = rng.normal(0, scale, V.shape).astype(np.float32)
        d[:, 2] -= 4 * scale
        out.append(d.ravel())
    return np.concatenate(out)


def _rows(a):
    return set(map(tuple, np.asarray(a).tolist()))


@pytest.mark.parametrize("scale", [0.0, 2e-3, 1e-2])
def test_broadphase_candidate_sets_identical(oracle, scale):
    w, ow, sheets = _scene(oracle)
    d = _disp(sheets, scale, 11)
    w.debug_refit(d)
    ow.refit(d)
    g = w.debug_candidates()
    o = ow.candidates()
    print(f"scale {scale}: {len(g)} candidates (oracle {len(o)})")
    assert len(g) > 0
    assert len(g) == len(_rows(g)), "duplicate candidate pairs"
    assert _rows(g) == _rows(o)


def test_dcd_contact_sets_identical(oracle):
    w, ow, sheets = _scene(oracle)
    d = _disp(sheets, 5e-3, 3)
    w.debug_refit(d)
    ow.refit(d)
    for t, dact in ((0.0, 0.02), (0.5, 0.02), (1.0, 0.01)):
        g = w.debug_dcd(t, dact)
        o = ow.dcd(t, dact)
        print(f"t={t}: {len(g)} active contacts")
        assert len(g) > 0
        np.testing.assert_array_equal(g, o)


def test_min_toi_identical(oracle):
    w, ow, sheets = _scene(oracle)
    d = _disp(sheets, 8e-3, 5)
    w.debug_refit(d)
    ow.refit(d)
    for ts, mt, ms in ((0.0, 1.0, 1e-4), (0.3, 0.7, 5e-4)):
        tg, nqg, nhg = w.debug_min_toi(ts, mt, ms)
        to, nqo, nho = ow.min_toi(ts, mt, ms)
        print(f"window ({ts},{mt}): toi {tg} queries {nqg} hits {nhg}")
        assert nqg == nqo and nhg == nho
        assert np.float32(tg) == np.float32(to)
        assert nhg > 0 and tg < mt
        # Pruned searches (the step's mode) give the same minimum.
        tp, nqp, _ = w.debug_min_toi(ts, mt, ms, prune=True)
        assert nqp == nqg and np.float32(tp) == np.float32(tg)


def _random_queries(rng, n, vf):
    base = rng.uniform(-1, 1, (n, 4, 3)).astype(np.float32)
    if vf:
        base[:, 1:, 2] = 0.0
        base[:, 0, 2] = rng.uniform(0.001, 0.2, n)
    motion = rng.normal(0, 0.4, (n, 4, 3)).astype(np.float32)
    motion[:, 0, 2] -= rng.uniform(0, 0.6, n)
    x = np.concatenate([base, base + motion], axis=1)
    return x.reshape(n, 24).astype(np.float32)


@pytest.mark.parametrize("vf", [True, False])
def test_ccd_batch_bit_exact(oracle, vf):
    rng = np.random.default_rng(42 if vf else 43)
    n = 3000
    x = _random_queries(rng, n, vf)
    err = np.array([4.053116e-06 if vf else 3.814698e-06] * 3, np.float32)
    ms = rng.choice([0.0, 1e-4, 1e-3], n).astype(np.float32)
    hit, toi, tup = N.ccd_batch(vf, x, err, ms, 1e-6, 4096, 1.0)
    hits = 0
    for i in range(n):
        oh, t4, small = oracle.ccd(vf, x[i], err, float(ms[i]))
        assert bool(hit[i]) == oh, i
        if oh:
            hits += 1
            exp_toi = t4[2] if small else t4[0]
            exp_up = t4[3] if small else t4[1]
            assert np.float32(toi[i]) == np.float32(exp_toi), (i, toi[i], exp_toi)
            assert np.float32(tup[i]) == np.float32(exp_up), (i, tup[i], exp_up)
    print(f"{'VF' if vf else 'EE'}: {hits} hits of {n}")
    assert 0 < hits < n


def test_coloring_valid_and_equal_to_oracle(oracle):
    rng = np.random.default_rng(9)
    n = 5000
    verts = rng.integers(-1, 1500, size=(n, 4)).astype(np.int32)
    prio = rng.integers(0, 2 ** 63, size=n, dtype=np.uint64)
    colors, nc = N.color_contacts(verts, prio)
    ocolors, onc = oracle.color_contacts(verts, prio)
    assert nc == onc
    np.testing.assert_array_equal(colors, ocolors)
    inc = {}
    for i, vs in enumerate(verts):
        for v in set(vs.tolist()):
            if v >= 0:
                inc.setdefault(int(v), []).append(i)
    for lst in inc.values():
        cs = [colors[i] for i in lst]
        assert len(cs) == len(set(cs))


def test_sheet_on_sphere_contacts_and_parity(oracle):
    """A 20x20 sheet dropped on an icosphere: over the first six steps (the
    sheet lands at step 3) the contact count, colour count and number of CCD
    rollbacks of each step equal the oracle's and positions agree within
    1e-3 m.  Later, FP32 rounding flips a rollback decision and contact
    trajectories diverge, as they do between two FP32 runs of the reference."""
    V, F = S.grid_sheet(20, side=0.5, z=0.312, jitter=1e-4, seed=4)
    SV, SF = S.icosphere(3, radius=0.3)
    g = N.GlobalConfig(max_inner_iteration=30)
    w = N.World()
    assert w.init()
    assert w.set_global_config(g)
    assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-5))
    r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(), V, F, [])
    r2, hs = w.add_obstacle(N.CollisionConfig(), SV, SF)
    assert r and r2
    perm, offs = w.cloth_partition(h, len(V))
    ow = oracle.OracleWorld(config=dict(max_inner_iteration=30, fixed_linear_rel_tol=1e-5))
    oh = ow.add_cloth(V, F, [], perm, offs)
    ow.add_obstacle(SV, SF)
    x = np.zeros(V.size, np.float32)
    saw_contacts = False
    for k in range(6):
        assert w.solver_step(), w
        assert ow.step() == 0
        st, so = w.step_stats(), ow.stats()
        assert w.get_cloth_position(h, x)
        err = np.abs(x.reshape(-1, 3) - ow.position(oh)).max()
        print(f"step {k + 1}: contacts {st.contacts}/{so['contacts']} colors "
              f"{st.colors}/{so['colors']} outer {st.outer_iterations}/"
              f"{so['outer_iterations']} err {err:.2e}")
        saw_contacts |= st.contacts > 0
        assert st.contacts == so["contacts"] and st.colors == so["colors"]
        assert st.outer_iterations == so["outer_iterations"]
        assert err < 1e-3
    assert saw_contacts


def test_moving_obstacle_parity(oracle):
    """A sphere pushed up under a resting sheet through set_obstacle_position
    (the prescribed obstacle displacement of dcd.cu:84-96 enters every
    contact): contact, colour and rollback counts equal the oracle's over the
    first three steps (afterwards FP32 rounding may move a pair across the
    activation distance: contact counts within 2 %) and positions agree
    within 1e-3 m over four steps (the lifted sheet's contact trajectory
    diverges from the oracle's after that, as two FP32 runs of the reference
    would)."""
    V, F = S.grid_sheet(20, side=0.5, z=0.305, jitter=1e-4, seed=5)
    SV, SF = S.icosphere(3, radius=0.3)
    g = N.GlobalConfig(max_inner_iteration=30)
    w = N.World()
    assert w.init()
    assert w.set_global_config(g)
    assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-5))
    r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(), V, F, [])
    r2, hs = w.add_obstacle(N.CollisionConfig(), SV, SF)
    assert r and r2
    perm, offs = w.cloth_partition(h, len(V))
    ow = oracle.OracleWorld(config=dict(max_inner_iteration=30, fixed_linear_rel_tol=1e-5))
    oh = ow.add_cloth(V, F, [], perm, offs)
    ohs = ow.add_obstacle(SV, SF)
    x = np.zeros(V.size, np.float32)
    saw = False
    for k in range(4):
        pos = (SV + np.array([0.0, 0.0, 0.004 * (k + 1)], np.float32)).astype(np.float32)
        assert w.set_obstacle_position(hs, pos)
        assert ow.set_obstacle_position(ohs, pos) == 0
        assert w.solver_step(), w
        assert ow.step() == 0
        st, so = w.step_stats(), ow.stats()
        assert w.get_cloth_position(h, x)
        err = np.abs(x.reshape(-1, 3) - ow.position(oh)).max()
        print(f"step {k + 1}: contacts {st.contacts}/{so['contacts']} outer "
              f"{st.outer_iterations}/{so['outer_iterations']} err {err:.2e}")
        saw |= st.contacts > 0
        if k < 3:
            assert st.contacts == so["contacts"] and st.colors == so["colors"]
            assert st.outer_iterations == so["outer_iterations"]
        else:
            # FP32 rounding may move a pair across the activation distance.
            assert abs(st.contacts - so["contacts"]) <= max(2, 0.02 * so["contacts"])
        assert err < 1e-3
    assert saw
    # The sheet was lifted with the sphere.
    assert x.reshape(-1, 3)[:, 2].max() > 0.305


def test_collision_groups_filter_candidates(oracle):
    """Objects collide only within one collision group (find_collision.cu:
    17-25): with the second sheet in its own group, no candidate pairs it
    with the first sheet or the sphere, and the candidate sets still equal the
    oracle's."""
    w = N.World()
    assert w.init()
    ow = oracle.OracleWorld()
    sheets = []
    for k, (z, grp) in enumerate(((0.35, 0), (0.365, 1))):
        V, F = S.grid_sheet(12, side=0.6, z=z, jitter=1e-3, seed=20 + k)
        col = N.CollisionConfig(group=grp)
        r, h = w.add_cloth(N.ClothConfig(), col, V, F, [])
        assert r
        perm, offs = w.cloth_partition(h, len(V))
        assert ow.add_cloth(V, F, [], perm, offs, collision=(1, 1, grp, 0.3, 0.3)) == h
        sheets.append((h, V))
    SV, SF = S.icosphere(2, radius=0.3)
    r, hs = w.add_obstacle(N.CollisionConfig(group=0), SV, SF)
    assert r and ow.add_obstacle(SV, SF, collision=(1, 1, 0, 0.3, 0.3)) == hs
    d = _disp([(h, V, None, None) for h, V in sheets], 5e-3, 7)
    w.debug_refit(d)
    ow.refit(d)
    g = w.debug_candidates()
    o = ow.candidates()
    assert _rows(g) == _rows(o)
    hb = sheets[1][0]
    # Records are (kind, handle a, primitive a, handle b, primitive b): the
    # second sheet may only pair with itself.
    pairs = {(int(c[1]), int(c[3])) for c in g}
    print(f"{len(g)} candidates; object pairs {sorted(pairs)}")
    assert len(g) > 0
    for a, b in pairs:
        if hb in (a, b):
            assert a == b == hb


def test_gs_forms_identical():
    """The single-block contact Gauss-Seidel (colour-ordered contacts on
    compact vertex slots) and the grid form give bit-identical positions on a
    pinned sheet draped on a sphere, where contacts also read pinned vertices
    and clamped (zero-weight) closest points."""
    out = []
    for form in (0, 1):
        V, F = S.grid_sheet(32, side=0.8, z=0.305, jitter=1e-4, seed=8)
        # Corners and the vertex over the sphere's top pinned: the sheet drapes
        # around a pinned vertex, so contacts also involve pinned vertices.
        P = np.concatenate([S.top_corner_pins(32), [16 * 32 + 16]]).astype(np.int32)
        SV, SF = S.icosphere(3, radius=0.3)
        w = N.World()
        assert w.init()
        assert w.set_global_config(N.GlobalConfig(acceleration_z=-9.81, max_inner_iteration=40))
        assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-5,
                                                    contact_gs_form=form))
        r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(), V, F, P)
        r2, _ = w.add_obstacle(N.CollisionConfig(), SV, SF)
        assert r and r2
        contacts = []
        for _ in range(10):
            assert w.solver_step(), w
            contacts.append(w.step_stats().contacts)
        x = np.zeros(V.size, np.float32)
        assert w.get_cloth_position(h, x)
        out.append((x, contacts))
    print(f"contacts per step: {out[0][1]}")
    assert max(out[0][1]) > 0
    assert out[0][1] == out[1][1]
    np.testing.assert_array_equal(out[0][0], out[1][0])


# Cloth side, obstacle side, gap in paddings: one batch of contacts on one
# warp; several batches with a remainder; more than the block's shared memory
# holds corrections for (226 KB / 16 B = 14,464 positions and corrections).
@pytest.mark.parametrize("s,so,few,many", [(2, 2, 1, 31), (12, 9, 100, 2000),
                                           (78, 78, 14464, 1 << 20)])
def test_gs_single_block_sizes_identical(s, so, few, many):
    """A sheet within contact distance of a flat obstacle, two ADMM
    iterations: the single-block Gauss-Seidel (contacts ordered by their
    vertices' counts) and the grid form (ordered by colour barriers) move
    every vertex alike, bit for bit."""
    out = []
    for form in (0, 1):
        V, F = S.grid_sheet(s, side=0.5 * (s - 1) / 77, z=1.0, jitter=1e-6, seed=4)
        OV, OF = S.grid_sheet(so, side=0.52 * (s - 1) / 77, z=0.0)
        OV[:, 2] = V[:, 2].min() - 0.3 * 0.05 * 0.5 / 77
        w = N.World()
        assert w.init()
        assert w.set_global_config(N.GlobalConfig(acceleration_z=-9.81, max_inner_iteration=3,
                                                  max_outer_iteration=1))
        assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-5,
                                                    contact_gs_form=form))
        r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(is_self_collision_on=False), V, F,
                           [])
        r2, _ = w.add_obstacle(N.CollisionConfig(), OV, OF)
        assert r and r2
        r = w.solver_step()
        assert r, r.to_string()
        x = np.zeros(V.size, np.float32)
        assert w.get_cloth_position(h, x)
        out.append((x, w.step_stats().contacts))
    print(f"{s} x {s} over {so} x {so}: {out[0][1]} contacts")
    assert few <= out[0][1] <= many
    assert out[0][1] == out[1][1]
    np.testing.assert_array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("s", [60, 118])
def test_gs_form_chosen_is_the_faster(s):
    """Many contacts per colour (about 560 and 2,200): the form that is chosen
    takes no longer than the grid form (event times of one step, the better of
    three, 10 % for their spread), and both move every vertex alike."""
    out = []
    for form in (0, 1):
        V, F = S.grid_sheet(s, side=0.5 * (s - 1) / 77, z=1.0, jitter=1e-6, seed=4)
        OV, OF = S.grid_sheet(s, side=0.52 * (s - 1) / 77, z=0.0)
        OV[:, 2] = V[:, 2].min() - 0.3 * 0.05 * 0.5 / 77
        w = N.World()
        assert w.init()
        assert w.set_global_config(N.GlobalConfig(acceleration_z=-9.81, max_inner_iteration=8,
                                                  max_outer_iteration=1, admm_abs_tol=0.0,
                                                  admm_rel_tol=0.0))
        assert w.set_solver_options(N.SolverOptions(fixed_linear_rel_tol=1e-5, profile=1,
                                                    contact_gs_form=form))
        r, h = w.add_cloth(N.ClothConfig(), N.CollisionConfig(is_self_collision_on=False), V, F,
                           [])
        r2, _ = w.add_obstacle(N.CollisionConfig(), OV, OF)
        assert r and r2
        ms = []
        for _ in range(3):
            assert w.set_cloth_state(h, V)
            w.profile(reset=True)
            assert w.solver_step()
            ms.append(w.profile()["contact_gs_ms"])
        x = np.zeros(V.size, np.float32)
        assert w.get_cloth_position(h, x)
        out.append((x, min(ms), w.step_stats()))
    print(f"{s}: {out[0][2].contacts} contacts, {out[0][2].colors} colours, "
          f"{out[0][1]:.2f} ms, grid {out[1][1]:.2f} ms")
    assert out[0][2].contacts > 14464
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1] <= 1.1 * out[1][1]


# Pending-box stores of the deep searches: 96 per thread in the first pass,
# heaps in shared memory (up to about 7,200 boxes), sorted arrays in global
# memory above that; the smallest cap, around the first pass's size, and both
# sides of the shared-memory limit.
@pytest.mark.parametrize("max_iter", [1, 94, 95, 96, 300, 7000, 7400])
@pytest.mark.parametrize("vf", [True, False])
def test_ccd_deep_search_stores_match_oracle(oracle, vf, max_iter):
    """Near-contact queries (searches of up to max_iter evaluations): hit,
    time of impact and upper bound equal the CPU restatement's bit for bit,
    whichever store holds the pending boxes; the allocation-free batch gives
    the same answers within its limit of 4,096."""
    import torch
    rng = np.random.default_rng(77)
    x = CC.near_contact_queries(rng, 40, vf)
    ms = np.full(40, 1e-3, np.float32)
    err = [CC.ERR[vf]] * 3
    hit, toi, tup = N.ccd_batch(vf, x, err, ms, max_iter=max_iter)
    for i in range(40):
        h, t = oracle.ccd_toi(vf, x[i], err, float(ms[i]), max_iter=max_iter)[:2]
        assert bool(h) == bool(hit[i])
        if h:
            assert np.float32(t) == toi[i]
    if max_iter > 4096:
        return
    d = {k: torch.from_numpy(v).cuda() for k, v in (("x", x), ("ms", ms))}
    o = [torch.zeros(40, dtype=t, device="cuda") for t in (torch.int32, torch.float32,
                                                           torch.float32)]
    r, _ = N.ccd_batch_noalloc(vf, d["x"].data_ptr(), 40, np.asarray(err, np.float32),
                               d["ms"].data_ptr(), *(b.data_ptr() for b in o),
                               max_iter=max_iter)
    assert r, r.to_string()
    np.testing.assert_array_equal(o[0].cpu().numpy().astype(bool), hit)
    np.testing.assert_array_equal(o[1].cpu().numpy(), toi)
    np.testing.assert_array_equal(o[2].cpu().numpy(), tup)
