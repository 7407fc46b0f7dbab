"""What the performance of this framework is measured on.

A user steps cloth scenes (``native.World`` and ``native.step_many``), and
some call the standalone operators: the CCD batch, on host arrays or on
device buffers, and the warm-start model's training step.  A pass of a scene
case restarts the scene from its stored state, advances it by one step and
reads positions and velocities back, as a host that replays or rolls out a
scene does.
"""
from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

from silk_physics_b200 import learned, native, scenes

ROOT = Path(__file__).resolve().parents[1]
DT = 1.0 / 60.0
ADMM_ABS = 1e-5
ADMM_REL = 1e-3
CCD_ERR = {True: (4.053116e-06,) * 3, False: (3.814698e-06,) * 3}


def listed():
    return [
        # The smallest calls: a handkerchief of 144 vertices, default
        # (adaptive) tolerances, no collision; launches and host time count.
        dict(name="sheet12_pinned", kind="sheet", s=12, pins="corners", collide=False, inner=20,
             tol=0.0),
        # The small configuration: 32 x 32, two pinned corners,
        # self-collision, 10 solver iterations.
        dict(name="sheet32_config1", kind="sheet", s=32, pins="corners", collide=True, inner=10,
             tol=1e-5),
        # A 6K garment-sized sheet hung by one edge at the default settings,
        # as the packaged dense-sheet scene.
        dict(name="sheet79_hung", kind="sheet", s=79, pins="line", collide=True, inner=50,
             tol=0.0),
        # The largest sheet, free and without an obstacle.
        dict(name="sheet316_free", kind="sheet", s=316, pins="none", collide=True, inner=100,
             tol=1e-5),
        # An interactive scene: a small sheet landing on a ball, default
        # tolerances, 50 solver iterations (the packaged cloth-ball scene's).
        dict(name="land41_default", kind="drape", s=41, side=0.6, radius=0.2, inner=50, tol=0.0,
             bf16=False, learned=False),
        # The 80 x 80 benchmark scene while the sheet settles over the ball:
        # thousands of contacts, hundreds of solver iterations.
        dict(name="settle80", kind="settle", inner=100, tol=1e-5, bf16=False, learned=False),
        # A mid-sized sheet landing, with the learned warm start and BF16
        # preconditioner blocks.
        dict(name="land112_learned_bf16", kind="drape", s=112, side=1.1, radius=0.33, inner=100,
             tol=1e-5, bf16=True, learned=True),
        # The 100K-vertex drape at its first contact: over twenty rollbacks.
        dict(name="land316", kind="drape", s=316, side=2.0, radius=0.6, inner=100, tol=1e-5,
             bf16=False, learned=False),
        # Independent scenes of uneven sizes stepped together.
        dict(name="batch6", kind="batch", worlds=6, smin=24, smax=56, inner=100, tol=1e-5),
        # The CCD operator: many queries from host arrays (vertex-face) ...
        dict(name="ccd_vf_host", kind="ccd", n=200003, vf=True, device=False),
        # ... and a frame's worth on caller-owned device buffers (edge-edge).
        dict(name="ccd_ee_device", kind="ccd", n=12007, vf=False, device=True),
        # Loss and gradient of the warm-start model over a batch of samples.
        dict(name="mlp_grad", kind="mlp", n=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sheet", "sheet", "drape", "drape", "drape", "settle", "batch", "ccd",
                       "ccd", "mlp"])
    tol = rng.choice([0.0, 1e-5])
    if kind == "sheet":
        return dict(kind=kind, s=_log(rng, 8, 316), pins=rng.choice(["corners", "line", "none"]),
                    collide=rng.random() < 0.5, inner=rng.randint(6, 50), tol=tol)
    if kind == "drape":
        s = _log(rng, 20, 180)
        side = round(s / 80.0 * rng.uniform(0.7, 1.1), 4)
        form = rng.choice(["plain", "plain", "bf16", "learned"])
        return dict(kind=kind, s=s, side=side, radius=round(0.3 * side, 4),
                    inner=rng.randint(20, 100), tol=tol, bf16=form != "plain",
                    learned=form == "learned")
    if kind == "settle":
        form = rng.choice(["plain", "bf16", "learned"])
        return dict(kind=kind, inner=rng.randint(30, 100), tol=1e-5, bf16=form != "plain",
                    learned=form == "learned")
    if kind == "batch":
        lo = rng.randint(12, 32)
        return dict(kind=kind, worlds=rng.randint(2, 7), smin=lo, smax=lo + rng.randint(4, 28),
                    inner=rng.randint(20, 100), tol=tol)
    if kind == "ccd":
        device = rng.random() < 0.5
        return dict(kind=kind, n=_log(rng, 100, 20000 if device else 200000),
                    vf=rng.random() < 0.5, device=device)
    return dict(kind="mlp", n=_log(rng, 500, 65536))


# ---------------------------------------------------------------- inputs

def _sheet_inputs(case, seed):
    """A seeded sheet (spacing of the 80 x 80 sheet) in gentle motion: rest
    shape, faces, pins, positions and velocities."""
    s = case["s"]
    rng = np.random.default_rng(seed)
    side = (s - 1) / 79.0
    V, F = scenes.grid_sheet(s, side=side, z=1.0, jitter=1e-4, seed=seed)
    pins = {"corners": scenes.top_corner_pins(s), "none": np.zeros(0, np.int32),
            "line": np.arange((s - 1) * s, s * s, dtype=np.int32)}[case["pins"]]
    u, v = V[:, 0] / side, V[:, 1] / side
    wave = np.zeros(len(V))
    for k in range(1, 4):
        wave += rng.normal(0, 1.0 / k) * np.sin(2.0 * k * u + rng.uniform(0, 6.3)) * \
            np.cos(2.0 * k * v + rng.uniform(0, 6.3))
    vel = np.zeros_like(V)
    vel[:, 2] = 0.3 * side * wave - 0.2
    vel[:, 0] = 0.05 * side * wave
    vel[pins] = 0.0
    return V, F, pins, V.copy(), vel.astype(np.float32)


def _drape_inputs(s, side, radius, seed):
    """A sheet in free fall 0.1 m above a ball, one step before contact."""
    V, F = scenes.grid_sheet(s, side=side, z=radius + 0.1, jitter=1e-4, seed=seed)
    SV, SF = scenes.icosphere(4, radius=radius)
    x, v = scenes.free_fall_state(V, 8, dt=DT)
    return V, F, SV, SF, x, v


def _settle_inputs(seed):
    """The stored benchmark state (27 steps into the 80 x 80 scene), the whole
    scene turned about the vertical by a seeded angle."""
    V, F, SV, SF = scenes.c2_scene()
    with np.load(ROOT / "tests" / "golden" / "c2_contact.npz") as g:
        x, v = g["x0"].reshape(-1, 3), g["v0"].reshape(-1, 3)
    a = np.random.default_rng(seed).uniform(0, 2 * math.pi)
    R = np.array([[math.cos(a), -math.sin(a), 0], [math.sin(a), math.cos(a), 0], [0, 0, 1]])
    turn = lambda p: (np.asarray(p, np.float64) @ R.T).astype(np.float32)  # noqa: E731
    return turn(V), F, turn(SV), SF, turn(x), turn(v)


def _ok(r):
    if not r:
        raise RuntimeError(r.to_string())


def _world(case, V, F, pins, x, v, collide=True, sphere=None):
    w = native.World()
    _ok(w.init())
    _ok(w.set_global_config(native.GlobalConfig(
        acceleration_z=-9.81, dt=DT, max_inner_iteration=case["inner"], admm_abs_tol=ADMM_ABS,
        admm_rel_tol=ADMM_REL)))
    _ok(w.set_solver_options(native.SolverOptions(
        fixed_linear_rel_tol=case["tol"], mas_bf16=case.get("bf16", False),
        learned_warm_start=case.get("learned", False))))
    r, h = w.add_cloth(native.ClothConfig(), native.CollisionConfig(
        is_collision_on=collide, is_self_collision_on=collide), V, F, pins)
    _ok(r)
    if sphere is not None:
        r, _ = w.add_obstacle(native.CollisionConfig(), *sphere)
        _ok(r)
    if case.get("learned"):
        _ok(w.set_warm_start_model(learned.load(
            str(Path(native.__file__).resolve().parent / "models" / "warm_start.npy"))))
    _ok(w.set_cloth_state(h, x, v))
    return dict(w=w, h=h, x0=x, v0=v)


def _batch_sizes(case):
    n = case["worlds"]
    r = (case["smax"] / case["smin"]) ** (1.0 / max(n - 1, 1))
    return [int(round(case["smin"] * r ** k)) for k in range(n)]


def _ccd_inputs(case, seed):
    """Crossing motions of unit-scale primitives; one in 200 starts within two
    minimum separations of contact, whose search is a deep one, about as rare
    as in a frame's candidates."""
    n, vf = case["n"], case["vf"]
    rng = np.random.default_rng(seed)
    base = rng.uniform(-1, 1, (n, 4, 3)).astype(np.float32)
    if vf:
        base[:, 1:, 2] = 0.0
        base[:, 0, 2] = rng.uniform(0.001, 0.2, n)
    motion = rng.normal(0, 0.4, (n, 4, 3)).astype(np.float32)
    motion[:, 0, 2] -= rng.uniform(0, 0.6, n)
    near = rng.random(n) < 0.005
    m = int(near.sum())
    if vf:
        base[near, 0, :2] = rng.uniform(-0.2, 0.2, (m, 2))
        base[near, 0, 2] = rng.uniform(0, 2e-3, m)
        base[near, 1:] = [(-1, -1, 0), (1, -1, 0), (0, 1, 0)]
    else:
        base[near, :2] = [(-1, 0, 0), (1, 0, 0)]
        base[near, 2, :2] = (0, -1)
        base[near, 3, :2] = (0, 1)
        base[near, 2:, 2] = rng.uniform(0, 2e-3, m)[:, None]
    motion[near] = rng.normal(0, 0.05, (m, 4, 3))
    motion[near, 0, 2] -= rng.uniform(0, 0.2, m)
    x = np.concatenate([base, base + motion], axis=1).reshape(n, 24).astype(np.float32)
    ms = np.where(near, 1e-3, rng.choice([0.0, 1e-4, 1e-3], n)).astype(np.float32)
    return x, ms


def _mlp_inputs(case, seed):
    n = case["n"]
    rng = np.random.default_rng(seed)
    f = np.zeros((n, learned.K_IN), np.float32)
    f[:, :learned.N_IN] = rng.normal(0, 1.5, (n, learned.N_IN))
    f[:, 12] = rng.random(n) < 0.02
    t = np.zeros((n, 4), np.float32)
    t[:, :3] = 0.5 * np.tanh(f[:, :3]) + 0.1 * rng.normal(0, 1, (n, 3))
    mean = np.zeros(learned.K_IN)
    std = np.ones(learned.K_IN)
    std[:learned.N_IN] = 1.5
    p = learned.initial_params(mean, std, np.full(learned.K_OUT, 0.5), seed=seed)
    return p, f, t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sheet":
        V, F, pins, x, v = _sheet_inputs(case, seed)
        return dict(kind=kind, scenes=[_world(case, V, F, pins, x, v, collide=case["collide"])])
    if kind == "drape":
        V, F, SV, SF, x, v = _drape_inputs(case["s"], case["side"], case["radius"], seed)
        return dict(kind=kind, scenes=[_world(case, V, F, [], x, v, sphere=(SV, SF))])
    if kind == "settle":
        V, F, SV, SF, x, v = _settle_inputs(seed)
        return dict(kind=kind, scenes=[_world(case, V, F, [], x, v, sphere=(SV, SF))])
    if kind == "batch":
        got = []
        for k, s in enumerate(_batch_sizes(case)):
            side = s / 80.0
            V, F, SV, SF, x, v = _drape_inputs(s, side, 0.3 * side, seed * 64 + k)
            got.append(_world(case, V, F, [], x, v, sphere=(SV, SF)))
        return dict(kind=kind, scenes=got)
    if kind == "ccd":
        x, ms = _ccd_inputs(case, seed)
        st = dict(kind=kind, vf=case["vf"], err=np.asarray(CCD_ERR[case["vf"]], np.float32))
        if not case["device"]:
            return dict(st, x=x, ms=ms)
        n = case["n"]
        return dict(st, x=torch.from_numpy(x).cuda(), ms=torch.from_numpy(ms).cuda(),
                    hit=torch.zeros(n, dtype=torch.int32, device="cuda"),
                    toi=torch.zeros(n, device="cuda"), tup=torch.zeros(n, device="cuda"))
    p, f, t = _mlp_inputs(case, seed)
    return dict(kind=kind, p=p, f=f, t=t)


# ---------------------------------------------------------------- a pass

def run(state):
    kind = state["kind"]
    if kind == "ccd":
        if isinstance(state["x"], np.ndarray):
            hit, toi, tup = native.ccd_batch(state["vf"], state["x"], state["err"], state["ms"])
            return dict(hit=hit, toi=toi, tup=tup)
        x, ms, hit, toi, tup = (state[k] for k in ("x", "ms", "hit", "toi", "tup"))
        r, _ = native.ccd_batch_noalloc(state["vf"], x.data_ptr(), ms.numel(), state["err"],
                                        ms.data_ptr(), hit.data_ptr(), toi.data_ptr(),
                                        tup.data_ptr(),
                                        stream=torch.cuda.current_stream().cuda_stream)
        _ok(r)
        return dict(hit=hit, toi=toi, tup=tup)
    if kind == "mlp":
        loss, grad = native.mlp_loss_grad(state["p"], state["f"], state["t"])
        return dict(loss=loss, grad=grad)
    for s in state["scenes"]:
        _ok(s["w"].set_cloth_state(s["h"], s["x0"], s["v0"]))
    if kind == "batch":
        for r in native.step_many([s["w"] for s in state["scenes"]]):
            _ok(r)
    else:
        _ok(state["scenes"][0]["w"].solver_step())
    out = {}
    for k, s in enumerate(state["scenes"]):
        x = np.empty(s["x0"].shape, np.float32)
        v = np.empty(s["x0"].shape, np.float32)
        _ok(s["w"].get_cloth_position(s["h"], x))
        _ok(s["w"].get_cloth_velocity(s["h"], v))
        out["x%d" % k], out["v%d" % k] = x, v
    return out


# ---------------------------------------------------------------- what it is held to

def _sizes(case):
    if case["kind"] == "settle":
        return [80]
    return _batch_sizes(case) if case["kind"] == "batch" else [case["s"]]


def work(case):
    """Steps: the state in and out and the scene's static data once (28 B per
    face, 7 doubles and the masses per vertex's share of the matrix), and the
    arithmetic of one solver iteration.  CCD: 24 floats and a separation in,
    three words out; at least one box evaluation per query."""
    if case["kind"] == "ccd":
        return dict(bytes=112.0 * case["n"], flops=250.0 * case["n"])
    if case["kind"] == "mlp":
        k = learned.K_IN * 64 + 2 * 64 * 64 + 64 * learned.K_OUT
        return dict(bytes=80.0 * case["n"] + 8.0 * learned.N_PARAMS, flops=6.0 * k * case["n"])
    nv = float(sum(s * s for s in _sizes(case)))
    nf = float(sum(2 * (s - 1) ** 2 for s in _sizes(case)))
    return dict(bytes=(48 + 8 * 19 + 24) * nv + 44.0 * nf, flops=(2 * 3 * 19 + 150) * nv + 250 * nf)


def tolerance(case):
    """Scenes are compared in positions and velocities; the velocities differ
    most.  Measured over these ranges between the solver's forms (which add in
    other orders) and with the linear systems solved to 1e-6 and 1e-7 instead:
    the largest relative difference of velocities was 1.4e-2 for sheets at the
    adaptive tolerance and 2e-3 at 1e-5, 6e-4 for the settled scene, and up to
    1.9e-2 for landing sheets, where a rollback lands elsewhere; single values
    7e-2, 1.5e-2, 4e-3 and 9e-2.  About four times that is allowed."""
    kind = case["kind"]
    if kind == "ccd":
        return "exact"
    if kind == "mlp":
        return dict(rel=4e-3, max=0.1)
    if kind == "sheet":
        return dict(rel=0.03, max=0.3) if case["tol"] == 0.0 else dict(rel=8e-3, max=0.06)
    if kind == "settle":
        return dict(rel=2.5e-3, max=2e-2)
    return dict(rel=0.03, max=0.4)


# ---------------------------------------------------------------- the same in 64 bits

def _assemble(V, F, cfg, dev):
    """Sparse matrix of the elastic and bending terms (COO), masses, bending
    right-hand side and the faces' chart rows."""
    V = torch.as_tensor(V, dtype=torch.float64, device=dev)
    F = torch.as_tensor(F, dtype=torch.int64, device=dev)
    n = len(V)
    p = V[F]
    e0, e1 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    nrm = torch.linalg.cross(e0, e1)
    area = 0.5 * nrm.norm(dim=1)
    l2 = torch.stack([(p[:, (i + 2) % 3] - p[:, (i + 1) % 3]).square().sum(1) for i in range(3)], 1)
    num = l2.sum(1, keepdim=True) - 2 * l2
    cot = num / (4 * area[:, None])
    obtuse = (num < 0)
    vor = torch.zeros(n, dtype=torch.float64, device=dev)
    for i in range(3):
        j, k = (i + 1) % 3, (i + 2) % 3
        m = torch.where(obtuse.any(1), torch.where(obtuse[:, i], 0.5 * area, 0.25 * area),
                        0.125 * (l2[:, k] * cot[:, k] + l2[:, j] * cot[:, j]))
        vor.index_add_(0, F[:, i], m)
    bx = e0 / e0.norm(dim=1, keepdim=True)
    by = torch.linalg.cross(nrm, e0)
    by = by / by.norm(dim=1, keepdim=True)
    a, b, c = (bx * e0).sum(1), (bx * e1).sum(1), (by * e1).sum(1)
    z = torch.zeros_like(a)
    B = torch.stack([torch.stack([-1 / a, 1 / a, z], 1),
                     torch.stack([b / (a * c) - 1 / c, -b / (a * c), 1 / c], 1)], 1)
    el = cfg.elastic_stiffness * area[:, None, None] * (B.transpose(1, 2) @ B)
    ii = F[:, :, None].expand(-1, 3, 3).reshape(-1)
    jj = F[:, None, :].expand(-1, 3, 3).reshape(-1)
    cr, cc, cv = [], [], []
    for i in range(3):
        u, v, w = F[:, (i + 1) % 3], F[:, (i + 2) % 3], 0.5 * cot[:, i]
        cr += [u, v, u, v]
        cc += [v, u, u, v]
        cv += [w, w, -w, -w]
    C = torch.sparse_coo_tensor(torch.stack([torch.cat(cr), torch.cat(cc)]), torch.cat(cv),
                                (n, n)).coalesce()
    ci = C.indices()
    MC = torch.sparse_coo_tensor(ci, C.values() / vor[ci[0]], (n, n)).coalesce()
    bend = torch.sparse.mm(C, MC) * cfg.bending_stiffness
    A = (torch.sparse_coo_tensor(torch.stack([ii, jj]), el.reshape(-1), (n, n)) + bend).coalesce()
    return A, cfg.density * vor, torch.sparse.mm(bend, V), B, F, area


def _clamp_projection(y):
    """Singular values of the 3 x 2 matrices (columns y[:, 0], y[:, 1])
    clamped to [0.9, 1.1]."""
    g11, g22, g12 = y[:, 0].square().sum(1), y[:, 1].square().sum(1), (y[:, 0] * y[:, 1]).sum(1)
    th = 0.5 * torch.atan2(2 * g12, g11 - g22)
    c, s = torch.cos(th)[:, None], torch.sin(th)[:, None]
    u1, u2 = y[:, 0] * c + y[:, 1] * s, y[:, 1] * c - y[:, 0] * s
    s1, s2 = u1.norm(dim=1, keepdim=True), u2.norm(dim=1, keepdim=True)
    u1, u2 = u1 / s1 * s1.clamp(0.9, 1.1), u2 / s2 * s2.clamp(0.9, 1.1)
    return torch.stack([u1 * c - u2 * s, u1 * s + u2 * c], 1)


def _solver(A, d):
    """x -> (A + diag(d))^-1 x: a dense factorisation, or for large systems
    conjugate gradients to 1e-13."""
    n = len(d)
    if n <= 8000:
        L = torch.linalg.cholesky(A.to_dense() + torch.diag(d))
        return lambda b, x: torch.cholesky_solve(b, L)
    i = A.indices()
    ad = torch.zeros_like(d)
    on = i[0] == i[1]
    ad[i[0][on]] = A.values()[on]
    inv = (1.0 / (ad + d))[:, None]
    M = A.to_sparse_csr()

    def cg(b, x):
        r = b - (M @ x + d[:, None] * x)
        z = inv * r
        p, rz = z.clone(), (r * z).sum()
        stop = 1e-26 * float((b * inv * b).sum())
        for k in range(4000):
            Ap = M @ p + d[:, None] * p
            al = rz / (p * Ap).sum()
            x = x + al * p
            r = r - al * Ap
            z = inv * r
            new = (r * z).sum()
            if k % 16 == 15 and float(new) <= stop:
                break
            p, rz = z + (new / rz) * p, new
        return x
    return cg


def _exact_step(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    V, F, pins, x0, v0 = _sheet_inputs(case, seed)
    cfg = native.ClothConfig()
    A, mass, bend_rhs, B, F, area = _assemble(V, F, cfg, dev)
    x0, v0 = (torch.as_tensor(q, dtype=torch.float64, device=dev) for q in (x0, v0))
    target = torch.as_tensor(V, dtype=torch.float64, device=dev)
    pin = torch.zeros(len(V), dtype=torch.float64, device=dev)
    pin[torch.as_tensor(pins, dtype=torch.int64, device=dev)] = 1.0
    pin = pin[:, None]
    acc = torch.tensor([0.0, 0.0, -9.81], dtype=torch.float64, device=dev)
    dt, rho, kp = DT, cfg.elastic_stiffness, 1e4
    vd = (1.0 - cfg.damping) * v0
    x = x0 + dt * vd + dt * dt * acc
    inertia = -x0 / dt ** 2 - vd / dt - acc
    w = area.sqrt()[:, None, None]
    nf, n = len(F), len(V)
    z = torch.zeros(nf, 2, 3, dtype=torch.float64, device=dev)
    u, lam = torch.zeros_like(z), torch.zeros_like(x)
    solve = _solver(A, mass / dt ** 2 + kp * pin[:, 0])
    gather = lambda q: torch.zeros_like(x).index_add_(  # noqa: E731
        0, F.reshape(-1), (B.transpose(1, 2) @ q).reshape(-1, 3))
    rhs = None
    for it in range(case["inner"]):
        if it:
            x = solve(rhs, x)
        S = B @ x[F]
        y = S + u / (rho * w)
        zo, z = z, 0.5 * y + 0.5 * _clamp_projection(y)
        u = (u + w * rho * (S - z)).clamp(-1e8, 1e8)
        lam = pin * (lam + kp * (x - target)).clamp(-1e8, 1e8)
        fz = rho * w * w
        gz = gather(fz * z)
        rhs = bend_rhs - mass[:, None] * inertia + pin * (kp * target - lam) + gz - gather(w * u)
        primal = math.sqrt(float((w * (S - z)).square().sum() + (pin * (x - target)).square().sum()))
        px = math.sqrt(float((w * S).square().sum() + (pin * x).square().sum()))
        pa = math.sqrt(float((w * z).square().sum() + (pin * target).square().sum()))
        gzo = gather(fz * zo)
        dual, dc, dp = (float(q.norm()) for q in (gz - gzo, gz, gzo))
        dof = 6 * nf + 3 * len(pins)
        if it and primal <= math.sqrt(dof) * ADMM_ABS + max(px, pa) * ADMM_REL and \
                dual <= math.sqrt(3 * n) * ADMM_ABS + max(dc, dp) * ADMM_REL:
            break
    x = torch.where(pin > 0, target, x)
    return dict(x0=x.cpu().numpy(), v0=((x - x0) / dt).cpu().numpy())


def _exact_mlp(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    p, f, t = _mlp_inputs(case, seed)
    q = torch.tensor(p, dtype=torch.float64, device=dev, requires_grad=True)
    part = {}
    for name, (o, shape) in learned.OFFSETS.items():
        part[name] = q[o:o + int(np.prod(shape))].reshape(shape)
    h = (torch.as_tensor(f, dtype=torch.float64, device=dev) - part["feat_mean"].detach()) / \
        part["feat_std"].detach()
    for i in (1, 2, 3):
        h = torch.nn.functional.gelu(h @ part["W%d" % i] + part["b%d" % i])
    y = (h @ part["W4"] + part["b4"])[:, :3]
    want = torch.as_tensor(t[:, :3], dtype=torch.float64, device=dev)
    loss = (y - want).square().mean()
    loss.backward()
    return dict(loss=float(loss.detach()), grad=q.grad.cpu().numpy())


def exact(case, seed):
    """Sheets without contact and the model's gradient.  Contact steps have no
    plain restatement that ends within seconds, and the CCD's answers are its
    own conservative intervals."""
    if case["kind"] == "sheet":
        return _exact_step(case, seed)
    if case["kind"] == "mlp":
        return _exact_mlp(case, seed)
    return None
