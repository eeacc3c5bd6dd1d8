"""The work a user of this framework has it do, as cases that can be measured.

Kinds (each through the entry points a program calls):

  step3d   the drop-in substep ``solve_mls_mpm_3d`` on CUDA tensors, called in a loop
  step2d   its 2D counterpart ``solve_mls_mpm_2d`` (elastic or snow)
  phases3d the reference's own three calls, ``three_d.p2g`` / ``grid_op`` / ``g2p``, on the caller's grid
  host3d   ``solve_mls_mpm_3d`` on pinned host arrays (what a CPU program that owns its arrays calls)
  solver   the resident ``MPMSolver`` replaying a captured graph, then reading the state (one frame)
  batch2d  many independent 2D scenes per launch (``Batch2D``)
  rollout  a differentiable rollout, forward and backward (``diff.simulate``)
  coarse   one corrected coarse step (``learned.Stepper.coarse_step`` with a ``Corrector``)
  train    one training step of the corrector network (``learned.Net``)

The states are those of a run that is under way: two bodies in motion with strain and velocity
gradients, not the rest state a scene starts from.  The single-substep kinds start every pass from
the same state (a program that reruns a scene), the resident ones go on from where they are (a
program that runs on).  The resident scenes use the textbook fixed-corotated stress, which stays
bounded however long a run goes on; the drop-in calls use the reference's model.
"""
import math

import numpy as np
import torch

from femflow_gb300 import batched, diff, learned
from femflow_gb300.solver import MPMSolver
from femflow_gb300.solvers.mpm import mls_mpm, three_d, two_d
from femflow_gb300.solvers.mpm.particle import ParticleSet

DEV = "cuda"
DTYPES = {"f32": torch.float32, "f64": torch.float64}
NU = 0.3


def listed():
    return [
        # the smallest call: a few thousand particles, one substep per call, latency and launches only
        dict(name="step3d_2k", kind="step3d", n=2048, res=32, dtype="f32", substeps=8),
        # the plain 2D block drop in the reference's own precision (8,192 particles on 128^2)
        dict(name="step2d_8k_f64", kind="step2d", n=8192, res=128, dtype="f64", model="neo_hookean", substeps=8),
        # the 2D snow model of two_d/g2p.py, an odd particle count
        dict(name="step2d_snow_65k", kind="step2d", n=65001, res=192, dtype="f32", model="snow", substeps=8),
        # a program that drives the three phases itself, a ragged count on a grid that is no power of two
        dict(name="phases3d_200k", kind="phases3d", n=199_999, res=96, dtype="f32", substeps=2),
        # the benchmark's end-to-end call: host arrays in, host arrays out
        dict(name="host3d_1M", kind="host3d", n=1_048_576, res=128, dtype="f32"),
        # a small scene played in real time from a graph
        dict(name="solver3d_16k", kind="solver", dim=3, n=16384, res=64, dtype="f32", substeps=40, deterministic=False),
        # the benchmark's resident run: 1M particles, 40-substep graphs
        dict(name="solver3d_1M", kind="solver", dim=3, n=1_048_576, res=128, dtype="f32", substeps=40,
             deterministic=False),
        # the bit-reproducible mode
        dict(name="solver3d_det_300k", kind="solver", dim=3, n=300_000, res=96, dtype="f32", substeps=20,
             deterministic=True),
        # the batched workload: 256 scenes of 2k to 64k particles
        dict(name="batch2d_256", kind="batch2d", scenes=256, n_lo=2048, n_hi=65536, dtype="f32", substeps=10),
        # the differentiable workload (131,072 particles on 64^3), a shorter rollout
        dict(name="rollout3d_131k", kind="rollout", dim=3, n=131_072, res=64, dtype="f32", substeps=20, checkpoint=10),
        # one corrected coarse step of the learned form at full size
        dict(name="coarse_1M", kind="coarse", n=1_048_576, res=128),
        # one Adam step of the corrector network at the batch its training uses
        dict(name="train_32k", kind="train", batch=32768),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step3d", "step2d", "phases3d", "host3d", "solver", "batch2d", "rollout", "coarse", "train"])
    if kind in ("step3d", "phases3d"):
        n = _log_int(rng, 1500, 500_000)
        return dict(kind=kind, n=n, res=_res3(rng, n), dtype="f64" if rng.random() < 0.2 and n < 100_000 else "f32",
                    substeps=rng.choice([2, 4, 8]))
    if kind == "step2d":
        n = _log_int(rng, 1500, 300_000)
        return dict(kind=kind, n=n, res=rng.randint(64, 256), dtype=rng.choice(["f32", "f64"]),
                    model=rng.choice(["neo_hookean", "neo_hookean", "snow"]), substeps=rng.choice([2, 4, 8]))
    if kind == "host3d":
        n = _log_int(rng, 262_144, 1_048_576)
        return dict(kind=kind, n=n, res=rng.choice([96, 112, 128]), dtype="f32")
    if kind == "solver":
        dim = rng.choice([3, 3, 2])
        n = _log_int(rng, 4000, 1_048_576 if dim == 3 else 300_000)
        return dict(kind=kind, dim=dim, n=n, res=_res3(rng, n) if dim == 3 else rng.randint(64, 256), dtype="f32",
                    substeps=rng.choice([8, 16, 40]), deterministic=dim == 3 and rng.random() < 0.25)
    if kind == "batch2d":
        hi = _log_int(rng, 8000, 65536)
        return dict(kind=kind, scenes=_log_int(rng, 8, 256), n_lo=2048, n_hi=hi, dtype="f32",
                    substeps=rng.choice([4, 10, 20]))
    if kind == "rollout":
        dim = rng.choice([3, 3, 2])
        n = _log_int(rng, 2000, 131_072)
        return dict(kind=kind, dim=dim, n=n, res=rng.choice([32, 48, 64]) if dim == 3 else rng.randint(48, 128),
                    dtype="f32", substeps=rng.choice([4, 8, 12]), checkpoint=rng.choice([4, 6]))
    if kind == "coarse":
        n = 2 * _log_int(rng, 8192, 500_000)
        return dict(kind=kind, n=n, res=rng.choice([64, 96, 128]))
    return dict(kind="train", batch=128 * rng.randint(8, 512))


def _res3(rng, n):
    """A 3D grid on which n particles fill the bodies at 2 to 40 particles per cell."""
    ok = [r for r in (32, 40, 48, 64, 80, 96, 128) if 2.0 <= n / (2 * (0.2 * r) ** 3) <= 40.0]
    return rng.choice(ok or [32])


# ------------------------------------------------------------------------------------------ scenes
def _lame(E, nu):
    return E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))


def _cfl_dt(res, E=4.5e3, cfl=0.5):
    """The time step at which the elastic wave of a unit-density body crosses half a cell (5e-5 at 128)."""
    c = math.sqrt(E * (1 - NU) / ((1 + NU) * (1 - 2 * NU)))
    return float("%.3g" % (cfl / (c * res)))


def _bodies(n, dim, seed, dtype, strain=0.01, spin=1.0, speed=1.0, edge=0.2):
    """Two cubes (squares) of edge `edge` moving toward each other, under way: x, v, F, C on the GPU."""
    g = torch.Generator(device=DEV).manual_seed(1_000_003 * seed + 17)
    f64 = dict(dtype=torch.float64, device=DEV)
    half = n // 2
    x = (torch.rand((n, dim), generator=g, **f64) - 0.5) * edge + 0.5
    side = torch.ones(n, **f64)
    side[:half] = -1.0
    x[:, 0] += 0.15 * side
    v = 0.05 * torch.randn((n, dim), generator=g, **f64)
    v[:, 0] -= speed * side
    F = torch.eye(dim, **f64) + strain * torch.randn((n, dim, dim), generator=g, **f64)
    C = spin * torch.randn((n, dim, dim), generator=g, **f64)
    return tuple(t.to(dtype).contiguous() for t in (x, v, F, C))


def _volume(n, dim, edge=0.2):
    return 2 * edge ** dim / n


def _material(n, dtype, vol, E=4.5e3):
    """Per-particle mass, mu and lambda: two bodies of one density and two stiffnesses."""
    mu, lam = _lame(E, NU)
    k = torch.ones(n, dtype=torch.float64, device=DEV)
    k[: n // 2] = 0.5
    return tuple((t * torch.ones_like(k)).to(dtype) for t in (vol, mu * k, lam * k))


# ------------------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, seed)
    s["case"] = case
    return s


def _prepare_step3d(c, seed):
    dt = DTYPES[c["dtype"]]
    vol = _volume(c["n"], 3)
    first = _bodies(c["n"], 3, seed, dt)
    m, mu, lam = _material(c["n"], dt, vol)
    now = [t.clone() for t in first]
    return dict(first=first, now=now, parts=ParticleSet(now[0], m, mu, lam), vol=vol, dt=_cfl_dt(c["res"]),
                Jp=torch.ones((c["n"], 1), dtype=dt, device=DEV))


def _prepare_phases3d(c, seed):
    s = _prepare_step3d(c, seed)
    R = c["res"] + 1
    s["gv"] = torch.zeros((R, R, R, 3), dtype=DTYPES[c["dtype"]], device=DEV)
    s["gm"] = torch.zeros((R, R, R, 1), dtype=DTYPES[c["dtype"]], device=DEV)
    return s


def _prepare_step2d(c, seed):
    dt = DTYPES[c["dtype"]]
    vol = _volume(c["n"], 2)
    # snow: most of the strain lies outside the range its singular values are clamped to
    first = _bodies(c["n"], 2, seed, dt)
    g = torch.Generator(device=DEV).manual_seed(seed + 5)
    Jp = (1 + 0.02 * torch.randn((c["n"], 1), generator=g, dtype=torch.float64, device=DEV)).to(dt)
    mu, lam = _lame(1e3, 0.2)
    return dict(first=first + (Jp,), now=[t.clone() for t in first + (Jp,)], vol=vol, mu=mu, lam=lam,
                hardening=10.0 if c["model"] == "snow" else 1.0, dt=_cfl_dt(c["res"], 4e3))


def _prepare_host3d(c, seed):
    dt = DTYPES[c["dtype"]]
    vol = _volume(c["n"], 3)
    pin = lambda t: t.cpu().pin_memory()
    x, v, F, C = (pin(t) for t in _bodies(c["n"], 3, seed, dt, strain=1e-3, spin=0.1))
    m, mu, lam = (pin(t) for t in _material(c["n"], dt, vol))
    return dict(parts=ParticleSet(x, m, mu, lam), now=[x, v, F, C], vol=vol, dt=_cfl_dt(c["res"]),
                Jp=pin(torch.ones((c["n"], 1), dtype=dt)))


def _prepare_solver(c, seed):
    dim, dt = c["dim"], DTYPES[c["dtype"]]
    x, v, F, C = _bodies(c["n"], dim, seed, dt, strain=1e-3, spin=0.1, speed=0.5)
    vol = _volume(c["n"], dim)
    mu, lam = _lame(4.5e3, NU)
    s = MPMSolver(x, res=c["res"], dt=_cfl_dt(c["res"]), gravity=-1.0, volume=vol, mass=vol, mu_0=mu, lambda_0=lam,
                  v=v, F=F, C=C, dtype=dt, model="fixed_corotated", deterministic=c["deterministic"])
    s.capture(c["substeps"])
    return dict(solver=s)


def _scenes(c, seed):
    """Scenes as batched.random_scenes draws them; their counts and grids belong to the case, the
    positions, velocities and materials to the seed."""
    size = np.random.default_rng(c["scenes"])
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(c["scenes"]):
        n = int(round(math.exp(size.uniform(math.log(c["n_lo"]), math.log(c["n_hi"])))))
        res = int(size.integers(64, 257))
        E, nu = math.exp(rng.uniform(math.log(1e3), math.log(1e5))), rng.uniform(0.1, 0.4)
        x = rng.uniform(0.1, 0.7, size=2) + rng.uniform(0, 0.2, size=(n, 2))
        v = rng.normal(0, 0.05, size=(n, 2)) + rng.uniform(-0.5, 0.5, size=2)
        mu, lam = _lame(E, nu)
        out.append(dict(x=x, v=v, res=res, dt=1e-4, mass=0.04 / n, volume=0.04 / n, mu_0=mu, lambda_0=lam, E=E, nu=nu,
                        model="fixed_corotated"))
    return batched.stable_variant(out)


def _prepare_batch2d(c, seed):
    b = batched.Batch2D(_scenes(c, seed), dtype=DTYPES[c["dtype"]])
    b.capture(c["substeps"])
    return dict(batch=b)


def _rollout_scene(c, seed):
    n, dim = c["n"], c["dim"]
    g = torch.Generator(device=DEV).manual_seed(seed + 23)
    x = torch.rand((n, dim), generator=g, dtype=torch.float64, device=DEV) * 0.25 + 0.375
    v = 0.1 * torch.randn((n, dim), generator=g, dtype=torch.float64, device=DEV)
    F = torch.eye(dim, dtype=torch.float64, device=DEV) + 0.01 * torch.randn((n, dim, dim), generator=g,
                                                                         dtype=torch.float64, device=DEV)
    mu, lam = _lame(4e3, NU)
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    dt = DTYPES[c["dtype"]]
    return tuple(t.to(dt) for t in (x, v, F, mu * one, lam * one)), 0.25 ** dim / n


def _target(dim, like):
    return torch.tensor([0.7, 0.3, 0.5][:dim], dtype=like.dtype, device=like.device)


def _prepare_rollout(c, seed):
    (x, v, F, mu, lam), vol = _rollout_scene(c, seed)
    cfg = diff.RolloutConfig(res=c["res"], dt=_cfl_dt(c["res"], 4e3), steps=c["substeps"], volume=vol,
                             checkpoint_every=c["checkpoint"], model="fixed_corotated")
    return dict(inputs=(x, v, F, mu, lam), cfg=cfg, vol=vol, target=_target(c["dim"], x))


def _coarse_state(c, seed):
    x, v, F, C = _bodies(c["n"], 3, seed, torch.float32)
    return diff.pack(x, v, F, C)


def _net(batch, seed):
    """A network as it is in the middle of a training: its scales fitted, its outputs of the size of its targets."""
    net = learned.Net(max_batch=batch, seed=seed)
    g = torch.Generator(device=DEV).manual_seed(seed + 31)
    net.params[40960:41152] = 0.1 * torch.randn(192, generator=g, device=DEV)
    net.repack()
    return net


def _prepare_coarse(c, seed):
    st = learned.Stepper(learned.SceneSpec(n_per_cube=c["n"] // 2, seed=seed), res=c["res"])
    net = _net(128, seed)
    net.in_scale.copy_(_coarse_in_scale())
    net.out_scale.fill_(1e-3)
    first = _coarse_state(c, seed)
    return dict(st=st, cor=learned.Corrector(net, st, 0.5), first=first, now=first.clone())


def _coarse_in_scale():
    s = torch.full((128,), 10.0, device=DEV)
    s[113:] = 0.0
    return s


def _train_data(c, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 41)
    X = torch.randn((c["batch"], 128), generator=g, device=DEV)
    X[:, 113:] = 0.0
    X = X.to(torch.bfloat16)
    M = 0.2 * torch.randn((113, 12), generator=g, device=DEV)
    T = torch.tanh(X[:, :113].float() @ M) + 0.3 * torch.randn((c["batch"], 12), generator=g, device=DEV)
    return X, T.contiguous()


def _prepare_train(c, seed):
    X, T = _train_data(c, seed)
    return dict(net=_net(c["batch"], seed), X=X, T=T, w=torch.ones(12, device=DEV),
                loss=torch.zeros(1, dtype=torch.float64, device=DEV))


# ---------------------------------------------------------------------------------------------- run
def run(s):
    return globals()["_run_" + s["case"]["kind"]](s)


def _restart(s):
    for a, b in zip(s["now"], s["first"]):
        a.copy_(b)


def _run_step3d(s):
    c, res = s["case"], s["case"]["res"]
    _restart(s)
    _, v, F, C = s["now"]
    for _ in range(c["substeps"]):
        mls_mpm.solve_mls_mpm_3d(res, float(res), 1.0, 1 / res, s["dt"], s["vol"], -9.8, s["parts"], v, F, C, s["Jp"])
    return dict(zip("xvFC", s["now"]))


def _run_step2d(s):
    c, res = s["case"], s["case"]["res"]
    _restart(s)
    x, v, F, C, Jp = s["now"]
    for _ in range(c["substeps"]):
        two_d.solve_mls_mpm_2d(res, float(res), s["hardening"], s["mu"], s["lam"], s["vol"], 1 / res, s["dt"],
                               s["vol"], -9.8, x, v, F, C, Jp, model=c["model"])
    return dict(x=x, v=v, F=F, C=C, Jp=Jp)


def _run_phases3d(s):
    c, res = s["case"], s["case"]["res"]
    _restart(s)
    _, v, F, C = s["now"]
    gv, gm, P, Jp, dx = s["gv"], s["gm"], s["parts"], s["Jp"], 1 / res
    for _ in range(c["substeps"]):
        gv.zero_()
        gm.zero_()
        three_d.p2g(float(res), 1.0, dx, s["dt"], s["vol"], gv, gm, P, v, F, C, Jp)
        three_d.grid_op(res, dx, s["dt"], -9.8, gv, gm)
        three_d.g2p(float(res), s["dt"], gv, P, v, F, C, Jp)
    return dict(zip("xvFC", s["now"]), grid_velocity=gv, grid_mass=gm)


def _run_host3d(s):
    res = s["case"]["res"]
    x, v, F, C = s["now"]
    mls_mpm.solve_mls_mpm_3d(res, float(res), 1.0, 1 / res, s["dt"], s["vol"], 0.0, s["parts"], v, F, C, s["Jp"])
    return dict(x=x, v=v, F=F, C=C)


def _run_solver(s):
    s["solver"].step(s["case"]["substeps"])
    return s["solver"].state()


def _run_batch2d(s):
    b = s["batch"]
    b.step(s["case"]["substeps"])
    return dict(x=b.x, v=b.v, F=b.F, C=b.C, Jp=b.Jp)


def _run_rollout(s):
    x, v, F, mu, lam = (t.detach().requires_grad_(True) for t in s["inputs"])
    xe, ve, Fe, _ = diff.simulate(x, v, mu, lam, s["cfg"], s["vol"], F0=F)
    loss = ((xe - s["target"]) ** 2).sum(1).mean()
    loss.backward()
    return dict(x=xe.detach(), v=ve.detach(), F=Fe.detach(), gx=x.grad, gv=v.grad, gF=F.grad, gmu=mu.grad, glam=lam.grad)


def _run_coarse(s):
    s["now"].copy_(s["first"])
    s["st"].coarse_step(s["now"], s["cor"])
    return s["now"]


def _run_train(s):
    net = s["net"]
    s["loss"].zero_()
    Y = net.forward_train(s["X"])
    net.backward_train(s["T"], s["w"], s["loss"])
    net.update(1e-3)
    return dict(Y=Y, loss=s["loss"], grads=net.grads, params=net.params)


# --------------------------------------------------------------------------------------------- work
def work(c):
    """Bytes: state and parameters read once and state written once per substep (per call for the
    kinds that hand the state over), float64 twice.  Operations: the weights, the stress, the 3^d
    scatter and gather and the F update, as multiply-adds counted twice."""
    k = c["kind"]
    if k == "train":
        B = c["batch"]
        macs = 113 * 64 + 64 * 64 * 2 + 64 * 12
        return dict(bytes=B * (256 + 48 + 48) + 41168 * 4 * 7, flops=2 * B * macs * 3 - 2 * B * 113 * 64)
    if k == "coarse":
        n = c["n"]
        return dict(bytes=192 * n, flops=n * (1600 + 2 * (113 * 64 + 64 * 64 * 2 + 64 * 12)))
    b = 8 if c.get("dtype") == "f64" else 4
    if k == "batch2d":
        n = int(c["scenes"] * (c["n_hi"] - c["n_lo"]) / math.log(c["n_hi"] / c["n_lo"]))
        return dict(bytes=26 * b * n * c["substeps"], flops=500 * n * c["substeps"])
    dim, n, steps = c.get("dim", 2 if k == "step2d" else 3), c["n"], c.get("substeps", 1)
    reals = 2 * dim + 2 * dim * dim
    flops = (1600 if dim == 3 else 500) * n * steps
    if k == "solver":
        # x and F travel every substep (v and C can be rebuilt from the grid), all of it at the ends
        return dict(bytes=b * n * (2 * (dim + dim * dim) * steps + 2 * reals), flops=flops)
    if k == "rollout":
        # forward, recomputation and reverse: the state in and out of each, the adjoint in and out
        return dict(bytes=b * n * reals * steps * 7, flops=5 * flops)
    extra = {"step3d": 3, "host3d": 3, "step2d": 2, "phases3d": 3}[k]
    grid = (c["res"] + 1) ** 3 * 4 * b * 4 * steps if k == "phases3d" else 0
    return dict(bytes=b * n * (2 * reals + extra) * steps + grid, flops=flops)


# -------------------------------------------------------------------------------------------- exact
def _polar(F):
    """Rotation of the polar decomposition of [n, d, d], by Newton's iteration (2D: closed form)."""
    if F.shape[-1] == 2:
        a, b = F[:, 0, 0] + F[:, 1, 1], F[:, 1, 0] - F[:, 0, 1]
        d = torch.sqrt(a * a + b * b) + 1e-10
        return torch.stack([a / d, -b / d, b / d, a / d], 1).reshape(-1, 2, 2)
    X = F
    for _ in range(9):
        r0, r1, r2 = X[:, 0], X[:, 1], X[:, 2]
        cof = torch.stack([torch.linalg.cross(r1, r2), torch.linalg.cross(r2, r0), torch.linalg.cross(r0, r1)], 1)
        det = (r0 * cof[:, 0]).sum(1)
        X = 0.5 * (X + cof / det[:, None, None])
    return X


def _det(F):
    if F.shape[-1] == 2:
        return F[:, 0, 0] * F[:, 1, 1] - F[:, 0, 1] * F[:, 1, 0]
    return (F[:, 0] * torch.linalg.cross(F[:, 1], F[:, 2])).sum(1)


def _stress(F, mu, lam, diagonal):
    J = _det(F)
    p = (lam * (J - 1) * J)[:, None, None]
    p = p * torch.eye(F.shape[-1], dtype=F.dtype, device=F.device) if diagonal else p
    return 2 * mu[:, None, None] * ((F - _polar(F)) @ F.transpose(1, 2)) + p


def _stencil(x, res):
    """Node indices [n, 3^d], weights [n, 3^d] and offsets (node - x) in cells [n, 3^d, d]."""
    d = x.shape[1]
    xs = x * res
    base = torch.trunc(xs.detach() - 0.5)
    fx = xs - base
    w = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2], 1)  # [n, 3, d]
    o = torch.cartesian_prod(*[torch.arange(3, device=x.device)] * d)  # [3^d, d]
    W = w[:, o[:, 0], 0]
    for a in range(1, d):
        W = W * w[:, o[:, a], a]
    idx = base.long()[:, None, :] + o
    flat = idx[..., 0]
    for a in range(1, d):
        flat = flat * (res + 1) + idx[..., a]
    return flat, W, o - fx[:, None, :]


def _p2g(x, v, F, C, m, mu, lam, res, dt, vol, diagonal):
    d = x.shape[1]
    flat, W, off = _stencil(x, res)
    A = -(dt * vol) * 4 * res * res * _stress(F, mu, lam, diagonal) + m[:, None, None] * C
    q = (m[:, None] * v)[:, None, :] + (off / res) @ A.transpose(1, 2)
    val = torch.cat([W[..., None] * q, (W * m[:, None])[..., None]], 2)
    grid = torch.zeros(((res + 1) ** d, d + 1), dtype=x.dtype, device=x.device)
    return grid.index_add(0, flat.reshape(-1), val.reshape(-1, d + 1))


def _grid(g, res, dt, gravity, d):
    mom, m = g[:, :d], g[:, d:]
    has = m > 0
    vel = torch.where(has, mom / torch.where(has, m, torch.ones_like(m)), mom)
    add = torch.zeros(d, dtype=g.dtype, device=g.device)
    add[1] = dt * gravity
    vel = torch.where(has, vel + add, vel)
    I = torch.arange(res + 1, device=g.device)
    at = torch.stack(torch.meshgrid(*[I] * d, indexing="ij"), -1).reshape(-1, d)
    if d == 3:
        top = 0.9 / res / dt
        vel = torch.where(has, vel.clamp(-top, top), vel)
        return torch.where((at < 1) | (at >= res - 1), torch.zeros_like(vel), vel)
    pos = at.double() / res
    stop = has & ((pos[:, :1] < 0.05) | (pos[:, :1] > 1 - 0.05) | (pos[:, 1:] > 1 - 0.05))
    vel = torch.where(stop, torch.zeros_like(vel), vel)
    low = has[:, 0] & (pos[:, 1] < 0.05)
    return torch.stack([vel[:, 0], torch.where(low, vel[:, 1].clamp(min=0), vel[:, 1])], 1)


def _g2p(vel, x, F, res, dt):
    d = x.shape[1]
    flat, W, off = _stencil(x, res)
    gv = W[..., None] * vel[flat]
    v = gv.sum(1)
    C = 4 * res * (gv.transpose(1, 2) @ off)
    return x + dt * v, v, F + dt * (C @ F), C


def _substep(x, v, F, C, m, mu, lam, res, dt, vol, gravity, diagonal):
    g = _p2g(x, v, F, C, m, mu, lam, res, dt, vol, diagonal)
    return _g2p(_grid(g, res, dt, gravity, x.shape[1]), x, F, res, dt)


def exact(case, seed):
    f = globals()["_exact_" + case["kind"]]
    if case["kind"] == "rollout":
        return f(case, seed)
    with torch.no_grad():
        return f(case, seed)


def _as64(ts):
    return [t.double() for t in ts]


def _exact_step3d(c, seed):
    dt, vol, res = DTYPES[c["dtype"]], _volume(c["n"], 3), c["res"]
    s = _as64(_bodies(c["n"], 3, seed, dt))
    mat = _as64(_material(c["n"], dt, vol))
    for _ in range(c["substeps"]):
        s = _substep(*s, *mat, res, _cfl_dt(res), vol, -9.8, False)
    return dict(zip("xvFC", s))


def _exact_phases3d(c, seed):
    dt, vol, res = DTYPES[c["dtype"]], _volume(c["n"], 3), c["res"]
    s = _as64(_bodies(c["n"], 3, seed, dt))
    mat = _as64(_material(c["n"], dt, vol))
    R, h = res + 1, _cfl_dt(res)
    for _ in range(c["substeps"]):
        g = _p2g(*s, *mat, res, h, vol, False)
        vel = _grid(g, res, h, -9.8, 3)
        s = _g2p(vel, s[0], s[2], res, h)
    return dict(zip("xvFC", s), grid_velocity=vel.reshape(R, R, R, 3), grid_mass=g[:, 3:].reshape(R, R, R, 1))


def _exact_host3d(c, seed):
    dt, vol, res = DTYPES[c["dtype"]], _volume(c["n"], 3), c["res"]
    s = _as64(_bodies(c["n"], 3, seed, dt, strain=1e-3, spin=0.1))
    mat = _as64(_material(c["n"], dt, vol))
    return dict(zip("xvFC", _substep(*s, *mat, res, _cfl_dt(res), vol, 0.0, False)))


def _exact_step2d(c, seed):
    s0 = _prepare_step2d(c, seed)
    x, v, F, C, Jp = _as64(s0["first"])
    n, res = c["n"], c["res"]
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    for _ in range(c["substeps"]):
        h = torch.exp(s0["hardening"] * (1 - Jp[:, 0])) if c["model"] == "snow" else s0["hardening"] * one
        x, v, F, C = _substep(x, v, F, C, s0["vol"] * one, s0["mu"] * h, s0["lam"] * h, res, s0["dt"], s0["vol"], -9.8,
                              False)
        J = _det(F)
        if c["model"] == "snow":
            F = _clamp_singular(F)
        Jp = (Jp * (J / (_det(F) + 1e-10))[:, None]).clamp(0.6, 20.0)
    return dict(x=x, v=v, F=F, C=C, Jp=Jp)


def _clamp_singular(F):
    """F with its singular values clamped to [1 - 0.025, 1 + 0.0075], through F = R S."""
    R = _polar(F)
    S = R.transpose(1, 2) @ F
    I = torch.eye(2, dtype=F.dtype, device=F.device)
    m = 0.5 * (S[:, 0, 0] + S[:, 1, 1])
    dev = 0.5 * (S + S.transpose(1, 2)) - m[:, None, None] * I
    r = torch.sqrt(dev[:, 0, 0] ** 2 + dev[:, 0, 1] ** 2)
    hi, lo = (m + r).clamp(1 - 2.5e-2, 1 + 7.5e-3), (m - r).clamp(1 - 2.5e-2, 1 + 7.5e-3)
    N = dev / r.clamp(min=1e-300)[:, None, None]
    return R @ ((0.5 * (hi + lo))[:, None, None] * I + (0.5 * (hi - lo))[:, None, None] * N)


def _exact_solver(c, seed):
    if c["n"] * c["substeps"] > 60_000_000:
        return None  # about 20 seconds
    n, dim, res = c["n"], c["dim"], c["res"]
    s = _as64(_bodies(n, dim, seed, DTYPES[c["dtype"]], strain=1e-3, spin=0.1, speed=0.5))
    vol = _volume(n, dim)
    mu, lam = _lame(4.5e3, NU)
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    Jp = one.clone()
    for _ in range(c["substeps"] + 2):  # capture() runs two substeps of its own first
        s = _substep(*s, vol * one, mu * one, lam * one, res, _cfl_dt(res), vol, -1.0, True)
        if dim == 2:
            J = _det(s[2])
            Jp = (Jp * J / (J + 1e-10)).clamp(0.6, 20.0)
    return dict(zip("xvFC", s), Jp=Jp)


def _exact_batch2d(c, seed):
    scenes = _scenes(c, seed)
    out = [[], [], [], [], []]
    if sum(len(s["x"]) for s in scenes) * c["substeps"] > 55_000_000:
        return None  # about 20 seconds
    for s in scenes:
        res, x0 = s["res"], s["x"]
        # each scene's particles in the order the batch documents: stably by base cell
        cell = np.clip(np.floor(x0 * res - 0.5), -1, res).astype(np.int64)
        at = np.argsort(cell[:, 0] * (res + 2) + cell[:, 1], kind="stable")
        f = lambda a: torch.tensor(a[at], dtype=DTYPES[c["dtype"]], device=DEV).double()
        n = len(x0)
        one = torch.ones(n, dtype=torch.float64, device=DEV)
        eye = torch.eye(2, dtype=torch.float64, device=DEV).expand(n, 2, 2)
        st = (f(x0), f(s["v"]), eye, torch.zeros_like(eye))
        Jp = one
        for _ in range(c["substeps"] + 1):  # capture() runs one substep of its own first
            st = _substep(*st, s["mass"] * one, s["mu_0"] * one, s["lambda_0"] * one, res, s["dt"], s["volume"], -9.8,
                          True)
            J = _det(st[2])
            Jp = (Jp * J / (J + 1e-10)).clamp(0.6, 20.0)
        for o, t in zip(out, (*st, Jp)):
            o.append(t.reshape(n, -1).T)
    x, v, F, C, Jp = (torch.cat(o, 1) for o in out)
    return dict(x=x, v=v, F=F, C=C, Jp=Jp[0])


def _exact_rollout(c, seed):
    (x, v, F, mu, lam), vol = _rollout_scene(c, seed)
    x, v, F, mu, lam = (t.double().requires_grad_(True) for t in (x, v, F, mu, lam))
    res, h = c["res"], _cfl_dt(c["res"], 4e3)
    m = torch.full_like(mu, vol)
    s = (x, v, F, torch.zeros_like(F))
    for _ in range(c["substeps"]):
        s = torch.utils.checkpoint.checkpoint(lambda *a: _substep(*a, m, mu, lam, res, h, vol, -9.8, True), *s,
                                              use_reentrant=False)
    ((s[0] - _target(c["dim"], x)) ** 2).sum(1).mean().backward()
    return dict(x=s[0].detach(), v=s[1].detach(), F=s[2].detach(), gx=x.grad, gv=v.grad, gF=F.grad, gmu=mu.grad,
                glam=lam.grad)


def _forward64(P, X, b4=None):
    W1, W2 = P[:8192].reshape(64, 128), P[16384:20480].reshape(64, 64)
    W3, W4 = P[24576:28672].reshape(64, 64), P[32768:33536].reshape(12, 64)
    h = X
    for W, b in ((W1, 40960), (W2, 41024), (W3, 41088)):
        h = torch.nn.functional.gelu(h @ W.T + P[b:b + 64])
    return h @ W4.T + (P[41152:41164] if b4 is None else b4)


def _exact_coarse(c, seed):
    n, res = c["n"], c["res"]
    st = _coarse_state(c, seed).double()
    x, v = st[0:3].T, st[3:6].T
    F, C = st[6:15].T.reshape(n, 3, 3), st[15:24].T.reshape(n, 3, 3)
    vol, h = _volume(n, 3), 5e-5 * 8
    mu, lam = _lame(150.0, NU)
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    PF = _stress(F, mu * one, lam * one, True)
    vel = _grid(_p2g(x, v, F, C, vol * one, mu * one, lam * one, res, h, vol, True), res, h, -9.8, 3)
    flat, _, _ = _stencil(x, res)
    xn, vn, Fn, Cn = _g2p(vel, x, F, res, h)
    u = vel[flat[:, 13]]
    k = h * h * res * res
    eye = torch.eye(3, dtype=torch.float64, device=DEV)
    feat = torch.cat([(Fn - eye).reshape(n, 9), Cn.reshape(n, 9) * h, (vn - u) * h * res,
                      ((vel[flat] - u[:, None]) * h * res).reshape(n, 81), (mu * k * one)[:, None],
                      (lam * k * one)[:, None], PF.reshape(n, 9) * k, torch.zeros((n, 15), dtype=torch.float64,
                                                                            device=DEV)], 1)
    net = _net(128, seed)
    P, scale = net.params.double(), _coarse_in_scale().double()
    rest = torch.zeros((1, 128), dtype=torch.float64, device=DEV)
    rest[0, 102], rest[0, 103] = mu * k, lam * k
    y = (_forward64(P, feat * scale) - _forward64(P, rest * scale)) * 5e-4
    dv = y[:, 9:12] / (h * res)
    Fn, vn, xn = Fn + y[:, :9].reshape(n, 3, 3), vn + dv, xn + h * dv
    return torch.cat([xn.T, vn.T, Fn.reshape(n, 9).T, Cn.reshape(n, 9).T], 0)


def _exact_train(c, seed):
    X, T = _train_data(c, seed)
    net = _net(c["batch"], seed)
    P = net.params.double()
    with torch.enable_grad():
        P.requires_grad_(True)
        Y = _forward64(P, X.double())
        loss = ((Y - T.double()) ** 2).sum() / c["batch"]
        (g,) = torch.autograd.grad(loss, P)
    return dict(Y=Y.detach(), loss=loss.detach().reshape(1), grads=g, params=None)
