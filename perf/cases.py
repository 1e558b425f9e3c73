"""Timing cases of the framework's main path, from a single collision check to trajectory optimisation.

Each case is a dict of plain values; ``listed`` gives the fixed ones, ``draw``
more of the same ranges.  ``prepare`` builds what a program has in hand before
a call (robot, scene, inputs on the GPU), ``run`` is one pass through the
public entry points, ``exact`` the same values in 64 bits by plain torch,
``work`` the bytes and operations a pass cannot do without and ``tolerance``
what another correct FP32 implementation may differ by.

The iterative solvers (``ik``, ``batch``, ``hjcd``, ``sqp``, ``chomp``) choose
between discrete alternatives -- a line-search step, the joint to move, to
accept or not -- so a change of rounding grows from iteration to iteration
(moving the inputs by one unit in the last place moves the 7-DOF benchmark's
configurations by 6e-5 after 4 iterations and 3e-3 after 30).  Their cases run
few iterations, every one of which does the work of any other; their iterates
depend on those choices and have no 64-bit value of their own.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from pyroffi_b200 import robot as R
from pyroffi_b200 import workloads as W

DEV = "cuda"
G64 = torch.float64


def listed():
    return [
        # one configuration of an arm against a small scene: the check inside a control loop
        dict(name="check_one", kind="check", out="min", B=1, per_link=8, Ms=64, Mc=0, Mb=0, Mh=0),
        # sphere-resolved distances of a large batch (a planner's or a learner's samples)
        dict(name="check_spheres", kind="check", out="spheres", B=65536, per_link=8, Ms=64, Mc=0, Mb=0, Mh=0),
        # per-link distances to a scanned scene of thousands of spheres and oriented boxes
        dict(name="check_links", kind="check", out="links", B=16384, per_link=16, Ms=4096, Mc=0, Mb=256, Mh=0),
        # forward kinematics of a 29-DOF humanoid over a ragged large batch
        dict(name="fk_humanoid", kind="fk", robot="humanoid", B=100003),
        # the drop-in distance operators on given sphere centres: world (all obstacle kinds) and self
        dict(name="world_self", kind="world", B=2048, per_link=12, Ms=201, Mc=33, Mb=32, Mh=2),
        # multi-seed collision-aware IK of one arm, the sizes of the repository's benchmark
        dict(name="ik_arm", kind="ik", P=256, Sd=128, iters=6, Ms=100, pairs=200),
        # uneven batch of IK problems over arms, a bimanual tree and a humanoid
        dict(name="ik_mixed", kind="batch", problems=512, iters=6),
        # HJCD-IK: coarse coordinate descent and LM refinement
        dict(name="hjcd", kind="hjcd", P=256, S=32, coarse=20, iters=6, Ms=100),
        # SQP-IK with hard joint limits
        dict(name="sqp", kind="sqp", P=256, S=32, iters=8, Ms=100),
        # the trajectory cost through autograd: forward, then backward
        dict(name="traj_grad", kind="traj", B=512, T=64, Ms=256, Mb=32),
        # one outer iteration of SCO and the ranking of its trajectories
        dict(name="sco_step", kind="sco", B=512, T=64, inner=30, Ms=256, Mc=16, Mb=32, Mh=1),
        # CHOMP steps: gradient, covariant direction, line search
        dict(name="chomp", kind="chomp", B=512, T=64, iters=5, Ms=256, Mb=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["check", "check", "fk", "world", "ik", "batch", "hjcd", "sqp", "traj", "sco", "chomp"])
    if kind == "check":
        out = rng.choice(["min", "spheres", "links"])
        c = dict(kind=kind, out=out, per_link=rng.randint(3, 16), Ms=_log(rng, 20, 4096), Mc=rng.choice([0, 0, 5, 17]),
                 Mb=rng.choice([0, 0, 31, 256]), Mh=rng.choice([0, 1, 2]))
        m = c["Ms"] + c["Mc"] + c["Mb"] + c["Mh"]
        # rows of at most 2 GB, at most the listed sweep's distances
        rows = 8 * (c["per_link"] if out == "spheres" else 1)
        most = min(65536, 5e8 / (m * rows) if out != "min" else 65536, 8e9 / (8 * c["per_link"] * m))
        return dict(c, B=_log(rng, 1, max(2, int(most))))
    if kind == "fk":
        return dict(kind=kind, robot=rng.choice(["chain", "bimanual", "humanoid"]), B=_log(rng, 1, 100000))
    if kind == "world":
        return dict(kind=kind, B=_log(rng, 1, 2048), per_link=rng.randint(2, 12), Ms=_log(rng, 8, 260),
                    Mc=rng.choice([0, 7, 33]), Mb=rng.choice([0, 9, 32]), Mh=rng.choice([0, 1, 2]))
    if kind == "ik":
        return dict(kind=kind, P=_log(rng, 1, 256), Sd=_log(rng, 16, 128), iters=rng.randint(2, 6),
                    Ms=rng.choice([0, 33, 100, 171]), pairs=rng.choice([0, 60, 200]))
    if kind == "batch":
        return dict(kind=kind, problems=_log(rng, 16, 512), iters=rng.randint(2, 6))
    if kind == "hjcd":
        return dict(kind=kind, P=_log(rng, 1, 256), S=_log(rng, 8, 40), coarse=rng.randint(4, 20),
                    iters=rng.randint(1, 6), Ms=rng.choice([0, 20, 100]))
    if kind == "sqp":
        return dict(kind=kind, P=_log(rng, 1, 256), S=_log(rng, 8, 40), iters=rng.randint(1, 8),
                    Ms=rng.choice([0, 20, 100]))
    if kind == "traj":
        return dict(kind=kind, B=_log(rng, 1, 512), T=rng.randint(9, 64), Ms=_log(rng, 16, 256), Mb=rng.randint(0, 32))
    if kind == "sco":
        return dict(kind=kind, B=_log(rng, 1, 512), T=rng.randint(9, 64), inner=rng.randint(5, 30),
                    Ms=_log(rng, 16, 256), Mc=rng.randint(1, 16), Mb=rng.randint(1, 32), Mh=1)
    return dict(kind=kind, B=_log(rng, 1, 512), T=rng.randint(9, 64), iters=rng.randint(1, 5), Ms=_log(rng, 16, 256),
                Mb=rng.randint(0, 32))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _t(x, dtype=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device=DEV)


@functools.lru_cache(maxsize=None)
def _ik_scene(P, Ms, pairs):
    """The benchmark's arm and feasible targets (fixed: not every random arm has a self-free posture)."""
    return W.ik(P=P, Sd=1, n_obstacles=Ms, n_self=pairs)


@functools.lru_cache(maxsize=None)
def _mixed_scene(problems):
    return W.mixed_ik(n_problems=problems)


def _world(rng, c):
    w = W.empty_world()
    w.spheres = W.random_sphere_world(rng, c["Ms"])
    if c.get("Mc"):
        w.capsules = W.random_capsules(rng, c["Mc"])
    if c.get("Mb"):
        w.boxes = W.random_boxes(rng, c["Mb"], oriented=True)
    if c.get("Mh"):
        hs = np.zeros((c["Mh"], 6), np.float32)
        hs[:, 2] = 1.0
        hs[:, 5] = -1.2 - 0.1 * np.arange(c["Mh"])
        w.halfspaces = hs
    return w


def _uniform(model, shape, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    lo, hi = _t(model.lower), _t(model.upper)
    return lo + (hi - lo) * torch.rand((*shape, model.n_act), device=DEV, generator=g)


def _trajectories(model, B, T, seed):
    """Noisy straight lines between random configurations, ends kept."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    ends = _uniform(model, (B, 2), seed + 1)
    s = torch.linspace(0.0, 1.0, T, device=DEV)[None, :, None]
    x = ends[:, :1] * (1 - s) + ends[:, 1:] * s
    noise = 0.1 * torch.randn(x.shape, device=DEV, generator=g)
    noise[:, 0] = 0.0
    noise[:, -1] = 0.0
    return (x + noise).contiguous()


def prepare(case, seed):
    c, k = case, case["kind"]
    rng = np.random.default_rng(seed)
    st = dict(case=c)
    if k == "check":
        from pyroffi_b200.device import DeviceRobot, DeviceSpheres, DeviceWorld

        model = R.serial_chain(7, rng)
        spheres = R.random_spheres(model, rng, per_link=c["per_link"], base_spheres=True)
        world = _world(rng, c)
        return dict(st, model=model, spheres=spheres, world=world, robot=DeviceRobot.upload(model, DEV),
                    dspheres=DeviceSpheres.upload(spheres, DEV), dworld=DeviceWorld.upload(world, DEV),
                    cfg=_uniform(model, (c["B"],), seed))
    if k == "fk":
        make = dict(chain=lambda r: R.serial_chain(7, r), bimanual=R.bimanual_tree, humanoid=R.humanoid_tree)
        model = make[c["robot"]](rng)
        i = torch.int32
        args = [_t(model.twists), _t(model.parent_tf), _t(model.parent_idx, i), _t(model.act_idx, i), _t(model.mimic_mul),
                _t(model.mimic_off), _t(model.mimic_act_idx, i), _t(model.topo_inv, i), _t(model.fk_level_starts, i),
                _t(model.fk_level_joints, i)]
        return dict(st, model=model, args=args, cfg=_uniform(model, (c["B"],), seed))
    if k == "world":
        model = R.humanoid_tree(rng)
        S, N, B = c["per_link"], model.n_links, c["B"]
        spheres = R.random_spheres(model, rng, per_link_range=(max(1, S // 3), S), base_spheres=True)
        g = torch.Generator(device=DEV).manual_seed(seed)
        links = 2.0 * torch.rand((B, 1, N, 3), device=DEV, generator=g) - 1.0
        cen = (links + _t(spheres.centers).transpose(0, 1)[None, :spheres.S]).contiguous()      # [B, S, N, 3]
        rad = _t(spheres.radii).T[None].expand(B, -1, -1).contiguous()                          # [B, S, N]
        S = spheres.S
        pairs = _t(W.active_link_pairs(model, spheres), torch.int32)
        world = _world(rng, c)
        return dict(st, cen=cen, rad=rad, soa=cen.reshape(B, S * N, 3).permute(2, 0, 1).contiguous(),
                    rk=rad.reshape(B, S * N).contiguous(), world=[_t(a) for a in world.arrays()], N=N,
                    pi=pairs[:, 0].contiguous(), pj=pairs[:, 1].contiguous())
    if k == "ik":
        from pyroffi_b200.ik import BatchIkSolver

        w = _ik_scene(c["P"], c["Ms"], c["pairs"])
        solver = BatchIkSolver(w.model, w.target_link, spheres=w.spheres, world=w.world, self_pairs=w.self_pairs,
                               max_iter=c["iters"], lambda_init=w.lambda_init, lambda_down=w.lambda_down,
                               lambda_up=w.lambda_up, device=DEV)
        return dict(st, solver=solver, target=_t(w.target_T[rng.permutation(c["P"])]),
                    seeds=_uniform(w.model, (c["P"], c["Sd"]), seed))
    if k == "batch":
        from pyroffi_b200.batch_ik import MixedIkBatch

        w = _mixed_scene(c["problems"])
        b = MixedIkBatch(w.classes, w.world, max_iter=c["iters"], lambda_init=w.lambda_init,
                         lambda_down=w.lambda_down, lambda_up=w.lambda_up, collision_weight=w.collision_weight,
                         collision_margin=w.collision_margin, device=DEV)
        b.prepare(w.problem_class, w.n_seeds)
        b.load([t[rng.permutation(len(t))] for t in w.target_T],
               [_uniform(cl.model, s.shape[:2], seed + i) for i, (cl, s) in enumerate(zip(w.classes, w.seeds))])
        return dict(st, batch=b)
    if k in ("hjcd", "sqp"):
        from pyroffi_b200.hjcd import HjcdSolver
        from pyroffi_b200.sqp import SqpSolver

        w = _ik_scene(c["P"], c["Ms"], 0)
        solver = (HjcdSolver if k == "hjcd" else SqpSolver)(w.model, w.target_link, spheres=w.spheres, world=w.world,
                                                            enable_collision=c["Ms"] > 0, device=DEV)
        g = torch.Generator(device=DEV).manual_seed(seed)
        noise = torch.randn((c["P"], c["S"], c["iters"], 7), device=DEV, generator=g) if k == "hjcd" else None
        return dict(st, solver=solver, target=_t(w.target_T[rng.permutation(c["P"])]),
                    seeds=_uniform(w.model, (c["P"], c["S"]), seed),
                    lm_seeds=_uniform(w.model, (c["P"], c["S"]), seed + 1), noise=noise)
    # trajectories of the 7-DOF arm, 8 spheres per moving link
    model = R.serial_chain(7, rng)
    spheres = R.random_spheres(model, rng, per_link=8)
    world = _world(rng, c)
    pairs = W.active_link_pairs(model, spheres)
    st.update(model=model, spheres=spheres, world=world, pairs=pairs, x=_trajectories(model, c["B"], c["T"], seed))
    if k == "sco":
        from pyroffi_b200.sco import ScoConfig, ScoOptimizer

        return dict(st, opt=ScoOptimizer(model, spheres, world, pairs, ScoConfig(n_inner_iters=c["inner"]), device=DEV))
    from pyroffi_b200.trajopt import TrajectoryCost

    cost = TrajectoryCost(model, spheres, world, pairs, device=DEV)
    if k == "traj":
        return dict(st, cost=cost)
    from pyroffi_b200.chomp import ChompConfig, ChompOptimizer

    return dict(st, opt=ChompOptimizer(cost, ChompConfig(n_iters=c["iters"])))


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(st):
    c, k = st["case"], st["case"]["kind"]
    if k == "check":
        from pyroffi_b200.collision import fk_sphere_collision

        r = fk_sphere_collision(st["robot"], st["dspheres"], st["dworld"], st["cfg"], per_sphere=c["out"] == "spheres",
                                per_link=c["out"] == "links", link_poses=c["out"] != "links")
        return dict(min_dist=r.min_dist, link_poses=r.link_poses, spheres=r.dist_bkm, links=r.dist_bnm)
    if k == "fk":
        from pyroffi_b200.cuda_kernels import fk_cuda

        return fk_cuda(st["cfg"], *st["args"])
    if k == "world":
        from pyroffi_b200.cuda_kernels import collision_self_sphere, collision_world_sphere_reduced

        return (collision_world_sphere_reduced(st["soa"], st["rk"], *st["world"], st["N"]),
                collision_self_sphere(st["cen"], st["rad"], st["pi"], st["pj"]))
    if k == "ik":
        r = st["solver"].solve(st["target"], st["seeds"])
        return dict(cfgs=r.cfgs, errs=r.errs, success=r.success)
    if k == "batch":
        b = st["batch"]
        res = b.solve()
        return dict(cfgs=b.out_cfg, errs=b.out_err, success=[None if r is None else r.success for r in res])
    if k == "hjcd":
        s = st["solver"]
        coarse = s.coarse(st["seeds"], st["target"], c["coarse"])
        fine = s.refine(st["lm_seeds"], st["noise"], st["target"], max_iter=c["iters"], lambda_init=1e-3,
                        limit_prior_weight=1e-4, kick_scale=0.02)
        return dict(coarse=coarse, fine=fine)
    if k == "sqp":
        return st["solver"].run(st["seeds"], st["target"], max_iter=c["iters"])
    if k == "traj":
        from pyroffi_b200.trajopt import TrajectoryCostFn

        x = st["x"].requires_grad_(True)
        x.grad = None
        J = TrajectoryCostFn.apply(x, st["cost"])
        J.sum().backward()
        return dict(cost=J.detach(), grad=x.grad)
    if k == "sco":
        o, x = st["opt"], st["x"]
        d, J, _ = o.linearize(x)
        y = o.inner(x, d, J, o.cfg.w_collision, x[0, 0], x[0, -1])
        return dict(dist=d, jac=J, traj=y, cost=o.final_cost(y))
    _, costs, final = st["opt"].run(st["x"], st["x"][0, 0], st["x"][0, -1])
    return dict(costs=costs, final=final)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

FK_JOINT = 130      # exp of one joint and two compositions
PLACE = 33          # one sphere moved by a pose
SPHERE = 12         # one sphere-sphere distance


def work(case):
    c, k = case, case["kind"]
    if k == "check":
        m, s = c["Ms"] + c["Mc"] + c["Mb"] + c["Mh"], 8 * c["per_link"]
        out = dict(min=1 + 56, spheres=1 + 56 + s * m, links=1 + 8 * m)[c["out"]]
        return dict(bytes=4 * c["B"] * (7 + out), flops=c["B"] * (7 * FK_JOINT + s * (PLACE + SPHERE * m)))
    if k == "fk":
        nj, n = dict(chain=(7, 7), bimanual=(16, 15), humanoid=(29, 29))[c["robot"]]
        return dict(bytes=4 * c["B"] * (n + 7 * nj), flops=c["B"] * nj * FK_JOINT)
    if k == "world":
        m, s = c["Ms"] + c["Mc"] + c["Mb"] + c["Mh"], 30 * c["per_link"]
        pairs = 30 * 29 // 2 - 29
        return dict(bytes=4 * c["B"] * (8 * s + 30 * m + pairs),
                    flops=c["B"] * SPHERE * s * (m + pairs * c["per_link"] / 30) / 2)
    if k in ("ik", "hjcd", "sqp"):
        seeds = c["P"] * (c["Sd"] if k == "ik" else c["S"])
        evals = 6 * c["iters"] + 1 + (c["coarse"] + 1 if k == "hjcd" else 0)
        sph = PLACE * 56 if c["Ms"] else 0
        return dict(bytes=4 * seeds * 15 * (2 if k == "hjcd" else 1),
                    flops=seeds * (evals * (7 * FK_JOINT + 60 + sph) + c["iters"] * (45 * 7 + 800)))
    if k == "batch":
        # mean seeds 144; joints, spheres and actuated joints averaged over the four classes
        seeds = 144 * c["problems"]
        nj, rs = 0.4 * 7 + 0.3 * 6 + 0.2 * 16 + 0.1 * 29, 0.4 * 56 + 0.3 * 48 + 0.2 * 128 + 0.1 * 232
        return dict(bytes=4 * seeds * 22, flops=seeds * ((6 * c["iters"] + 1) * (nj * FK_JOINT + 60 + PLACE * rs)
                                                          + c["iters"] * 3000))
    wp = c["B"] * c["T"]
    m = c["Ms"] + c.get("Mc", 0) + c["Mb"] + c.get("Mh", 0)
    # a bounding test per (link, obstacle); the sphere tests follow for the near ones
    wpf = 7 * FK_JOINT + 56 * PLACE + 7 * m * SPHERE
    if k == "traj":
        return dict(bytes=4 * wp * 14 + 4 * c["B"], flops=2 * wp * wpf)
    if k == "sco":
        lin = wp * (wpf + 7 * m * 8 * SPHERE)
        return dict(bytes=4 * wp * (7 + 5 + 35 + 7), flops=lin + wp * wpf + c["inner"] * wp * 7 * 60)
    return dict(bytes=4 * wp * 14, flops=c["iters"] * 7 * wp * wpf)


def tolerance(case):
    """About four times what one unit in the last place of the inputs does (measured at the listed sizes);
    for the smooth-minimum Jacobian four times its distance from 64 bits (3e-4): where two spheres of a link
    are equally near an obstacle to within rounding, either one's gradient is right."""
    k = case["kind"]
    if k in ("check", "fk", "world"):
        return dict(rel=2e-6, max=2e-5)
    if k in ("ik", "batch"):
        return dict(rel=4e-3, max=0.9, differ=0.01)
    if k == "hjcd":
        return dict(rel=3e-3, max=0.6, differ=0.01)
    if k == "sqp":
        return dict(rel=1e-3, max=0.2)
    if k == "traj":
        return dict(rel=1e-5, max=2e-4)
    if k == "sco":
        return dict(rel=1.5e-3, max=0.5)
    return dict(rel=1e-3, max=0.2)


# ---------------------------------------------------------------------------
# the same values in 64 bits
# ---------------------------------------------------------------------------

def _qmul(a, b):
    w1, x1, y1, z1 = a.unbind(-1)
    w2, x2, y2, z2 = b.unbind(-1)
    return torch.stack([w1 * w2 - x1 * x2 - y1 * y2 - z1 * z2, w1 * x2 + x1 * w2 + y1 * z2 - z1 * y2,
                        w1 * y2 - x1 * z2 + y1 * w2 + z1 * x2, w1 * z2 + x1 * y2 - y1 * x2 + z1 * w2], -1)


def _rot4(q, v):
    u, w = q[..., 1:4], q[..., :1]
    t = 2.0 * torch.linalg.cross(u, v)
    return v + w * t + torch.linalg.cross(u, t)


def _fk64(model, cfg):
    """Joint poses [..., n_j, 7] of revolute, prismatic and fixed joints."""
    d = lambda a: torch.as_tensor(np.asarray(a), dtype=G64, device=DEV)  # noqa: E731
    q = cfg.to(G64)
    lead = q.shape[:-1]
    poses = [None] * model.n_joints
    for j in (int(v) for v in model.topo_inv):
        ptf, tw = d(model.parent_tf[j]), d(model.twists[j])
        quat, tr = ptf[:4].expand(*lead, 4), ptf[4:].expand(*lead, 3)
        a = int(model.act_idx[j])
        if a >= 0:
            nw = torch.linalg.norm(tw[3:])
            if float(nw) > 0:
                h = 0.5 * q[..., a:a + 1] * nw
                quat = _qmul(quat, torch.cat([torch.cos(h), torch.sin(h) * (tw[3:] / nw)], -1))
            else:
                tr = tr + _rot4(quat, q[..., a:a + 1] * tw[:3])
        p = int(model.parent_idx[j])
        if p >= 0:
            pq, pt = poses[p]
            quat, tr = _qmul(pq, quat), pt + _rot4(pq, tr)
        poses[j] = (quat, tr)
    return torch.stack([torch.cat(p, -1) for p in poses], -2)


def _links64(model, cfg):
    T = _fk64(model, cfg)
    ident = torch.zeros((*T.shape[:-2], 1, 7), dtype=G64, device=DEV)
    ident[..., 0] = 1.0
    return torch.cat([T, ident], -2)[..., [int(j) if j >= 0 else model.n_joints for j in model.parent_joint_indices], :]


def _centres64(links, centers):
    """Sphere centres [..., N, S, 3] of link poses [..., N, 7] and link-frame centres [N, S, 3]."""
    c = torch.as_tensor(centers, dtype=G64, device=DEV)
    T = links[..., None, :].expand(*links.shape[:-1], c.shape[1], 7)
    return _rot4(T[..., :4], c.expand(*T.shape[:-1], 3)) + T[..., 4:]


def _dist64(p, r, world):
    """Signed distances [..., M] of spheres (p [..., 3], r [...]) to the obstacle arrays, as a list by kind."""
    ws, wc, wb, wh = (torch.as_tensor(a, dtype=G64, device=DEV) for a in world)
    p, r, out = p[..., None, :], r[..., None], []
    out.append(torch.linalg.norm(p - ws[:, :3], dim=-1) - r - ws[:, 3] if len(ws) else None)
    if len(wc):
        v = wc[:, 3:6] - wc[:, :3]
        t = (((p - wc[:, :3]) * v).sum(-1) / (v * v).sum(-1)).clamp(0.0, 1.0)
        out.append(torch.linalg.norm(wc[:, :3] + t[..., None] * v - p, dim=-1) - r - wc[:, 6])
    else:
        out.append(None)
    if len(wb):
        e = p - wb[:, :3]
        q = torch.stack([(e * wb[:, 3 + 3 * i:6 + 3 * i]).sum(-1).abs() - wb[:, 12 + i] for i in range(3)], -1)
        m2 = q.clamp(min=0.0).square().sum(-1)
        outside = torch.where(m2 > 0, torch.where(m2 > 0, m2, 1.0).sqrt(), 0.0)
        out.append(outside + q.amax(-1).clamp(max=0.0) - r)
    else:
        out.append(None)
    out.append(((p - wh[:, 3:]) * wh[:, :3]).sum(-1) - r if len(wh) else None)
    return out


def _cat(parts):
    return torch.cat([x for x in parts if x is not None], -1)


def _exact_check(st):
    c, m = st["case"], st["model"]
    r = torch.as_tensor(st["spheres"].radii, dtype=G64, device=DEV)                  # [N, S]
    M = c["Ms"] + c["Mc"] + c["Mb"] + c["Mh"]
    step = max(1, int(4e7 // (r.numel() * M)))
    mins, poses, rows = [], [], []
    for i in range(0, c["B"], step):
        links = _links64(m, st["cfg"][i:i + step])
        d = _cat(_dist64(_centres64(links, st["spheres"].centers), r, st["world"].arrays()))   # [b, N, S, M]
        mins.append(d.amin((1, 2, 3)))
        poses.append(links)
        if c["out"] == "links":
            rows.append(d.amin(2))
        elif c["out"] == "spheres":
            rows.append(d.transpose(1, 2).reshape(d.shape[0], -1, M))                # sphere k = s * N + n
    rows = torch.cat(rows) if rows else None
    return dict(min_dist=torch.cat(mins), link_poses=torch.cat(poses) if c["out"] != "links" else None,
                spheres=rows if c["out"] == "spheres" else None, links=rows if c["out"] == "links" else None)


def _exact_world(st):
    cen, rad, pi, pj = st["cen"].to(G64), st["rad"].to(G64), st["pi"].long(), st["pj"].long()
    world, selfd = [], []
    for i in range(0, cen.shape[0], 32):
        p, r = cen[i:i + 32], rad[i:i + 32]                                          # [b, S, N, 3], [b, S, N]
        d = _cat(_dist64(p, r, st["world"]))
        world.append(torch.where((r < 0)[..., None], math.inf, d).amin(1))
        a, b, ra, rb = p[:, :, None, pi], p[:, None, :, pj], r[:, :, None, pi], r[:, None, :, pj]
        s = torch.linalg.norm(a - b, dim=-1) - ra - rb
        selfd.append(torch.where((ra < 0) | (rb < 0), math.inf, s).amin((1, 2)))
    return torch.cat(world), torch.cat(selfd)


def _exact_traj(st):
    m, o = st["model"], st["cost"].opt
    r = torch.as_tensor(st["spheres"].radii, dtype=G64, device=DEV)
    has = torch.as_tensor((st["spheres"].radii > 0).any(1), device=DEV)
    lo, hi = (torch.as_tensor(a, dtype=G64, device=DEV) for a in (m.lower, m.upper))
    pi, pj = (torch.as_tensor(st["pairs"][:, i], dtype=torch.long, device=DEV) for i in (0, 1))
    f = lambda v: float(np.float32(v))  # noqa: E731
    costs, grads = [], []
    for i in range(0, st["x"].shape[0], 8):
        x = st["x"][i:i + 8].detach().to(G64).requires_grad_(True)
        acc = (-x[:, :-4] + 16 * x[:, 1:-3] - 30 * x[:, 2:-2] + 16 * x[:, 3:-1] - x[:, 4:]) / 12
        jerk = acc[:, 1:] - acc[:, :-1]
        over = (x - hi).clamp(min=0) + (lo - x).clamp(min=0)
        cen = _centres64(_links64(m, x), st["spheres"].centers)                      # [b, T, N, S, 3]
        hinge = lambda d: (f(o.margin) - d).clamp(min=0).square()  # noqa: E731
        d = _cat(_dist64(cen[:, :, has], r[has], st["world"].arrays())).amin(3)
        s = (torch.linalg.norm(cen[:, :, pi] - cen[:, :, pj], dim=-1) - r[pi] - r[pj]).amin(-1)
        J = (f(o.w_smooth) * (f(o.w_acc) * acc.square().sum((1, 2)) + f(o.w_jerk) * jerk.square().sum((1, 2)))
             + f(o.w_limits) * over.square().sum((1, 2)) + f(o.w_coll) * (hinge(d).sum((1, 2, 3)) + hinge(s).sum((1, 2))))
        (g,) = torch.autograd.grad(J.sum(), x)
        costs.append(J.detach())
        grads.append(g)
    return dict(cost=torch.cat(costs), grad=torch.cat(grads))


def _exact_linearise(st):
    m, tau = st["model"], float(np.float32(st["opt"].cfg.smooth_min_temperature))
    r = torch.as_tensor(st["spheres"].radii, dtype=G64, device=DEV)
    has = torch.as_tensor((st["spheres"].radii > 0).any(1), device=DEV)
    pi, pj = (torch.as_tensor(st["pairs"][:, i], dtype=torch.long, device=DEV) for i in (0, 1))
    q = st["x"].reshape(-1, m.n_act)
    ds, js = [], []
    for i in range(0, q.shape[0], 512):
        x = q[i:i + 512].detach().to(G64).requires_grad_(True)
        cen = _centres64(_links64(m, x), st["spheres"].centers)
        s = torch.linalg.norm(cen[:, pi][:, :, :, None] - cen[:, pj][:, :, None], dim=-1) - r[pi][:, :, None] - r[pj][:, None]
        groups = [s.amin((2, 3))] + [d.amin(2).flatten(1) for d in _dist64(cen[:, has], r[has], st["world"].arrays())]
        soft = [-tau * torch.logsumexp(-g / tau, 1) for g in groups]
        js.append(torch.stack([torch.autograd.grad(v.sum(), x, retain_graph=True)[0] for v in soft], 1))
        ds.append(torch.stack([v.detach() for v in soft], 1))
    lead = st["x"].shape[:2]
    return dict(dist=torch.cat(ds).reshape(*lead, 5), jac=torch.cat(js).reshape(*lead, 5, m.n_act), traj=None, cost=None)


def exact(case, seed):
    k = case["kind"]
    if k not in ("check", "fk", "world", "traj", "sco"):
        return None
    st = prepare(case, seed)
    if k == "check":
        return _exact_check(st)
    if k == "fk":
        return torch.cat([_fk64(st["model"], q) for q in st["cfg"].split(20000)])
    if k == "world":
        return _exact_world(st)
    return _exact_traj(st) if k == "traj" else _exact_linearise(st)
