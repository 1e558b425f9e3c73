"""GPU parity of the LM IK kernels and the FP64 verification / winner
selection against the oracle.

The LM is iterative and its accept/reject and line-search decisions are
discontinuous, so an FP32 GPU run and the FP64 oracle can part ways on a
few seeds; the tests therefore check (a) one iteration seed by seed,
(b) the FP64 verification exactly, and (c) the solved problems' success
against the oracle's on the same inputs."""

import numpy as np
import pytest
import torch

from error_report import record
from oracle import kinematics as okin
from oracle import lm as olm
from pyroffi_b200 import robot as R
from pyroffi_b200 import workloads as W
from pyroffi_b200.cuda_kernels import ls_ik_cuda
from pyroffi_b200.ik import BatchIkSolver

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def tt(x, dtype=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device=DEV)


def small_ik(P=6, Sd=32, seed=1002):
    return W.ik(P=P, Sd=Sd, seed=seed)


def solver_for(w, **kw):
    opts = dict(max_iter=w.max_iter, lambda_init=w.lambda_init, lambda_down=w.lambda_down,
                lambda_up=w.lambda_up, collision_weight=w.collision_weight,
                collision_margin=w.collision_margin, pos_tol=w.pos_tol, rot_tol=w.rot_tol)
    opts.update(kw)
    return BatchIkSolver(w.model, w.target_link, spheres=w.spheres, world=w.world,
                         self_pairs=w.self_pairs, device=DEV, **opts)


def oracle_run(w, p, max_iter, seeds=None, lam_down=None, lam_up=None, self_pairs=True, coll=True,
               fixed_mask=None):
    m = w.model.as_dict()
    tj = w.model.link_joint(w.target_link)
    return olm.ls_ik(w.seeds[p] if seeds is None else seeds, w.target_T[p][None, None], m, [tj],
                     [w.model.ancestor_mask(w.target_link)], lower=w.model.lower, upper=w.model.upper,
                     fixed_mask=fixed_mask, max_iter=max_iter, lambda_init=w.lambda_init,
                     lambda_down=w.lambda_down if lam_down is None else lam_down,
                     lambda_up=w.lambda_up if lam_up is None else lam_up, enable_collision=coll,
                     collision_weight=w.collision_weight, collision_margin=w.collision_margin,
                     spheres_local=w.spheres_local, sphere_joint=w.sphere_joint, ws=w.world.spheres,
                     self_i=w.self_pairs[:, 0] if self_pairs else None,
                     self_j=w.self_pairs[:, 1] if self_pairs else None)


@pytest.mark.parametrize("tps", [0, 1, 2, 4, 5, 8])
@pytest.mark.parametrize("max_iter", [0, 1, 2])
def test_lm_few_iterations_seed_by_seed(tps, max_iter):
    w = small_ik(P=3, Sd=40)
    s = solver_for(w, max_iter=max_iter, threads_per_seed=tps)
    cfgs, errs = s.run_lm(tt(w.target_T), tt(w.seeds))
    cfgs, errs = cfgs.cpu().numpy(), errs.cpu().numpy()
    ok = 0
    for p in range(3):
        oc_, oe = oracle_run(w, p, max_iter)
        close = (np.abs(cfgs[p] - oc_).max(axis=1) < 2e-4) & (np.abs(errs[p] - oe) <= 1e-3 * np.abs(oe) + 1e-4)
        ok += close.sum()
    # decisions on the edge of the accept test may flip between FP32 and FP64
    assert ok >= 0.95 * 3 * 40, ok


@pytest.mark.parametrize("tps", [0, 2])
def test_lm_thirty_iterations_seed_by_seed(tps):
    """A whole 30-iteration solve, seed by seed, against the FP64 oracle: the
    FP64 normal equations keep the FP32 kernel on the oracle's path."""
    w = small_ik(P=3, Sd=40)
    s = solver_for(w, threads_per_seed=tps)
    cfgs, errs = s.run_lm(tt(w.target_T), tt(w.seeds))
    cfgs, errs = cfgs.cpu().numpy(), errs.cpu().numpy()
    ok = 0
    for p in range(3):
        oc_, oe = oracle_run(w, p, w.max_iter)
        close = (np.abs(cfgs[p] - oc_).max(axis=1) < 2e-4) & (np.abs(errs[p] - oe) <= 1e-3 * np.abs(oe) + 1e-4)
        ok += close.sum()
    record("IK seed disagreement with the FP64 oracle after 30 iterations (fraction)", 1.0 - ok / 120.0,
           f"3 x 40 seeds, threads_per_seed {tps}")
    assert ok >= 0.95 * 3 * 40, ok


@pytest.mark.parametrize("max_iter", [0, 1, 2, 30])
def test_lm_fp64_solve_seed_by_seed(max_iter):
    """The FP64 option of the damped step (the precision of the reference's
    normal equations) against the FP64 oracle, seed by seed."""
    w = small_ik(P=3, Sd=40)
    s = solver_for(w, max_iter=max_iter, fp64_solve=True)
    cfgs, errs = s.run_lm(tt(w.target_T), tt(w.seeds))
    cfgs, errs = cfgs.cpu().numpy(), errs.cpu().numpy()
    ok = 0
    for p in range(3):
        oc_, oe = oracle_run(w, p, max_iter)
        close = (np.abs(cfgs[p] - oc_).max(axis=1) < 2e-4) & (np.abs(errs[p] - oe) <= 1e-3 * np.abs(oe) + 1e-4)
        ok += close.sum()
    assert ok >= 0.95 * 3 * 40, ok


def test_lm_fp32_default_success_matches_fp64_solve():
    """30 iterations on 32 problems x 128 seeds: the default FP32 dual solve
    (with its conditional FP64 refinement) finds as many solutions (1 mm /
    0.01 rad, FP64-verified) as the FP64 solve, within 2."""
    w = small_ik(P=32, Sd=128)
    r64 = solver_for(w, fp64_solve=True).solve(tt(w.target_T), tt(w.seeds))
    r32 = solver_for(w).solve(tt(w.target_T), tt(w.seeds))
    n64, n32 = int(r64.success.sum()), int(r32.success.sum())
    assert n32 >= n64 - 2, (n32, n64)


@pytest.mark.parametrize("tps", [0, 2])
@pytest.mark.parametrize("max_iter", [2, 30])
def test_lm_fixed_joints_seed_by_seed(tps, max_iter):
    """Joints 0 and 5 fixed: 5 free columns against 6 residual rows, so the
    damped step goes through the primal system (the dual one would be
    rank-deficient); seed by seed against the FP64 oracle, and the fixed
    joints keep their seed values."""
    w = small_ik(P=3, Sd=40)
    mask = np.zeros(w.model.n_act, np.int32)
    mask[[0, 5]] = 1
    s = solver_for(w, max_iter=max_iter, threads_per_seed=tps)
    s.set_fixed_mask(mask)
    cfgs, errs = s.run_lm(tt(w.target_T), tt(w.seeds))
    cfgs, errs = cfgs.cpu().numpy(), errs.cpu().numpy()
    np.testing.assert_array_equal(cfgs[..., [0, 5]], w.seeds[..., [0, 5]])
    ok = 0
    for p in range(3):
        oc_, oe = oracle_run(w, p, max_iter, fixed_mask=mask)
        close = (np.abs(cfgs[p] - oc_).max(axis=1) < 2e-4) & (np.abs(errs[p] - oe) <= 1e-3 * np.abs(oe) + 1e-4)
        ok += close.sum()
    record("IK seed disagreement with the FP64 oracle, joints 0 and 5 fixed (fraction)", 1.0 - ok / 120.0,
           f"3 x 40 seeds, {max_iter} iterations, threads_per_seed {tps}")
    assert ok >= 0.95 * 3 * 40, ok


@pytest.mark.parametrize("tps", [0, 2])
def test_lm_obstacle_grid_resolution_leaves_results_unchanged(tps):
    """The default grid of the 100-sphere world (14 cells per axis), 8 and 10
    cells, 16 cells (whose lists overflow their capacity here and fall back
    to 8) and no grid: the grid only decides which obstacles take the
    bounding test.  With one lane per seed each joint's hinge terms are
    summed in increasing obstacle order, so the bits are the same; lanes
    sharing a seed take the candidates by list position, so their partial
    sums may round differently."""
    w = small_ik(P=4, Sd=64)
    s = solver_for(w, max_iter=8, threads_per_seed=tps)
    base = None
    for grid in (0, 8, 10, 16, -1):
        s.opt.obstacle_grid = grid
        c, e = s.run_lm(tt(w.target_T), tt(w.seeds))
        if base is None:
            base = (c.clone(), e.clone())
        elif tps == 0:
            assert torch.equal(c, base[0]) and torch.equal(e, base[1]), grid
        else:
            a, b = e.cpu().numpy(), base[1].cpu().numpy()
            assert np.mean(np.abs(a - b) <= 1e-4 * np.abs(b) + 1e-5) >= 0.95, grid


@pytest.mark.parametrize("n_obstacles", [40, 600])
def test_lm_grid_offsets_in_small_blocks(n_obstacles):
    """Blocks of 32 seeds have few pose slots, and the grid's 16-bit offsets are made in the place of the 32-bit
    ones: the bits are the same with every grid and without one."""
    w = W.ik(P=2, Sd=40, n_obstacles=n_obstacles)
    s = solver_for(w, max_iter=4, threads_per_seed=1, seeds_per_block=32)
    base = None
    for grid in (-1, 0, 1, 9, 14, 16):
        s.opt.obstacle_grid = grid
        c, e = s.run_lm(tt(w.target_T), tt(w.seeds))
        if base is None:
            base = c, e
        assert torch.equal(c, base[0]) and torch.equal(e, base[1]), grid


def test_lm_fp64_solve_rejects_other_mappings():
    w = small_ik(P=1, Sd=8)
    with pytest.raises(Exception, match="fp64_solve"):
        solver_for(w, fp64_solve=True, threads_per_seed=2).run_lm(tt(w.target_T), tt(w.seeds))


def test_lm_initial_error_matches_oracle_exactly_enough():
    w = small_ik(P=4, Sd=64)
    s = solver_for(w, max_iter=0)
    cfgs, errs = s.run_lm(tt(w.target_T), tt(w.seeds))
    np.testing.assert_array_equal(cfgs.cpu().numpy(), w.seeds)
    for p in range(4):
        _, oe = oracle_run(w, p, 0)
        np.testing.assert_allclose(errs[p].cpu().numpy(), oe, rtol=2e-5, atol=1e-5)


def test_verify_select_fp64():
    w = small_ik(P=8, Sd=16)
    s = solver_for(w)
    rng = np.random.default_rng(4)
    cfgs = np.clip(w.target_cfgs[:, None, :] + rng.normal(0, 1e-3, size=(8, 16, 7)), -2.8, 2.8).astype(np.float32)
    errs = rng.uniform(0, 1, size=(8, 16)).astype(np.float32)
    errs[3, 5] = errs[3, 9] = -1.0                      # tie -> smallest seed index
    winner, pos, rot, ok = s.verify_select(tt(cfgs), tt(errs), tt(w.target_T))
    idx = np.argmin(errs, axis=1)
    assert idx[3] == 5
    np.testing.assert_array_equal(winner.cpu().numpy(), cfgs[np.arange(8), idx])
    pe, re = olm.pose_errors(cfgs[np.arange(8), idx].astype(np.float64), w.target_T.astype(np.float64),
                             w.model.as_dict(), w.model.link_joint(w.target_link))
    np.testing.assert_allclose(pos.cpu().numpy(), pe, rtol=1e-9, atol=1e-12)
    np.testing.assert_allclose(rot.cpu().numpy(), re, rtol=1e-7, atol=1e-10)
    np.testing.assert_array_equal(ok.cpu().numpy(), ((pe < 1e-3) & (re < 1e-2)).astype(np.int32))


def test_continuity_weight_selection():
    w = small_ik(P=2, Sd=8)
    s = solver_for(w)
    cfgs = np.tile(w.seeds[:, :1], (1, 8, 1)) + np.arange(8)[None, :, None] * 0.1
    errs = np.zeros((2, 8), np.float32)
    prev = cfgs[:, 5]
    winner, *_ = s.verify_select(tt(cfgs), tt(errs), tt(w.target_T), prev=tt(prev), continuity_weight=1.0)
    np.testing.assert_allclose(winner.cpu().numpy(), prev, atol=0)


def test_full_solve_success_matches_oracle():
    """Config-2 semantics on 8 problems x 64 seeds: GPU success >= oracle's - 1."""
    w = small_ik(P=8, Sd=64)
    s = solver_for(w)
    res = s.solve(tt(w.target_T), tt(w.seeds))
    gpu_ok = int(res.success.sum())
    m = w.model.as_dict()
    tj = w.model.link_joint(w.target_link)
    or_ok = 0
    best_agree = 0
    gpu_best = res.errs.min(dim=1).values.cpu().numpy()
    for p in range(8):
        oc_, oe = oracle_run(w, p, w.max_iter)
        win, _ = olm.select_winner(oc_[None], oe[None])
        pe, re = olm.pose_errors(win, w.target_T[p][None].astype(np.float64), m, tj)
        or_ok += int(pe[0] < 1e-3 and re[0] < 1e-2)
        best_agree += int(abs(gpu_best[p] - oe.min()) <= 1e-3 * abs(oe.min()) + 1e-6)
    assert gpu_ok >= or_ok - 1, (gpu_ok, or_ok)
    # the best weighted error found per problem agrees with the oracle's
    assert best_agree >= 6, best_agree


def test_drop_in_ls_ik_cuda_reference_semantics():
    """pk_ls_ik_cuda: reference damping (x0.5 / x3), no self pairs, world spheres."""
    w = small_ik(P=3, Sd=32)
    md = w.model
    tj = md.link_joint(w.target_link)
    anc = md.ancestor_mask(w.target_link)[None]
    z = lambda k: tt(np.zeros((0, k), np.float32))  # noqa: E731
    cfgs, errs = ls_ik_cuda(
        tt(w.seeds), tt(md.twists), tt(md.parent_tf), tt(md.parent_idx, torch.int32), tt(md.act_idx, torch.int32),
        tt(md.mimic_mul), tt(md.mimic_off), tt(md.mimic_act_idx, torch.int32), tt(md.topo_inv, torch.int32),
        tt([tj], torch.int32), tt(anc, torch.int32), tt(w.target_T[:, None, :]), tt(w.spheres_local),
        tt(w.sphere_joint, torch.int32), tt(w.world.spheres), z(7), z(15), z(6), tt(md.lower), tt(md.upper),
        tt(np.zeros(7), torch.int32), max_iter=2, pos_weight=50.0, ori_weight=10.0, lambda_init=5e-3,
        eps_pos=1e-8, eps_ori=1e-8, enable_collision=True, collision_weight=1e4, collision_margin=0.02)
    cfgs, errs = cfgs.cpu().numpy(), errs.cpu().numpy()
    ok = 0
    for p in range(3):
        m = md.as_dict()
        oc_, oe = olm.ls_ik(w.seeds[p], w.target_T[p][None, None], m, [tj], [anc[0]], lower=md.lower,
                            upper=md.upper, max_iter=2, lambda_init=5e-3, enable_collision=True,
                            collision_weight=1e4, collision_margin=0.02, spheres_local=w.spheres_local,
                            sphere_joint=w.sphere_joint, ws=w.world.spheres)
        ok += ((np.abs(cfgs[p] - oc_).max(axis=1) < 2e-4) & (np.abs(errs[p] - oe) <= 1e-3 * np.abs(oe) + 1e-4)).sum()
    assert ok >= 0.95 * 96, ok


def test_tree_robot_two_ees():
    """15-DOF bimanual tree, two EE targets (16-DOF kernel bucket)."""
    rng = np.random.default_rng(21)
    model = R.bimanual_tree(rng)
    links = (10, 16)
    P, Sd = 4, 48
    tcfg = model.random_cfgs(rng, P)
    m = model.as_dict()
    Tj = okin.fk_joints(tcfg, m["twists"], m["parent_tf"], m["parent_idx"], m["act_idx"], m["mimic_mul"],
                        m["mimic_off"], m["mimic_act_idx"], m["topo_inv"])
    tj = [model.link_joint(l) for l in links]
    target = Tj[:, tj].astype(np.float32)                 # [P, 2, 7]
    seeds = model.random_cfgs(rng, P * Sd).reshape(P, Sd, -1)
    s = BatchIkSolver(model, links, max_iter=40, lambda_init=1e-2, lambda_down=0.1, lambda_up=10.0, device=DEV)
    res = s.solve(tt(target), tt(seeds))
    cfgs, errs = res.cfgs.cpu().numpy(), res.errs.cpu().numpy()
    anc = [model.ancestor_mask(l) for l in links]
    agree = 0
    for p in range(P):
        oc_, oe = olm.ls_ik(seeds[p], target[p][None], m, tj, anc, lower=model.lower, upper=model.upper,
                            max_iter=1, lambda_init=1e-2, lambda_down=0.1, lambda_up=10.0)
        s1 = BatchIkSolver(model, links, max_iter=1, lambda_init=1e-2, lambda_down=0.1, lambda_up=10.0, device=DEV)
        c1, e1 = s1.run_lm(tt(target[p:p + 1]), tt(seeds[p:p + 1]))
        agree += (np.abs(c1.cpu().numpy()[0] - oc_).max(axis=1) < 2e-4).sum()
    assert agree >= 0.95 * P * Sd
    # FP64 re-check of the winners matches the oracle
    idx = np.argmin(errs, axis=1)
    win = cfgs[np.arange(P), idx].astype(np.float64)
    Tw = okin.fk_joints(win, m["twists"], m["parent_tf"], m["parent_idx"], m["act_idx"], m["mimic_mul"],
                        m["mimic_off"], m["mimic_act_idx"], m["topo_inv"])
    pe = np.max(np.linalg.norm(Tw[:, tj, 4:] - target[..., 4:], axis=-1), axis=1)
    np.testing.assert_allclose(res.pos_err.cpu().numpy(), pe, rtol=1e-6, atol=1e-9)


@pytest.mark.parametrize("max_iter", [1, 3])
def test_tree_robot_two_ees_fixed_joints(max_iter):
    """15-DOF bimanual tree, two EE targets, five joints fixed: 10 free
    columns against 12 residual rows, so the 16-DOF kernel solves the primal
    system (out of line) instead of its usual dual one; seed by seed against
    the FP64 oracle with the same fixed joints."""
    rng = np.random.default_rng(23)
    model = R.bimanual_tree(rng)
    links = (10, 16)
    P, Sd = 3, 32
    tcfg = model.random_cfgs(rng, P)
    m = model.as_dict()
    Tj = okin.fk_joints(tcfg, m["twists"], m["parent_tf"], m["parent_idx"], m["act_idx"], m["mimic_mul"],
                        m["mimic_off"], m["mimic_act_idx"], m["topo_inv"])
    tj = [model.link_joint(l) for l in links]
    target = Tj[:, tj].astype(np.float32)
    seeds = model.random_cfgs(rng, P * Sd).reshape(P, Sd, -1).astype(np.float32)
    mask = np.zeros(model.n_act, np.int32)
    mask[[0, 3, 6, 9, 12]] = 1
    s = BatchIkSolver(model, links, max_iter=max_iter, lambda_init=1e-2, lambda_down=0.1, lambda_up=10.0,
                      device=DEV)
    s.set_fixed_mask(mask)
    cfgs, errs = s.run_lm(tt(target), tt(seeds))
    cfgs, errs = cfgs.cpu().numpy(), errs.cpu().numpy()
    np.testing.assert_array_equal(cfgs[..., mask == 1], seeds[..., mask == 1])
    anc = [model.ancestor_mask(l) for l in links]
    ok = 0
    for p in range(P):
        oc_, oe = olm.ls_ik(seeds[p], target[p][None], m, tj, anc, lower=model.lower, upper=model.upper,
                            fixed_mask=mask, max_iter=max_iter, lambda_init=1e-2, lambda_down=0.1,
                            lambda_up=10.0)
        ok += ((np.abs(cfgs[p] - oc_).max(axis=1) < 2e-4) & (np.abs(errs[p] - oe) <= 1e-3 * np.abs(oe) + 1e-4)).sum()
    assert ok >= 0.95 * P * Sd, ok


def test_lm_ragged_seed_counts():
    """Seeds per problem not a multiple of the block's seed count."""
    w = small_ik(P=2, Sd=37)
    s = solver_for(w, max_iter=1, threads_per_seed=4)
    cfgs, errs = s.run_lm(tt(w.target_T), tt(w.seeds))
    _, oe = oracle_run(w, 1, 1)
    assert np.isfinite(errs.cpu().numpy()).all()
    close = np.abs(errs[1].cpu().numpy() - oe) <= 1e-3 * np.abs(oe) + 1e-4
    assert close.mean() >= 0.9


@pytest.mark.parametrize("Sd", [1, 31, 129])
@pytest.mark.parametrize("n_self", [0, 7, 200])
@pytest.mark.parametrize("iters", [0, 3])
def test_trial_lanes_equal_one_lane(Sd, n_self, iters):
    """Two trial lanes per seed (the default mapping) against one lane per seed (asked for by
    seeds_per_block): the same evaluations, so the same results but for roundings that the compiler
    places differently in the two kernels."""
    w = W.ik(P=3, Sd=Sd, n_self=n_self)
    kw = dict(spheres=w.spheres, world=w.world, self_pairs=w.self_pairs, max_iter=iters, lambda_init=w.lambda_init,
              lambda_down=w.lambda_down, lambda_up=w.lambda_up, device=DEV)
    a = BatchIkSolver(w.model, w.target_link, **kw).run_lm(tt(w.target_T), tt(w.seeds))
    b = BatchIkSolver(w.model, w.target_link, threads_per_seed=1, seeds_per_block=128, **kw).run_lm(tt(w.target_T),
                                                                                                   tt(w.seeds))
    close = ((a[0] - b[0]).abs().amax(-1) < 2e-4) & ((a[1] - b[1]).abs() <= 1e-3 * b[1].abs() + 1e-4)
    assert close.float().mean() >= 0.97


def test_negative_collision_weight_takes_one_lane():
    """With a negative weight the skipped trials depend on the order they are seen in: one lane per seed."""
    w = W.ik(P=3, Sd=64)
    kw = dict(spheres=w.spheres, world=w.world, self_pairs=w.self_pairs, max_iter=4, lambda_init=w.lambda_init,
              lambda_down=w.lambda_down, lambda_up=w.lambda_up, collision_weight=-1e4, device=DEV)
    a = BatchIkSolver(w.model, w.target_link, **kw).run_lm(tt(w.target_T), tt(w.seeds))
    b = BatchIkSolver(w.model, w.target_link, threads_per_seed=1, seeds_per_block=128, **kw).run_lm(tt(w.target_T),
                                                                                                   tt(w.seeds))
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
