"""GPU parity of the trajectory cost and its hand-written adjoint: cost
against the FP64 oracle, gradient against the oracle's analytic smoothness /
limit gradient plus FP64 central differences of the collision cost
(relative error <= 1e-4), and the torch.autograd adapter."""

import numpy as np
import pytest
import torch

from error_report import record
from oracle import traj as otr
from pyroffi_b200 import workloads as W
from pyroffi_b200.trajopt import TrajectoryCost, TrajectoryCostFn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def setup(Bt=4, T=16, seed=1003):
    w = W.trajectories(Bt=Bt, T=T, seed=seed)
    tc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=w.margin, w_smooth=w.w_smooth,
                        w_acc=w.w_acc, w_jerk=w.w_jerk, w_limits=w.w_limits, w_coll=w.w_collision, device=DEV)
    return w, tc


def oracle_cost(w, x):
    return otr.total_cost(x, w.model.as_dict(), w.spheres.centers, w.spheres.radii, w.link_pairs, w.world.arrays(),
                          margin=w.margin, w_smooth=w.w_smooth, w_acc=w.w_acc, w_jerk=w.w_jerk,
                          w_limits=w.w_limits, w_coll=w.w_collision, lower=w.model.lower, upper=w.model.upper)


def test_cost_matches_oracle():
    w, tc = setup(Bt=16, T=32)
    c = tc.cost(torch.as_tensor(w.traj, device=DEV)).cpu().numpy()
    ref = np.array([oracle_cost(w, w.traj[b].astype(np.float64)) for b in range(16)])
    record("trajectory cost (relative)", np.abs(c - ref) / np.abs(ref), "16 x 32 x 7")
    np.testing.assert_allclose(c, ref, rtol=1e-4, atol=1e-5)
    wp = tc.waypoint_collision(torch.as_tensor(w.traj, device=DEV)).cpu().numpy()
    assert (wp > 0).any(), "the workload should touch obstacles"


@pytest.mark.parametrize("Ms", [1, 63, 64, 65, 129])
def test_cost_over_obstacle_chunks(Ms):
    """A lane tests its obstacles 32 at a time: counts around one and two chunks of a 4-lane group's
    share (4 x 32 = 128 obstacles) and partial ones, every sphere of the scene within reach."""
    w, _ = setup(Bt=2, T=6)
    w.world.spheres = W.random_sphere_world(np.random.default_rng(Ms), Ms, lo=-0.4, hi=0.4)
    tc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=w.margin, w_smooth=0.0, w_acc=0.0,
                        w_jerk=0.0, w_limits=0.0, w_coll=1.0, device=DEV)
    c = tc.cost(torch.as_tensor(w.traj, device=DEV)).cpu().numpy()
    ref = np.array([otr.collision_cost(w.traj[b], w.model.as_dict(), w.spheres.centers, w.spheres.radii, w.link_pairs,
                                       w.world.arrays(), w.margin) for b in range(2)])
    np.testing.assert_allclose(c, ref, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("n", [1, 31, 33, 65])
def test_listed_capsules_and_boxes(n):
    """A warp lists the capsules and boxes near its waypoints 32 at a time by their bounding spheres: counts
    around one and two rounds, long thin ones among them, some out of reach and some not; the cost of the
    launch without a gradient and of the one with it."""
    rng = np.random.default_rng(n)
    w, _ = setup(Bt=2, T=9)
    a = rng.uniform(-1.0, 1.0, (n, 3))
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    w.world.capsules = np.concatenate([a, a + rng.uniform(0.0, 2.0, (n, 1)) * u, rng.uniform(0.01, 0.1, (n, 1))],
                                      axis=1).astype(np.float32)
    axes = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    w.world.boxes = np.concatenate([rng.uniform(-1.5, 1.5, (n, 3)), axes.transpose(0, 2, 1).reshape(n, 9),
                                    rng.uniform(0.01, 0.7, (n, 3))], axis=1).astype(np.float32)
    tc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=w.margin, w_smooth=0.0, w_acc=0.0,
                        w_jerk=0.0, w_limits=0.0, w_coll=1.0, device=DEV)
    x = torch.as_tensor(w.traj, device=DEV)
    ref = np.array([otr.collision_cost(w.traj[b], w.model.as_dict(), w.spheres.centers, w.spheres.radii, w.link_pairs,
                                       w.world.arrays(), w.margin) for b in range(2)])
    np.testing.assert_allclose(tc.cost(x).cpu().numpy(), ref, rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(tc.cost_and_grad(x)[0].cpu().numpy(), ref, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("scale", [(0.5, 0.5, 0.5), (1.0, 0.3, 1.0)])
@pytest.mark.parametrize("n_boxes,every", [(12, 1), (40, 1), (40, 13)])
def test_boxes_with_short_axes(scale, n_boxes, every):
    """Axes shorter than 1, of all boxes or a few, stretch a box past its half lengths: none of it may be lost to
    the balls of a list (32 boxes and more, here)."""
    rng = np.random.default_rng(8)
    w, _ = setup(Bt=2, T=9)
    w.world.spheres = w.world.spheres[:1]
    w.world.boxes = W.random_boxes(rng, n_boxes, oriented=True)
    short = w.world.boxes[every - 1::every]
    short[:, 3:12] = (short[:, 3:12].reshape(-1, 3, 3) * np.array(scale, np.float32)[:, None]).reshape(-1, 9)
    tc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=w.margin, w_smooth=0.0, w_acc=0.0,
                        w_jerk=0.0, w_limits=0.0, w_coll=1.0, device=DEV)
    x = torch.as_tensor(w.traj, device=DEV)
    ref = np.array([otr.collision_cost(w.traj[b], w.model.as_dict(), w.spheres.centers, w.spheres.radii, w.link_pairs,
                                       w.world.arrays(), w.margin) for b in range(2)])
    np.testing.assert_allclose(tc.cost(x).cpu().numpy(), ref, rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(tc.cost_and_grad(x)[0].cpu().numpy(), ref, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("total", [700, 10000])
def test_worlds_with_and_without_a_list(total):
    """Spheres out of reach pad the world.  10,000 of them and two warps' lists of them are more than a block
    holds, so that every obstacle is tested: cost and gradient as of the world without the padding."""
    rng = np.random.default_rng(6)
    w, _ = setup(Bt=3, T=9)
    w.world.spheres = W.random_sphere_world(rng, 40, lo=-0.5, hi=0.5)
    w.world.capsules = W.random_capsules(rng, 9)
    w.world.boxes = W.random_boxes(rng, 9, oriented=True)
    x = torch.as_tensor(w.traj, device=DEV)
    make = lambda: TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=w.margin, w_smooth=0.0,  # noqa: E731
                                  w_acc=0.0, w_jerk=0.0, w_limits=0.0, w_coll=1.0, device=DEV)
    c, g = make().cost_and_grad(x)
    near = w.world.spheres
    w.world.spheres = np.tile(np.array([[100.0, 0, 0, 0.1]], np.float32), (total, 1))
    w.world.spheres[::total // len(near)][:len(near)] = near
    padded = make()
    c2, g2 = padded.cost_and_grad(x)
    np.testing.assert_allclose(c2.cpu().numpy(), c.cpu().numpy(), rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(padded.cost(x).cpu().numpy(), c.cpu().numpy(), rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(g2.cpu().numpy(), g.cpu().numpy(), rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("n_boxes", [0, 1])
def test_working_sets_around_48_kb(n_boxes, tmp_path, monkeypatch):
    """Worlds that take a block's working set past 48 KB in steps of 32 bytes, through a copy of the library
    whose kernels have not been launched with more before."""
    import shutil

    from pyroffi_b200 import _lib
    w, _ = setup(Bt=2, T=33)
    w.world.boxes = W.random_boxes(np.random.default_rng(0), n_boxes, oriented=True)
    x = torch.as_tensor(w.traj, device=DEV)
    monkeypatch.setattr(_lib, "LIB_PATH", type(_lib.LIB_PATH)(shutil.copy(_lib.LIB_PATH, tmp_path)))
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "_fns", {})
    for n in range(100, 420):
        w.world.spheres = np.tile(np.array([[100.0, 0, 0, 0.1]], np.float32), (n, 1))
        TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, device=DEV).cost(x)


def test_gradient_matches_finite_differences():
    w, tc = setup(Bt=3, T=12)
    x = torch.as_tensor(w.traj, device=DEV)
    c, g = tc.cost_and_grad(x)
    g = g.cpu().numpy().astype(np.float64)
    md = w.model.as_dict()
    for b in range(3):
        xb = w.traj[b].astype(np.float64)
        ref = (w.w_smooth * otr.smoothness_grad(xb, w.w_acc, w.w_jerk)
               + w.w_limits * otr.limits_grad(xb, w.model.lower, w.model.upper)
               + w.w_collision * otr.collision_grad_fd(xb, md, w.spheres.centers, w.spheres.radii, w.link_pairs,
                                                       w.world.arrays(), w.margin))
        rel = np.linalg.norm(g[b] - ref) / max(np.linalg.norm(ref), 1e-12)
        record("trajectory gradient vs FP64 finite differences (relative)", rel, "3 x 12 x 7, full cost")
        assert rel < 1e-4, (b, rel)
    # the fused launch and the separate ones agree
    np.testing.assert_allclose(tc.cost(x).cpu().numpy(), c.cpu().numpy(), rtol=0, atol=0)
    np.testing.assert_allclose(tc.grad(x).cpu().numpy(), g.astype(np.float32), rtol=0, atol=0)


def test_collision_gradient_alone_matches_fd():
    """Collision-only weights, waypoints that touch obstacles."""
    w, _ = setup(Bt=8, T=8)
    tc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=w.margin, w_smooth=0.0, w_acc=0.0,
                        w_jerk=0.0, w_limits=0.0, w_coll=1.0, device=DEV)
    x = torch.as_tensor(w.traj, device=DEV)
    wp = tc.waypoint_collision(x).cpu().numpy()
    b = int(np.argmax(wp.sum(1)))
    assert wp[b].sum() > 0
    g = tc.grad(x).cpu().numpy()[b].astype(np.float64)
    ref = otr.collision_grad_fd(w.traj[b].astype(np.float64), w.model.as_dict(), w.spheres.centers,
                                w.spheres.radii, w.link_pairs, w.world.arrays(), w.margin)
    rel = np.linalg.norm(g - ref) / np.linalg.norm(ref)
    record("trajectory gradient vs FP64 finite differences (relative)", rel, "8 x 8 x 7, collision only")
    assert rel < 1e-4, rel


def test_autograd_adapter():
    w, tc = setup(Bt=4, T=16)
    x = torch.as_tensor(w.traj, device=DEV).requires_grad_(True)
    J = TrajectoryCostFn.apply(x, tc)
    (J * torch.arange(1, 5, device=DEV, dtype=J.dtype)).sum().backward()
    _, g = tc.cost_and_grad(x.detach())
    np.testing.assert_allclose(x.grad.cpu().numpy(), (g * torch.arange(1, 5, device=DEV)[:, None, None]).cpu().numpy(),
                               rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("margin,n_spheres", [(0.01, 24), (0.3, 23)])
def test_all_obstacle_kinds_match_oracle(margin, n_spheres):
    """Spheres, capsules, oriented boxes and a halfspace (each kind has its own
    broad-phase loop; the spheres go two per packed test, so an odd count pads
    the last pair); the large margin keeps most (link, obstacle) pairs and puts
    link bounding centres inside boxes."""
    w = W.mixed_trajectories(Bt=6, T=12, n_spheres=n_spheres)
    tc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=margin, w_smooth=1.0, w_acc=0.5,
                        w_jerk=0.1, w_limits=1.0, w_coll=3.0, device=DEV)
    x = torch.as_tensor(w.traj, device=DEV)
    c, g = tc.cost_and_grad(x)
    md = w.model.as_dict()
    for b in range(6):
        xb = w.traj[b].astype(np.float64)
        ref = otr.total_cost(xb, md, w.spheres.centers, w.spheres.radii, w.link_pairs, w.world.arrays(),
                             margin=margin, w_smooth=1.0, w_acc=0.5, w_jerk=0.1, w_limits=1.0, w_coll=3.0,
                             lower=w.model.lower, upper=w.model.upper)
        assert abs(float(c[b]) - ref) <= 1e-4 * abs(ref) + 1e-5, (b, float(c[b]), ref)
    b = int(np.argmax(tc.waypoint_collision(x).cpu().numpy().sum(1)))
    tcc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=margin, w_smooth=0.0, w_acc=0.0,
                         w_jerk=0.0, w_limits=0.0, w_coll=1.0, device=DEV)
    gc = tcc.grad(x).cpu().numpy()[b].astype(np.float64)
    ref = otr.collision_grad_fd(w.traj[b].astype(np.float64), md, w.spheres.centers, w.spheres.radii, w.link_pairs,
                                w.world.arrays(), margin)
    assert np.linalg.norm(ref) > 0
    assert np.linalg.norm(gc - ref) / np.linalg.norm(ref) < 1e-4


def test_large_batch_two_lane_path_matches_oracle():
    """Batches above 2 x SMs run 2 lanes per waypoint (config 3 and the CHOMP
    line search take that path); smaller ones 4.  Both against the oracle, and
    against each other on the same trajectories."""
    w, tc = setup(Bt=320, T=16)
    x = torch.as_tensor(w.traj, device=DEV)
    c_big, g_big = tc.cost_and_grad(x)
    c_small, g_small = tc.cost_and_grad(x[:12].contiguous())
    np.testing.assert_allclose(c_big[:12].cpu().numpy(), c_small.cpu().numpy(), rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(g_big[:12].cpu().numpy(), g_small.cpu().numpy(), rtol=1e-4, atol=1e-5)
    idx = [0, 5, 77, 150, 233, 319]
    ref = np.array([oracle_cost(w, w.traj[b].astype(np.float64)) for b in idx])
    np.testing.assert_allclose(c_big.cpu().numpy()[idx], ref, rtol=1e-4, atol=1e-5)
    md = w.model.as_dict()
    for b in (77, 319):
        xb = w.traj[b].astype(np.float64)
        ref_g = (w.w_smooth * otr.smoothness_grad(xb, w.w_acc, w.w_jerk)
                 + w.w_limits * otr.limits_grad(xb, w.model.lower, w.model.upper)
                 + w.w_collision * otr.collision_grad_fd(xb, md, w.spheres.centers, w.spheres.radii, w.link_pairs,
                                                         w.world.arrays(), w.margin))
        rel = np.linalg.norm(g_big[b].cpu().numpy() - ref_g) / max(np.linalg.norm(ref_g), 1e-12)
        assert rel < 1e-4, (b, rel)


@pytest.mark.parametrize("T", [5, 8, 9])
@pytest.mark.parametrize("n_spheres", [3, 65])
def test_short_trajectories_in_large_batches(T, n_spheres):
    """Two lanes for each of up to 8 waypoints make blocks of half a warp (9: a whole one), whose candidate
    list needs its own shared memory: cost and gradient of a large batch as of its parts, which take four
    lanes, and as the oracle's.  All obstacles are within reach of the arm, capsules and boxes among them."""
    rng = np.random.default_rng(T)
    w = W.trajectories(Bt=320, T=T)
    w.world.spheres = W.random_sphere_world(rng, n_spheres, lo=-0.5, hi=0.5)
    w.world.capsules = W.random_capsules(rng, 7)
    w.world.boxes = W.random_boxes(rng, 5, oriented=True)
    tc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=w.margin, w_smooth=0.0, w_acc=0.0,
                        w_jerk=0.0, w_limits=0.0, w_coll=1.0, device=DEV)
    x = torch.as_tensor(w.traj, device=DEV)
    c, g = (v.cpu().numpy() for v in tc.cost_and_grad(x))
    np.testing.assert_array_equal(tc.cost(x).cpu().numpy(), c)
    part = [tc.cost_and_grad(x[i:i + 160].contiguous()) for i in (0, 160)]
    np.testing.assert_allclose(c, torch.cat([v[0] for v in part]).cpu().numpy(), rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(g, torch.cat([v[1] for v in part]).cpu().numpy(), rtol=1e-4, atol=1e-4)
    args = (w.model.as_dict(), w.spheres.centers, w.spheres.radii, w.link_pairs, w.world.arrays(), w.margin)
    ref = np.array([otr.collision_cost(w.traj[b].astype(np.float64), *args) for b in range(0, 320, 16)])
    np.testing.assert_allclose(c[::16], ref, rtol=1e-4, atol=1e-5)
    b = int(np.argmax(c))
    ref = otr.collision_grad_fd(w.traj[b].astype(np.float64), *args)
    assert np.linalg.norm(g[b] - ref) / np.linalg.norm(ref) < 1e-4


@pytest.mark.parametrize("per_link", [8, 16, 20])
def test_sphere_count_variants_match_oracle(per_link):
    """Kernels for up to 8, 16 and 32 spheres per link (register pairs)."""
    w = W.mixed_trajectories(Bt=3, T=10, per_link=per_link)
    margin = 0.05
    tc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=margin, w_smooth=1.0, w_acc=0.5,
                        w_jerk=0.1, w_limits=1.0, w_coll=3.0, device=DEV)
    x = torch.as_tensor(w.traj, device=DEV)
    c = tc.cost(x).cpu().numpy()
    md = w.model.as_dict()
    for b in range(3):
        ref = otr.total_cost(w.traj[b].astype(np.float64), md, w.spheres.centers, w.spheres.radii, w.link_pairs,
                             w.world.arrays(), margin=margin, w_smooth=1.0, w_acc=0.5, w_jerk=0.1, w_limits=1.0,
                             w_coll=3.0, lower=w.model.lower, upper=w.model.upper)
        assert abs(float(c[b]) - ref) <= 1e-4 * abs(ref) + 1e-5, (b, float(c[b]), ref)
    tcc = TrajectoryCost(w.model, w.spheres, w.world, w.link_pairs, margin=margin, w_smooth=0.0, w_acc=0.0,
                         w_jerk=0.0, w_limits=0.0, w_coll=1.0, device=DEV)
    b = int(np.argmax(tcc.waypoint_collision(x).cpu().numpy().sum(1)))
    g = tcc.grad(x).cpu().numpy()[b].astype(np.float64)
    ref = otr.collision_grad_fd(w.traj[b].astype(np.float64), md, w.spheres.centers, w.spheres.radii, w.link_pairs,
                                w.world.arrays(), margin)
    assert np.linalg.norm(ref) > 0
    assert np.linalg.norm(g - ref) / np.linalg.norm(ref) < 1e-4
