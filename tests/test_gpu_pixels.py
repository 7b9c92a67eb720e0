"""Multi-pose pixel-list renderer with optical flow (fm_render.py render_func_idx_quattrans and
_flow, argument order fixed) against the float64 oracle, and against the image renderer."""

import numpy as np
import pytest
import torch

import fuzzy_ellipses as fe
from fuzzy_ellipses import synthetic as S
from oracle import fm_render_np as O
from tests.helpers import TOL_ALPHA, TOL_DEPTH_REL, DEPTH_MASK_ALPHA, scene_to_dev

pytestmark = pytest.mark.gpu


def pose_list(cams):
    return np.stack([np.concatenate([c.quat, c.trans]) for c in cams]).astype(np.float32)


def grid_rays(H, W, k, step=1):
    v, u = np.mgrid[0:H:step, 0:W:step]
    n = u.size
    return np.stack([u.ravel() - W / 2, v.ravel() - H / 2, np.ones(n), np.full(n, k)], 1)


def test_mixed_pose_rays_match_oracle_with_flow(cuda_device):
    rng = np.random.default_rng(0)
    scene, cams = S.config0(seed=3)
    cams = [S.Camera(64, 64, 64.0, 64.0, 32.0, 32.0, *S.look_at(0.5 * d))
            for d in S.random_unit_vectors(3, rng)]
    poses = pose_list(cams)
    inv_f = 1.0 / 64.0
    rays = np.concatenate([grid_rays(64, 64, k, step=2) for k in range(3)])
    rays = rays[rng.permutation(len(rays))].astype(np.float32)  # poses interleaved
    m, p, w = scene_to_dev(scene, cuda_device)
    d, a, _, _, fp, fm = fe.render_pixels(m, p, w, torch.from_numpy(rays), inv_f,
                                          torch.from_numpy(poses), flow=True)
    d, a, fp, fm = (x.cpu().numpy().astype(np.float64) for x in (d, a, fp, fm))
    rd, ra, _, _, rfp, rfm = O.render_func_idx_quattrans_flow(scene.means, scene.prec,
                                                              scene.logw, rays, inv_f, poses,
                                                              21.4, 2.66)
    assert np.max(np.abs(a - ra)) <= TOL_ALPHA
    mask = ra > DEPTH_MASK_ALPHA
    assert np.max(np.abs(d - rd)[mask] / rd[mask]) <= TOL_DEPTH_REL
    # the flow arithmetic itself (given the depths): float32 against float64
    # (a depth-0 ray whose neighbour pose clamps to its own pose reprojects 0/0: NaN, as in the
    # reference; the NaNs must sit on the same rays)
    with np.errstate(invalid="ignore"):
        gfp, gfm = O.flow_from_depth(rays, inv_f, poses, d)
    for got, want in ((fp, gfp), (fm, gfm)):
        assert np.array_equal(np.isnan(got), np.isnan(want))
        ok = ~np.isnan(want)
        assert np.max(np.abs(got - want)[ok]) <= 1e-3
    # and end to end where depth is defined
    assert np.max(np.abs(fp - rfp)[mask]) <= 2e-2 and np.max(np.abs(fm - rfm)[mask]) <= 2e-2


def test_pixel_grid_equals_image_render(cuda_device):
    scene, cams = S.config0(seed=4)
    c = cams[0]
    H, W, f = 48, 80, 60.0
    m, p, w = scene_to_dev(scene, cuda_device)
    rays = grid_rays(H, W, 0).astype(np.float32)
    pose = pose_list([c])
    d, a, _, _ = fe.render_pixels(m, p, w, torch.from_numpy(rays), 1.0 / f, torch.from_numpy(pose))
    di, ai = fe.render_forward(m, p, w, f, f, W / 2, H / 2, c.quat, c.trans, H, W)
    assert torch.allclose(a.reshape(H, W), ai, atol=2e-6, rtol=0)
    ok = ai > DEPTH_MASK_ALPHA
    assert torch.allclose(d.reshape(H, W)[ok], di[ok], rtol=2e-5, atol=0)


def test_scaled_rays_weights_and_features(cuda_device):
    """Rays (x c, y c, c): the same line as (x, y, 1), so alpha is unchanged, while the ray
    parameter (and with it the softmax logits -beta2 z) scales by 1/c, as in fm_render; depth,
    the dense weights and the weighted features agree with the oracle's."""
    rng = np.random.default_rng(5)
    scene, cams = S.config0(seed=5)
    c = cams[0]
    pose = pose_list([c])
    inv_f = 1.0 / 40.0
    base = grid_rays(40, 40, 0, step=3)
    scaled = base.copy()
    scaled[:, :3] *= 2.0
    feats = rng.normal(size=(scene.n, 5)).astype(np.float32)
    m, p, w = scene_to_dev(scene, cuda_device)
    out1 = fe.render_pixels(m, p, w, torch.from_numpy(base.astype(np.float32)), inv_f,
                            torch.from_numpy(pose))
    out2 = fe.render_pixels(m, p, w, torch.from_numpy(scaled.astype(np.float32)), inv_f,
                            torch.from_numpy(pose), weights=True, features=torch.from_numpy(feats))
    d1, a1 = out1[0].cpu().numpy(), out1[1].cpu().numpy()
    d2, a2, wts, of = out2[0].cpu().numpy(), out2[1].cpu().numpy(), out2[3].cpu().numpy(), out2[4].cpu().numpy()
    assert np.allclose(a2, a1, atol=1e-6)
    rd, ra, _, rw = O.render_func_idx_quattrans(scene.means, scene.prec, scene.logw, scaled, inv_f,
                                                pose, 21.4, 2.66, return_weights=True)
    mask = ra > DEPTH_MASK_ALPHA
    assert np.max(np.abs(a2 - ra)) <= TOL_ALPHA
    assert np.max(np.abs(d2 - rd)[mask] / rd[mask]) <= TOL_DEPTH_REL
    assert np.max(np.abs(wts - rw)[:, mask]) <= 1e-4
    assert np.allclose(wts.sum(0)[mask], 1.0, atol=1e-5)
    assert np.max(np.abs(of - (rw.T @ feats.astype(np.float64)))[mask]) <= 1e-3


@pytest.mark.parametrize("n,n_rays,n_poses", [(41, 20011, 3), (130, 12345, 70), (1100, 9729, 1),
                                             (500, 40001, 70)])
def test_long_lists_match_their_pieces(cuda_device, n, n_rays, n_poses):
    """A ray's result does not depend on the list around it: a long shuffled list (bucketed by
    pose and cell, 64 rays per warp or fewer) equals, bit for bit, the same rays rendered in short
    pieces (a few rays per warp, in the order given); a sample agrees with the oracle."""
    rng = np.random.default_rng(n)
    scene = S.random_gaussians(n, 0.15, rng)
    cams = [S.Camera(96, 160, 120.0, 120.0, 80.0, 48.0, *S.look_at(0.6 * d))
            for d in S.random_unit_vectors(n_poses, rng)]
    poses, inv_f = pose_list(cams), 1.0 / 120.0
    rays = np.stack([rng.uniform(-90, 90, n_rays), rng.uniform(-60, 60, n_rays), np.ones(n_rays),
                     rng.integers(0, n_poses, n_rays)], 1).astype(np.float32)
    m, p, w = scene_to_dev(scene, cuda_device)
    feats = torch.from_numpy(rng.normal(size=(n, 5)).astype(np.float32))
    rd, pd = torch.from_numpy(rays), torch.from_numpy(poses)
    whole = fe.render_pixels(m, p, w, rd, inv_f, pd, flow=True, features=feats)
    for lo, hi in ((0, 1), (1, 63), (63, 127), (127, 5000), (5000, n_rays - 7001),
                   (n_rays - 33, n_rays)):
        part = fe.render_pixels(m, p, w, rd[lo:hi], inv_f, pd, flow=True, features=feats)
        for x, y in zip(whole, part):
            if x is not None:
                torch.testing.assert_close(x[lo:hi], y, rtol=0, atol=0, equal_nan=True)
    pick = rng.choice(n_rays, 200, replace=False)
    ref_d, ref_a, _, _ = O.render_func_idx_quattrans(scene.means, scene.prec, scene.logw,
                                                     rays[pick], inv_f, poses, 21.4, 2.66)
    d, a = (x.cpu().numpy().astype(np.float64)[pick] for x in whole[:2])
    seen = ref_a > DEPTH_MASK_ALPHA
    assert np.max(np.abs(a - ref_a)) <= TOL_ALPHA
    assert np.max(np.abs(d - ref_d)[seen] / ref_d[seen]) <= TOL_DEPTH_REL


@pytest.mark.parametrize("n,n_poses,step", [(60, 2, 2), (700, 3, 1), (1000, 1, 9)])
def test_culled_lists_equal_the_thread_per_ray_kernel(cuda_device, n, n_poses, step):
    """With dense weights every ray tests every Gaussian by itself, with IEEE divisions; without
    them warps cull for their rays and evaluate in pairs. Depth and alpha are the same bits: the
    same operations in the same order."""
    rng = np.random.default_rng(n)
    scene = S.random_gaussians(n, 0.3, rng)
    cams = [S.Camera(120, 160, 150.0, 150.0, 80.0, 60.0, *S.look_at(1.0 * d))
            for d in S.random_unit_vectors(n_poses, rng)]
    rays = np.concatenate([grid_rays(120, 160, k, step) for k in range(n_poses)]).astype(np.float32)
    args = scene_to_dev(scene, cuda_device) + (torch.from_numpy(rays).to(cuda_device), 1.0 / 150.0,
                                               torch.from_numpy(pose_list(cams)).to(cuda_device))
    d0, a0 = fe.render_pixels(*args, weights=True)[:2]
    d1, a1 = fe.render_pixels(*args)[:2]
    assert torch.equal(d0, d1) and torch.equal(a0, a1)


@pytest.mark.parametrize("thickness", [8e-20, 1e19])
def test_discs_at_the_ends_of_the_float_range(cuda_device, thickness):
    """Discs facing the camera whose precision along the view is the reciprocal of 8e-20 or 1e19:
    the squared ray term is then within a factor of 4 of the largest or smallest normal float32,
    and its reciprocal is not normal. Depths as with the division (which has 22 bits there)."""
    n, rng = 60, np.random.default_rng(1)
    means = np.concatenate([rng.uniform(-0.2, 0.2, (n, 2)), rng.uniform(0.8, 1.2, (n, 1))], 1)
    prec = np.tile(np.diag([1.0, 1.0, 1.0 / thickness]), (n, 1, 1))
    if thickness > 1:
        prec[:, 0, 0] = prec[:, 1, 1] = 0.02 / thickness
    arrays = [torch.from_numpy(x.astype(np.float32)).to(cuda_device)
              for x in (means, prec, rng.normal(0, 0.5, n))]
    rays = torch.from_numpy(grid_rays(100, 100, 0, 2).astype(np.float32)).to(cuda_device)
    pose = torch.tensor([[1.0, 0, 0, 0, 0, 0, 0]], device=cuda_device)
    d0, a0 = fe.render_pixels(*arrays, rays, 0.01, pose, weights=True)[:2]
    d1, a1 = fe.render_pixels(*arrays, rays, 0.01, pose)[:2]
    assert float(d0.max()) > 0.5 and bool(torch.isfinite(d0).all())
    assert bool(((d1 - d0).abs() <= 2e-5 * d0.abs()).all())
    assert bool(((a1 - a0).abs() <= 2e-5).all())


@pytest.mark.parametrize("step", [1, 2])
def test_list_features_do_not_depend_on_the_kernel(cuda_device, step):
    """Features of the culled kernel and of the thread-per-ray one (taken with dense weights) are the
    same bits. A Gaussian whose weight underflows still multiplies its feature, so an infinite one
    gives NaN along its rays in both."""
    n, rng = 600, np.random.default_rng(2)
    scene = S.random_gaussians(n, 0.2, rng)
    means = scene.means.copy()
    prec = scene.prec.copy()
    means[-1], prec[-1] = [0.0, 0.0, 9.0], np.eye(3)  # 10 m away: e^-200 of the others' weight
    m, p, w = (torch.from_numpy(x).to(cuda_device) for x in (means, prec, scene.logw))
    feats = rng.normal(size=(n, 5)).astype(np.float32)
    feats[-1, 2] = np.inf
    pose = torch.tensor([[1.0, 0, 0, 0, 0, 0, -1.0]], device=cuda_device)
    rays = torch.from_numpy(grid_rays(120, 120, 0, step).astype(np.float32)).to(cuda_device)
    args = (m, p, w, rays, 1.0 / 120.0, pose)
    feats = torch.from_numpy(feats).to(cuda_device)
    f0 = fe.render_pixels(*args, weights=True, features=feats)[4]
    f1 = fe.render_pixels(*args, features=feats)[4]
    assert bool(torch.isnan(f0[:, 2]).any()) and not bool(torch.isnan(f0[:, :2]).any())
    assert torch.equal(torch.isnan(f0), torch.isnan(f1))
    assert torch.equal(torch.nan_to_num(f0), torch.nan_to_num(f1))


@pytest.mark.parametrize("n,n_rays,nf", [(41, 3000, 3), (129, 3000, 0), (600, 3000, 7),
                                         (600, 12000, 7), (1153, 200000, 0)])
def test_rays_in_the_camera_plane_leave_the_others_alone(cuda_device, n, n_rays, nf):
    """Rays with c = 0 have infinite pixel offsets, so the box around a warp's rays can be the whole
    plane. The warp still takes the pose's own Gaussians only (their number is no multiple of the 128
    it looks at together, and the next pose's follow): every ray has the bits of the kernel that tests
    each Gaussian for each ray."""
    rng = np.random.default_rng(n)
    scene = S.random_gaussians(n, 0.3, rng)
    cams = [S.Camera(100, 100, 100.0, 100.0, 50.0, 50.0, *S.look_at(0.6 * d))
            for d in S.random_unit_vectors(4, rng)]
    rays = np.concatenate([rng.uniform(-50, 50, (n_rays, 2)), np.ones((n_rays, 1)),
                           rng.integers(0, 4, (n_rays, 1))], 1).astype(np.float32)
    rays[::3, 2] = 0.0
    m, p, w = scene_to_dev(scene, cuda_device)
    rays = torch.from_numpy(rays).to(cuda_device)
    feats = torch.from_numpy(rng.normal(size=(n, nf)).astype(np.float32)).to(cuda_device) if nf else None
    args = (m, p, w, rays, 0.01, torch.from_numpy(pose_list(cams)).to(cuda_device))
    want = fe.render_pixels(*args, weights=True, features=feats)
    got = fe.render_pixels(*args, features=feats)
    for i in (0, 1, 4)[:3 if nf else 2]:
        assert torch.equal(torch.isnan(want[i]), torch.isnan(got[i]))
        assert torch.equal(torch.nan_to_num(want[i]), torch.nan_to_num(got[i]))


def test_overflow_does_not_depend_on_the_kernel(cuda_device):
    """Gaussians 1e36 and 1e19 m away overflow the ray products: depth and alpha are NaN at the same
    rays with the culled kernel and the thread-per-ray one, and the same bits elsewhere."""
    n, rng = 300, np.random.default_rng(6)
    scene = S.random_gaussians(n, 0.2, rng)
    means, prec = scene.means.copy(), scene.prec.copy()
    prec[::3] *= 0.02
    means[::10, 0], means[5::20, 2] = 1e36, -1e19
    m, p, w = (torch.from_numpy(x).to(cuda_device) for x in (means, prec, scene.logw))
    poses = np.stack([np.concatenate(S.look_at(0.15 * d)) for d in S.random_unit_vectors(3, rng)])
    rays = np.concatenate([grid_rays(50, 60, k) for k in range(3)]).astype(np.float32)
    args = (m, p, w, torch.from_numpy(rays).to(cuda_device), 0.02,
            torch.from_numpy(poses.astype(np.float32)).to(cuda_device))
    want = fe.render_pixels(*args, weights=True)[:2]
    assert bool(torch.isnan(want[0]).any())
    for a, b in zip(want, fe.render_pixels(*args)[:2]):
        assert torch.equal(torch.isnan(a), torch.isnan(b))
        assert torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
