"""Softmax-weighted features of an image render (fm_render's w applied to per-Gaussian features)
against the float64 oracle's w @ f, against the pixel-list path, and the weight sum."""

import numpy as np
import pytest
import torch

import fuzzy_ellipses as fe
from fuzzy_ellipses import synthetic as S
from oracle import fm_render_np as O
from tests.helpers import DEPTH_MASK_ALPHA, scene_to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,H,W", [((16, 16), 64, 64), ((8, 8), 37, 53), ((32, 8), 45, 70)])
def test_features_match_oracle_weights(cuda_device, tile, H, W):
    rng = np.random.default_rng(sum(tile) + H)
    scene, cams = S.config0(seed=7)
    c = cams[0]
    f = float(max(H, W))
    feats = rng.normal(size=(scene.n, 6)).astype(np.float32)  # two chunks of four
    m, p, w = scene_to_dev(scene, cuda_device)
    d, a, out = fe.render_features(m, p, w, torch.from_numpy(feats), f, f, W / 2, H / 2, c.quat,
                                   c.trans, H, W, tile=tile)
    out = out.cpu().numpy().reshape(-1, 6)
    rays = O.pinhole_rays(H, W, f, f, W / 2, H / 2)
    _, ra, _, rw = O.render_func_quat(scene.means, scene.prec, scene.logw, rays, c.quat, c.trans,
                                      21.4, 2.66, return_weights=True)
    mask = ra > DEPTH_MASK_ALPHA
    ref = rw.T @ feats.astype(np.float64)
    assert np.max(np.abs(out - ref)[mask]) <= 1e-3
    # all-ones feature: the weights sum to one wherever a front Gaussian exists (to 5e-5: this
    # pass re-evaluates each weight in scalar arithmetic, the forward summed its normaliser with
    # packed arithmetic associated differently)
    ones = fe.render_features(m, p, w, torch.ones(scene.n, 1), f, f, W / 2, H / 2, c.quat, c.trans,
                              H, W, tile=tile)[2].cpu().numpy().ravel()
    assert np.allclose(ones[mask], 1.0, atol=5e-5)
    assert np.all((ones == 0) | (np.abs(ones - 1) < 5e-5))


def test_features_equal_the_pixel_list_path(cuda_device):
    rng = np.random.default_rng(3)
    scene, cams = S.config0(seed=8)
    c = cams[0]
    H, W, f = 48, 64, 60.0
    feats = torch.from_numpy(rng.normal(size=(scene.n, 3)).astype(np.float32))
    m, p, w = scene_to_dev(scene, cuda_device)
    _, a, out = fe.render_features(m, p, w, feats, f, f, W / 2, H / 2, c.quat, c.trans, H, W)
    v, u = np.mgrid[0:H, 0:W]
    rays = np.stack([u.ravel() - W / 2, v.ravel() - H / 2, np.ones(H * W), np.zeros(H * W)], 1)
    pose = np.concatenate([c.quat, c.trans])[None].astype(np.float32)
    res = fe.render_pixels(m, p, w, torch.from_numpy(rays.astype(np.float32)), 1.0 / f,
                           torch.from_numpy(pose), features=feats)
    ok = (a > DEPTH_MASK_ALPHA).reshape(-1)
    assert torch.allclose(out.reshape(-1, 3)[ok], res[4][ok], rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("tile", [(16, 16), (8, 8), (32, 8)])
@pytest.mark.parametrize("nf", [1, 4, 5, 8, 17, 33, 64])
def test_feature_widths_agree(cuda_device, tile, nf):
    """Every width's kernel and its last, partial pass: column j of a wide table equals the same
    column rendered alone (the weights are the same bits; a sum over at most 70 keys is reassociated
    only where the table's padding differs, so to 70 ulp), and a constant column gives the constant
    times the weights' sum. More than one stage of keys per tile, odd image sides."""
    rng = np.random.default_rng(nf)
    scene = S.random_gaussians(150, 0.08, rng)
    H, W, f = 43, 61, 60.0
    quat, trans = S.look_at(0.5 * S.random_unit_vectors(1, rng)[0])
    m, p, w = scene_to_dev(scene, cuda_device)
    feats = torch.from_numpy(rng.normal(size=(scene.n, nf)).astype(np.float32)).to(cuda_device)
    cam = (f, f, W / 2, H / 2, quat, trans, H, W)
    wide = fe.render_features(m, p, w, feats, *cam, tile=tile)[2]
    for j in {0, nf // 2, nf - 1}:
        one = fe.render_features(m, p, w, feats[:, j:j + 1].contiguous(), *cam, tile=tile)[2]
        torch.testing.assert_close(wide[..., j], one[..., 0], rtol=0,
                                   atol=70 * 6e-8 * float(feats.abs().max()))


@pytest.mark.parametrize("tile", [(16, 16), (8, 8), (32, 8)])
def test_features_where_an_infinite_logit_reaches(cuda_device, tile):
    """A log-weight of +inf leaves no finite normaliser at the pixels its tiles cover: they take no
    weights, so their features are 0, as where no Gaussian is in front."""
    rng = np.random.default_rng(5)
    scene = S.random_gaussians(90, 0.05, rng)
    H, W, f = 43, 61, 60.0
    quat, trans = S.look_at(0.5 * S.random_unit_vectors(1, rng)[0])
    m, p, w = scene_to_dev(scene, cuda_device)
    feats = torch.from_numpy(rng.normal(size=(scene.n, 5)).astype(np.float32)).to(cuda_device)
    cam = (f, f, W / 2, H / 2, quat, trans, H, W)
    w[17] = float("inf")
    stats = torch.empty((3, H, W), device=cuda_device)
    fe.render_forward(m, p, w, *cam, tile=tile, stats=stats)
    dead = ~(stats[1] > 0)
    assert bool(stats[1].isnan().any())
    out = fe.render_features(m, p, w, feats, *cam, tile=tile)[2]
    assert bool((out[dead] == 0).all()) and bool(torch.isfinite(out).all())


@pytest.mark.parametrize("tile", [(16, 16), (8, 8), (32, 8)])
@pytest.mark.parametrize("nf", [5, 17, 33])
def test_wide_features_match_oracle_weights(cuda_device, tile, nf):
    """Tables whose last pass is partial, over more than one stage of keys, an odd number of them
    included: the float64 oracle's w @ f on pixels that see the scene (to 1e-3: a logit of 40 to
    float32's 1e-6), and a constant column gives the constant where a front Gaussian exists (the
    weights sum to one to 5e-5, as against the forward's normaliser), else 0."""
    rng = np.random.default_rng(nf)
    scene = S.random_gaussians(151, 0.08, rng)
    H, W, f = 43, 61, 60.0
    quat, trans = S.look_at(0.5 * S.random_unit_vectors(1, rng)[0])
    m, p, w = scene_to_dev(scene, cuda_device)
    feats = rng.normal(size=(scene.n, nf)).astype(np.float32)
    feats[:, nf - 1] = 3.0
    out = fe.render_features(m, p, w, torch.from_numpy(feats), f, f, W / 2, H / 2, quat, trans, H, W,
                             tile=tile)[2].cpu().numpy().reshape(-1, nf)
    rays = O.pinhole_rays(H, W, f, f, W / 2, H / 2)
    _, ra, _, rw = O.render_func_quat(scene.means, scene.prec, scene.logw, rays, quat, trans, 21.4,
                                      2.66, return_weights=True)
    seen = ra > DEPTH_MASK_ALPHA
    assert np.max(np.abs(out - rw.T @ feats.astype(np.float64))[seen]) <= 1e-3
    ones = out[:, nf - 1] / 3.0
    assert np.all(np.abs(ones[seen] - 1) < 5e-5)
    assert np.all((ones == 0) | (np.abs(ones - 1) < 5e-5))
