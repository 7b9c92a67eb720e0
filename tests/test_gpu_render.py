"""Forward parity of the CUDA render path against the float64 restatement of fm_render."""

import numpy as np
import pytest
import torch

import fuzzy_ellipses as fe
from fuzzy_ellipses import synthetic as S
from oracle import fm_render_np as O
from tests.helpers import (TOL_ALPHA, TOL_DEPTH_REL, floor_dominated, oracle_pixels, parity_errors,
                           scene_to_dev, tile_lists_from_keys, to_dev)

pytestmark = pytest.mark.gpu
TILES = [(8, 8), (16, 16), (32, 8)]


def render_np(dev, scene, cam, **kw):
    m, p, w = scene_to_dev(scene, dev)
    d, a = fe.render_forward(m, p, w, cam.fx, cam.fy, cam.cx, cam.cy, cam.quat, cam.trans,
                             cam.height, cam.width, **kw)
    torch.cuda.synchronize()
    assert fe.device_status() == 0
    return d.cpu().numpy(), a.cpu().numpy()


@pytest.fixture(scope="module")
def cfg0():
    scene, cams = S.config0(seed=0)
    cam = cams[0]
    d, a = O.render_pinhole(scene.means, scene.prec, scene.logw, cam.height, cam.width, cam.fx,
                            cam.fy, cam.cx, cam.cy, cam.quat, cam.trans)
    return scene, cam, d, a


@pytest.mark.parametrize("tile", TILES)
def test_config0_matches_fm_render(cuda_device, cfg0, tile):
    scene, cam, d_ref, a_ref = cfg0
    d, a = render_np(cuda_device, scene, cam, tile=tile)
    ea, ed = parity_errors(d, a, d_ref, a_ref)
    assert ea <= TOL_ALPHA, ea
    assert ed <= TOL_DEPTH_REL, ed


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_more_config0_scenes(cuda_device, seed):
    scene, cams = S.config0(seed=seed)
    cam = cams[0]
    d_ref, a_ref = O.render_pinhole(scene.means, scene.prec, scene.logw, cam.height, cam.width,
                                    cam.fx, cam.fy, cam.cx, cam.cy, cam.quat, cam.trans)
    d, a = render_np(cuda_device, scene, cam)
    ea, ed = parity_errors(d, a, d_ref, a_ref)
    assert ea <= TOL_ALPHA and ed <= TOL_DEPTH_REL, (ea, ed)


def test_config1_cameras_on_pixel_samples(cuda_device):
    scene, cams = S.config1(seed=0)
    rng = np.random.default_rng(0)
    for ci in (0, 7, 15):
        cam = cams[ci]
        d, a = render_np(cuda_device, scene, cam)
        pix = rng.choice(cam.height * cam.width, 6000, replace=False)
        d_ref, a_ref = oracle_pixels(scene, cam, pix)
        ea, ed = parity_errors(d.ravel()[pix], a.ravel()[pix], d_ref, a_ref)
        assert ea <= TOL_ALPHA and ed <= TOL_DEPTH_REL, (ci, ea, ed)


@pytest.mark.parametrize("tile", TILES)
def test_nstd_cull_matches_culled_oracle(cuda_device, cfg0, tile):
    """3-sigma mode: the kernel matches fm_render restricted to its own tile lists; the tail it
    drops (culled oracle vs dense oracle) is large and is reported, not hidden."""
    scene, cam, d_ref, a_ref = cfg0
    m, p, w = scene_to_dev(scene, cuda_device)
    keys, ranges = fe.render_binning(m, p, w, cam.fx, cam.fy, cam.cx, cam.cy, cam.quat, cam.trans,
                                     cam.height, cam.width, cull="nstd", cull_param=3.0, tile=tile)
    lists = tile_lists_from_keys(keys, ranges.shape[0])
    dc, ac = O.render_culled(scene.means, scene.prec, scene.logw, cam.height, cam.width, cam.fx,
                             cam.fy, cam.cx, cam.cy, cam.quat, cam.trans, lists, tile[0], tile[1])
    d, a = render_np(cuda_device, scene, cam, cull="nstd", cull_param=3.0, tile=tile)
    ea = float(np.abs(a - ac).max())
    mask = ac > 1e-3
    ed = float((np.abs(d - dc)[mask] / dc[mask]).max())
    assert ea <= TOL_ALPHA and ed <= TOL_DEPTH_REL, (ea, ed)
    tail = float(np.abs(ac - a_ref).max())
    assert 1e-3 < tail < 5e-2, tail  # the 3-sigma tail error is of order exp(-4.5)


def test_eps_binning_is_conservative(cuda_device, cfg0):
    """Every Gaussian whose peak density along a pixel ray exceeds the cut-off is listed for that
    pixel's tile."""
    scene, cam, _, _ = cfg0
    eps = 1e-7
    m, p, w = scene_to_dev(scene, cuda_device)
    keys, ranges = fe.render_binning(m, p, w, cam.fx, cam.fy, cam.cx, cam.cy, cam.quat, cam.trans,
                                     cam.height, cam.width, cull="eps", cull_param=eps, tile=(8, 8))
    lists = tile_lists_from_keys(keys, ranges.shape[0])
    rays = O.pinhole_rays(cam.height, cam.width, cam.fx, cam.fy, cam.cx, cam.cy) @ O.quat_to_rot(cam.quat)
    _, stds = O.ray_gaussian_terms(rays, np.tile(cam.trans.astype(np.float64), (rays.shape[0], 1)),
                                   scene.means, scene.prec, scene.logw)
    gx = (cam.width + 7) // 8
    v, u = np.divmod(np.arange(cam.height * cam.width), cam.width)
    tile = (v // 8) * gx + u // 8
    need = stds > np.log(eps) + 1e-6
    for g in range(scene.n):
        tiles_needed = np.unique(tile[need[g]])
        for t in tiles_needed:
            assert g in set(lists[t].tolist()), (g, t)


def test_keys_sorted_and_ranges_consistent(cuda_device):
    scene, cams = S.config1(seed=0)
    cam = cams[3]
    m, p, w = scene_to_dev(scene, cuda_device)
    for tile in TILES:
        keys, ranges = fe.render_binning(m, p, w, cam.fx, cam.fy, cam.cx, cam.cy, cam.quat,
                                         cam.trans, cam.height, cam.width, tile=tile)
        k = keys.cpu().numpy().view(np.uint64)
        assert np.all(k[1:] > k[:-1])
        tiles = (k >> np.uint64(32)).astype(np.int64)
        r = ranges.cpu().numpy()
        assert tiles.max() < r.shape[0] and (k & np.uint64(0xFFFFFFFF)).max() < scene.n
        counts = np.bincount(tiles, minlength=r.shape[0])
        assert np.array_equal(r[:, 1] - r[:, 0], counts)
        nz = counts > 0
        assert np.array_equal(r[nz, 0], np.searchsorted(tiles, np.nonzero(nz)[0]))


def test_empty_scene_and_tiny_images(cuda_device):
    dev = cuda_device
    z = torch.zeros((0, 3), device=dev)
    d, a = fe.render_forward(z, torch.zeros((0, 3, 3), device=dev), torch.zeros(0, device=dev),
                             10.0, 10.0, 5.0, 5.0, [1, 0, 0, 0], [0, 0, 0], 7, 9)
    torch.cuda.synchronize()
    assert torch.all(d == 0) and torch.all(a == 0)
    scene, cams = S.config0(seed=4)
    cam = cams[0]
    for (H, W) in [(1, 1), (3, 17), (37, 23), (64, 1)]:
        f = float(max(H, W)) + 1.0
        cam2 = S.Camera(H, W, f, f, W / 2, H / 2, cam.quat, cam.trans)
        d_ref, a_ref = O.render_pinhole(scene.means, scene.prec, scene.logw, H, W, f, f, W / 2,
                                        H / 2, cam.quat, cam.trans)
        for tile in TILES:
            d, a = render_np(dev, scene, cam2, tile=tile)
            ea, ed = parity_errors(d, a, d_ref, a_ref)
            assert ea <= TOL_ALPHA and ed <= TOL_DEPTH_REL, (H, W, tile, ea, ed)


def test_single_gaussian_and_behind_camera(cuda_device):
    dev = cuda_device
    H, W, f = 40, 48, 60.0
    quat, trans = np.array([1, 0, 0, 0], np.float32), np.zeros(3, np.float32)
    prec = np.stack([np.triu(np.eye(3) / 0.02)] * 2).astype(np.float32)
    # One Gaussian in front; one behind the camera whose ray *line* still passes close to it:
    # fm_render counts it in alpha (no z>0 mask, fm_render.py:89) but not in depth.
    means = np.array([[0.01, -0.02, 0.5], [0.0, 0.0, -0.4]], np.float32)
    logw = np.array([0.2, -1.0], np.float32)
    sc = S.Scene(means, prec, logw)
    cam = S.Camera(H, W, f, f, W / 2, H / 2, quat, trans)
    d_ref, a_ref = O.render_pinhole(means, prec, logw, H, W, f, f, W / 2, H / 2, quat, trans)
    floor = floor_dominated(sc, cam)
    assert floor.any()  # the scene does exercise fm_render's weight floor
    n_tiles = ((W + 7) // 8) * ((H + 7) // 8)
    d_front, _ = O.render_culled(means, prec, logw, H, W, f, f, W / 2, H / 2, quat, trans,
                                 [np.arange(2)] * n_tiles, 8, 8)
    for tile in TILES:
        d, a = render_np(dev, sc, cam, tile=tile)
        ea, ed = parity_errors(d, a, d_ref, a_ref, exclude=floor)
        assert ea <= TOL_ALPHA and ed <= TOL_DEPTH_REL, (tile, ea, ed)
        # Where the floor governs fm_render, the renderer keeps the front-only softmax depth (the
        # culled oracle's definition), or 0 where the front Gaussian is culled from the tile.
        df = d.ravel()[floor]
        dc = d_front.ravel()[floor]
        listed = df != 0
        assert np.all(np.abs(df[listed] - dc[listed]) <= TOL_DEPTH_REL * dc[listed])


def test_gaussian_straddling_camera_plane_covers_image(cuda_device):
    dev = cuda_device
    H, W, f = 32, 32, 32.0
    quat, trans = np.array([1, 0, 0, 0], np.float32), np.zeros(3, np.float32)
    means = np.array([[0.3, 0.0, 0.02], [0.0, 0.0, 0.6]], np.float32)
    prec = np.stack([np.triu(np.eye(3) / 0.1), np.triu(np.eye(3) / 0.05)]).astype(np.float32)
    logw = np.array([0.0, 0.5], np.float32)
    sc = S.Scene(means, prec, logw)
    cam = S.Camera(H, W, f, f, W / 2, H / 2, quat, trans)
    d_ref, a_ref = O.render_pinhole(means, prec, logw, H, W, f, f, W / 2, H / 2, quat, trans)
    d, a = render_np(dev, sc, cam)
    ea, ed = parity_errors(d, a, d_ref, a_ref, exclude=floor_dominated(sc, cam))
    assert ea <= TOL_ALPHA and ed <= TOL_DEPTH_REL, (ea, ed)


def test_stream_ordering_and_repeatability(cuda_device):
    scene, cams = S.config0(seed=5)
    cam = cams[0]
    m, p, w = scene_to_dev(scene, cuda_device)
    s = torch.cuda.Stream()
    outs = []
    with torch.cuda.stream(s):
        for _ in range(3):
            outs.append(fe.render_forward(m, p, w, cam.fx, cam.fy, cam.cx, cam.cy, cam.quat,
                                          cam.trans, cam.height, cam.width))
    s.synchronize()
    for d, a in outs[1:]:
        assert torch.equal(d, outs[0][0]) and torch.equal(a, outs[0][1])


@pytest.mark.parametrize("tile", TILES)
def test_subpixel_gaussians(cuda_device, tile):
    """Gaussians a quarter of a pixel wide: the Mahalanobis polynomial is evaluated around each
    Gaussian's own projected centre, so float32 keeps the stated tolerance."""
    rng = np.random.default_rng(11)
    scene = S.random_gaussians(80, 0.1, rng, scale_lo=0.002, scale_hi=0.006)
    q, t = S.look_at(0.5 * S.random_unit_vectors(1, rng)[0])
    cam = S.Camera(64, 64, 64.0, 64.0, 32.0, 32.0, q, t)
    d_ref, a_ref = O.render_pinhole(scene.means, scene.prec, scene.logw, 64, 64, 64.0, 64.0, 32.0,
                                    32.0, q, t)
    d, a = render_np(cuda_device, scene, cam, tile=tile)
    ea, ed = parity_errors(d, a, d_ref, a_ref)
    assert ea <= TOL_ALPHA and ed <= TOL_DEPTH_REL, (ea, ed)


def test_large_scene_beyond_the_key_budget(cuda_device):
    """24,000 Gaussians at 1280x720 with 16x16 tiles: the worst-case key plan (N x tiles = 86 M
    keys, ~8 GB of key scratch) exceeds the 4 GiB key budget, so the plain call reads the exact
    key count back and sizes the keys from it. Sampled pixels against the float64 oracle; the
    backward goes through the same path."""
    rng = np.random.default_rng(21)
    scene = S.random_gaussians(24000, 0.35, rng)
    cam = S.Camera(720, 1280, 900.0, 900.0, 640.0, 360.0, *S.look_at([0.2, -0.3, 1.1]))
    m, p, w = scene_to_dev(scene, cuda_device)
    depth, alpha = fe.render_forward(m, p, w, cam.fx, cam.fy, cam.cx, cam.cy, cam.quat, cam.trans,
                                     cam.height, cam.width)
    assert fe.device_status() == 0
    pix = rng.choice(cam.height * cam.width, 600, replace=False)
    d_ref, a_ref = oracle_pixels(scene, cam, pix)
    ea, ed = parity_errors(depth.cpu().numpy().ravel()[pix], alpha.cpu().numpy().ravel()[pix],
                           d_ref, a_ref)
    assert ea <= TOL_ALPHA and ed <= TOL_DEPTH_REL, (ea, ed)
    mr, pr, wr = [t.clone().requires_grad_() for t in (m, p, w)]
    d2, a2 = fe.render(mr, pr, wr, cam.fx, cam.fy, cam.cx, cam.cy, cam.quat, cam.trans,
                       cam.height, cam.width)
    assert torch.equal(a2.detach(), alpha)
    a2.sum().backward()
    for g in (mr.grad, pr.grad, wr.grad):
        assert torch.isfinite(g).all() and float(g.abs().sum()) > 0


@pytest.mark.parametrize("kind", ["array", "list", "cpu tensor", "double"])
def test_host_pose_equals_device_pose(cuda_device, kind):
    """A pose in host memory goes to the kernels by value: the same bits as the same pose in device
    tensors, in the forward, the features and the gradients, also when the caller overwrites its
    array between the forward and the backward."""
    scene, cams = S.config0(seed=2)
    c = cams[0]
    m, p, w = scene_to_dev(scene, cuda_device)
    q, t = c.quat.copy(), c.trans.copy()
    if kind == "list":
        q, t = [float(x) for x in q], [float(x) for x in t]
    elif kind == "cpu tensor":
        q, t = torch.from_numpy(q), torch.from_numpy(t)
    elif kind == "double":
        q, t = q.astype(np.float64), t.astype(np.float64)
    dq, dt = to_dev(c.quat, cuda_device), to_dev(c.trans, cuda_device)
    size = (c.height, c.width)
    feats = torch.rand(scene.n, 3, device=cuda_device)
    a = fe.render_features(m, p, w, feats, c.fx, c.fy, c.cx, c.cy, q, t, *size)
    b = fe.render_features(m, p, w, feats, c.fx, c.fy, c.cx, c.cy, dq, dt, *size)
    assert all(torch.equal(x, y) for x, y in zip(a, b))
    fwd = fe.render_forward(m, p, w, c.fx, c.fy, c.cx, c.cy, q, t, *size)
    assert torch.equal(fwd[0], b[0]) and torch.equal(fwd[1], b[1])
    grads = []
    for quat, trans in ((q, t), (dq, dt)):
        mm = m.clone().requires_grad_()
        depth, alpha = fe.render(mm, p, w, c.fx, c.fy, c.cx, c.cy, quat, trans, *size)
        if quat is q and not isinstance(q, list):
            q[0], t[0] = 9.0, 9.0
        (alpha.sum() + depth.sum()).backward()
        grads.append(mm.grad)
    # (the backward's atomics leave the order of a Gaussian's tile sums open)
    torch.testing.assert_close(grads[0], grads[1], rtol=1e-5, atol=1e-5 * float(grads[1].abs().max()))


@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("n,H,W", [(256, 16, 16), (1000, 33, 50), (2600, 64, 64), (5000, 37, 129)])
def test_few_tiles_of_many_gaussians(cuda_device, tile, n, H, W):
    """Launches of few tiles cut each tile's keys into pieces and merge their sums: depth and alpha
    within the stated tolerance of the float64 oracle, and the statistics they leave give the
    gradients of the same view blended whole (a batch with 16-pair stages; both backwards
    accumulate in float32 with open order, so to 1e-4 of the largest entry)."""
    rng = np.random.default_rng(n)
    scene = S.random_gaussians(n, 0.12, rng)
    cam = S.Camera(H, W, float(max(H, W)), float(max(H, W)), W / 2, H / 2,
                   *S.look_at(0.5 * S.random_unit_vectors(1, rng)[0]))
    m, p, w = [x.requires_grad_() for x in scene_to_dev(scene, cuda_device)]
    depth, alpha = fe.render(m, p, w, cam.fx, cam.fy, cam.cx, cam.cy, cam.quat, cam.trans, H, W,
                             tile=tile)
    assert fe.device_status() == 0
    d, a = depth.detach().cpu().numpy().ravel(), alpha.detach().cpu().numpy().ravel()
    pix = rng.choice(H * W, min(400, H * W), replace=False)
    ea, ed = parity_errors(d[pix], a[pix], *oracle_pixels(scene, cam, pix))
    assert ea <= TOL_ALPHA and ed <= TOL_DEPTH_REL, (ea, ed)
    gd, ga = torch.rand(H, W, device=cuda_device), torch.rand(H, W, device=cuda_device)
    got = torch.autograd.grad((depth, alpha), (m, p, w), (gd, ga))
    view = dict(scene=0, height=H, width=W, fx=cam.fx, fy=cam.fy, cx=cam.cx, cy=cam.cy,
                quat=cam.quat, trans=cam.trans)
    b = fe.Batch([(0, n)], [view], tile=tile, px=2, chunk=16)
    args = [x.detach() for x in (m, p, w)]
    stats = torch.empty(3 * b.n_pixels, device=cuda_device)
    bd, ba = b.forward(*args, stats=stats)
    want = b.backward(*args, bd, ba, stats, gd.ravel(), ga.ravel())
    for x, y in zip(got, want):
        assert float((x - y).abs().max()) <= 1e-4 * float(y.abs().max())
    b.close()


@pytest.mark.parametrize("n,H,W", [(2500, 64, 80), (2501, 64, 80), (2501, 500, 700), (5000, 730, 1090)])
def test_chained_launches_replay_from_a_graph(cuda_device, n, H, W):
    """Calls of more than 2500 Gaussians launch their kernels chained (each may start before the one
    before has ended): captured and replayed, on other data, they render as the eager call does."""
    rng = np.random.default_rng(n + H)
    q, t = S.look_at(0.7 * S.random_unit_vectors(1, rng)[0])
    q, t = [torch.tensor(np.asarray(x), dtype=torch.float32, device=cuda_device) for x in (q, t)]
    a, b = [scene_to_dev(S.random_gaussians(n, 0.2, rng), cuda_device) for _ in range(2)]
    data = [x.clone() for x in a]
    out = [torch.empty((H, W), device=cuda_device) for _ in range(2)]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())

    def go():
        fe.render_forward(*data, float(W), float(W), W / 2, H / 2, q, t, H, W, out=out)

    with torch.cuda.stream(s):
        go()
        go()
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        go()
    for x, y in zip(data, b):
        x.copy_(y)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    got = [x.clone() for x in out]
    want = fe.render_forward(*b, float(W), float(W), W / 2, H / 2, q, t, H, W)
    assert fe.device_status() == 0
    assert got[1].max() > 0.1
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
