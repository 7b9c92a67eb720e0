"""Which binning a call takes, and that the images do not depend on it. Routes are read off the
number of kernels: preprocess, emission and blend with a block per tile row; preprocess, counts,
bases, keys and blend in segments of the records; eight or more through emission and sort."""

import ctypes

import numpy as np
import pytest
import torch

import fuzzy_ellipses as fe
from fuzzy_ellipses import _native as N
from fuzzy_ellipses import synthetic as S
from tests.helpers import to_dev

pytestmark = pytest.mark.gpu


def kernels_of(call):
    """Number of kernels `call(stream handle)` launches: it runs once for the scratch to grow, then
    under capture, and the captured graph's kernel nodes are counted."""
    cu = ctypes.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    handle = ctypes.c_void_p(stream.cuda_stream)
    call(handle)
    stream.synchronize()
    graph = ctypes.c_void_p()
    relaxed = 2  # CU_STREAM_CAPTURE_MODE_RELAXED
    assert cu.cuStreamBeginCapture_v2(handle, relaxed) == 0
    try:
        call(handle)
    finally:
        rc = cu.cuStreamEndCapture(handle, ctypes.byref(graph))
    assert rc == 0
    count = ctypes.c_size_t()
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(count)) == 0
    kinds = []
    for node in nodes:
        kind = ctypes.c_int()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kinds.append(kind.value)
    cu.cuGraphDestroy(graph)
    return kinds.count(0)  # CU_GRAPH_NODE_TYPE_KERNEL


@pytest.mark.parametrize("n,views,h,w", [(2600, 1, 480, 640), (4000, 2, 200, 300),
                                         (8000, 6, 480, 640)])
def test_exact_key_plans_keep_a_block_per_row(cuda_device, n, views, h, w):
    """Plans whose keys are sized on the device have no room for segment counts: above 2500
    Gaussians they take a block per tile row as far as that applies (4096 Gaussians; 16384 from
    152 rows on), with the images and gradients of the sorted plan."""
    rng = np.random.default_rng(n)
    sc = S.random_gaussians(n, 0.3, rng)
    arrays = [to_dev(x, cuda_device) for x in (sc.means, sc.prec, sc.logw)]
    vs = []
    for d in S.random_unit_vectors(views, rng):
        q, t = S.look_at(1.0 * d)
        vs.append(dict(scene=0, height=h, width=w, fx=float(w), fy=float(w), cx=w / 2, cy=h / 2,
                       quat=q, trans=t))
    out = []
    for binning in ("tiles", "radix"):
        b = fe.Batch([(0, n)], vs, exact_keys=True, binning=binning)
        assert (b.launches_per_forward == 3) == (binning == "tiles")
        depth, alpha = b.forward(*arrays)
        st = b.status()
        assert st["device_error"] == 0 and st["num_keys"] == st["want_keys"]
        out.append((depth, alpha, st["num_keys"]))
        b.close()
    assert out[0][2] == out[1][2]
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


def legacy_inputs(n, culled, h, w, dev, seed=0):
    """Arrays of a legacy call: n Gaussians in view, then `culled` ones behind the near cut."""
    rng = np.random.default_rng(seed)
    z = rng.uniform(0.5, 1.5, n)
    means = np.stack([rng.uniform(-0.3, 0.3, n) * z, rng.uniform(-0.3, 0.3, n) * z * h / w, z], 1)
    quats = rng.standard_normal((n, 4))
    quats /= np.linalg.norm(quats, axis=1, keepdims=True)
    logw, scales = rng.normal(0, 0.5, n), np.exp(rng.uniform(-5.3, -3.5, (n, 3)))

    def pad(x, row):
        return np.concatenate([x, np.tile([row], (culled,) + (1,) * (x.ndim - 1))])
    f = float(w)
    rays = np.stack(list(np.meshgrid((np.arange(w) - w / 2) / f, (np.arange(h) - h / 2) / f)) +
                    [np.ones((h, w))], -1).reshape(-1, 3)
    arrays = (pad(means, [0.0, 0.0, -1.0]), pad(logw, 0.0), pad(scales, [0.01] * 3),
              pad(quats, [1.0, 0.0, 0.0, 0.0]), rays, np.eye(3), np.zeros(3))
    return [to_dev(x.astype(np.float32), dev) for x in arrays]


def legacy_call(ins, h, w, out):
    """A call of the native legacy entry on a stream, with host matrices and cleaned outputs."""
    f = float(w)
    tx, ty, view, proj = fe.api._legacy_scalars(h, w, f, f, w / 2, h / 2, 0.01, 4.5)
    d = N.LegacyDesc(h, w, ins[0].shape[0], float(tx), float(ty))

    def call(stream):
        N.check(N.load().fe_rasterize_legacy_host(
            ctypes.byref(d), *[x.data_ptr() for x in ins], view.ctypes.data, proj.ctypes.data, 1,
            out[0].data_ptr(), out[1].data_ptr(), stream))
    return call


# Gaussians in view, culled ones appended, image and the kernels of the call: 3000 on a block per
# row, in segments (4200 over few rows) and sorted (more rows x records than segments are for);
# 8000 with 152 tile rows the same.
LEGACY = [(3000, [(0, 3), (1200, 5)], 480, 640), (3000, [(0, 3), (1900, None)], 28000, 8),
          (8000, [(0, 3), (9000, 5), (52000, None)], 1216, 64)]


@pytest.mark.parametrize("n,routes,h,w", LEGACY)
def test_legacy_routes(cuda_device, n, routes, h, w):
    """The legacy call takes one emission launch as far as a block per row applies, then segments,
    then the sort; Gaussians that reach no tile change nothing, so all give the same image."""
    images = []
    for culled, kernels in routes:
        ins = legacy_inputs(n, culled, h, w, cuda_device)
        out = [torch.empty(h, w, device=cuda_device) for _ in range(2)]
        torch.cuda.synchronize()
        count = kernels_of(legacy_call(ins, h, w, out))
        assert count == kernels if kernels else count >= 8
        torch.cuda.synchronize()
        images.append([x.clone() for x in out])
    assert float(images[0][1].max()) > 0.1
    for z, a in images[1:]:
        assert torch.equal(z, images[0][0]) and torch.equal(a, images[0][1])


def _view(scene, h, w):
    return dict(scene=scene, height=h, width=w, fx=float(w), fy=float(w), cx=w / 2, cy=h / 2,
                quat=[1.0, 0.0, 0.0, 0.0], trans=[0.0, 0.0, -1.0])


@pytest.mark.parametrize("views,tile,limit", [
    # one view of 512 tile rows among 1000 of one tile: 1001 x 513 row totals of 8 bytes, and
    # everything else by the 1512 tiles and 1001 records there are
    ([_view(0, 8192, 16)] + [_view(0, 16, 16)] * 1000, (16, 16), 16 << 20),
    # 262144 tiles: lists, entry, range, key and its twin at 256 + 16 + 8 + 16 bytes a tile, grown
    # buffers a quarter larger
    ([_view(0, 4096, 4096)], (8, 8), 296 * 262144 * 5 // 4 + (8 << 20)),
    # the same through the sort: no lists, entries or spans
    ([_view(0, 4096, 16384)], (8, 8), 32 * 2 * 524288 * 5 // 4 + (8 << 20))])
def test_batch_scratch_follows_what_the_plan_uses(cuda_device, views, tile, limit):
    fe.Batch([(0, 1)], [_view(0, 64, 64)]).close()  # (the library's kernels are loaded)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    b = fe.Batch([(0, 1)], views, tile=tile)
    used = free - torch.cuda.mem_get_info()[0]
    b.close()
    assert used <= limit


@pytest.mark.parametrize("n,views,h,w,kw,binning,pieces", [
    (300, 4, 480, 640, {}, "rows", False), (300, 40, 100, 100, {}, "rows", False),
    (1300, 1, 64, 64, {}, "rows", True), (6000, 4, 480, 640, {}, "segments", False),
    (3000, 1, 64, 64, {}, "segments", True), (300, 4, 480, 640, {"binning": "radix"}, "sort", False),
    (1300, 1, 64, 64, {"binning": "radix"}, "sort", True),
    (3000, 1, 64, 64, {"heavy_first": True}, "segments", True)])
def test_plan_names_the_kernels(cuda_device, n, views, h, w, kw, binning, pieces):
    """Batch.plan says which binning a forward takes, whether its blend is cut into pieces and how
    many kernels it launches."""
    rng = np.random.default_rng(n)
    sc = S.random_gaussians(n, 0.3, rng)
    arrays = [to_dev(x, cuda_device) for x in (sc.means, sc.prec, sc.logw)]
    b = fe.Batch([(0, n)], [_view(0, h, w)] * views, **kw)
    plan = b.plan
    assert plan["binning"] == binning and (plan["pieces"] > 1) == pieces
    out = [torch.empty(b.n_pixels, device=cuda_device) for _ in range(2)]
    torch.cuda.synchronize()

    def call(stream):
        N.check(N.load().fe_batch_fwd(b._h, *[x.data_ptr() for x in arrays + out], None, stream))
    assert kernels_of(call) == plan["kernels"] == b.launches_per_forward + pieces
    b.close()


@pytest.mark.parametrize("n,h,w,whole", [(1300, 64, 64, False), (3000, 64, 64, False),
                                         (1300, 480, 640, True), (3000, 720, 1280, True)])
def test_asking_for_the_heaviest_tiles_first(cuda_device, n, h, w, whole):
    """Blends of whole tiles take the order that is asked for; a blend in pieces has none and lists no
    tiles for it. The images do not depend on it."""
    sc = S.random_gaussians(n, 0.3, np.random.default_rng(n))
    arrays = [to_dev(x, cuda_device) for x in (sc.means, sc.prec, sc.logw)]
    images = []
    for heavy in (False, True):
        b = fe.Batch([(0, n)], [_view(0, h, w)], heavy_first=heavy)
        plan = b.plan
        assert (plan["pieces"] == 1) == whole
        if heavy or not whole:
            assert plan["heavy_first"] == whole
        images.append(b.forward(*arrays))
        b.close()
    assert torch.equal(images[0][0], images[1][0]) and torch.equal(images[0][1], images[1][1])
