"""Small ray batches over a CWBVH: the shares a warp takes of a batch that does not fill the GPU, and the traversal with eight
lanes per ray that finishes a warp's last rays, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 4, 5, 33, 1000, 4737, 18945, 18951, 37889, 151553]   # around 1, 4, 5 and 32 rays per warp of 148 x 8 x 4 warps


@pytest.fixture(scope="module")
def rays(cwp):
    rng = np.random.default_rng(3)
    n = max(SIZES)
    o = np.zeros((n, 4), np.float32); d = np.empty((n, 4), np.float32)
    o[:, :3] = rng.uniform([-18, -18, 0.2], [18, 18, 6], (n, 3)); o[:, 3] = np.where(rng.random(n) < 0.25, 0.5, 0.0)
    v = rng.normal(size=(n, 3)); v[rng.random(n) < 0.1, 2] = 0.0   # and rays along an axis plane
    d[:, :3] = v / np.linalg.norm(v, axis=1, keepdims=True); d[:, 3] = np.where(rng.random(n) < 0.3, 5.0, 1e30)
    return o, d


@pytest.mark.parametrize("tri,spatial", [(1, 0.0), (0, 0.0), (1, 1e-3)])
def test_small_batches_bitexact_vs_oracle(gpu, cwp, oracle, rays, tri, spatial):
    _, bvh = cwp.scene(1024, variant=8, bins=32, spatial=spatial)
    acc = cwp.Accel(bvh, tri=tri)
    o, d = rays
    tv = bvh.woop if tri else bvh.tris
    want = oracle.trace(8, tri, False, bvh.nodes, tv, o, d).view(np.uint32)
    want_any = oracle.trace(8, tri, True, bvh.nodes, tv, o, d)
    to, td = gpu.from_numpy(o).cuda(), gpu.from_numpy(d).cuda()
    for n in SIZES:
        hits = gpu.full((n, 4), -7.0, dtype=gpu.float32, device="cuda"); occ = gpu.full((n,), -7, dtype=gpu.int32, device="cuda")
        acc.trace_closest(to.data_ptr(), td.data_ptr(), hits.data_ptr(), n)
        acc.trace_any(to.data_ptr(), td.data_ptr(), occ.data_ptr(), n)
        gpu.cuda.synchronize(); acc.status()
        assert np.array_equal(hits.cpu().numpy().view(np.uint32), want[:n]), n
        assert np.array_equal(occ.cpu().numpy(), want_any[:n]), n


def test_precision_shares_bitexact_vs_oracle(gpu, cwp, oracle, rays):
    """precision any-hit rays: even shares up to five rays a warp, whole fetches above; closest hits beside them"""
    _, bvh = cwp.scene(1024, variant=8, bins=32)
    acc = cwp.Accel(bvh)
    acc.set_precision(1)
    o, d = rays
    warps = gpu.cuda.get_device_properties(0).multi_processor_count * 8 * 4
    sizes = [1, 3, warps - 1, 5 * warps, 5 * warps + 1, 32 * warps]
    assert sizes[-1] <= len(o)
    want = oracle.trace_prec(bvh.nodes, bvh.verts, o, d).view(np.uint32)
    want_any = oracle.trace_prec(bvh.nodes, bvh.verts, o, d, any_hit=True)
    to, td = gpu.from_numpy(o).cuda(), gpu.from_numpy(d).cuda()
    for n in sizes:
        hits = gpu.full((n, 4), -7.0, dtype=gpu.float32, device="cuda"); occ = gpu.full((n,), -7, dtype=gpu.int32, device="cuda")
        acc.trace_closest(to.data_ptr(), td.data_ptr(), hits.data_ptr(), n)
        acc.trace_any(to.data_ptr(), td.data_ptr(), occ.data_ptr(), n)
        gpu.cuda.synchronize(); acc.status()
        assert np.array_equal(hits.cpu().numpy().view(np.uint32), want[:n]), n
        assert np.array_equal(occ.cpu().numpy(), want_any[:n]), n
