"""Frames in every form of path order and traversal that the options choose: runs of up to 32 samples of one pixel, refill or one
fetch per warp, top levels of the tree in shared memory, fewer bounces than the renderer was set up for. All are the same samples of
the same paths, so each is compared with the oracle and with the frame of one sample per pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def render(cwp, p, bvh, variant, spp, **kw):
    r = cwp.Renderer()
    r.init(p, bvh, variant=variant, **kw)
    st = r.render(spp)
    return st, r.read_accum()


def same_sums(a, b, terms):
    """the same float contributions per pixel added in another order: each addition rounds by at most 2^-24 of the sum"""
    return np.all(np.abs(a - b) <= 2 * terms * 2.0 ** -24 * np.maximum(np.abs(b), 1e-30))


@pytest.mark.parametrize("w,h", [(24, 12), (13, 7)])   # whole 8 x 4 tiles, and rows of pixels
@pytest.mark.parametrize("batch,spp", [(32, 32), (64, 64), (96, 192), (24, 24), (7, 7)])   # runs of 32, 32, 32, 8 and 1; one and several runs per pixel
def test_sample_runs(gpu, cwp, oracle, w, h, batch, spp):
    mesh, bvh = cwp.scene(1024, variant=8, bins=32)
    p = cwp.frame_params(mesh, w, h, bounces=3)
    st, acc = render(cwp, p, bvh, 8, spp, batch=batch, bounces=3)
    s1, one = render(cwp, p, bvh, 8, spp, batch=1, bounces=3)
    assert (st.rays, st.shadow_rays) == (s1.rays, s1.shadow_rays)
    assert same_sums(acc, one, spp * 5 * 2)
    want, counts = oracle.render(p, 8, 1, bvh, 3, spp)
    assert cwp.imageio.psnr(acc[:, :3] / spp, want[:, :3] / spp) >= 60.0
    assert abs(st.rays - counts[0]) <= 1e-3 * counts[0] and abs(st.shadow_rays - counts[1]) <= 1e-3 * counts[1]


FORMS = [(2, 1, -1), (2, 2, -1), (4, 2, -1), (8, 1, -1), (8, 2, -1), (8, 0, 1), (8, 1, 2), (8, 2, 2), (8, 0, 3)]


@pytest.mark.parametrize("variant,traversal,stage", FORMS)
@pytest.mark.parametrize("tri", [0, 1])
@pytest.mark.parametrize("max_b", [3, 1, 0])   # 3: the limit of the set-up; below it several depths trace rays beyond the limit
def test_traversal_forms(gpu, cwp, variant, traversal, stage, tri, max_b):
    w, h, spp = 40, 20, 32
    mesh, bvh = cwp.scene(1024, variant=variant, bins=32)
    p = cwp.frame_params(mesh, w, h, bounces=max_b)
    base, want = render(cwp, p, bvh, variant, spp, batch=16, bounces=3, tri=tri, stage_levels=-1)
    for graph in (0, 1):
        st, acc = render(cwp, p, bvh, variant, spp, batch=16, bounces=3, tri=tri, traversal=traversal, stage_levels=stage, graph=graph)
        assert (st.rays, st.shadow_rays) == (base.rays, base.shadow_rays)
        assert same_sums(acc, want, spp * (max_b + 2) * 2)


@pytest.mark.parametrize("variant", [2, 8])
@pytest.mark.parametrize("traversal", [0, 2])
def test_fewer_bounces_than_the_limit(gpu, cwp, oracle, variant, traversal):
    mesh, bvh = cwp.scene(1024, variant=variant, bins=32)
    p = cwp.frame_params(mesh, 40, 20, bounces=1)
    st, acc = render(cwp, p, bvh, variant, 8, batch=8, bounces=4, traversal=traversal)
    want, counts = oracle.render(p, variant, 1, bvh, 4, 8)
    assert cwp.imageio.psnr(acc[:, :3] / 8, want[:, :3] / 8) >= 60.0
    assert abs(st.rays - counts[0]) <= 1e-3 * counts[0] and abs(st.shadow_rays - counts[1]) <= 1e-3 * counts[1]


@pytest.mark.parametrize("boxes", [682, 683])   # 8,186 and 8,198 triangles: either side of the line between the bounce kernels
@pytest.mark.parametrize("spatial", [0.0, 1e-3])
def test_bounce_kernels_on_either_side_of_the_line(gpu, cwp, oracle, boxes, spatial):
    mesh, bvh = cwp.scene(boxes, variant=8, bins=32, spatial=spatial)
    p = cwp.frame_params(mesh, 40, 20, bounces=3)
    st, acc = render(cwp, p, bvh, 8, 8, batch=8, bounces=3)
    s1, refill = render(cwp, p, bvh, 8, 8, batch=8, bounces=3, traversal=1)
    assert (st.rays, st.shadow_rays) == (s1.rays, s1.shadow_rays)
    assert same_sums(acc, refill, 8 * 5 * 2)
    want, counts = oracle.render(p, 8, 1, bvh, 3, 8)
    assert cwp.imageio.psnr(acc[:, :3] / 8, want[:, :3] / 8) >= 60.0
    assert abs(st.rays - counts[0]) <= 1e-3 * counts[0] and abs(st.shadow_rays - counts[1]) <= 1e-3 * counts[1]
