"""The captured frame against the host loop: shadow passes on a branch of their own (small passes), one graph for every sample
range, at image sizes and depths where a branch or a queue can be empty."""
import numpy as np
import pytest

from conftest import only_free

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [2, 4, 8])
@pytest.mark.parametrize("w,h,batch,bounces", [(1, 1, 1, 0), (33, 17, 1, 1), (64, 48, 2, 4), (257, 131, 3, 2)])
def test_graph_frame_equals_host_loop(gpu, cwp, variant, w, h, batch, bounces):
    mesh, bvh = cwp.scene(64, variant=variant, bins=16)
    p = cwp.frame_params(mesh, w, h, bounces=bounces)
    r, loop = cwp.Renderer(), cwp.Renderer()
    r.init(p, bvh, variant=variant, batch=batch, bounces=bounces, graph=1)
    loop.init(p, bvh, variant=variant, batch=batch, bounces=bounces, graph=0)
    for s_base, clear in ((0, True), (2 * batch, False), (7, False), (3, True)):   # one graph, four sample ranges
        a, b = r.render(2 * batch, s_base, clear), loop.render(2 * batch, s_base, clear)
        assert (a.rays, a.shadow_rays) == (b.rays, b.shadow_rays)
        x, y = r.read_accum(), loop.read_accum()
        # the same float contributions per pixel, at most 6 samples x (bounces + 2) x 2, added in another order: each addition
        # rounds by at most 2^-24 of the sum
        n = 6 * batch * (bounces + 2) * 2
        assert np.all(np.abs(x - y) <= n * 2.0 ** -24 * np.maximum(np.abs(y), 1e-30) * 2)


def test_scarce_memory_keeps_one_shadow_queue(gpu, cwp):
    """a shadow queue per depth is taken from plenty only: with little memory free the frame keeps one and is the same"""
    mesh, bvh = cwp.scene(64, variant=8, bins=16)
    w, h, bounces = 1024, 512, 4                       # 0.5 M paths: 21 MB a queue, 105 MB for all depths
    p = cwp.frame_params(mesh, w, h, bounces=bounces)
    roomy, scarce = cwp.Renderer(), cwp.Renderer()
    roomy.init(p, bvh, variant=8, batch=1, bounces=bounces)
    with only_free(gpu, 1 << 30):
        scarce.init(p, bvh, variant=8, batch=1, bounces=bounces)
    assert roomy.info().vram_mb - scarce.info().vram_mb >= 0.9 * bounces * 40 * w * h / 2 ** 20
    a, b = roomy.render(4), scarce.render(4)
    assert (a.rays, a.shadow_rays) == (b.rays, b.shadow_rays)
    x, y = roomy.read_accum(), scarce.read_accum()
    n = 4 * (bounces + 2) * 2   # the same float contributions in another order, as above
    assert np.all(np.abs(x - y) <= n * 2.0 ** -24 * np.maximum(np.abs(y), 1e-30) * 2)
