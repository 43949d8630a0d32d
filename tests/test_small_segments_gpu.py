"""Builds whose segments all fit one block each sort and start the tree in one kernel; a build with one larger segment takes the
general passes. The trees of the same meshes must be the same either way: sizes around the block sizes, coincident and equal
centroids among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def soup(n, seed, mat, kind):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-10, 10, (n, 1, 3))
    if kind == "fives":
        c = np.repeat(c[:(n + 4) // 5], 5, 0)[:n]    # five centroids in one place: only positions order them
    if kind == "pairs":
        c[1::2] = c[:n // 2 * 2:2][:len(c[1::2])]    # equal keys in pairs
    tri = np.array([[0, 0, 0], [0.5, 0, 0], [0, 0.5, 0]]) if kind != "random" else rng.uniform(-0.3, 0.3, (n, 3, 3))
    v = (c + tri).reshape(-1, 3).astype(np.float32)
    return v, np.arange(3 * n, dtype=np.int32).reshape(n, 3), np.full(n, mat, np.int32), None


@pytest.mark.parametrize("sizes", [(1, 2, 3), (1023, 1024), (1025, 5), (4095, 4096, 33)])
@pytest.mark.parametrize("kind", ["random", "fives", "pairs"])
def test_small_segments_build_the_general_tree(gpu, cwp, sizes, kind):
    meshes = [soup(n, 10 + i, i, kind) for i, n in enumerate(sizes)]
    small = cwp.Batch(meshes)
    general = cwp.Batch(meshes + [soup(4097, 99, len(meshes), "random")])
    for width in (2, 4, 8):
        a, b = (x.download(width)[1].reshape(-1, 3, 4) for x in (small, general))
        for i in range(len(meshes)):   # the leaf order of each mesh's triangles, which the whole tree decides
            mine = [t[t[:, 1, 3].view(np.int32) == i] for t in (a, b)]
            assert np.array_equal(mine[0].view(np.uint32), mine[1].view(np.uint32)), (width, i)


@pytest.mark.parametrize("sizes", [(127, 128, 1), (129, 2), (2047, 2048), (2049, 1)])   # around the other block sizes
@pytest.mark.parametrize("kind", ["random", "pairs"])
def test_block_sizes_build_the_general_tree(gpu, cwp, sizes, kind):
    test_small_segments_build_the_general_tree(gpu, cwp, sizes, kind)
