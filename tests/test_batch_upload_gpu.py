"""Meshes of a batch go up as they are and a kernel gathers the triangle records: sizes at the edges of a block, meshes with and
without material ids, and the first offending corner of bad input."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def strip(n, mat, seed):
    rng = np.random.default_rng(seed)
    v = rng.uniform(-5, 5, (n + 2, 3)).astype(np.float32)
    f = np.stack([np.arange(n), np.arange(n) + 1, np.arange(n) + 2], 1).astype(np.int32)
    return v, f, (np.arange(n) % 7).astype(np.int32) if mat else None, None


@pytest.mark.parametrize("sizes", [(1,), (2, 1), (255, 1, 256), (257, 3, 1000)])
@pytest.mark.parametrize("leaf", [1, 4])
def test_records_of_every_mesh(gpu, cwp, sizes, leaf):
    meshes = [strip(n, i % 2 == 0, i) for i, n in enumerate(sizes)]
    b = cwp.Batch(meshes, leaf=leaf)
    for width in (2, 4, 8):
        _, tris = b.download(width)
        rec = tris.reshape(-1, 3, 4)
        # each mesh's records, by mesh-local id (its triangles are placed together, mesh after mesh, level by level within)
        want = np.concatenate([np.concatenate([v[f[:, 0]], v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]], np.arange(len(f))[:, None],
                                               (np.zeros(len(f)) if m is None else m)[:, None]], 1) for v, f, m, _ in meshes]).astype(np.float32)
        got = np.concatenate([rec[:, 0, :3], rec[:, 1, :3], rec[:, 2, :3], rec[:, 0, 3].view(np.int32)[:, None].astype(np.float32),
                              rec[:, 1, 3].view(np.int32)[:, None].astype(np.float32)], 1)
        assert np.array_equal(want[np.lexsort(want.T)], got[np.lexsort(got.T)])


@pytest.mark.parametrize("mesh,tri,corner,what", [(0, 0, 0, "index"), (1, 299, 2, "index"), (2, 5, 1, "nan"), (1, 0, 0, "negative")])
@pytest.mark.parametrize("builder", [0, 1])
def test_first_bad_corner_is_named(gpu, cwp, mesh, tri, corner, what, builder):
    meshes = [strip(n, True, i) for i, n in enumerate((256, 300, 10))]
    v, f, m, _ = meshes[mesh]
    v, f = v.copy(), f.copy()
    if what == "nan":
        v[f[tri, corner], 1] = np.inf
    else:
        f[tri, corner] = len(v) if what == "index" else -1
    meshes[mesh] = (v, f, m, None)
    with pytest.raises(cwp.CwpError) as e:
        cwp.Batch(meshes, builder=builder)
    assert e.value.code == cwp.ERR_INVALID
    text = f"mesh {mesh}: non-finite vertex {f[tri, corner]}" if what == "nan" else f"mesh {mesh} triangle {tri}: vertex index {f[tri, corner]} out of range"
    assert text in str(e.value)


def parts(n_verts, counts, half=5.0, size=None):
    """meshes that each use a few vertices of one array of n_verts, from its start to its end, and the same meshes compacted"""
    big = np.zeros((n_verts, 3), np.float32)   # (pages that nothing touches take no memory)
    rng = np.random.default_rng(5)
    shared, alone = [], []
    for i, n in enumerate(counts):
        at = (n_verts - 3 * n) * i // max(1, len(counts) - 1)
        big[at:at + 3 * n] = rng.uniform(-half, half, (3 * n, 3)) if size is None else (rng.uniform(-half, half, (n, 1, 3)) + rng.uniform(-size, size, (n, 3, 3))).reshape(-1, 3)
        f = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
        mat = np.full(n, i, np.int32)
        shared.append((big, f + at, mat, None)); alone.append((big[at:at + 3 * n], f, mat, None))
    return shared, alone


def same_layouts(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for w in (2, 4, 8) for x, y in zip(a.download(w), b.download(w)))


@pytest.mark.parametrize("counts", [(1, 2, 3), (255, 1, 257)])
@pytest.mark.parametrize("builder", [0, 1])
def test_parts_of_one_vertex_array(gpu, cwp, counts, builder):
    shared, alone = parts(5000, counts)
    v, f, m, _ = alone[0]
    strip_of = (v, np.concatenate([f, f[:1]]), np.concatenate([m, m[:1]]), None)   # and one mesh that goes up as it is
    assert same_layouts(cwp.Batch(shared + [strip_of], builder=builder), cwp.Batch(alone + [strip_of], builder=builder))


def test_parts_of_a_large_vertex_array_fit(gpu, cwp):
    shared, alone = parts(1 << 27, [4] * 128)   # 1.6 GB of vertices: once per mesh they would be more than the device holds
    assert same_layouts(cwp.Batch(shared), cwp.Batch(alone))


@pytest.mark.parametrize("what", ["index", "negative", "nan"])
def test_first_bad_corner_of_a_part(gpu, cwp, what):
    shared, _ = parts(5000, (10, 300))
    v, f, m, _ = shared[1]
    f = f.copy()
    if what == "nan":
        v[f[7, 1]] = np.nan
    else:
        f[7, 1] = len(v) if what == "index" else -1
    shared[1] = (v, f, m, None)
    with pytest.raises(cwp.CwpError) as e:
        cwp.Batch(shared)
    assert e.value.code == cwp.ERR_INVALID
    assert (f"mesh 1: non-finite vertex {f[7, 1]}" if what == "nan" else f"mesh 1 triangle 7: vertex index {f[7, 1]} out of range") in str(e.value)


@pytest.mark.parametrize("sizes", [(5000, 3, 6000, 1, 2), (1200,) * 30 + (4000,)])   # meshes that go up alone and, before, after and between them, together
@pytest.mark.parametrize("builder", [0, 1])
def test_small_meshes_between_large_ones(gpu, cwp, sizes, builder):
    rng = np.random.default_rng(7)
    meshes = []
    for i, n in enumerate(sizes):
        v = (rng.uniform(-50, 50, (n, 1, 3)) + rng.uniform(-0.2, 0.2, (n, 3, 3))).astype(np.float32)
        meshes.append((v.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(n, 3), rng.integers(0, 9, n).astype(np.int32), None))
    b = cwp.Batch(meshes, builder=builder)
    for width in (2, 4, 8):
        rec = b.download(width)[1].reshape(-1, 3, 4)
        got = np.concatenate([rec[:, 0, :3], rec[:, 1, :3], rec[:, 2, :3], rec[:, :2, 3].copy().view(np.int32).astype(np.float32)], 1)
        want = np.concatenate([np.concatenate([(t := v.reshape(-1, 3, 3))[:, 0], t[:, 1] - t[:, 0], t[:, 2] - t[:, 0], np.arange(len(f))[:, None], m[:, None]], 1)
                               for v, f, m, _ in meshes]).astype(np.float32)
        assert np.array_equal(want[np.lexsort(want.T)], got[np.lexsort(got.T)])


def test_large_and_small_parts(gpu, cwp):
    shared, alone = parts(200000, (2500, 3, 3000, 2), 50, 0.2)   # 90 KB of corners and more alone, the small ones together
    assert same_layouts(cwp.Batch(shared), cwp.Batch(alone))
