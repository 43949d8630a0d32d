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
