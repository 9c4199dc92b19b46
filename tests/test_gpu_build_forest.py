"""The device builder builds all meshes' trees and the instances' tree as one forest: meshes from
one triangle up, many more trees than a block has threads, sizes at the edges of a block's tile
and of the clusters one block finishes alone, and coinciding triangles (equal keys, no extent)."""
import numpy as np
import pytest

from imbatracer_b200 import scene as S
from imbatracer_b200 import scenegen as G
from oracle import oracle as O
from tests import helpers as H
from tests.test_gpu_build import _DeviceBytes, trace


def soup(rng, n, extent=6.0, size=0.7):
    c = rng.uniform(-extent, extent, (n, 1, 3))
    v = (c + rng.normal(scale=size, size=(n, 3, 3))).reshape(-1, 3)
    idx = np.concatenate([np.arange(3 * n).reshape(n, 3), np.zeros((n, 1), int)], 1)
    return S.Mesh(v.astype(np.float32), idx.astype(np.int32))


def placed(rng, mesh):
    m = np.eye(4)
    m[:3, :3] = G.rotation(rng) * rng.uniform(0.4, 1.5)
    m[:3, 3] = rng.uniform(-8, 8, 3)
    return S.Instance(mesh, m.astype(np.float32))


def forest(name):
    rng = np.random.default_rng(17)
    if name == "one":
        return [soup(rng, 1)], [S.Instance(0)]
    if name == "tiny trees":
        meshes = [soup(rng, int(n), 1.0, 1.0) for n in rng.integers(1, 5, 700)]
        return meshes, [placed(rng, i % 700) for i in range(900)]
    if name == "edges":
        meshes = [soup(rng, n) for n in (2, 3, 4, 31, 255, 256, 257, 2047, 2048, 2049, 4500)]
        return meshes, [placed(rng, i) for i in range(len(meshes))]
    if name == "coinciding":
        m = soup(rng, 1, 0.0, 3.0)
        v = np.tile(m.vertices, (1500, 1))
        idx = np.concatenate([np.arange(4500).reshape(1500, 3), np.zeros((1500, 1), int)], 1).astype(np.int32)
        return [S.Mesh(v, idx), soup(rng, 40)], [S.Instance(0), S.Instance(1)]
    if name == "many instances":       # fewer blocks an instance than the larger mesh has chunks of vertices
        meshes = [soup(rng, 3, 0.5, 0.3), soup(rng, 8000, 6.0, 0.1)]
        return meshes, [placed(rng, int(k in (17, 4321))) for k in range(6000)]
    return [soup(rng, 70000, 10.0, 0.1)], [S.Instance(0)]      # "large": several blocks, one tree


def records(ds, which, count, size):
    import torch
    raw = torch.as_tensor(_DeviceBytes(ds.device_arrays()[which], count * size), device="cuda").cpu().numpy()
    return raw.reshape(count, size)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["one", "tiny trees", "edges", "coinciding", "large", "many instances"])
def test_forest_build_and_refit(cuda, name):
    build_and_refit(name)


@pytest.mark.gpu
@pytest.mark.parametrize("name,limit", [("one", 1), ("tiny trees", 500), ("tiny trees", 100000), ("edges", 3000),
                                        ("edges", 4512), ("coinciding", 1500)])
def test_forest_in_batches(cuda, monkeypatch, name, limit):
    """Scenes above the batch limit: meshes above it alone, instances in the last batch or, where
    they do not fit there, in one of their own; the same hits, and refits of records and nodes that
    several batches wrote."""
    monkeypatch.setenv("IMBART_BUILD_BATCH", str(limit))
    build_and_refit(name)


def build_and_refit(name):
    meshes, instances = forest(name)
    n_tris = sum(m.triangle_count for m in meshes)
    ds = S.DeviceScene.build_gpu(meshes, instances)
    assert ds.info.triangles == n_tris and ds.info.instances == len(instances)
    ids = records(ds, 1, n_tris, 48)[:, 12:16].copy().view(np.int32)[:, 0]
    assert np.array_equal(np.sort(ids), np.arange(n_tris))                 # every triangle in one leaf
    nodes = records(ds, 0, int(ds.info.wide_nodes), 80)
    bottom = int(ds.info.wide_nodes - ds.info.top_nodes)
    counts = nodes[:, 24:32] >> 5
    assert counts[:bottom].sum() == n_tris and counts[bottom:].sum() == len(instances)
    assert counts.max() <= 3 and counts[bottom:].max() == 1
    internal = np.unpackbits(nodes[:, 15]).sum()
    assert internal == len(nodes) - len(meshes) - 1                        # every node but the roots has a parent
    layout = np.concatenate([[0], np.cumsum([m.triangle_count for m in meshes])[:-1]]).astype(np.int32)
    rays = G.random_rays(np.random.default_rng(3), 1500, [-9] * 3, [9] * 3)
    want = O.trace_brute(meshes, instances, layout, rays)
    got, _ = trace(ds, rays)
    assert (want["tri_id"] >= 0).any() or name == "one"
    assert H.hits_equal(want, got).all()
    # Moved twice: the second refit finds the counters the first one left.
    for step in (1, 2):
        moved = [S.Mesh((m.vertices * np.float32(1 + 0.1 * step)), m.indices, m.normals, m.texcoords, m.geom_normals)
                 for m in meshes]
        ds.refit(moved)
        want = O.trace_brute(moved, instances, layout, rays)
        got, _ = trace(ds, rays)
        assert H.hits_equal(want, got).all()
    ds.close()


@pytest.mark.gpu
def test_scratch_between_builds(cuda):
    """The scratch kept from one build to the next: smaller and larger scenes after each other, given
    back between builds, and two threads building at once; every build's arrays are the first one's."""
    import threading
    import torch
    from imbatracer_b200 import native as N
    scenes = [forest(n) for n in ("tiny trees", "one", "large", "edges")]

    def arrays(k, stream=None):
        ds = S.DeviceScene.build_gpu(*scenes[k], stream=stream)
        out = [records(ds, 0, int(ds.info.wide_nodes), 80), records(ds, 1, int(ds.info.triangles), 48)]
        ds.close()
        return out

    def same(k, stream=None):
        return all(np.array_equal(a, b) for a, b in zip(first[k], arrays(k, stream)))

    first = [arrays(k) for k in range(4)]
    for k in (1, 2, 0, 3, 2):
        assert same(k), k
        if k == 2:
            N.load().imbart_invalidate_scenes()
    wrong = []

    def work(order):
        try:
            stream = torch.cuda.Stream()       # of the thread's own: the builds overlap on the device
            wrong.extend(k for k in order if not same(k, stream))
        except Exception as e:          # shown by the assertion below
            wrong.append(repr(e))
    threads = [threading.Thread(target=work, args=(o,)) for o in ([0, 1, 2, 3] * 2, [2, 3, 0, 1] * 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == []


def slivers(x):
    """A small triangle at each x along an axis, all alike."""
    v = np.zeros((len(x), 3, 3))
    v[:, :, 0] = np.asarray(x)[:, None]
    v += np.array([[0, 0, 0], [0.25, 0, 0], [0, 0.25, 0.125]])
    n = len(x)
    idx = np.concatenate([np.arange(3 * n).reshape(n, 3), np.zeros((n, 1), int)], 1)
    return S.Mesh(v.reshape(-1, 3).astype(np.float32), idx.astype(np.int32))


def levels(ds, root):
    """Levels of wide nodes below `root`."""
    nodes = records(ds, 0, int(ds.info.wide_nodes), 80)
    internal = np.unpackbits(nodes[:, 15:16], axis=1).sum(1).astype(np.int64)
    base = nodes[:, 16:20].copy().view(np.uint32)[:, 0].astype(np.int64)
    at, n = np.array([root]), 0
    while len(at):
        n += 1
        at = np.concatenate([np.arange(base[i], base[i] + internal[i]) for i in at])
    return n


@pytest.mark.gpu
@pytest.mark.parametrize("name,n", [("coinciding", 1500), ("points", 5000), ("even", 4096), ("even", 30011),
                                    ("growing", 30000)])
def test_trees_of_tied_neighbours_are_shallow(cuda, name, n):
    """Every round adds at most one level and takes one pass over the clusters. Equally near
    neighbours pair up, so coinciding, extentless and evenly spaced triangles halve every round or
    nearly; spacings that grow along the row (no ties, each nearest to the one before) merge one pair
    a round until the positions pair up as they stand, after 128 rounds. Half as many rounds as
    triangles took 100 ms, these take 3."""
    if name == "points":
        m = slivers(np.zeros(n))
        mesh = S.Mesh(np.repeat(np.arange(n, dtype=np.float32), 3)[:, None] * np.float32([1, 0, 0]), m.indices)
    else:
        mesh = slivers({"coinciding": np.zeros(n), "even": np.arange(n), "growing": np.arange(n) ** 2 / 1024.0}[name])
    ds = S.DeviceScene.build_gpu([soup(np.random.default_rng(1), 3), mesh], [S.Instance(0), S.Instance(1)])
    halvings = int(np.ceil(np.log2(n)))
    if name == "points":
        assert ds.info.wide_nodes <= 0.3 * n           # no box has an area; a node per binary one: n / 2
    assert levels(ds, 1) <= (2 * halvings if name != "growing" else 128 + 2 * halvings)
    if name == "growing":
        times = []
        for _ in range(3):
            again = S.DeviceScene.build_gpu([soup(np.random.default_rng(1), 3), mesh], [S.Instance(0), S.Instance(1)])
            times.append(again.build_ms)
            again.close()
        assert min(times) < 30.0
    if name != "points":
        rng = np.random.default_rng(2)
        pick = rng.integers(0, n, 500)
        target = mesh.vertices.reshape(n, 3, 3)[pick].mean(1)
        org = target + rng.normal(size=target.shape)
        from imbatracer_b200 import native as N
        rays = np.zeros(500, N.RAY_DTYPE)
        rays["org"][:, :3], rays["dir"][:, :3], rays["dir"][:, 3] = org, target - org, 3.0e38
        meshes = [soup(np.random.default_rng(1), 3), mesh]
        want = O.trace_brute(meshes, [S.Instance(0), S.Instance(1)], np.array([0, 3], np.int32), rays)
        got, _ = trace(ds, rays)
        assert (want["tri_id"] >= 0).sum() > 400 and H.hits_equal(want, got).all()
    ds.close()


@pytest.mark.gpu
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_a_triangle_without_a_position_leaves_the_tree_as_good(cuda, sign):
    """NaN vertices (of either sign) stay out of the box that the order along the curve is cut from:
    rays visit as many nodes of the others' tree as without them."""
    import torch
    from imbatracer_b200 import native as N
    lib = N.load()
    mesh = soup(np.random.default_rng(4), 20000, 10.0, 0.1)
    v = np.concatenate([mesh.vertices, np.full((3, 3), np.copysign(np.float32(np.nan), np.float32(sign)))])
    lost = S.Mesh(v.astype(np.float32), np.concatenate([mesh.indices, [[60000, 60001, 60002, 0]]]).astype(np.int32))
    rays = G.random_rays(np.random.default_rng(5), 4000, [-10] * 3, [10] * 3)
    r = torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()).cuda()
    visits, hits = [], []
    for m in (mesh, lost):
        ds = S.DeviceScene.build_gpu([m], [S.Instance(0)])
        h = torch.zeros((len(rays), 4), dtype=torch.int32, device="cuda")
        counts = torch.zeros(3, dtype=torch.int64, device="cuda")
        N.check(lib.imbart_trace_stats(ds.handle, N.ptr(r), N.ptr(h), len(rays), N.TRACE_CLOSEST, N.ptr(counts), None),
                "imbart_trace_stats")
        torch.cuda.synchronize()
        visits.append(int(counts[0]))
        hits.append(h.cpu().numpy())
        ds.close()
    assert np.array_equal(hits[0], hits[1]) and (hits[0][:, 0] >= 0).sum() > 500
    assert visits[1] <= 1.1 * visits[0], visits
