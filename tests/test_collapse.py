"""The collapse of the converter into wide nodes: every triangle in one leaf, every node below one
parent, and the node slots filled (opening the child of largest area left 4.2-4.3 of 8 filled)."""
import numpy as np
import pytest

from imbatracer_b200 import scene as S
from tests import helpers as H


@pytest.mark.parametrize("name,width,fill", [("tiny", 8, 0.0), ("config1", 8, 5.8), ("config1", 4, 3.3),
                                             ("config2", 8, 5.5), ("config2", 4, 3.2)])
def test_collapse_is_a_tree_with_filled_nodes(name, width, fill):
    td = H.traversal_data(name)
    nodes, tris, insts, root = H.wide_arrays(td, width)[:4]
    raw = np.ascontiguousarray(nodes).view(np.uint8).reshape(-1, 80)
    imask, meta = raw[:, 15], raw[:, 24:32]
    internal = np.unpackbits(imask[:, None], axis=1, bitorder="little").sum(1)
    leaves = (meta >> 5 > 0).sum(1)
    base = raw[:, 16:20].copy().view(np.uint32)[:, 0]
    below = np.concatenate([np.arange(b, b + k) for b, k in zip(base, internal)])
    assert len(np.unique(below)) == len(below)                       # one parent each
    assert len(raw) - len(below) == len(set(td.instances["next"].tolist())) + 1   # but the roots
    assert (meta >> 5).sum() == len(np.ascontiguousarray(tris).view(np.uint8).reshape(-1, 48)) + len(
        np.ascontiguousarray(insts).view(np.uint8).reshape(-1, 64))
    assert (internal + leaves).max() <= width
    assert (internal + leaves).mean() >= fill


@pytest.mark.parametrize("width,most", [(8, 0.15), (4, 0.3)])
def test_collapse_of_extentless_geometry(width, most):
    """Boxes without area cost nothing either way: their nodes are filled all the same, instead of one
    wide node for every binary one (0.76 n of them)."""
    n = 3000
    v = np.zeros((3 * n, 3), np.float32)
    v[:, 0] = np.repeat(np.arange(n), 3)
    idx = np.concatenate([np.arange(3 * n).reshape(n, 3), np.zeros((n, 1), int)], 1).astype(np.int32)
    td = S.build_traversal_data([S.Mesh(v, idx)], [S.Instance(0)])
    nodes, tris = H.wide_arrays(td, width)[:2]
    assert len(tris) == n and len(nodes) <= most * n
