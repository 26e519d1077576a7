"""Flattening a scene to the C ABI's node array: field by field (few nodes)
and column by column give the same array, also for transforms that are not
4x4 and nodes without a material."""
import numpy as np
import pytest

import edge_scenes as E
from minirender_gb300 import scene as S


def _scene(k):
    if k >= 0:
        return E.random_scene(k)[1]
    sc = S.Scene()
    tri = np.eye(3, dtype=np.float32)
    for j in range(3):
        m = S.TriMesh(tri, tri, np.arange(3), material=None if j == 1 else S.Material(diffuse=[0.1, 0.2, 0.3 + j]))
        m.transform = (np.arange(16, dtype=np.float64) / 7).reshape((16,) if j else (4, 4))
        sc.add(m).add(S.SceneNode())
    return sc


@pytest.mark.parametrize("k", [-1, 0, 3, 11])
def test_node_columns_equal_node_fields(k, monkeypatch):
    sc = _scene(k)
    got = {}
    for name, fill in (("fields", S._fill_nodes), ("columns", S._fill_columns)):
        monkeypatch.setattr(S, "_fill_nodes", fill)
        monkeypatch.setattr(S, "_fill_columns", fill)
        got[name] = bytes(S.flatten(sc).nodes)
        monkeypatch.undo()
    assert got["fields"] == got["columns"]
