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


def _coloured(values, name):
    sc = S.Scene()
    tri = np.eye(3, dtype=np.float32)
    for v in values:
        m = S.TriMesh(tri, tri, np.arange(3), material=S.Material())
        setattr(m.material, name, v)
        sc.add(m)
    return sc


_ROW = np.float32([0.1, 0.2, 0.3])
_COLOURS = {
    "scalar": np.float32(0.4), "zero_d": np.array(0.4), "one_element": np.float32([0.4]), "row_of_rows": _ROW[None],
    "column": _ROW[:, None], "four": np.float32([0.1, 0.2, 0.3, 0.4]), "none": None, "list": [0.1, 0.2, 0.3],
    "short_list": [0.1, 0.2], "texts": ["0.1", "0.2", "0.3"], "whole": np.array([1, 0, 2**40 + 1]),
    "objects": np.array([0.1, None, 0.3], object), "double": np.array([0.1, 1e300, -1e300]), "half": np.float16([0.1, 0.2, 0.3]),
}


def _outcome(sc):
    """The material fields of every mesh, or the type of the error."""
    try:
        nodes = S.flatten(sc).nodes
    except Exception as e:
        return type(e)
    return [bytes(nd.material) for nd in nodes if nd.mesh >= 0]


@pytest.mark.parametrize("name", ["diffuse", "specular", "emissive"])
@pytest.mark.parametrize("kind", sorted(_COLOURS))
def test_a_colour_is_taken_alike_at_any_node_count(kind, name):
    """A colour is three numbers, whatever else the scene holds: scalars, rows
    of another length or shape and other values are refused (or taken) as in a
    scene of one mesh, alone, in company and beside good ones."""
    v = _COLOURS[kind]
    alone = _outcome(_coloured([v], name))
    refused = {"scalar": TypeError, "zero_d": TypeError, "one_element": ValueError, "row_of_rows": TypeError,
               "four": ValueError, "none": TypeError, "short_list": ValueError, "objects": TypeError}
    if kind in refused:
        assert alone is refused[kind]
    for n in (1, 2, 3, 4, 9):
        many = _outcome(_coloured([v] * n, name))
        beside = _outcome(_coloured([_ROW] * n + [v] + [_ROW] * n, name))
        if isinstance(alone, type):
            assert many is alone and beside is alone
        else:
            assert many == alone * n
            assert beside == _outcome(_coloured([_ROW], name)) * n + alone + _outcome(_coloured([_ROW], name)) * n


@pytest.mark.parametrize("value", [None, "x", np.float32([1.0, 2.0])], ids=["none", "text", "pair"])
@pytest.mark.parametrize("name", ["shininess", "opacity"])
def test_a_number_is_taken_alike_at_any_node_count(name, value):
    alone = _outcome(_coloured([value], name))
    assert isinstance(alone, type)
    for n in (2, 3, 4, 9):
        assert _outcome(_coloured([value] * n, name)) is alone
