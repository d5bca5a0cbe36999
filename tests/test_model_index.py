"""ID lookups of a model: the table and the difference for IDs that fill a range give
what the sort and search give, and refuse what they refuse."""

import numpy as np
import pytest

from lightfem_gb300 import mesh

IDS = {"from one": np.arange(1, 13), "negative": np.arange(-5, 7), "gap": np.r_[1:7, 8:14],
       "far gap": np.r_[1:12, 2**62], "low end": np.iinfo(np.int64).min + np.arange(12),
       "high end": np.iinfo(np.int64).max - 11 + np.arange(12)}


def model_with(node_ids, element_ids=None, material_ids=None):
    model = mesh.cantilever(3, 2)
    model.sort_and_index()
    assert model.n_nodes == node_ids.shape[0]
    model.node_ids = node_ids
    if element_ids is not None:
        model.element_ids = element_ids
        model.material_ids = material_ids
    return model


def searched(ids, wanted):
    order = np.argsort(ids, kind="stable")
    where = np.clip(np.searchsorted(ids[order], wanted), 0, ids.shape[0] - 1)
    assert np.all(ids[order][where] == wanted)
    return order[where]


@pytest.mark.parametrize("name", IDS)
@pytest.mark.parametrize("shuffle", [False, True])
def test_lookups(name, shuffle):
    rng = np.random.default_rng(4)
    ids = IDS[name].astype(np.int64)
    nodes = rng.permutation(ids) if shuffle else ids
    model = model_with(nodes, ids, ids)
    wanted = rng.choice(ids, 40)
    for got, base in ((model.node_index(wanted), nodes), (model.element_index(wanted), ids),
                      (model.material_index(wanted), ids)):
        np.testing.assert_array_equal(got, searched(base, wanted))
        assert got.dtype == np.int64
    for lookup in (model.node_index, model.element_index, model.material_index):
        assert lookup(np.empty(0, np.int64)).shape == (0,)
        for missing in {0, 7, 40, -6, 2**63 - 1, -2**63} - set(ids.tolist()):
            with pytest.raises(ValueError):
                lookup(np.r_[ids[0], missing].astype(np.int64))


def test_duplicate_node_ids_take_the_general_path():
    ids = np.array([1, 2, 2, 4, 5, 6, 7, 8, 9, 10, 11, 12])
    model = model_with(ids)
    np.testing.assert_array_equal(model.node_index(np.array([4, 2, 12])), [3, 1, 11])
    with pytest.raises(ValueError):
        model.node_index(np.array([3]))


def test_node_order_with_a_duplicate_is_refused():
    model = model_with(np.arange(1, 13))
    with pytest.raises(ValueError):
        model.index_with_node_order(np.r_[1:12, 1])
    model.index_with_node_order(np.arange(12, 0, -1))
    np.testing.assert_array_equal(model.node_ids, np.arange(12, 0, -1))
