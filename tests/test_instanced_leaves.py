"""Instanced traversal over leaves of every size.  What is left of a leaf when one of its records is an instance waits on
the traversal stack; with leaves of more than three records its mask reaches bits 24 to 31, where a node group keeps its
children, and the two must not be taken for one another."""
import numpy as np
import pytest

from conftest import assert_hits_equal
from selas_gb300 import make_rayhits, make_rays
from test_instances import INVALID, _build, _oracle, _release, graph_rays, scene_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [2, 3, 5, 6, 7, 8])
def test_leaves_of_instances(device, leaf):
    import selas_gb300 as sel
    g = scene_graph()
    built = _build(sel, device, g, leaf=leaf)
    org, d = graph_rays(8000)
    want = _oracle(g, org, d)
    assert (want["geomID"] != INVALID).sum() > 2000 and (want["instID1"] != INVALID).sum() > 20
    got = make_rayhits(org, d)
    built[0].intersect1M(got)
    assert_hits_equal(got, want)
    want = _oracle(g, org, d, any_hit=True)
    got = make_rays(org, d)
    built[0].occluded1M(got)
    np.testing.assert_array_equal(np.isneginf(got["tfar"]), np.isneginf(want["tfar"]))
    _release(built)
