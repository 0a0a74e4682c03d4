"""The streamed 8-wide traversal (lanes refilled with new rays, work taken over from blocks that have not started)
against the brute-force oracle, bit for bit, at the sizes where its ranges change."""
import numpy as np
import pytest

import oracle
import selas_gb300 as sel
from conftest import assert_hits_equal
from edge_scenes import grid_rays, grid_scene, segment_rayhits, segment_rays
from selas_gb300 import scenes

pytestmark = pytest.mark.gpu

RESIDENT = 152 * 32 * 32  # rays of a grid whose one-warp blocks all run at once on 152 SMs
GROUPS = 152 * 32 * 4 * 3  # rays of the largest batch traced by eight lanes a ray


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 1000, GROUPS, GROUPS + 1, RESIDENT, RESIDENT + 1,
                               2 * RESIDENT + 37])
def test_batch_sizes(device, n):
    data = scenes.displaced_icospheres(count=2, level=2, seed=21)
    sc = sel.Scene(device)
    data.attach_to(sc)
    sc.commit()
    org, d = scenes.surface_rays(data, n, seed=22)
    d[5::97] = 0.0        # untraceable rays among the others
    org[7::89] = np.nan
    for make, query, ref in ((sel.make_rayhits, sc.intersect1M, oracle.intersect_bruteforce),
                             (sel.make_rays, sc.occluded1M, oracle.occluded_bruteforce)):
        got, want = make(org, d), make(org, d)
        query(got)
        ref(data.soup(), want)
        assert_hits_equal(got, want, fields=("tfar",) if make is sel.make_rays else
                          ("tfar", "u", "v", "Ng_x", "primID", "geomID"))
    sc.release()


@pytest.mark.parametrize("scale,distance", [(1.0, 1e2), (1.0, 1e4), (1e-6, 1.0), (1e8, 3.0), (1e8, 1e3)])
def test_box_tests_stay_outside_the_boxes(device, scale, distance):
    """Origins far from small nodes (the offset's rounding) and huge scenes met by axis-parallel rays (the offset
    overflows): no hit may be lost.  Exact: the boxes only grow, so the answer is brute force's."""
    rng = np.random.default_rng(5)
    data = scenes.displaced_icospheres(count=6, level=2, seed=23, ground=False)
    data.meshes = [(g, (v * np.float32(scale)).astype(np.float32), f) for g, v, f in data.meshes]
    sc = sel.Scene(device)
    data.attach_to(sc)
    sc.commit()
    verts = data.soup()[0].reshape(-1, 3, 3)
    target = verts[rng.integers(0, verts.shape[0], 3000)].mean(axis=1, dtype=np.float64)
    d = rng.normal(size=(3000, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    axes = np.repeat(np.eye(3), 500, axis=0) * np.where(rng.random((1500, 1)) < 0.5, -1.0, 1.0)
    d[:1500] = axes
    org = (target - d * (100.0 * scale * distance)).astype(np.float32)
    d = d.astype(np.float32)
    got, want = sel.make_rayhits(org, d), sel.make_rayhits(org, d)
    sc.intersect1M(got)
    oracle.intersect_bruteforce(data.soup(), want)
    if distance <= 1e4:
        assert (want["geomID"] != sel.INVALID_ID).mean() > 0.9
    assert_hits_equal(got, want, fields=("tfar", "u", "v", "primID", "geomID"))
    sc.release()


def test_ties_and_edges_in_long_batches(device):
    """The edge-case rays (shared edges and vertices, ties, segment ends) among enough copies to be streamed."""
    data = grid_scene()
    sc = sel.Scene(device)
    data.attach_to(sc)
    sc.commit()
    org, d, _ = grid_rays()
    for make, query, ref in ((lambda: sel.make_rayhits(org, d), sc.intersect1M, oracle.intersect_bruteforce),
                             (segment_rayhits, sc.intersect1M, oracle.intersect_bruteforce),
                             (segment_rays, sc.occluded1M, oracle.occluded_bruteforce)):
        want = make()
        ref(data.soup(), want)
        copies = GROUPS // want.size + 2
        got = np.tile(make(), copies)
        query(got)
        assert_hits_equal(got, np.tile(want, copies), fields=("tfar",) if want.dtype == sel.RAY_DTYPE else
                          ("tfar", "u", "v", "Ng_x", "primID", "geomID"))
    sc.release()
