"""The device BVH builder at the sizes where its kernels hand over to one another, against brute force."""
import numpy as np
import pytest

import oracle
import selas_gb300 as sel
from conftest import assert_hits_equal
from selas_gb300.scenes import TriangleScene

pytestmark = pytest.mark.gpu


def _soup(n, seed, kind):
    rng = np.random.default_rng(seed)
    if kind == "same":  # one triangle n times over: no plane separates them
        v = np.repeat(rng.uniform(-1, 1, (1, 3, 3)), n, axis=0)
    elif kind == "line":  # centroids on a line, sizes from tiny to huge
        c = np.zeros((n, 1, 3))
        c[:, 0, 0] = np.sort(rng.uniform(-50, 50, n))
        v = c + rng.uniform(-1, 1, (n, 3, 3)) * np.exp(rng.uniform(-6, 2, (n, 1, 1)))
    else:
        v = rng.uniform(-10, 10, (n, 1, 3)) + rng.uniform(-0.7, 0.7, (n, 3, 3))
    return v.astype(np.float32)


@pytest.mark.parametrize("leaf", [1, 3, 8])
@pytest.mark.parametrize("n", [1, 2, 8, 9, 16, 17, 32, 33, 1023, 1024, 1025, 2047, 2049, 6145])
def test_sizes(device, n, leaf):
    for kind in ("cloud", "line", "same"):
        tris = _soup(n, n + leaf, kind)
        data = TriangleScene()
        cut = n // 3  # two meshes, one of them possibly empty
        for gid, part in ((4, tris[:cut]), (2, tris[cut:])):
            data.add(gid, part.reshape(-1, 3), np.arange(3 * part.shape[0], dtype=np.uint32).reshape(-1, 3))
        sc = sel.Scene(device)
        sc.set_leaf_size(leaf)
        data.attach_to(sc)
        sc.commit()
        info = sc.info()
        assert info.triangle_count == n and info.max_depth <= 24
        flat = tris.reshape(-1, 3)
        assert tuple(info.bounds_lo) == tuple(flat.min(axis=0)) and tuple(info.bounds_hi) == tuple(flat.max(axis=0))
        rng = np.random.default_rng(7)
        target = tris[rng.integers(0, n, 700)].mean(axis=1)
        org = (target + rng.normal(size=(700, 3)) * 20.0).astype(np.float32)
        d = (target - org).astype(np.float32)
        got, want = sel.make_rayhits(org, d), sel.make_rayhits(org, d)
        sc.intersect1M(got)
        oracle.intersect_bruteforce(data.soup(), want)
        assert_hits_equal(got, want, fields=("tfar", "u", "v", "primID", "geomID"))
        sc.release()


def test_refuses_non_finite_vertices_in_use(device):
    v = np.zeros((4, 3), np.float32)
    v[1, 0] = v[2, 1] = 1.0
    v[3] = np.nan
    sc = sel.Scene(device)
    sc.attach_triangle_mesh(0, v, np.array([[0, 1, 2]], np.uint32))  # the NaN vertex is not referenced
    sc.commit()
    sc.attach_triangle_mesh(1, v, np.array([[0, 1, 3]], np.uint32))
    with pytest.raises(sel.SelError) as e:
        sc.commit()
    assert e.value.code == sel.SEL_ERR_INVALID_OPERATION and "non-finite" in str(e.value)
    sc.release()
