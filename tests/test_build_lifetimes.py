"""Scenes of one small subtree committed by several threads at once: what a build copies to the GPU (the subtree's task,
the tables, small meshes gathered into one copy) has to outlive the copies whatever else the host does meanwhile."""
import threading

import numpy as np
import pytest

import oracle
import selas_gb300 as sel
from conftest import assert_hits_equal
from selas_gb300.scenes import TriangleScene

pytestmark = pytest.mark.gpu


def test_small_scenes_built_by_several_threads(device):
    results, errors = {}, []

    def build(k):
        try:
            for n in (1, 7, 500, 1024, 1025, 3000):
                rng = np.random.default_rng(1000 * k + n)
                tris = (rng.uniform(-10, 10, (n, 1, 3)) + rng.uniform(-0.7, 0.7, (n, 3, 3))).astype(np.float32)
                data = TriangleScene()
                for gid, part in enumerate(np.array_split(tris, 3)):  # several small meshes, some empty
                    data.add(gid, part.reshape(-1, 3), np.arange(3 * len(part), dtype=np.uint32).reshape(-1, 3))
                sc = sel.Scene(device)
                data.attach_to(sc)
                sc.commit()
                target = tris[rng.integers(0, n, 300)].mean(axis=1)
                org = (target + rng.normal(size=(300, 3)) * 20.0).astype(np.float32)
                got = sel.make_rayhits(org, (target - org).astype(np.float32))
                want = got.copy()
                sc.intersect1M(got)
                results[k, n] = (data, got, want, sc.info().triangle_count)
                sc.release()
        except Exception as exc:  # reported by the test's own thread
            errors.append(exc)

    threads = [threading.Thread(target=build, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert len(results) == 36
    for (_, n), (data, got, want, count) in results.items():
        assert count == n
        oracle.intersect_bruteforce(data.soup(), want)
        assert_hits_equal(got, want, fields=("tfar", "u", "v", "primID", "geomID"))
