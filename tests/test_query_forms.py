"""The forms a query batch is traced in (eight lanes a ray, packets, streams) at the sizes where one gives way to the next,
over rays that run side by side, part, or do both, against brute force, bit for bit: records in GPU memory and in host
memory, whose limits differ.

The limits are rays for each warp that runs at once: 32 one-warp blocks a multiprocessor for flat scenes, 16 for scenes
with instances.
"""
import numpy as np
import pytest

import oracle
import selas_gb300 as sel
from conftest import HIT_FIELDS, assert_hits_equal
from selas_gb300 import scenes
from test_instances import _build, _release, graph_rays, scene_graph

pytestmark = pytest.mark.gpu


def _warps(per_sm):
    import torch
    return per_sm * torch.cuda.get_device_properties(0).multi_processor_count


def _camera(data, n, seed):
    """n rays of a frame in pixel order, neighbours well within a degree of one another."""
    rng = np.random.default_rng(seed)
    w = max(1, int(np.sqrt(n)))
    i = np.arange(n)
    verts = data.soup()[0].reshape(-1, 3)
    lo, hi = verts.min(axis=0), verts.max(axis=0)
    eye = (lo + hi) / 2 + (hi - lo).max() * np.array([0.1, 0.4, -1.5]) + rng.normal(size=3)
    at = np.stack([lo[0] + (hi[0] - lo[0]) * (i % w + 0.5) / w, lo[1] + (hi[1] - lo[1]) * (i // w + 0.5) / max(1, n // w),
                   np.full(n, (lo[2] + hi[2]) / 2)], axis=1)
    d = at - eye
    return np.broadcast_to(eye, (n, 3)).astype(np.float32), (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def _rays(data, n, kind, seed):
    org, d = _camera(data, n, seed) if kind != "surface" else scenes.surface_rays(data, n, seed=seed)
    org, d = np.array(org), np.array(d)
    if kind == "mixed":  # ranges of 32 that run side by side, that do not, and that just about do
        o2, d2 = scenes.surface_rays(data, n, seed=seed + 1)
        part = np.random.default_rng(seed).integers(0, 4, n // 32 + 1)[np.arange(n) // 32]
        swap = (part == 1) | ((part == 2) & (np.arange(n) % 8 == 0)) | ((part == 3) & (np.arange(n) % 7 == 0))
        org[swap], d[swap] = o2[swap], d2[swap]
    d[5::97] = 0.0  # untraceable rays among the others
    org[7::89] = np.nan
    return org.astype(np.float32), d.astype(np.float32)


def _trace(scene, recs, where):
    """The records after their query, from host memory or from a copy in GPU memory."""
    closest = recs.dtype == sel.RAYHIT_DTYPE
    if where == "host":
        got = recs.copy()
        (scene.intersect1M if closest else scene.occluded1M)(got)
        return got
    import torch
    dev = torch.from_numpy(recs.view(np.uint8).reshape(-1).copy()).cuda()
    (scene.intersect_device if closest else scene.occluded_device)(dev.data_ptr(), recs.size, None)
    torch.cuda.synchronize()
    return dev.cpu().numpy().view(recs.dtype)


@pytest.mark.parametrize("kind", ["camera", "surface", "mixed"])
@pytest.mark.parametrize("where,per_warp", [("device", 7), ("device", 8), ("device", 20), ("device", 64), ("host", 12),
                                            ("host", 32), ("host", 64)])
def test_flat_scenes_around_each_limit(device, kind, where, per_warp):
    data = scenes.displaced_icospheres(count=2, level=2, seed=41)
    limit = per_warp * _warps(32)
    org, d = _rays(data, limit + 37, kind, per_warp)
    sc = sel.Scene(device)
    data.attach_to(sc)
    sc.commit()
    for make, ref in ((sel.make_rayhits, oracle.intersect_bruteforce), (sel.make_rays, oracle.occluded_bruteforce)):
        want = make(org, d)
        ref(data.soup(), want)
        for n in (limit - 1, limit, limit + 1, limit + 37):
            assert_hits_equal(_trace(sc, make(org[:n], d[:n]), where), want[:n],
                              fields=("tfar",) if make is sel.make_rays else HIT_FIELDS)
    sc.release()


@pytest.mark.parametrize("per_warp", [9, 256])
@pytest.mark.parametrize("kind", ["camera", "surface"])
def test_large_scenes_around_their_limits(device, kind, per_warp):
    """Scenes of more than 2^20 triangles stay with eight lanes a ray a little longer, and their largest closest-hit batches
    are streams whatever the rays; against smaller batches."""
    data = scenes.displaced_icospheres(count=13, level=6, seed=43)
    limit = per_warp * _warps(32)
    org, d = _rays(data, limit + 37, kind, 9)
    sc = sel.Scene(device)
    data.attach_to(sc)
    sc.commit()
    assert sc.info().triangle_count > 1 << 20
    for make in (sel.make_rayhits, sel.make_rays):
        recs = make(org, d)
        want = np.concatenate([_trace(sc, part.copy(), "device") for part in np.array_split(recs, 10 * (per_warp // 8))])
        for n in (limit - 1, limit, limit + 1, limit + 37):
            assert_hits_equal(_trace(sc, recs[:n].copy(), "device"), want[:n],
                              fields=("tfar",) if make is sel.make_rays else HIT_FIELDS)
    sc.release()


@pytest.mark.parametrize("kind", ["camera", "surface"])
def test_records_in_gpu_memory_with_ties_and_segments(device, kind):
    """The same limits over device-resident records, whose segments end at, before and beyond their hits."""
    data = scenes.displaced_icospheres(count=2, level=1, seed=42)
    sc = sel.Scene(device)
    data.attach_to(sc)
    sc.commit()
    for per_warp in (8, 20, 64):
        n = per_warp * _warps(32) + 5
        org, d = _rays(data, n, kind, 100 + per_warp)
        first = sel.make_rayhits(org, d)
        oracle.intersect_bruteforce(data.soup(), first)
        pick = np.arange(n) % 4
        hit = np.isfinite(first["tfar"]) & (first["geomID"] != sel.INVALID_ID)
        t = np.where(hit, first["tfar"], np.float32(50.0)).astype(np.float32)
        tnear = np.where(pick == 3, t, np.float32(0.0)).astype(np.float32)
        tfar = np.choose(pick, [t, np.nextafter(t, np.float32(0.0)), np.full(n, np.inf, np.float32),
                                np.full(n, np.inf, np.float32)]).astype(np.float32)
        for make, ref in ((sel.make_rayhits, oracle.intersect_bruteforce), (sel.make_rays, oracle.occluded_bruteforce)):
            recs = make(org, d, tnear, tfar)
            want = recs.copy()
            ref(data.soup(), want)
            assert_hits_equal(_trace(sc, recs, "device"), want, fields=HIT_FIELDS if make is sel.make_rayhits else ("tfar",))
    sc.release()


@pytest.mark.parametrize("per_warp", [2, 32])
def test_instanced_scenes_around_each_limit(device, per_warp):
    g = scene_graph()
    built = _build(sel, device, g)
    limit = per_warp * _warps(16)
    org, d = graph_rays(limit + 37)
    side = np.arange(limit + 37) // 32 % 3 == 0  # every third range of 32 runs side by side
    org[side] = org[(np.arange(limit + 37) // 32 * 32)[side]]
    d[side] = d[(np.arange(limit + 37) // 32 * 32)[side]] + np.float32(0.001) * d[side]
    for make, any_hit in ((sel.make_rayhits, False), (sel.make_rays, True)):
        want = make(org, d)
        oracle.instanced_query(g, 0, want, any_hit=any_hit)
        for n in (limit - 1, limit, limit + 1, limit + 37):
            for where in ("device", "host"):
                got = _trace(built[0], make(org[:n], d[:n]), where)
                assert_hits_equal(got, want[:n], fields=("tfar",) if any_hit else HIT_FIELDS)
    _release(built)
