"""Host-memory queries that go through copies in GPU memory: one copy, and chunks of 262,144 records in turn on four
streams, whose last chunk is short.  Batches take them with the zero-copy option off, from records the GPU cannot read in
place (not 16-byte aligned) and, for closest hits, from more than 2,097,152 page-locked records that run nearly parallel.
"""
import numpy as np
import pytest

import oracle
import selas_gb300 as sel
from conftest import HIT_FIELDS, assert_hits_equal
from selas_gb300 import scenes

pytestmark = pytest.mark.gpu

CHUNK = 1 << 18
FIELDS = {96: HIT_FIELDS, 48: ("tfar",)}


@pytest.fixture(scope="module")
def scene(device):
    data = scenes.displaced_icospheres(count=2, level=2, seed=51)
    sc = sel.Scene(device)
    data.attach_to(sc)
    sc.commit()
    yield data, sc
    sc.release()


def _want(data, recs):
    want = recs.copy()
    (oracle.intersect_bruteforce if recs.dtype.itemsize == 96 else oracle.occluded_bruteforce)(data.soup(), want)
    return want


def _query(sc, address, n, size):
    sel.check((sel.lib().sel_intersect1M if size == 96 else sel.lib().sel_occluded1M)(sc.handle, address, n, size))


@pytest.mark.parametrize("n", [700, 2 * CHUNK, 2 * CHUNK + 1, 5 * CHUNK + 17])
@pytest.mark.parametrize("make", [sel.make_rayhits, sel.make_rays])
def test_copies_return_what_brute_force_does(device, scene, make, n):
    data, sc = scene
    recs = make(*scenes.surface_rays(data, n, seed=52))
    size = recs.dtype.itemsize
    want = _want(data, recs)
    try:
        for zero_copy, offset in ((0, 0), (1, 4), (1, 0)):
            device.set_option(sel.SEL_OPTION_ZERO_COPY, zero_copy)
            raw = np.full(n * size + 96, 0xA5, np.uint8)
            start = (-raw.ctypes.data) % 16 + 16 + offset
            raw[start:start + n * size] = recs.view(np.uint8).reshape(-1)
            _query(sc, raw.ctypes.data + start, n, size)
            assert_hits_equal(raw[start:start + n * size].copy().view(recs.dtype), want, fields=FIELDS[size])
            assert (raw[:start] == 0xA5).all() and (raw[start + n * size:] == 0xA5).all()
    finally:
        device.set_option(sel.SEL_OPTION_ZERO_COPY, 1)


@pytest.mark.parametrize("n", [8 * CHUNK, 8 * CHUNK + 1])
def test_page_locked_parallel_records_around_the_staging_limit(scene, n):
    """2,097,152 records are traced in place, one more goes through the copies."""
    import torch
    data, sc = scene
    w = 1449
    i = np.arange(n)
    org = np.broadcast_to(np.array([0.0, 70.0, -170.0]), (n, 3)).astype(np.float32)
    at = np.stack([(i % w) / w * 160.0 - 80.0, (i // w) / w * 80.0, np.zeros(n)], axis=1)
    d = at - org
    recs = sel.make_rayhits(org, (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))
    pinned = torch.from_numpy(recs.view(np.uint8).reshape(-1)).pin_memory()
    _query(sc, pinned.data_ptr(), n, 96)
    got = pinned.numpy().view(recs.dtype)
    resident = torch.from_numpy(recs.view(np.uint8).reshape(-1)).cuda()
    sc.intersect_device(resident.data_ptr(), n)
    torch.cuda.synchronize()
    assert_hits_equal(got, resident.cpu().numpy().view(recs.dtype))
    some = np.r_[0:2000, n - 2000:n]
    assert_hits_equal(got[some], _want(data, recs[some]))
    assert (got["geomID"] != sel.INVALID_ID).any()


@pytest.mark.parametrize("stride", [96, 128])
def test_page_locked_and_pageable_records_in_place_and_copied(device, scene, stride):
    """Every way of a 30,000-record batch, dense and embedded in a larger struct, against brute force (not against one
    another)."""
    import torch
    data, sc = scene
    n = 30000
    recs = sel.make_rayhits(*scenes.surface_rays(data, n, seed=53))
    want = _want(data, recs)
    try:
        for zero_copy in (1, 0):
            device.set_option(sel.SEL_OPTION_ZERO_COPY, zero_copy)
            for pinned in (True, False):
                raw = torch.full((n * stride,), 0xA5, dtype=torch.uint8)
                raw = (raw.pin_memory() if pinned else raw).numpy()
                body = raw.reshape(n, stride)
                body[:, :96] = recs.view(np.uint8).reshape(n, 96)
                sel.check(sel.lib().sel_intersect1M(sc.handle, raw.ctypes.data, n, stride))
                assert_hits_equal(np.ascontiguousarray(body[:, :96]).view(recs.dtype).reshape(n), want)
                assert (body[:, 96:] == 0xA5).all()
    finally:
        device.set_option(sel.SEL_OPTION_ZERO_COPY, 1)
