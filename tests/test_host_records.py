"""Host-memory queries on ordinary (pageable) records at every alignment and stride: traced in place where the GPU can
address them, staged otherwise, with the same bits as brute force and nothing else in the buffer touched."""
import numpy as np
import pytest

import oracle
import selas_gb300 as sel
from conftest import HIT_FIELDS, assert_hits_equal
from selas_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 700])
@pytest.mark.parametrize("stride,offset", [(0, 0), (0, 4), (0, 16), (16, 0), (4, 0), (32, 8), (160, 16)])
def test_alignments_and_strides(device, n, stride, offset):
    data = scenes.displaced_icospheres(count=3, level=2, seed=31)
    sc = sel.Scene(device)
    data.attach_to(sc)
    sc.commit()
    org, d = scenes.surface_rays(data, n, seed=32)
    lib = sel.lib()
    for make, call, ref in ((sel.make_rayhits, lib.sel_intersect1M, oracle.intersect_bruteforce),
                            (sel.make_rays, lib.sel_occluded1M, oracle.occluded_bruteforce)):
        recs = make(org, d)
        want = recs.copy()
        ref(data.soup(), want)
        step = recs.dtype.itemsize + stride
        raw = np.full(64 + offset + n * step + 64, 0xA5, np.uint8)
        start = (-raw.ctypes.data) % 16 + 16 + offset
        at = lambda i: slice(start + i * step, start + i * step + recs.dtype.itemsize)
        before = raw.copy()
        for i in range(n):
            raw[at(i)] = recs[i:i + 1].view(np.uint8)
        sel.check(call(sc.handle, raw.ctypes.data + start, n, step))
        got = np.concatenate([raw[at(i)] for i in range(n)]).view(recs.dtype)
        assert_hits_equal(got, want, fields=HIT_FIELDS if recs.dtype == sel.RAYHIT_DTYPE else ("tfar",))
        for i in range(n):
            raw[at(i)] = before[at(i)]
        assert np.array_equal(raw, before)
    sc.release()
