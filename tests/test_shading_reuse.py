"""Shading kernels: what they skip and how they split a queue.

The Disney Fresnel term of a surface with metallic 0 ends at its dielectric part without running the Schlick part.

A denormal metallic runs the whole interpolation, (1 - m) * fd + m * fm, and rounds to the same floats as metallic 0:
1 - m is 1 and m * fm is far below half an ulp of fd, which is at least 1e-3 for the indices used here.  So both must
agree bit for bit, in every evaluation and sample.

One block of 512 or 640 threads per SM steps through the queue, all blocks with equally many entries a step (a multiple
of 32).  However a batch falls into blocks and steps, its paths are the same: only the order of the FP64 additions to a
pixel differs (about 1e-15 relative each), so images agree to one rounding of the result to FP32, 2^-23.
"""
from pathlib import Path

import numpy as np
import pytest

import oracle

BASE, METALLIC, RELATIVE_IOR, SPECULAR_TINT, IOR = slice(9, 12), 19, 24, 25, 28
GOLDEN = Path(__file__).resolve().parent / "golden" / "bsdf_golden.npz"


def _run(fn_name, surf, a, b, width):
    import torch

    import selas_gb300 as sel
    from selas_gb300._build import build_library
    build_library()
    dev = [torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda() for x in (oracle.surface_records(surf), a, b)]
    out = torch.zeros((len(surf), width), dtype=torch.float32, device="cuda")
    sel.check(getattr(sel.lib(), fn_name)(*(t.data_ptr() for t in dev), len(surf), out.data_ptr(), None))
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("base", [None, 0.0, 1e-38, 1e-31, 1.0])
@pytest.mark.parametrize("tint", [0.0, 1.0])
def test_metallic_zero_equals_denormal_metallic(base, tint):
    golden = dict(np.load(GOLDEN))
    for name, kind, second, width in (("sel_bsdf_evaluate_device", "e", "wi_e", 5),
                                      ("sel_bsdf_sample_device", "s", "u_s", 16)):
        surf = golden[f"surf_{kind}"].copy()
        surf[:, IOR] = np.linspace(1.2, 2.4, len(surf))
        surf[:, RELATIVE_IOR] = 1.0 / surf[:, IOR]
        surf[:, SPECULAR_TINT] = tint
        if base is not None:
            surf[:, BASE] = base
        got = []
        for metallic in (0.0, 1e-42):
            surf[:, METALLIC] = metallic
            got.append(_run(name, surf, golden[f"wo_{kind}"], golden[second], width))
        assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))


# batches around one warp, around the most that the forms with a thread for each part of an entry take (160 and 256 a
# block on 152 SMs), around the wave of 512- and 640-thread blocks, and two steps with a remainder
@pytest.mark.gpu
@pytest.mark.parametrize("size,batch", [((9, 7), 1), ((9, 7), 31), ((9, 7), 33), ((400, 250), 24320), ((400, 250), 24321),
                                        ((400, 250), 38912), ((400, 250), 38913), ((400, 250), 77823),
                                        ((400, 250), 77825), ((400, 250), 97279), ((400, 250), 97281)])
def test_batches_of_any_size_give_one_image(device, size, batch):
    import selas_gb300 as sel
    from selas_gb300 import scenes
    rs = scenes.textured_spheres(count=4, level=3)
    sc = rs.build(sel, device)
    cam = rs.sel_camera(sel, *size)
    imgs = []
    for paths in (batch, 0):
        st, df = sel.pt_settings(1, 5, seed=3), sel.deferred_settings(1, 6, seed=3)
        st.pathsInFlight = df.pathsInFlight = paths
        imgs.append((sc.pt_generate_image(cam, st), sc.deferred_generate_image(cam, df)))
    sc.release()
    for got, want in zip(*imgs):
        np.testing.assert_allclose(got, want, rtol=2.0 ** -22, atol=1e-12)
