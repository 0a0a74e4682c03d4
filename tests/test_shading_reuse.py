"""The Disney Fresnel term of a surface with metallic 0 ends at its dielectric part without running the Schlick part.

A denormal metallic runs the whole interpolation, (1 - m) * fd + m * fm, and rounds to the same floats as metallic 0:
1 - m is 1 and m * fm is far below half an ulp of fd, which is at least 1e-3 for the indices used here.  So both must
agree bit for bit, in every evaluation and sample.
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
