"""VCM renders of one scene before and after its 2D base-colour images change: the captured passes must follow.

The passes of a render are captured once and replayed while nothing that they were made from has changed.  A scene whose
images come or go keeps the addresses and sizes of all its buffers, so only the textures themselves tell the captures apart.
"""
import dataclasses

import numpy as np
import pytest

import ref_scenes

pytestmark = pytest.mark.gpu


def _scene():
    # two material classes (the glass boxes are transparent), so that the hits are sorted with and without images
    return dataclasses.replace(ref_scenes.textured_cornell(), materials=ref_scenes.media_cornell().materials)


@pytest.mark.parametrize("sort", [1, 0])
def test_images_set_and_removed_between_renders(device, sort):
    import selas_gb300 as sel
    rs = _scene()
    cam, settings = rs.sel_camera(sel, 40, 32), sel.vcm_settings(2, 6, 3, 0, True, 1.25)
    device.set_option(sel.SEL_OPTION_MATERIAL_SORT, sort)
    try:
        want = []
        for textures in ({}, rs.textures):  # freshly built scenes
            sc = dataclasses.replace(rs, textures=textures).build(sel, device)
            want.append(sc.vcm_generate_image(cam, settings))
            sc.release()
        assert not np.allclose(want[0], want[1], rtol=1e-2)
        sc = dataclasses.replace(rs, textures={}).build(sel, device)
        for step in (0, 1, 0, 1):
            for gid, image in rs.textures.items():
                sc.set_texture(gid, image if step else None)
            # the same paths; only the order of the FP64 additions to a pixel differs
            np.testing.assert_allclose(sc.vcm_generate_image(cam, settings), want[step], rtol=1e-5, atol=1e-8)
        sc.release()
    finally:
        device.set_option(sel.SEL_OPTION_MATERIAL_SORT, 1)
