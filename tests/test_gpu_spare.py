"""Render()'s images over memory used before: kept ones stay as they were,
and every array is written whole, also where the scene covers nothing."""
import numpy as np
import pytest

from polyred_gb300 import procedural, render

pytestmark = pytest.mark.gpu
FIELDS = ("rgba", "tri_id", "depth", "mat_id", "shadow_maps")


@pytest.mark.parametrize("size", [(1, 1), (333, 77)])
@pytest.mark.parametrize("shadows", [False, True])
def test_kept_images(device, size, shadows):
    s, cam = procedural.small_scene(width=size[0], height=size[1])

    def renderer():
        return render.NewRenderer(render.Size(*size), render.Camera(cam), render.Scene(s), render.ShadowMap(shadows),
                                  render.GammaCorrection(True), render.Outputs_(*FIELDS), render.CUDA(device))

    r = renderer()
    r.Render()
    want = {k: a.copy() for k, a in r.outputs().items()}
    kept = []
    for k in range(6):
        r.Render()
        if k % 2:
            kept.append(r.outputs())
    for a in r.outputs().values():
        a.view(np.uint8)[...] = 0xA5  # the memory's next frame overwrites this
    last = kept.pop()
    del last
    r.Render()
    for got in kept + [r.outputs()]:
        for k in FIELDS:
            assert np.array_equal(got[k].view(np.uint8), want[k].view(np.uint8)), k
