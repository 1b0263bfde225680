"""Gaussians of an infinite scale, or of one whose square is (`-m gpu`): cylinders and slabs without end, whose box has no middle.  The tile
lists have to hold them, and the march to test them, wherever a ray can meet them: hits, counted and hashed, against the search of all
Gaussians."""
import math

import pytest
import torch

from raygaussx_b200 import _lib, scenes

pytestmark = pytest.mark.gpu


def check(sc, cam, height):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from raygaussx_b200 import render_optix as ro
    dev = torch.device("cuda")
    cam.to(dev)
    cs = ro.camera_struct(cam)
    tens = [t.to(dev).contiguous() for t in sc.tensors()]
    r = ro.Renderer(dev)
    r.build(*tens[:4])
    got = {}
    for label, flags in (("lists", 0), ("all", _lib.FLAG_BRUTE_FORCE)):
        r.reset_counters()
        rgb, alpha, _ = r.forward(*tens, cs, r._march(0.01, False, 2048, False, 1e-3, None, height, flags | _lib.FLAG_COUNT_WORK),
                                  want_alpha=True)
        got[label] = (rgb.clone(), alpha.clone(), r.read_counters())
    for k in ("rays", "slabs", "slabs_hit", "hits", "hits_hash"):
        assert got["lists"][2][k] == got["all"][2][k], k
    assert got["lists"][2]["hits"] > 0
    for a, b in zip(got["lists"][:2], got["all"][:2]):     # hits are met in another order: the sums' last bits
        assert (a - b).abs().max().item() < 1e-5


@pytest.mark.parametrize("axes", [1, 2])
@pytest.mark.parametrize("width,height", [(1, 1), (61, 40), (150, 131), (230, 201)])
def test_infinite_gaussians_are_met(axes, width, height):
    sc = scenes.tiny_scene(n=600, width=width, height=height, log_scale_mean=-3.0, density_scale=1.0, seed=width + axes)
    sc.scales[::60, :axes] = math.inf
    check(sc, sc.cameras[0], height)


@pytest.mark.parametrize("width,height", [(6, 5), (150, 131), (230, 201)])
def test_slabs_across_the_view_are_met(width, height):
    """Seen along their normal: endless ranges of ray parameters, and no width across the patch's cone at all."""
    sc = scenes.tiny_scene(n=600, width=width, height=height, log_scale_mean=-3.0, density_scale=1.0, seed=width)
    sc.scales[::60] = torch.tensor([0.2, 3e19, 3e19])
    sc.quaternions[::60] = torch.tensor([1.0, 0.0, 0.0, 0.0])
    check(sc, scenes.SimpleCamera((4.0, 0.0, 0.0), target=(0.0, 0.0, 0.0), width=width, height=height), height)
