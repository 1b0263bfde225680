"""Images of few rays (`-m gpu`): the nearest Gaussians, on which the first of a view's two depths of lists is spent, may be met by no ray
of the view, and its lists be empty; what lies behind them is seen all the same."""
import pytest
import torch

from raygaussx_b200 import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 1500, 6000])
@pytest.mark.parametrize("width,height", [(1, 1), (1, 2), (2, 1), (3, 3), (1, 37), (5, 4), (9, 8)])
def test_views_of_few_rays_are_whole(width, height, n):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from raygaussx_b200 import render_optix as ro
    dev = torch.device("cuda")
    sc = scenes.tiny_scene(n=n, width=width, height=height, log_scale_mean=-2.6, sh_degree=1, seed=width)
    cs, m = ro.camera_struct(sc.cameras[0].to(dev)), sc.march
    tens = [t.to(dev).contiguous() for t in sc.tensors()]

    def view(flags):
        r = ro.Renderer(dev)                       # nothing learnt from views before
        r.build(*tens[:4])
        return r.forward(*tens, cs, r._march(m.dt_step, m.dynamic_sampling, m.max_prim_slice, False, m.transmittance_eps, None, height, flags),
                         want_alpha=True, want_depth=True)

    two_depths, complete = view(0), view(_lib.FLAG_COUNT_WORK)
    assert complete[1].max().item() > 0.5
    for a, b in zip(two_depths, complete):
        assert torch.equal(a, b)
