"""How deep the lists of recording forwards are (`-m gpu`): deeper after rays went beyond them, shallower again after a while without, and
what was asked for with a set of another size."""
import pytest
import torch

from raygaussx_b200 import _lib, scenes

pytestmark = pytest.mark.gpu


def test_lists_get_shallower_again():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from raygaussx_b200 import render_optix as ro
    dev = torch.device("cuda")
    sc = scenes.unbounded_scene(n=1_000_000, n_cameras=3, width=628, height=414)
    tens = [t.to(dev).contiguous() for t in sc.tensors()]
    tens[1] = tens[1] * 3.0 ** (1.0 / 3.0)                  # as large as their distances: some 30 pairs per ray
    cam, m = sc.cameras[0], sc.march
    cam.to(dev)
    cs = ro.camera_struct(cam)
    rays = cs.width * cs.height
    march = ro.Renderer._march(m.dt_step, m.dynamic_sampling, m.max_prim_slice, m.white_background, m.transmittance_eps, None, cs.height,
                               _lib.FLAG_SAVE_HITS)
    r = ro.Renderer(dev)

    def views(n, t=tens):
        """(pairs in the lists per ray, whether rays went beyond) of n views."""
        out = []
        for _ in range(n):
            r.near_lists()                                  # forgets the cached lists and the figures
            r.forward(*t, cs, march)
            st = r.near_lists()
            out.append((r.read_binning()["pairs"] / rays, st["views_with_rays_beyond"] > 0))
        return out

    r.build(*tens[:4])
    r.near_lists(1, 0)                                      # one pair per ray: too shallow
    first = views(12)
    assert any(beyond for _, beyond in first)
    deep = first[-1][0]
    assert deep > 2.5 and not first[-1][1]                  # 3 pairs per ray or more suffice here: deepened to 4
    later = views(80)
    assert min(k for k, _ in later) < 0.75 * deep           # after 64 views without such rays they were tried half as deep
    few = [t[:-1].contiguous() for t in tens]
    r.build(*few[:4])
    again = views(2, few)
    assert again[1][0] < 1.6                                # a set of another size begins where the first one did
