"""The march by patches of rays on the GPU (`-m gpu`): image sizes on either side of every line at which the shape of a patch or
of a tile changes, ragged edges, and row ranges that cut patches, against the per-ray search."""
import pytest
import torch

from raygaussx_b200 import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,rows", [(1, 1, None), (3, 5, (1, 4)), (37, 19, (3, 18)), (128, 128, None), (129, 128, None),
                                               (200, 200, (7, 150)), (201, 200, None), (256, 256, None), (259, 255, (2, 253))])
def test_patches_of_every_shape_match_the_per_ray_search(width, height, rows):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from raygaussx_b200 import render_optix as ro
    dev = torch.device("cuda")
    sc = scenes.tiny_scene(n=1500, width=width, height=height, log_scale_mean=-2.7, seed=width, dynamic_sampling=True, dt_step=0.005,
                           max_prim_slice=512)
    tens = [t.to(dev).contiguous() for t in sc.tensors()]
    sc.cameras[0].to(dev)
    cs = ro.camera_struct(sc.cameras[0])
    m = sc.march
    march = lambda flags: ro.Renderer._march(m.dt_step, m.dynamic_sampling, m.max_prim_slice, True, m.transmittance_eps, rows,
                                             cs.height, flags)
    r = ro.get_renderer()
    r.build(*tens[:4])
    lo, hi = (0, height) if rows is None else rows
    seg = slice(lo * width, hi * width)
    got = {}
    for label, flags in (("patches", 0), ("per_ray", _lib.FLAG_PER_RAY_SEARCH)):
        r.reset_counters()
        rgb, alpha, depth = r.forward(*tens, cs, march(flags | _lib.FLAG_COUNT_WORK), want_alpha=True, want_depth=True)
        got[label] = (rgb[seg].clone(), alpha[seg].clone(), depth[seg].clone(), r.read_counters())
    for k in ("rays", "slabs", "slabs_hit", "closest_queries", "hits", "hits_hash", "overflow_slabs"):
        assert got["patches"][3][k] == got["per_ray"][3][k], k
    for a, b, tol in zip(got["patches"][:3], got["per_ray"][:3], (1e-5, 1e-5, 1e-4)):
        assert (a - b).abs().max().item() < tol
    plain, _, _ = r.forward(*tens, cs, march(0))
    assert torch.equal(plain[seg], got["patches"][0])
    rgb, _, _ = r.forward(*tens, cs, march(_lib.FLAG_SAVE_HITS))
    assert torch.equal(rgb[seg], plain[seg])
    dl = torch.sign(rgb - 0.5) / (3 * rgb.shape[0])
    grads = []
    for flags in (0, _lib.FLAG_PER_RAY_SEARCH):
        out = [torch.zeros_like(t) for t in tens]
        r.backward(*tens, cs, march(flags), rgb, dl, tuple(out))
        grads.append(out)
    for a, b in zip(*(g[:5] for g in grads)):
        assert ((a - b).abs().max() / b.abs().max().clamp_min(1e-30)).item() < 3e-4
