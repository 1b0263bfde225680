"""The gradient tensors of a backward (`-m gpu`): each in memory of its own, and zero where no ray came, at sizes around the blocks that
clear them and on addresses that are not 16-byte aligned."""
import pytest
import torch

from raygaussx_b200 import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ro():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from raygaussx_b200 import render_optix
    return render_optix


def scene(n, degree, lobes):
    dev = torch.device("cuda")
    sc = scenes.tiny_scene(n=n, width=12, height=12, log_scale_mean=-2.5, sh_degree=degree, lobes=lobes)
    sc.cameras[0].to(dev)
    return sc, [t.to(dev).contiguous() for t in sc.tensors()]


def test_a_kept_gradient_keeps_no_other(ro):
    sc, tens = scene(1500, 3, 2)
    leaves = [t.requires_grad_() for t in tens]
    m = sc.march
    st = ro.RenderOptixSettings(None, False, None, None, None, None, None, m.dt_step, m.dynamic_sampling, sc.cameras[0], m.max_prim_slice, 2)
    grads = torch.autograd.grad(ro.RenderOptixFunction.apply(*leaves, st).sum(), leaves)
    assert len({g.untyped_storage().data_ptr() for g in grads}) == 8
    assert all(g.untyped_storage().nbytes() < 4 * g.numel() + 16 for g in grads)


@pytest.mark.parametrize("n,degree,lobes,offset", [(1, 0, 0, 0), (31, 1, 1, 1), (2048, 2, 0, 3), (2049, 3, 2, 0), (2731, 2, 3, 2), (8192, 0, 1, 1)])
def test_gradients_are_cleared_before_they_are_written(ro, n, degree, lobes, offset):
    sc, tens = scene(n, degree, lobes)
    cs, m = ro.camera_struct(sc.cameras[0]), sc.march
    r = ro.get_renderer()
    r.build(*tens[:4])
    march = ro.Renderer._march(m.dt_step, m.dynamic_sampling, m.max_prim_slice, m.white_background, m.transmittance_eps, None, cs.height,
                               _lib.FLAG_SAVE_HITS)
    rgb, _, _ = r.forward(*tens, cs, march)
    dl = torch.sign(rgb - 0.5) / rgb.numel()
    out = []
    for value, at in ((0.0, 0), (float("nan"), offset)):
        room = [torch.full((t.numel() + 8,), value, device=t.device) for t in tens]
        grads = [q[at:at + t.numel()].view(t.shape) for q, t in zip(room, tens)]
        march.flags = _lib.FLAG_ACCUMULATE if at == 0 and value == 0.0 else 0
        r.backward(*tens, cs, march, rgb, dl, tuple(grads))
        if march.flags == 0:                                    # nothing outside the tensors is written to
            for q, t in zip(room, tens):
                assert torch.isnan(q[:at]).all() and (t.numel() == 0 or torch.isnan(q[at + t.numel():]).all())
        out.append(grads)
    for a, b in zip(*out):
        assert torch.isfinite(b).all()
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-5 * float(a.abs().max()) if a.numel() else 0.0)
        if a.numel():
            assert torch.equal(a.reshape(n, -1).any(dim=1), b.reshape(n, -1).any(dim=1))
