"""The fused kernels of the training iteration against the operators they stand for (`-m gpu`)."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tr():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    from raygaussx_b200 import _lib, training
    _lib.lib()
    return training


@pytest.mark.parametrize("w,h,factor,lam", [(1, 1, (1, 1), 0.2), (5, 3, (1, 1), 1.0), (32, 32, (1, 1), 0.2), (33, 31, (2, 3), 0.2),
                                            (100, 45, (1, 1), 0.0), (70, 129, (3, 1), 0.5)])
def test_image_loss_and_its_gradient(tr, w, h, factor, lam):
    g = torch.Generator(device="cuda").manual_seed(w * 1000 + h)
    target = torch.rand(3, h, w, generator=g, device="cuda")
    rays = torch.rand(w * h * factor[0] * factor[1], 3, generator=g, device="cuda").requires_grad_(True)
    loss = tr.image_loss(rays, target, w, h, factor, lam)
    (loss * 0.05).backward()
    got = rays.grad.clone()
    r64 = rays.detach().double().requires_grad_(True)
    image = tr.reduce_supersampling(w, h, r64, factor).permute(2, 0, 1)
    want = (1 - lam) * tr.l1_loss(image, target.double()) + lam * (1 - tr.ssim(image, target.double()))
    (want * 0.05).backward()
    assert loss.item() == pytest.approx(want.item(), rel=2e-5, abs=1e-6)
    assert (got.double() - r64.grad).norm() <= 2e-4 * r64.grad.norm()


@pytest.mark.parametrize("n,degree,lobes", [(1, 3, 0), (255, 0, 7), (257, 1, 3), (1000, 2, 1), (4099, 3, 0)])
@pytest.mark.parametrize("normalize", [True, False])
def test_parameterisation_and_its_gradient(tr, n, degree, lobes, normalize):
    g = torch.Generator().manual_seed(n + degree)
    k = (degree + 1) ** 2
    args = [torch.randn(n, 3, generator=g), torch.exp(torch.randn(n, 3, generator=g)), torch.randn(n, 4, generator=g),
            torch.rand(n, generator=g), torch.randn(n, 3, k, generator=g)]
    if lobes:
        args += [torch.randn(n, 3, lobes, generator=g), 30 * torch.rand(n, lobes, generator=g), torch.randn(n, lobes, 3, generator=g)]
    dev = tr.SimplePointCloud(*[a.cuda() for a in args])
    ref = tr.SimplePointCloud(*[a.double() for a in args])          # on the CPU: composed of operators
    for a, b in zip((dev.scales, dev.bandwidth_sharpness), (ref.scales, ref.bandwidth_sharpness)):
        b.data.copy_(a.data)
    outs, wants = dev.get_data(normalize, normalize), ref.get_data(normalize, normalize)
    total = total_ref = 0.0
    for i, (a, b) in enumerate(zip(outs, wants)):
        assert a.shape == b.shape
        if b.numel():
            assert torch.allclose(a.detach().double().cpu(), b.detach(), rtol=3e-6, atol=1e-6), i
            weight = torch.randn(b.shape, generator=g, dtype=torch.float64)
            total = total + (a * weight.float().cuda()).sum()
            total_ref = total_ref + (b * weight).sum()
    total.backward()
    total_ref.backward()
    for name in ("positions", "scales", "quaternions", "densities", "rgb", "spherical_harmonics", "bandwidth_sharpness", "lobe_axis"):
        a, b = getattr(dev, name).grad, getattr(ref, name).grad
        if b is not None and b.numel():
            assert torch.allclose(a.double().cpu(), b, rtol=2e-5, atol=1e-5), name


def test_adam_steps_like_the_base_class(tr):
    g = torch.Generator(device="cuda").manual_seed(1)
    shapes = [(4099, 3), (4096,), (1,), (7, 5, 3), (4097,)]
    ours = [torch.randn(s, generator=g, device="cuda").requires_grad_(True) for s in shapes]
    odd = torch.randn(1002, generator=g, device="cuda")[1:].requires_grad_(True)       # off a 16-byte boundary
    ours.append(odd)
    theirs = [p.detach().clone().requires_grad_(True) for p in ours]
    groups = lambda ps: [dict(params=[p], lr=10.0 ** -(1 + i % 4), name=str(i)) for i, p in enumerate(ps)]
    a, b = tr._Adam(groups(ours), eps=1e-15), torch.optim.Adam(groups(theirs), eps=1e-15)
    for it in range(4):
        for i, (p, q) in enumerate(zip(ours, theirs)):
            p.grad = q.grad = None
            if (i + it) % 5:                                                             # now and then a tensor without a gradient
                grad = torch.randn(p.shape, generator=g, device="cuda") * 10.0 ** (it - 3)
                p.grad, q.grad = grad, grad.clone()
        versions = [p._version for p in ours]
        a.step()
        b.step()
        for p, q, v in zip(ours, theirs, versions):
            assert torch.allclose(p, q, rtol=2e-6, atol=2e-7)
            assert p.grad is None or p._version > v
    copy.deepcopy(a.state_dict())
    b.load_state_dict(a.state_dict())                                                   # same state layout


@pytest.mark.parametrize("n", [1, 255, 1000])
def test_densification_statistics(tr, n):
    g = torch.Generator().manual_seed(n)
    args = [torch.randn(n, 3, generator=g) * 3, torch.rand(n, 3, generator=g) + 0.1, torch.randn(n, 4, generator=g),
            torch.rand(n, generator=g), torch.randn(n, 3, 4, generator=g)]
    grad = torch.randn(n, 3, generator=g) * (torch.rand(n, 1, generator=g) > 0.3)
    from types import SimpleNamespace
    clouds = [tr.SimplePointCloud(*[a.to(d) for a in args]) for d in ("cuda", "cpu")]
    for pc, d in zip(clouds, ("cuda", "cpu")):
        cam = SimpleNamespace(camera_center=torch.tensor([0.5, -1.0, 2.0], device=d))
        for _ in range(3):
            pc.accumulate_gradient(grad.to(d), cam)
            pc.accumulate_gradient_gaussians_not_visible(grad.to(d))
    a, b = clouds
    assert torch.allclose(a.xyz_gradient_accum_norm.cpu(), b.xyz_gradient_accum_norm, rtol=1e-5)
    assert torch.equal(a.num_accum.cpu(), b.num_accum) and torch.equal(a.num_accum_gnv.cpu(), b.num_accum_gnv)


@pytest.mark.parametrize("coeffs,lobes,normalize,factor", [(1, 0, False, 1), (16, 0, True, 1), (4, 2, False, 2), (4, 3, True, 1)])
def test_iteration_without_a_graph_is_the_one_with(tr, coeffs, lobes, normalize, factor):
    """training_iteration calls its Functions itself where nothing asks for a graph; a hook asks for one."""
    from raygaussx_b200 import scenes
    sc = scenes.tiny_scene(n=700, width=33, height=21, log_scale_mean=-2.5, sh_degree=int(coeffs ** 0.5) - 1, lobes=lobes, seed=coeffs)
    cam = sc.cameras[0].to("cuda")
    cam.original_image = torch.rand(3, 21, 33, generator=torch.Generator().manual_seed(1))
    cfg = tr.default_config(dt=0.01)
    cfg.training.normalize_quaternion = cfg.training.normalize_lobe_axis = normalize
    cfg.training.supersampling_x = factor
    got = []
    for hooked in (False, True):
        pc = tr.SimplePointCloud(*[t.cuda() for t in sc.tensors()])
        if hooked:
            pc.positions.register_hook(lambda g: None)
        grads = {}
        step = pc.optim_managers.step
        names = [g["name"] for g in pc.optim_managers.optimizer.param_groups]
        pc.optim_managers.step = lambda: (grads.update({k: getattr(pc, k).grad.clone() for k in names}), step())
        loss, stepped = tr.training_iteration(pc, cam, cfg, 0, tr.AccumulationSchedule())
        assert stepped and not loss.requires_grad and all(getattr(pc, k).grad is None for k in names)
        got.append((loss, grads, pc))
    assert torch.equal(got[0][0], got[1][0])
    for k, a in got[0][1].items():
        b = got[1][1][k]
        assert a.shape == b.shape and (a - b).abs().max() <= 2e-5 * b.abs().max().clamp_min(1e-30), k
    assert torch.equal(got[0][2].num_accum, got[1][2].num_accum)
