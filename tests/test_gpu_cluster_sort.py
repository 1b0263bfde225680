"""Sets of the sizes that one cluster of blocks sorts, and on either side of them (`-m gpu`).  Neighbour distances against brute force
(every point gets its own), and the march: a set together with Gaussians below the threshold, which take no part, is sorted by the library once
it has more than some 80 thousand members, and must give the same image, bit for bit where the lists' keys have as many bits, and the same gradients."""
import pytest
import torch

from raygaussx_b200 import scenes

pytestmark = pytest.mark.gpu


def gpu():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    return torch.device("cuda")


@pytest.mark.parametrize("n", [4096, 4097, 4864, 4865, 16384, 16385, 65535, 65536, 78000, 78001, 81920, 81921])
def test_every_point_gets_its_own_distance(n):
    dev = gpu()
    from simple_knn._C import distCUDA2
    g = torch.Generator().manual_seed(n)
    pts = torch.randn(n, 3, generator=g)
    pts[: n // 8] = pts[: n // 8] * 0.001          # many equal keys
    pts = pts[torch.randperm(n, generator=g)].to(dev)
    got, p = distCUDA2(pts).double(), pts.double()
    pick = torch.randperm(n, generator=g)[:2048].to(dev)
    for who in pick.split(256):
        d = torch.cdist(p[who], p, compute_mode="donot_use_mm_for_euclid_dist") ** 2
        d[torch.arange(len(who), device=dev), who] = float("inf")
        assert torch.allclose(got[who], d.topk(3, dim=1, largest=False).values.mean(dim=1), rtol=1e-5, atol=0)
    assert torch.isfinite(got).all() and (got > 0).all()


@pytest.mark.parametrize("n,cluster", [(4096, False), (4864, False), (4865, True), (65535, True), (65536, True), (78000, True), (78001, False)])
def test_the_cluster_sorts_what_it_is_for(n, cluster):
    """Own kernels of a call: bounds, keys, gather, upper boxes, query, and the cluster's sort; those of the library are not counted."""
    dev = gpu()
    from raygaussx_b200 import _lib
    from simple_knn._C import distCUDA2
    pts = torch.randn(n, 3, generator=torch.Generator().manual_seed(n)).to(dev)
    before = _lib.lib().rgx_kernel_launches()
    distCUDA2(pts)
    assert _lib.lib().rgx_kernel_launches() - before == 5 + cluster


@pytest.mark.parametrize("n,bits,cluster", [(4864, 10, False), (4865, 10, True), (81_920, 10, True), (81_921, 10, False),
                                            (4096, 20, False), (4097, 20, True), (78_000, 20, True), (78_001, 20, False)])
def test_the_cluster_sorts_what_it_is_for_in_a_build(n, bits, cluster):
    """Own kernels of a build: bounds, keys, gather, refit, and the cluster's sort."""
    dev = gpu()
    from raygaussx_b200 import _lib
    from raygaussx_b200 import render_optix as ro
    tens = [t.to(dev).contiguous() for t in scenes.tiny_scene(n=n, width=8, height=8, seed=n).tensors()]
    r = ro.Renderer(dev)
    before = _lib.lib().rgx_kernel_launches()
    r.build(*tens[:4], morton_bits=bits)
    assert _lib.lib().rgx_kernel_launches() - before == 4 + cluster


@pytest.mark.parametrize("n,bits", [(4097, 10), (4097, 20), (4865, 10), (30_000, 10), (30_000, 20), (70_001, 10), (78_000, 20), (81_920, 10), (81_920, 20)])
def test_same_image_and_gradients_as_with_the_library(n, bits):
    dev = gpu()
    from raygaussx_b200 import render_optix as ro
    sc = scenes.tiny_scene(n=n, width=96, height=80, log_scale_mean=-3.7, seed=n)
    tens = [t.to(dev).contiguous() for t in sc.tensors()]
    extra = 100_000 - n
    more = [torch.cat([t, t[torch.arange(extra, device=dev) % n]]).contiguous() for t in tens]
    more[3][n:] = 0.01                             # below the threshold: hit by no ray
    cam = sc.cameras[0].to(dev)
    cs, r = ro.camera_struct(cam), ro.Renderer(dev)
    march = r._march(0.0025, False, 2048, True, 1e-3, None, cs.height, 0)
    out = []
    for t in (tens, more):
        r.build(*t[:4], morton_bits=bits)
        rgb, alpha, _ = r.forward(*t, cs, march, want_alpha=True)
        grads = [torch.zeros_like(x) for x in t]
        r.backward(*t, cs, march, rgb, torch.sign(rgb - 0.5) / rgb.numel(), tuple(grads))
        out.append((rgb.clone(), alpha.clone(), [x[:n] for x in grads[:5]]))
    a, b = out
    if n > 65536:                                  # as many bits for the slot either way
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    else:
        assert (a[0] - b[0]).abs().max().item() < 1e-5
    assert (a[1] > 0.1).any()
    for x, y in zip(a[2], b[2]):                   # sums of a few thousand fp32 terms in no fixed order
        assert ((x - y).abs().max() / y.abs().max()).item() < 3e-4
