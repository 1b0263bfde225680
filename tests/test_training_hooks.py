"""What a caller hangs on a point cloud still runs in a training iteration: hooks on gradient accumulators, accessors and statistics of
a class of their own."""
import pytest
import torch

from raygaussx_b200 import training as tr
from tests.helpers import make_scene


def accumulator(p):
    return p.view_as(p).grad_fn.next_functions[0][0]


def test_held_accumulators_are_noticed():
    params = [torch.zeros(k, 3, requires_grad=True) for k in range(4)]
    assert not tr._accumulators_held(params)
    for p in params:
        node = accumulator(p)                       # as a wrapper with hooks there keeps it
        assert tr._accumulators_held(params) and tr._accumulators_held(params) and not node.metadata
        del node
        assert not tr._accumulators_held(params)
    graph = params[2] * 2                           # or a graph that is still in use
    assert tr._accumulators_held(params)
    del graph
    assert not tr._accumulators_held(params)


def cloud(cls=tr.SimplePointCloud, device="cpu"):
    return cls(*[t.to(device) for t in make_scene("small_static").tensors()[:5]])


def test_replaced_methods_are_noticed():
    class Same(tr.SimplePointCloud):
        pass

    class Other(tr.SimplePointCloud):
        def get_density(self):
            return super().get_density() * 2

    assert all(tr._as_defined(cloud(c), m) for c in (tr.SimplePointCloud, Same) for m in (tr._ACCESSORS, tr._STATISTICS))
    assert not tr._as_defined(cloud(Other), tr._ACCESSORS) and tr._as_defined(cloud(Other), tr._STATISTICS)
    pc = cloud()
    pc.accumulate_gradient = lambda *a: None
    assert not tr._as_defined(pc, tr._STATISTICS) and not tr._as_defined(object(), tr._ACCESSORS)


def test_onlookers_are_noticed():
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    assert not tr._autograd_watched()
    same = lambda t: t
    for onlooker in (torch.autograd.graph.saved_tensors_hooks(same, same), torch.autograd.detect_anomaly(check_nan=False),
                     TorchFunctionMode(), TorchDispatchMode()):
        with onlooker:
            assert tr._autograd_watched(), onlooker
    assert not tr._autograd_watched()


@pytest.fixture
def iteration():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path")
    sc = make_scene("small_static")
    cam, m = sc.cameras[0], sc.march
    cam.to(torch.device("cuda"))
    g = torch.Generator().manual_seed(3)
    cam.original_image = torch.rand(3, cam.image_height, cam.image_width, generator=g).cuda()
    cfg = tr.default_config(dt=m.dt_step, dynamic_sampling=m.dynamic_sampling, white_background=m.white_background,
                            max_prim_slice=m.max_prim_slice)
    return lambda pc: tr.training_iteration(pc, cam, cfg, 0, tr.AccumulationSchedule())


@pytest.mark.gpu
def test_hooks_on_accumulators_run(iteration):
    plain, hooked = cloud(device="cuda"), cloud(device="cuda")
    seen = {}
    nodes = {k: accumulator(getattr(hooked, k)) for k in ("positions", "spherical_harmonics", "scales")}
    for k, node in nodes.items():
        node.register_prehook(lambda grads, k=k: seen.__setitem__(k, grads[0].clone()))
    iteration(plain)
    iteration(hooked)
    assert set(seen) == set(nodes) and all(float(v.abs().sum()) > 0 for v in seen.values())
    for k in ("positions", "scales", "rgb", "spherical_harmonics", "densities", "quaternions"):      # and nothing else changes
        a, b = getattr(plain, k).detach(), getattr(hooked, k).detach()
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-6), k


@pytest.mark.gpu
def test_accessors_of_the_callers_own_run(iteration):
    called = []
    pc = cloud(device="cuda")
    data, stats = pc.get_data, pc.accumulate_gradient
    pc.get_data = lambda *a, **k: called.append("data") or data(*a, **k)
    pc.accumulate_gradient = lambda grad, camera: called.append("statistics") or stats(grad, camera)
    iteration(pc)
    assert called == ["data", "statistics"] and float(pc.num_accum.sum()) > 0 and float(pc.num_accum_gnv.sum()) > 0


@pytest.mark.gpu
def test_hooks_on_saved_tensors_run(iteration):
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t, lambda t: t):
        iteration(cloud(device="cuda"))
    assert packed
