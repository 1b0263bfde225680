"""One training iteration around the ray-marching operator: the counterpart of the
loop body of the reference's ``scripts/train.py:83-165`` without its OptiX, cupy
and ``fused_ssim`` imports.

What an iteration does there, and here: pick a random training camera, render it
through ``RenderOptixFunction`` (``optix_raycasting/render_optix.py``), average the
supersampled rays, form the loss ``(1 - l) L1 + l (1 - SSIM) + l_iso * isotropy``,
divide it by the number of accumulated views once accumulation is on
(20 views per optimizer step from iteration 20,000), back-propagate, feed the
position gradients to the densification statistics
(``classes/point_cloud.py:468-479``) and step the optimizers when the window is
full.  The reference's OptiX context, pipelines and acceleration structure
(``scripts/train.py:95-115``) have no counterpart: the operator keeps its own
workspace.

``pointcloud`` is any object with the reference's interface: ``get_data(...)``,
``optim_managers`` (``zero_grad()``, ``step()``), ``positions``,
``accumulate_gradient(grad, cam)``, ``accumulate_gradient_gaussians_not_visible(grad)``
and ``num_sph_gauss``.  ``SimplePointCloud`` is a small one for tests and benchmarks.
"""
from __future__ import annotations

import ctypes as C
import math
import random
from types import SimpleNamespace
from typing import Callable, List, Optional

import torch
import torch.nn.functional as F

from . import _lib
from . import render_optix as r_ox
from .inference import reduce_supersampling


# ----------------------------------------------------------------------------- losses
def l1_loss(image, target):
    return (image - target).abs().mean()


def _gaussian_taps(size: int, sigma: float, like: torch.Tensor) -> torch.Tensor:
    x = torch.arange(size, dtype=torch.float64) - size // 2
    g = torch.exp(-(x * x) / (2.0 * sigma * sigma))
    return (g / g.sum()).to(like.dtype).to(like.device)


def _blur(x: torch.Tensor, taps: torch.Tensor) -> torch.Tensor:
    """Separable Gaussian blur of ``[B, C, H, W]`` with zero padding, one pass per axis."""
    c = x.shape[1]
    k = taps.numel()
    kx = taps.view(1, 1, 1, k).expand(c, 1, 1, k)
    ky = taps.view(1, 1, k, 1).expand(c, 1, k, 1)
    x = F.conv2d(x, kx, padding=(0, k // 2), groups=c)
    return F.conv2d(x, ky, padding=(k // 2, 0), groups=c)


def ssim(img1: torch.Tensor, img2: torch.Tensor, window_size: int = 11, sigma: float = 1.5) -> torch.Tensor:
    """Mean structural similarity (Wang et al. 2004) of ``[B, 3, H, W]`` or ``[3, H, W]`` images in [0, 1] with
    the 11-tap, sigma 1.5 Gaussian window, zero padding and the constants (0.01^2, 0.03^2) that the reference's
    loss uses (``scripts/train.py:134`` through ``fused_ssim``; same definition as ``utils/loss_utils.py:37-62``)."""
    squeeze = img1.dim() == 3
    if squeeze:
        img1, img2 = img1.unsqueeze(0), img2.unsqueeze(0)
    taps = _gaussian_taps(window_size, sigma, img1)
    mu1, mu2 = _blur(img1, taps), _blur(img2, taps)
    mu1_sq, mu2_sq, mu12 = mu1 * mu1, mu2 * mu2, mu1 * mu2
    s1 = _blur(img1 * img1, taps) - mu1_sq
    s2 = _blur(img2 * img2, taps) - mu2_sq
    s12 = _blur(img1 * img2, taps) - mu12
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    value = ((2 * mu12 + c1) * (2 * s12 + c2)) / ((mu1_sq + mu2_sq + c1) * (s1 + s2 + c2))
    return value.mean()


def isotropy_loss(scales: torch.Tensor) -> torch.Tensor:
    """``scripts/train.py:139-142``: mean over Gaussians of ``max(r, 10) - 10`` with
    ``r = 2 / (pi sqrt 3) * |s|^3 / (s_x s_y s_z)`` (the reference writes pi as 3.14159265359)."""
    r = (2 / (3.14159265359 * (3 ** 0.5))) * ((scales[:, 0] ** 2 + scales[:, 1] ** 2 + scales[:, 2] ** 2) ** (3 / 2)) / (
        scales[:, 0] * scales[:, 1] * scales[:, 2])
    return (torch.clamp(r, min=10) - 10).mean()


# ----------------------------------------------------------------------------- the same on the device, fused (csrc/train.cu)
def _stream(t: torch.Tensor):
    return _lib.raw_stream(t.device)


def _check(rc: int, what: str):
    if rc != 0:
        raise _lib.RgxError(rc, what + " failed")


def _fusable(*tensors) -> bool:
    """fp32 CUDA tensors of one device, contiguous: what the fused kernels take."""
    index = tensors[0].get_device()                      # -1: not on a GPU
    for t in tensors:
        if t.layout != torch.strided or t.get_device() != index or t.dtype != torch.float32 or not t.is_contiguous():
            return False
    return index >= 0


class _ImageLoss(torch.autograd.Function):
    """``(1 - l) L1 + l (1 - SSIM)`` of the supersampled rays ``[R, 3]`` against ``[3, H, W]``: one kernel and a small sum
    forward, one kernel backward, in place of some hundred operators on images."""

    @staticmethod
    def forward(ctx, rays, target, width, height, factor, lambda_ssim):
        lib, dev = _lib.lib(), rays.device
        maps = torch.empty(9 * width * height, device=dev) if lambda_ssim != 0 and ctx.needs_input_grad[0] else None
        scratch = torch.empty(int(lib.rgx_image_loss_scratch_floats(width, height)), device=dev)
        loss = torch.empty((), device=dev)
        _check(lib.rgx_image_loss(dev.index or 0, rays.data_ptr(), target.data_ptr(), width, height, factor[0], factor[1],
                                  lambda_ssim, maps.data_ptr() if maps is not None else None, scratch.data_ptr(),
                                  loss.data_ptr(), _stream(rays)), "rgx_image_loss")
        ctx.args = (width, height, factor, lambda_ssim)
        ctx.save_for_backward(rays, target, maps)
        return loss

    @staticmethod
    def backward(ctx, grad_loss):
        rays, target, maps = ctx.saved_tensors
        width, height, factor, lambda_ssim = ctx.args
        grad = torch.empty_like(rays)
        _check(_lib.lib().rgx_image_loss_backward(rays.device.index or 0, rays.data_ptr(), target.data_ptr(), width, height, factor[0],
                                                  factor[1], lambda_ssim, maps.data_ptr() if maps is not None else None,
                                                  grad_loss.contiguous().data_ptr() if grad_loss is not None else None,
                                                  grad.data_ptr(), _stream(rays)),
               "rgx_image_loss_backward")
        return grad, None, None, None, None, None


def image_loss(rays, target, width: int, height: int, supersampling=(1, 1), lambda_ssim: float = 0.2):
    """``(1 - l) L1 + l (1 - SSIM)`` of the rays' image (``scripts/train.py:128-137``): fused where the tensors allow it,
    else composed of :func:`l1_loss` and :func:`ssim`."""
    if _fusable(rays, target) and target.dim() == 3:
        return _ImageLoss.apply(rays, target, int(width), int(height), (int(supersampling[0]), int(supersampling[1])),
                                float(lambda_ssim))
    image = reduce_supersampling(width, height, rays, supersampling).permute(2, 0, 1)
    loss = (1.0 - lambda_ssim) * l1_loss(image, target)
    return loss + lambda_ssim * (1.0 - ssim(image, target)) if lambda_ssim != 0 else loss


class _Activate(torch.autograd.Function):
    """Parameters -> the operator's inputs that are not parameters themselves (``rgx_activate``), one kernel each way."""

    @staticmethod
    def forward(ctx, log_scales, quaternions, rgb, sh, sharpness, axis, normalize_q, normalize_axis):
        n, g = log_scales.shape[0], sharpness.shape[1]
        a = _lib.Activation()
        a.n, a.sh_coeffs, a.num_lobes = n, 1 + sh.shape[2], g
        scales, color = torch.empty_like(log_scales), torch.empty(n, 3, a.sh_coeffs, device=rgb.device)
        sharp = torch.empty_like(sharpness)
        quats = torch.empty_like(quaternions) if normalize_q else None
        ax = torch.empty_like(axis) if normalize_axis else None
        a.log_scales, a.raw_quaternions, a.rgb, a.sh = (r_ox._ptr(t) for t in (log_scales, quaternions, rgb, sh))
        a.raw_sharpness, a.raw_axis = r_ox._ptr(sharpness), r_ox._ptr(axis)
        a.scales, a.quaternions, a.color, a.sharpness, a.lobe_axis = (r_ox._ptr(t) for t in (scales, quats, color, sharp, ax))
        _check(_lib.lib().rgx_activate(rgb.device.index or 0, C.byref(a), _stream(rgb)), "rgx_activate")
        ctx.sizes = (a.n, a.sh_coeffs, a.num_lobes)
        ctx.save_for_backward(scales, quaternions, sharpness, axis, rgb, sh)
        ctx.set_materialize_grads(False)
        return scales, quats, color, sharp, ax

    @staticmethod
    def backward(ctx, d_scales, d_quats, d_color, d_sharp, d_axis):
        scales, quaternions, sharpness, axis, rgb, sh = ctx.saved_tensors
        a, g = _lib.Activation(), _lib.ActivationGrads()
        a.n, a.sh_coeffs, a.num_lobes = ctx.sizes
        a.raw_quaternions, a.raw_sharpness, a.raw_axis, a.scales = (r_ox._ptr(t) for t in (quaternions, sharpness, axis, scales))
        given = [r_ox._aligned(t) if t is not None else None for t in (d_scales, d_quats, d_color, d_sharp, d_axis)]
        g.scales, g.quaternions, g.color, g.sharpness, g.lobe_axis = (r_ox._ptr(t) for t in given)
        need = ctx.needs_input_grad
        wanted = [torch.empty_like(like) if need[i] and given[src] is not None else None for i, src, like in (
            (0, 0, scales), (1, 1, quaternions), (2, 2, rgb), (3, 2, sh), (4, 3, sharpness), (5, 4, axis))]
        g.log_scales, g.raw_quaternions, g.rgb, g.sh, g.raw_sharpness, g.raw_axis = (r_ox._ptr(t) for t in wanted)
        _check(_lib.lib().rgx_activate_backward(rgb.device.index or 0, C.byref(a), C.byref(g), _stream(rgb)), "rgx_activate_backward")
        return (*wanted, None, None)


class _Node:
    """What a Function keeps between its forward and its backward."""

    def __init__(self, needs_input_grad=()):
        self.needs_input_grad = needs_input_grad
        self.saved_tensors = ()

    def save_for_backward(self, *tensors):
        self.saved_tensors = tensors

    def set_materialize_grads(self, _):
        pass


class _Edges(torch.autograd.Function):
    """A graph node that leads to the accumulators of the parameters given."""

    @staticmethod
    def forward(ctx, *params):
        return params[0].new_empty(0)


def _accumulators_held(params) -> bool:
    """Whether something else holds a parameter's gradient accumulator -- a hook on it, a graph that is still in use.  Autograd
    makes an accumulator when one is asked for and drops it with its last holder, so one that something is written on is
    found again only if it has another."""
    for again in (False, True):
        end = _Edges.apply(*params)
        nodes = [node for node, _ in end.grad_fn.next_functions]
        if again:
            return any([node.metadata.pop("rgx_seen", False) for node in nodes])
        for node in nodes:
            node.metadata["rgx_seen"] = True
        del end, nodes, node


def _autograd_watched() -> bool:
    """Whether somebody looks on: hooks on saved tensors (``torch.autograd.graph.saved_tensors_hooks``), anomaly detection, a mode."""
    return (torch._C._autograd._top_saved_tensors_default_hooks(True) is not None or torch.is_anomaly_enabled()
            or torch._C._is_torch_function_mode_enabled() or torch._C._len_torch_dispatch_stack() > 0)


def _gradients_directly(pc, settings, target, cam, supersampling, t):
    """Loss, and the gradients left in the parameters' empty ``.grad``: the iteration's three Functions called one after the
    other.  Built and run by autograd they cost a small scene's iteration more host time than its kernels take (4 k Gaussians
    at 64x64: 0.70 ms of host time around 0.35 ms of kernels, 0.41 this way).  None: something here is for autograd to look after -- a
    point cloud with accessors of its own, frozen parameters, hooks on them or on saved tensors, gradients to add to, another loss.  Where something holds
    an accumulator, autograd hands the gradients over, and with them to the hooks there."""
    params = (pc.positions, pc.scales, pc.quaternions, pc.densities, pc.rgb, pc.spherical_harmonics, pc.sph_gauss_features,
              pc.bandwidth_sharpness, pc.lobe_axis) if _as_defined(pc, _ACCESSORS) else ()
    if (not params or t.lambda_iso != 0 or target.dim() != 3 or target.requires_grad or not _fusable(*params, target)
            or not torch.is_grad_enabled() or _autograd_watched()):
        return None
    for p in params:
        if not p.requires_grad or not p.is_leaf or p.grad is not None or p._backward_hooks or p._post_accumulate_grad_hooks:
            return None
    positions, scales, quaternions, densities, rgb, sh, sg, sharpness, axis = params
    with_q, with_axis = not t.normalize_quaternion, not t.normalize_lobe_axis and axis.numel() > 0
    with torch.no_grad():
        activate, render, compare = _Node((True,) * 6), _Node(), _Node((True,))
        act_scales, act_q, color, act_sharp, act_axis = _Activate.forward(activate, scales, quaternions, rgb, sh, sharpness, axis,
                                                                          with_q, with_axis)
        image = r_ox.RenderOptixFunction.forward(render, positions, act_scales, act_q if with_q else quaternions, densities, color,
                                                 sg, act_sharp, act_axis if with_axis else axis, settings)
        loss = _ImageLoss.forward(compare, image, target, int(cam.image_width), int(cam.image_height),
                                  (int(supersampling[0]), int(supersampling[1])), float(t.lambda_ssim))
        d_image = _ImageLoss.backward(compare, None)[0]
        g_pos, g_scales, g_q, g_dens, g_color, g_sg, g_sharp, g_axis, _ = r_ox.RenderOptixFunction.backward(render, d_image)
        d = _Activate.backward(activate, g_scales, g_q if with_q else None, g_color, g_sharp, g_axis if with_axis else None)
    grads = (g_pos, d[0], d[1] if with_q else g_q, g_dens, d[2], d[3], g_sg, d[4], d[5] if with_axis else g_axis)
    if _accumulators_held([p for p in params if p.numel() > 0]):
        there = [(p, g) for p, g in zip(params, grads) if g is not None]
        torch.autograd.backward([p for p, _ in there], [g for _, g in there])
    else:
        for p, g in zip(params, grads):
            p.grad = g
    return loss


# ----------------------------------------------------------------------------- the iteration
class AccumulationSchedule:
    """Gradient accumulation of ``scripts/train.py:77-85,150-161``: from ``accum_start`` on, ``accum_steps``
    views share one optimizer step."""

    def __init__(self, accum_steps: int = 20, accum_start: int = 20000):
        self.accum_steps = accum_steps
        self.accum_start = accum_start
        self.counter = 0

    def use_accum(self, iteration: int) -> bool:
        return iteration >= self.accum_start and self.accum_steps > 1


def pick_camera(stack: List, cameras: Callable[[], List]):
    """``scripts/train.py:90-94``: cameras are drawn without replacement; the stack is refilled when empty."""
    if not stack:
        stack.extend(cameras())
    return stack.pop(random.randint(0, len(stack) - 1))


def training_iteration(pointcloud, viewpoint_cam, config, iteration: int, schedule: AccumulationSchedule,
                       hit_prim_idx=None):
    """The body of the reference's training loop for one camera (``scripts/train.py:86-165``).  ``config`` has the
    reference's fields: ``scene.dt``, ``scene.dynamic_sampling``, ``scene.white_background``,
    ``training.max_prim_slice``, ``training.jitter``, ``training.rnd_sample``, ``training.supersampling_x/_y``,
    ``training.lambda_ssim``, ``training.lambda_iso``, ``training.normalize_quaternion``,
    ``training.normalize_lobe_axis``.  Returns ``(loss, stepped)``: the detached loss as back-propagated and
    whether the optimizers stepped."""
    t = config.training
    use_accum = schedule.use_accum(iteration)
    if (not use_accum) or schedule.counter == 0:
        pointcloud.optim_managers.zero_grad()
    gt_image = viewpoint_cam.original_image.to(pointcloud.positions.device)
    supersampling = (t.supersampling_x, t.supersampling_y)
    settings = r_ox.RenderOptixSettings(None, False, None, None, None, None, None, config.scene.dt,
                                        config.scene.dynamic_sampling, viewpoint_cam, t.max_prim_slice,
                                        pointcloud.num_sph_gauss, iteration=iteration, jitter=t.jitter,
                                        rnd_sample=t.rnd_sample, supersampling=supersampling,
                                        white_background=config.scene.white_background, hit_prim_idx=hit_prim_idx)
    loss = None if use_accum else _gradients_directly(pointcloud, settings, gt_image, viewpoint_cam, supersampling, t)
    if loss is None:
        (positions, scales, quaternions, densities, color_features, sph_gauss_features, bandwidth_sharpness,
         lobe_axis) = pointcloud.get_data(normalized_quaternion=not t.normalize_quaternion,
                                          normalized_lobe_axis=not t.normalize_lobe_axis)
        image = r_ox.RenderOptixFunction.apply(positions, scales, quaternions, densities, color_features,
                                               sph_gauss_features, bandwidth_sharpness, lobe_axis, settings)
        loss = image_loss(image, gt_image, viewpoint_cam.image_width, viewpoint_cam.image_height, supersampling, t.lambda_ssim)
        if t.lambda_iso != 0:
            loss = loss + t.lambda_iso * isotropy_loss(scales)
        if use_accum:
            loss = loss / float(schedule.accum_steps)
        loss.backward()
    if pointcloud.positions.grad is not None:
        grad = pointcloud.positions.grad
        if _as_defined(pointcloud, _STATISTICS) and _fusable(grad, pointcloud.num_accum_gnv):     # both statistics in one pass
            if not pointcloud.accumulate_gradient(grad, viewpoint_cam, pointcloud.num_accum_gnv.data_ptr()):
                pointcloud.accumulate_gradient_gaussians_not_visible(grad)
        else:
            pointcloud.accumulate_gradient(grad, viewpoint_cam)
            pointcloud.accumulate_gradient_gaussians_not_visible(grad)
    stepped = False
    if use_accum:
        schedule.counter += 1
        if schedule.counter >= schedule.accum_steps:
            pointcloud.optim_managers.step()
            pointcloud.optim_managers.zero_grad()
            schedule.counter = 0
            stepped = True
    else:
        pointcloud.optim_managers.step()
        pointcloud.optim_managers.zero_grad()
        stepped = True
    return loss.detach(), stepped


# ----------------------------------------------------------------------------- a small point cloud
class _Adam(torch.optim.Adam):
    """``torch.optim.Adam`` whose step is one kernel over all tensors (``rgx_adam_step``) where the parameters are contiguous
    fp32 CUDA tensors and nothing but the plain algorithm is asked for; state and results are those of the base class."""

    @staticmethod
    def _plain(grp) -> bool:
        return not (grp["weight_decay"] or grp["amsgrad"] or grp["maximize"] or grp["capturable"] or grp["differentiable"]
                    or grp["fused"] or torch.is_tensor(grp["lr"]))

    @torch.no_grad()
    def step(self, closure=None):
        work = [(p, p.grad, grp) for grp in self.param_groups for p in grp["params"] if p.grad is not None]
        if closure is not None or not work or not all(self._plain(grp) for grp in self.param_groups) or not _fusable(
                *[p for p, _, _ in work], *[g for _, g, _ in work]):
            return super().step(closure)
        batches = {}
        for p, grad, grp in work:
            st = self.state[p]
            if len(st) == 0:
                st["step"] = torch.tensor(0.0)
                st["exp_avg"] = torch.zeros_like(p, memory_format=torch.preserve_format)
                st["exp_avg_sq"] = torch.zeros_like(p, memory_format=torch.preserve_format)
            t = st["step"].add_(1).item()                # a host tensor
            beta1, beta2 = grp["betas"]
            batches.setdefault((beta1, beta2, grp["eps"]), []).append(
                (p.data_ptr(), st["exp_avg"].data_ptr(), st["exp_avg_sq"].data_ptr(), grad.data_ptr(), p.numel(),
                 grp["lr"] / (1 - beta1 ** t), 1.0 / math.sqrt(1 - beta2 ** t)))
        dev = work[0][0].device
        for (beta1, beta2, eps), rows in batches.items():
            for lo in range(0, len(rows), _lib.ADAM_MAX):
                part = rows[lo:lo + _lib.ADAM_MAX]
                table = (_lib.AdamTensor * len(part))(*part)
                _check(_lib.lib().rgx_adam_step(dev.index or 0, table, len(part), beta1, beta2, eps, _stream(work[0][0])),
                       "rgx_adam_step")
        torch.autograd.graph.increment_version([p for p, _, _ in work])       # written to behind torch's back


class _Optimizers:
    """The part of the reference's optimizer manager the loop uses (``zero_grad``, ``step``, ``get_lrs``)."""

    def __init__(self, groups):
        self.optimizer = _Adam(groups, eps=1e-15)

    def zero_grad(self):
        for group in self.optimizer.param_groups:
            for p in group["params"]:
                p.grad = None

    def step(self):
        self.optimizer.step()

    def get_lrs(self):
        return {g["name"]: g["lr"] for g in self.optimizer.param_groups}


class SimplePointCloud:
    """Gaussians in the reference's parameterisation (``classes/point_cloud.py:509-559``): positions, logarithms
    of the scales, raw quaternions, densities, colour as DC term plus higher SH bands, lobe tensors -- with one
    Adam group per tensor and the densification statistics of ``classes/point_cloud.py:468-479``."""

    def __init__(self, positions, scales, quaternions, densities, color_features, sph_gauss_features=None,
                 bandwidth_sharpness=None, lobe_axis=None, lrs: Optional[dict] = None):
        dev = positions.device
        n = positions.shape[0]
        leaf = lambda x: x.detach().clone().contiguous().requires_grad_(True)
        self.positions = leaf(positions)
        self.scales = leaf(torch.log(scales))
        self.quaternions = leaf(quaternions)
        self.densities = leaf(densities)
        self.rgb = leaf(color_features[:, :, 0])
        self.spherical_harmonics = leaf(color_features[:, :, 1:])
        g = 0 if sph_gauss_features is None else sph_gauss_features.shape[2]
        self.num_sph_gauss = g
        self.sph_gauss_features = leaf(sph_gauss_features if g else torch.zeros(n, 3, 0, device=dev))
        # softplus is undone so that get_bandwidth_sharpness returns what was passed in
        sharp = bandwidth_sharpness if g else torch.zeros(n, 0, device=dev)
        self.bandwidth_sharpness = leaf(torch.where(sharp > 20, sharp, torch.log(torch.expm1(sharp.clamp_min(1e-6)))))
        self.lobe_axis = leaf(lobe_axis if g else torch.zeros(n, 0, 3, device=dev))
        lr = dict(positions=1.6e-4, scales=5e-3, quaternions=1e-3, densities=5e-2, rgb=2.5e-3,
                  spherical_harmonics=1.25e-4, sph_gauss_features=2.5e-3, bandwidth_sharpness=1e-3, lobe_axis=1e-3)
        lr.update(lrs or {})
        self.optim_managers = _Optimizers([dict(params=[getattr(self, k)], lr=v, name=k) for k, v in lr.items()
                                           if getattr(self, k).numel() > 0])
        self.reset_gradient_accum()

    # accessors of classes/point_cloud.py:509-559
    def get_color_features(self):
        return torch.cat([self.rgb[:, :, None], self.spherical_harmonics], dim=2)

    def get_scale(self):
        return torch.exp(self.scales)

    def get_normalized_quaternion(self):
        return self.quaternions / torch.norm(self.quaternions, dim=1)[:, None]

    def get_density(self):
        return self.densities

    def get_bandwidth_sharpness(self):
        return F.softplus(self.bandwidth_sharpness)

    def get_normalized_lobe_axis(self):
        if self.lobe_axis.numel() == 0:
            return self.lobe_axis
        return self.lobe_axis / torch.norm(self.lobe_axis, dim=2)[:, :, None]

    def get_data(self, normalized_quaternion=True, normalized_lobe_axis=True):
        raw = (self.scales, self.quaternions, self.rgb, self.spherical_harmonics, self.bandwidth_sharpness, self.lobe_axis)
        if _fusable(*raw):
            with_axis = normalized_lobe_axis and self.lobe_axis.numel() > 0
            scales, q, color, sharp, a = _Activate.apply(*raw, normalized_quaternion, with_axis)
            return (self.positions, scales, q if normalized_quaternion else self.quaternions, self.get_density(), color,
                    self.sph_gauss_features, sharp, a if with_axis else self.lobe_axis)
        q = self.get_normalized_quaternion() if normalized_quaternion else self.quaternions
        a = self.get_normalized_lobe_axis() if normalized_lobe_axis else self.lobe_axis
        return (self.positions, self.get_scale(), q, self.get_density(), self.get_color_features(),
                self.sph_gauss_features, self.get_bandwidth_sharpness(), a)

    def renderer_inputs(self):
        """The operator's eight inputs, activated (``inference.py``)."""
        return self.get_data()

    # statistics of classes/point_cloud.py:468-485
    @torch.no_grad()
    def reset_gradient_accum(self):
        n, dev = self.positions.shape[0], self.positions.device
        self.xyz_gradient_accum_norm = torch.zeros(n, device=dev)
        self.num_accum = torch.zeros(n, device=dev)
        self.num_accum_gnv = torch.zeros(n, device=dev)

    @torch.no_grad()
    def accumulate_gradient(self, grad, camera, _also=None):
        eye = camera.camera_center
        if _fusable(self.positions, grad, eye, self.xyz_gradient_accum_norm, self.num_accum):
            _check(_lib.lib().rgx_gradient_stats(grad.device.index or 0, grad.shape[0], self.positions.data_ptr(), grad.data_ptr(),
                                                 eye.data_ptr(), self.xyz_gradient_accum_norm.data_ptr(),
                                                 self.num_accum.data_ptr(), _also, _stream(grad)), "rgx_gradient_stats")
            return True
        dist = torch.clamp(torch.norm(self.positions - camera.camera_center[None, :], dim=1), min=1.0)
        norm = torch.norm(grad, dim=1)
        self.xyz_gradient_accum_norm += norm * dist
        self.num_accum += torch.where(norm > 0, 1.0, 0.0)
        return False

    @torch.no_grad()
    def accumulate_gradient_gaussians_not_visible(self, grad):
        if _fusable(grad, self.num_accum_gnv):
            _check(_lib.lib().rgx_gradient_stats(grad.device.index or 0, grad.shape[0], None, grad.data_ptr(), None, None,
                                                 self.num_accum_gnv.data_ptr(), None, _stream(grad)), "rgx_gradient_stats")
            return
        self.num_accum_gnv += torch.where(torch.norm(grad, dim=1) > 0, 1.0, 0.0)


#: What the fused paths above take the place of, as it is defined here.
_ACCESSORS = {k: vars(SimplePointCloud)[k] for k in (
    "get_data", "get_color_features", "get_scale", "get_normalized_quaternion", "get_density", "get_bandwidth_sharpness",
    "get_normalized_lobe_axis")}
_STATISTICS = {k: vars(SimplePointCloud)[k] for k in ("accumulate_gradient", "accumulate_gradient_gaussians_not_visible")}


def _as_defined(pc, methods) -> bool:
    """A SimplePointCloud, or a class derived from it, that has replaced none of ``methods``, neither in its class nor on the object."""
    own = getattr(pc, "__dict__", {})
    return isinstance(pc, SimplePointCloud) and all(getattr(type(pc), k) is f and k not in own for k, f in methods.items())


def default_config(dt=0.01, dynamic_sampling=False, white_background=False, max_prim_slice=512, lambda_ssim=0.2,
                   lambda_iso=0.0) -> SimpleNamespace:
    """A configuration with the fields ``training_iteration`` reads, named as in the reference's YAML
    (``configs/base.yml``)."""
    return SimpleNamespace(
        scene=SimpleNamespace(dt=dt, dynamic_sampling=dynamic_sampling, white_background=white_background),
        training=SimpleNamespace(max_prim_slice=max_prim_slice, jitter=False, rnd_sample=0, supersampling_x=1,
                                 supersampling_y=1, lambda_ssim=lambda_ssim, lambda_iso=lambda_iso,
                                 normalize_quaternion=False, normalize_lobe_axis=False))
