"""``distCUDA2`` of the reference's simple-knn extension (submodules/simple-knn/ext.cpp, simple_knn.cu), on
``rgx_knn_mean_dist2``: mean squared distance from every point to its three nearest other points."""
import torch

from raygaussx_b200 import _lib


def distCUDA2(points: torch.Tensor) -> torch.Tensor:
    if not points.is_cuda:
        raise RuntimeError("distCUDA2 needs a CUDA tensor: there is no CPU path")
    pts = points.detach().to(torch.float32).contiguous()
    if pts.dim() != 2 or pts.shape[1] != 3:
        raise ValueError("points must be [N, 3]")
    n, dev = pts.shape[0], pts.device
    out = torch.empty(n, device=dev, dtype=torch.float32)
    lib = _lib.lib()
    # scratch from torch's own allocator: no cudaMalloc, no cudaFree and no wait for the stream in the call
    need = int(lib.rgx_knn_scratch_bytes(n))
    scratch = torch.empty(need, device=dev, dtype=torch.uint8)
    rc = lib.rgx_knn_mean_dist2_scratch(dev.index or 0, pts.data_ptr(), n, out.data_ptr(), scratch.data_ptr(), need,
                                        _lib.raw_stream(dev))
    if rc != 0:
        raise _lib.RgxError(rc, "rgx_knn_mean_dist2 failed")
    return out
