"""Brute-force KNN as an autograd Function (no backward), call-compatible with the reference's
``Swin3D.sparse_dl.knn.KNN`` (microsoft/Swin3D, Swin3D/sparse_dl/knn/knn.py:9-26):
``KNN.apply(K, src_xyz, query_xyz, src_offset, query_offset) -> (idx int32 [Nq,K], dist [Nq,K])``
with ``dist`` the Euclidean distance (sqrt of the kernel's squared distance, knn.py:25).
"""
import torch
from torch.autograd.function import Function

from ... import _lib, _stream


def _search(K: int, src_xyz, query_xyz, src_offset, query_offset, root: bool, out=None):
    for name, t in (("src_xyz", src_xyz), ("query_xyz", query_xyz)):
        if not t.is_cuda:
            raise RuntimeError(f"{name} must be a CUDA tensor")
        if t.dtype != torch.float32 or t.dim() != 2 or t.shape[1] != 3:
            raise ValueError(f"{name} must be float32 [n, 3]")
    assert src_xyz.is_contiguous() and query_xyz.is_contiguous()
    if src_offset.shape != query_offset.shape:
        raise ValueError("src_offset and query_offset must have one entry per scene")
    K = int(K)
    so = src_offset.to(torch.int32).contiguous()
    qo = query_offset.to(torch.int32).contiguous()
    dev = query_xyz.device
    B, Nq, Ns = so.shape[0], query_xyz.shape[0], src_xyz.shape[0]
    if out is None:
        out = (torch.empty((Nq, K), dtype=torch.int32, device=dev), torch.empty((Nq, K), dtype=torch.float32, device=dev))
    idx, dist = out
    nbytes = _lib.lib.s3d_knn_workspace_bytes(K, B, Ns, Nq)
    work = torch.empty(nbytes, dtype=torch.uint8, device=dev) if nbytes else None
    rc = _stream.call(dev, _lib.lib.s3d_knn_search, K, src_xyz.data_ptr(), query_xyz.data_ptr(), so.data_ptr(), qo.data_ptr(),
                      B, Ns, Nq, int(root), idx.data_ptr(), dist.data_ptr(), None if work is None else work.data_ptr(), nbytes)
    _lib.check(rc, "s3d_knn")
    return idx, dist


def knn_raw(K: int, src_xyz, query_xyz, src_offset, query_offset):
    """-> (idx int32 [Nq,K], squared distance float32 [Nq,K])."""
    return _search(K, src_xyz, query_xyz, src_offset, query_offset, False)


class KNN(Function):
    @staticmethod
    def forward(ctx, K, src_xyz, query_xyz, src_offset, query_offset):
        idx, dist = _search(K, src_xyz, query_xyz, src_offset, query_offset, True)
        ctx.mark_non_differentiable(idx, dist)
        return idx, dist
