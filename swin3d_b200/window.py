"""Host wrapper of the window builders (s3d_window_groups, s3d_window_build).

``build_windows`` produces, for one (stage, shift), what the reference's
``BasicLayer.get_index01`` (microsoft/Swin3D, Swin3D/modules/swin3d_layers.py:789-822) produces
through MinkowskiEngine: the window-sorted voxel order ``n2n_indices``, the per-window sizes and
offsets, and ``n_coords`` (cell + in-voxel position, then the colour / normal signals) in sorted
order.  Windows are emitted in lexicographic (batch, wx, wy, wz) order; the reference's order is
whatever MinkowskiEngine's pooling returns and attention does not depend on it.
"""
import ctypes
from dataclasses import dataclass, field
from typing import Optional

import torch

from . import _lib, _stream


@dataclass
class WindowIndex:
    n2n: torch.Tensor        # int32 [N]  sorted position -> voxel row
    n_coords: torch.Tensor   # float32 [N, F]  sorted order
    w_sizes: torch.Tensor    # int32 [W]
    w2n: torch.Tensor        # int32 [W]  first sorted position of each window
    num_pairs: int           # M = sum w^2
    max_window: int
    w2m: Optional[torch.Tensor] = field(default_factory=lambda: None)   # int64 [W]  exclusive sum of w^2; made when asked for

    def __post_init__(self):
        if self.w2m is None:
            del self.w2m

    def __getattr__(self, name):
        if name != "w2m":
            raise AttributeError(name)
        w2 = self.w_sizes.to(torch.int64) ** 2
        self.w2m = torch.cumsum(w2, 0) - w2
        return self.w2m

    def reference_indices(self, n_crse: torch.Tensor):
        """The six-tensor list ``SelfAttnAIOFunction.apply`` takes for IndexMode.INDIRECT.
        ``m2w`` (one entry per attention pair in the reference) is never read by the fused
        kernels, so an empty tensor stands in for it; ``w2m`` is the exclusive sum of w^2."""
        m2w = torch.empty(0, dtype=torch.int64, device=self.n2n.device)
        return [m2w, self.w_sizes, self.w2m, self.w2n, self.n2n, n_crse]


_RANGE_ERROR = ("s3d_window_build: a batch index or window coordinate is outside the "
                "supported key range (batch < 1024, |window index| < 16384)")


def _build(coords, xyz, rest, feats, window_size: int, shift: int, stride: int) -> WindowIndex:
    """coords int32 [N,4]; xyz [N,3] and rest [N,F-3] float32 with unit column stride; feats() -> the two
    as one contiguous [N,F] array (only asked for on the sorting path)."""
    N, F = coords.shape[0], 3 + rest.shape[1]
    dev = coords.device
    n2n = torch.empty(N, dtype=torch.int32, device=dev)
    n_coords = torch.empty((N, F), dtype=torch.float32, device=dev)
    w_sizes = torch.empty(max(N, 1), dtype=torch.int32, device=dev)
    w2n = torch.empty(max(N, 1), dtype=torch.int32, device=dev)
    w2m = torch.empty(max(N, 1), dtype=torch.int64, device=dev)
    lib = _lib.lib
    # distinct voxels that fill their box of windows reasonably well are not sorted (others are, after a second
    # look); the library reads the window count back itself
    wbytes = lib.s3d_window_groups_workspace_bytes(N, window_size)
    if wbytes:
        work = torch.empty(wbytes, dtype=torch.uint8, device=dev)
        host = (ctypes.c_int64 * 4)()
        rc = _stream.call(dev, lib.s3d_window_groups, coords.data_ptr(), xyz.data_ptr(), xyz.stride(0) if N else F,
                          rest.data_ptr() if F > 3 else None, rest.stride(0) if N else F, N, F, stride, window_size, shift,
                          n2n.data_ptr(), n_coords.data_ptr(), w_sizes.data_ptr(), w2n.data_ptr(), w2m.data_ptr(),
                          ctypes.addressof(host), work.data_ptr(), wbytes)
        _lib.check(rc, "s3d_window_groups")
        W, M, mx, flags = host
        if flags & 1:
            raise ValueError(_RANGE_ERROR)
        return WindowIndex(n2n, n_coords, w_sizes[:W], w2n[:W], M, mx, None if flags else w2m[:W])
    counts = torch.empty(4, dtype=torch.int64, device=dev)
    wbytes = lib.s3d_window_build_workspace_bytes(N)
    work = torch.empty(wbytes, dtype=torch.uint8, device=dev)
    rc = _stream.call(dev, lib.s3d_window_build, coords.data_ptr(), feats().data_ptr(), N, F, stride, window_size, shift,
                      n2n.data_ptr(), n_coords.data_ptr(), w_sizes.data_ptr(), w2n.data_ptr(), counts.data_ptr(),
                      work.data_ptr(), wbytes)
    _lib.check(rc, "s3d_window_build")
    W, M, mx, err = (int(x) for x in counts.tolist())
    if err:
        raise ValueError(_RANGE_ERROR)
    return WindowIndex(n2n, n_coords, w_sizes[:W], w2n[:W], M, mx)


def build_windows(coords: torch.Tensor, feats: torch.Tensor, window_size: int, shift: int = 0,
                  stride: int = 1) -> WindowIndex:
    """coords int32 [N,4] (batch,x,y,z; multiples of ``stride``); feats float32 [N,F] with the
    in-voxel position in columns 0..2 and the other cRSE signals after it."""
    if not coords.is_cuda or not feats.is_cuda:
        raise RuntimeError("coords and feats must be CUDA tensors")
    if coords.dtype != torch.int32 or coords.dim() != 2 or coords.shape[1] != 4:
        raise ValueError("coords must be int32 [N, 4]")
    N = coords.shape[0]
    if feats.dtype != torch.float32 or feats.dim() != 2 or feats.shape[0] != N:
        raise ValueError("feats must be float32 [N, F]")
    feats = feats.contiguous()
    return _build(coords.contiguous(), feats[:, :3], feats[:, 3:], lambda: feats, int(window_size), int(shift), int(stride))


def _tensor_stride(sp) -> int:
    """Tensor stride of a MinkowskiEngine-style sparse tensor (or of any object that mimics
    ``sp.coordinate_map_key.get_tensor_stride()`` / ``sp.tensor_stride``)."""
    key = getattr(sp, "coordinate_map_key", None)
    if key is not None and hasattr(key, "get_tensor_stride"):
        s = key.get_tensor_stride()
    else:
        s = getattr(sp, "tensor_stride", 1)
    return int(s[0]) if isinstance(s, (list, tuple)) else int(s)


def get_index01(sp, local_xyz: torch.Tensor, colors: torch.Tensor, window_size: int,
                shift_size: int = 0):
    """Call-compatible replacement of ``BasicLayer.get_index01`` (Swin3D/modules/swin3d_layers.py:
    789-822) that does not go through MinkowskiEngine: ``sp`` only needs ``.C`` (int [N,4]: batch,
    x, y, z) and its tensor stride.  Returns the same 8-tuple ``WindowAttention.forward``
    (:490-500) unpacks:

        (x_offset, y_offset, m2w_indices, w_sizes, w2n_indices, n2n_indices, w2m_indices, n_coords)

    ``x_offset`` and ``y_offset`` are not read by ``WindowAttention`` and ``m2w_indices`` (one entry
    per attention pair) is not read by the fused kernels: they are None / an empty tensor.  The
    index tensors are int32, which ``SelfAttnAIOFunction`` takes as they are (the reference converts
    int64 to int32 inside every call, self_attn_aio_fwd.cu:395-400).

    ``shift_size`` (in voxels of this stage) may be given instead of building a shifted copy of
    ``sp`` as ``BasicLayer.get_shifted_sp`` does; a shifted ``sp`` with ``shift_size=0`` groups
    the same way."""
    xyz, rest = local_xyz.float(), colors.float()
    if not sp.C.is_cuda or not xyz.is_cuda or not rest.is_cuda:
        raise RuntimeError("coords and feats must be CUDA tensors")
    N = sp.C.shape[0]
    if sp.C.dim() != 2 or sp.C.shape[1] != 4:
        raise ValueError("coords must be int32 [N, 4]")
    if xyz.dim() != 2 or rest.dim() != 2 or xyz.shape[0] != N or rest.shape[0] != N:
        raise ValueError("local_xyz and colors must be [N, columns]")
    if xyz.shape[1] != 3:                       # the signals count as one row wherever they are cut
        both = torch.cat([xyz, rest], dim=1)
        xyz, rest = both[:, :3], both[:, 3:]
    xyz = xyz if xyz.stride(1) == 1 else xyz.contiguous()
    rest = rest if rest.stride(1) == 1 else rest.contiguous()
    wi = _build(sp.C.int().contiguous(), xyz, rest, lambda: torch.cat([xyz, rest], dim=1), int(window_size), int(shift_size),
                _tensor_stride(sp))
    m2w = torch.empty(0, dtype=torch.int64, device=wi.n2n.device)
    return (None, None, m2w, wi.w_sizes, wi.w2n, wi.n2n, wi.w2m, wi.n_coords)
