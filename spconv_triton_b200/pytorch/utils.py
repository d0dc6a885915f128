"""Point cloud voxelisation (reference: spconv_triton/pytorch/utils.py).

``PointToVoxel`` keeps the reference's constructor, persistent buffers, return
values and first-come-first-served semantics; the work is done by
``spc_voxelize_number`` / ``spc_voxelize_store`` of the CUDA library (hash table,
prefix sums, ranks inside a voxel) and its results equal the reference's bit for bit.  CUDA tensors
only: there is no CPU path.
"""

from __future__ import annotations

import torch

from ._impl import host as _host


class PointToVoxel:
    """WARNING: you MUST construct PointToVoxel AFTER set device."""

    def __init__(self, vsize_xyz: list[float], coors_range_xyz: list[float], num_point_features: int,
                 max_num_voxels: int, max_num_points_per_voxel: int,
                 device: torch.device = torch.device("cpu:0")):
        self.ndim = len(vsize_xyz)
        self.device = torch.device(device)
        self.num_point_features = num_point_features
        self.max_num_voxels = max_num_voxels
        self.max_num_points_per_voxel = max_num_points_per_voxel
        if self.device.type != "cuda":
            raise NotImplementedError("spconv_triton_b200 voxelises on CUDA devices only (no CPU path)")

        cmin = coors_range_xyz[: self.ndim]
        cmax = coors_range_xyz[self.ndim:]
        grid_size_xyz = [round((cmax[i] - cmin[i]) / vsize_xyz[i]) for i in range(self.ndim)]
        self._vsize_xyz = list(vsize_xyz)
        self._grid_size_xyz = grid_size_xyz
        self._coors_range_xyz = list(coors_range_xyz)
        # public metadata is stored reversed (z, y, x), as upstream (reference: utils.py:44-52)
        self.vsize = list(reversed(vsize_xyz))
        self.grid_size = list(reversed(grid_size_xyz))
        self.coors_range = list(reversed(cmin)) + list(reversed(cmax))
        stride = [1] * self.ndim
        for i in range(self.ndim - 2, -1, -1):
            stride[i] = stride[i + 1] * self.grid_size[i + 1]
        self.grid_stride = stride

        self.voxels = torch.zeros([max_num_voxels, max_num_points_per_voxel, num_point_features],
                                  dtype=torch.float32, device=self.device)
        self.indices = torch.zeros([max_num_voxels, self.ndim], dtype=torch.int32, device=self.device)
        self.num_per_voxel = torch.zeros([max_num_voxels], dtype=torch.int32, device=self.device)

    def __call__(self, pc: torch.Tensor, clear_voxels: bool = True, empty_mean: bool = False):
        res = self.generate_voxel_with_id(pc, clear_voxels, empty_mean)
        return res[0], res[1], res[2]

    def generate_voxel_with_id(self, pc: torch.Tensor, clear_voxels: bool = True, empty_mean: bool = False):
        """``(voxels [M, P, F], indices [M, ndim] zyx, num_per_voxel [M], pc_voxel_id [N])``
        (reference: utils.py:72-163)."""
        if pc.device != self.voxels.device:
            raise AssertionError("your pc device is wrong")
        if pc.dtype != torch.float32:
            raise NotImplementedError("points must be float32 (voxel boundaries are computed in the points' dtype)")
        if pc.dim() != 2 or pc.shape[1] < max(self.ndim, self.num_point_features):
            raise AssertionError("points must be [N, >= max(ndim, num_point_features)]")
        return _host.ext().voxelize(pc, self.voxels, self.indices, self.num_per_voxel, self._coors_range_xyz[:self.ndim], self._vsize_xyz,
                                    self._grid_size_xyz, bool(clear_voxels), bool(empty_mean))


def gather_features_by_pc_voxel_id(seg_res_features: torch.Tensor, pc_voxel_id: torch.Tensor,
                                   invalid_value: int | float = 0):
    """Per-voxel results back onto the points they came from; points without a
    voxel receive ``invalid_value`` (reference: utils.py:166-192)."""
    if seg_res_features.device != pc_voxel_id.device:
        pc_voxel_id = pc_voxel_id.to(seg_res_features.device)
    shape = (pc_voxel_id.shape[0], *seg_res_features.shape[1:])
    res = torch.full(shape, invalid_value, dtype=seg_res_features.dtype, device=seg_res_features.device)
    valid = torch.nonzero(pc_voxel_id != -1).view(-1)
    res[valid] = seg_res_features[pc_voxel_id[valid]]
    return res
