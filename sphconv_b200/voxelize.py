"""Points -> range-voxel tensor on the GPU.

Host mirror of the reference's voxel generator for a given resolution (``VoxelGeneratorV3``,
sphconv/utils/voxel_generator.py:6-70, with ``points_to_voxel_v2``, sphconv/utils/voxelize.py:122-219) fused with
the mean of the kept points (``SimpleVoxel``, sphconv/vfe.py:210-228) and with ``init_tensor``: what
``VoxelizationVFE.generate`` + ``merge_batch_torch`` + ``SparseConvTensor(...)`` do in the reference's tests
(sphconv/datagen.py:77-108, test/common.py:33-59), for a whole batch of scans in a few kernel launches.

Differences from the reference, all on purpose: the points are a CUDA tensor (a batch is one tensor plus
``scan_ptr``); voxels come out in range-voxel row order (ascending b, c0, c1, c2), not in first-come order; the
per-voxel point lists (``voxels`` [V, max_points, C]) are not materialised, only their mean is.  Which points a
voxel keeps, which voxels survive ``max_voxels`` and every cell index are the reference's.
"""
from typing import List, Optional, Sequence

import numpy as np
import torch

from . import _capi as C
from .tensor import SparseConvTensor

SYSTEMS = {"spherical": 0, "l-spherical": 1, "cylinder": 2, "l-cylinder": 3, "hybrid": 4, "l-hybrid": 5}


def system_range(point_cloud_range: Sequence[float], point_cloud_sphere_range: Sequence[float],
                 coord_system: str) -> np.ndarray:
    """float32 [6] bounds of the three system coordinates, as the reference's transform functions return them
    (sphconv/utils/coord_transform.py:17-23 and the five siblings): degrees -> radians, logarithm of the range
    bounds for the l- systems, the Cartesian z bounds for the cylinders.  All in float32, like the reference."""
    c = np.asarray(point_cloud_range, dtype=np.float32)
    s = np.asarray(point_cloud_sphere_range, dtype=np.float32)
    logarithmic = coord_system.startswith("l-")
    first = (np.log(s[0]), np.log(s[3])) if logarithmic else (s[0], s[3])
    third = (c[2], c[5]) if coord_system.endswith("cylinder") else (np.radians(s[2]), np.radians(s[5]))
    return np.array([first[0], np.radians(s[1]), third[0], first[1], np.radians(s[4]), third[1]], dtype=np.float32)


class VoxelGenerator:
    """``VoxelGenerator(point_cloud_range, point_cloud_sphere_range, max_num_points, max_voxels, resolution_HWD,
    coord_system)``: the arguments of the reference's VoxelGeneratorV3 that its resolution path reads.
    ``resolution_HWD`` = cells along the (first, second, third) system coordinate, e.g. (r, phi, theta)."""

    def __init__(self, point_cloud_range, point_cloud_sphere_range, max_num_points: int, max_voxels: int = 30000,
                 resolution_HWD: Optional[List[int]] = None, coord_system: str = "spherical", append_mode: int = 0):
        if resolution_HWD is None:
            raise ValueError("resolution_HWD is required (the cell-size path of the reference is not provided)")
        if coord_system not in SYSTEMS:
            raise ValueError("unknown coord_system %r" % (coord_system,))    # the reference prints and exits
        self.coord_system = coord_system
        self.grid_size = [int(v) for v in resolution_HWD]
        self.max_num_points = int(max_num_points)
        self.max_voxels = int(max_voxels)
        self.append_mode = int(append_mode)
        self.system_range = system_range(point_cloud_range, point_cloud_sphere_range, coord_system)
        self._range = [float(v) for v in self.system_range]

    @property
    def spatial_shape(self) -> List[int]:
        """[s0, s1, s2] of the tensor ``to_tensor`` returns (what the reference calls spatial_shape_DWH)."""
        g = self.grid_size
        return [g[2], g[1], g[0]]

    def transform(self, points: torch.Tensor) -> torch.Tensor:
        """[N,4] system coordinates + intensity of the points (coord_transform.py of the reference)."""
        return C.host().voxel_transform(points, SYSTEMS[self.coord_system])

    def generate(self, points: torch.Tensor, scan_ptr: Optional[torch.Tensor] = None,
                 system_points: Optional[torch.Tensor] = None, with_coordinates: bool = True) -> dict:
        """points float32 [N, F] on the device; scan_ptr int32 [B+1] (device or host; None = one scan).
        Returns feature [NNZ, C], z_idx, z_ptr [B, s0, s1], coordinates int32 [NNZ,4] = (b, c0, c1, c2),
        num_points_per_voxel int32 [NNZ], voxel_num, batch_size, spatial_shape."""
        sys_pts = self.transform(points) if system_points is None else system_points
        feature, z_idx, z_ptr, coords, num = C.host().voxelize(
            points, scan_ptr, sys_pts, self.grid_size, self._range, self.max_num_points, self.max_voxels, self.append_mode,
            with_coordinates)
        return {"feature": feature, "z_idx": z_idx, "z_ptr": z_ptr, "coordinates": coords,
                "num_points_per_voxel": num, "voxel_num": feature.shape[0], "batch_size": z_ptr.shape[0],
                "spatial_shape": self.spatial_shape}

    def to_tensor(self, points: torch.Tensor, scan_ptr: Optional[torch.Tensor] = None,
                  dtype: Optional[torch.dtype] = None) -> SparseConvTensor:
        """The SparseConvTensor the encoder takes, straight from the points."""
        r = self.generate(points, scan_ptr, with_coordinates=False)
        feature = r["feature"] if dtype is None else r["feature"].to(dtype)
        return SparseConvTensor(feature, r["spatial_shape"], r["batch_size"], z_idx=r["z_idx"], z_ptr=r["z_ptr"])
