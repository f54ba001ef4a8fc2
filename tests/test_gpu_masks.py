"""The label mask and majorant passes (GPU) at the sizes where their splits end:
volumes whose rows are no multiple of a 4-voxel group or an 8-voxel brick, soft
grids that leave the scratch room for the nodes' records, for their flags only,
or for neither, flipped and permuted grid axes, the smallest and largest
smoothing radius, each label mode and storage.

Tolerances: masks within one code step of the oracle's with 99.9 % of the codes
equal (its expf differs from CUDA's in the last bit, which a code boundary can
show), majorants bit-exact on the device's masks.
"""
import numpy as np
import pytest

from oracle import oracle as O
from volview_gb300 import abi, scene
from volview_gb300 import renderer as R

pytestmark = pytest.mark.gpu

# (volume x, y, z; soft grid: the voxels per node, its dims, or None; source
# axes; flips; radius; label mode; storage)
CASES = {
    "ragged_third": ((37, 26, 19), 3, (0, 1, 2), (0, 0, 0), 1, abi.LABEL_HYBRID, (0, 0)),
    "ragged_half_radius8": ((41, 33, 17), 2, (0, 1, 2), (0, 0, 0), 8, abi.LABEL_HYBRID, (0, 0)),
    "per_voxel_nodes": ((35, 21, 14), 1, (0, 1, 2), (0, 0, 0), 2, abi.LABEL_ISOLATE, (0, 0)),
    "nodes_beyond_scratch": ((5, 3, 2), (31, 30, 29), (0, 1, 2), (0, 0, 0), 1, abi.LABEL_HYBRID, (0, 0)),
    "permuted_flipped": ((30, 23, 45), (12, 17, 9), (2, 0, 1), (1, 0, 1), 3, abi.LABEL_HYBRID, (0, 0)),
    "tint_margin": ((33, 18, 27), 3, (0, 1, 2), (0, 1, 0), 0, abi.LABEL_TINT, (0, 0)),
    "no_grid": ((29, 34, 9), None, (0, 1, 2), (0, 0, 0), 4, abi.LABEL_HYBRID, (0, 0)),
    "labels_off": ((27, 9, 11), None, (0, 1, 2), (0, 0, 0), 1, abi.LABEL_OFF, (3, 0)),
    "bf16_mask_radius5": ((18, 39, 21), 2, (0, 1, 2), (0, 0, 1), 5, abi.LABEL_HYBRID, (2, 2)),
    "fp32": ((39, 20, 25), 2, (0, 1, 2), (0, 0, 0), 1, abi.LABEL_HYBRID, (3, 0)),
    "one_voxel": ((1, 1, 1), None, (0, 1, 2), (0, 0, 0), 1, abi.LABEL_HYBRID, (0, 0)),
}


def _inputs(dims, soft, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    z, y, x = np.mgrid[:nz, :ny, :nx]
    # Slanted layers of six labels (0, 1 and 4 .. 7) around a core, HU by label.
    lab = (((x + 2 * y + z) // 9) % 6).astype(np.uint8)
    lab[lab > 1] += 2
    hu = np.clip(lab * 150.0 - 200.0 + 60.0 * rng.standard_normal(lab.shape), -1024, 3071).astype(np.int16)
    if soft is None:
        return hu, lab, None
    if isinstance(soft, int):
        grid = scene.soft_grid(lab, (1.0, 1.0, 1.0), soft)
    else:
        grid = np.zeros(soft[::-1] + (4,), np.uint8)
        band = np.add.outer(np.add.outer(np.arange(soft[2]), np.arange(soft[1])), np.arange(soft[0])) // 4
        grid[..., 0], grid[..., 1] = band % 3 + 4, (band + 1) % 3 + 4
        grid[..., 2] = rng.integers(0, 255, band.shape)
    grid[..., 3] = rng.random(grid.shape[:3]) < 0.03  # some nodes replaced by finer labels
    return hu, lab, grid


@pytest.mark.parametrize("name", list(CASES))
def test_masks_and_majorants(name, gpu_ctx):
    dims, soft, axes, flips, radius, mode, (density, mask) = CASES[name]
    hu, lab, grid = _inputs(dims, soft, 5)
    vol, tf = abi.volume_struct(hu, (1.0, 1.0, 1.0)), abi.tf_struct(abi.PRESETS["bone"])
    labels = scene.label_params(lab, hu, {v: (scene.OTHER, (0.5, 0.4, 0.3), 0.4) for v in (1, 4, 5, 6, 7)}, mode=mode)
    labels.smoothing = radius
    labels.ghost[5] = 1
    labels.colors[6][3] = 0.0
    r = R.Renderer(gpu_ctx, vol, tf, abi.precision(density_format=density, mask_format=mask))
    cpu = O.CpuRenderer(vol, tf, hu, density_format=density, mask_format=mask)
    try:
        if mode != abi.LABEL_OFF:
            r.set_labels(lab, abi.soft_struct(grid, axes, flips) if grid is not None else None)
            cpu.set_labels(lab, grid, axes, flips)
        r.resize(16, 16)
        p = abi.frame_params(abi.camera_framing(list(r.center), r.diagonal), 0.5, labels, abi.lighting_default(),
                             abi.path_tracing_default(), abi.clipping_default())
        r.probe_bspline(p, np.zeros((1, 3), np.float32))  # runs record's mask and majorant passes
        cpu.prepare(p, 16, 16)
        if mode != abi.LABEL_OFF:
            got = r.read_volume(abi.VOLUME_MASK)
            d = np.abs(got.astype(np.int32) - cpu.mask.astype(np.int32))
            assert d.max() <= 1 and (d == 0).mean() >= 0.999, (d.max(), (d == 0).mean())
            cpu.mask = got
        u = cpu.uniforms(p, 1, 16, 16)
        maj = np.zeros_like(cpu.majorant)
        O.lib().vvo_majorant(O.ptr(u), O.C.byref(cpu.scene()), O.ptr(maj))
        assert np.array_equal(r.read_volume(abi.VOLUME_MAJORANT), maj)
    finally:
        r.destroy()
