"""The real-time ray marcher (path tracing off) against the reference's own
shaders (GPU): the occlusion volume (ao.comp), the shadow volume swept towards
the key light (shadow.comp with record_shadow_sweep) and the image (dvr.comp),
for point-sampled and pre-integrated transfer functions and a light map,
against tests/golden/small_raymarch.npz (made by tests/golden/make_golden.py
from the reference's shaders compiled as CPU code).

Tolerances: uniforms bit-exact; the half-precision volumes and image within
2e-3 absolute (plus 1e-2 relative) for >= 99 % of their values, and the whole
image's mean radiance within 1 %. The device evaluates expf/powf/sqrtf and
contracts multiply-adds, so last bits differ, and a voxel at the masks'
zero boundary may land one quantum off (see the mask parity test).
"""
import os

import numpy as np
import pytest

from oracle import oracle as O
from volview_gb300 import abi, scene
from volview_gb300 import renderer as R

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "small_raymarch.npz")


def _half(a):
    return np.asarray(a).view(np.float16).astype(np.float32)


def _close(a, b, what):
    d = np.abs(a - b)
    ok = d <= 2e-3 + 1e-2 * np.abs(b)
    assert ok.mean() >= 0.99, f"{what}: {ok.mean():.4f} within tolerance, max diff {d.max():.4g}"


@pytest.fixture(scope="module")
def golden():
    if not os.path.exists(GOLDEN):
        pytest.skip("ray marcher fixture not generated")
    return np.load(GOLDEN)


@pytest.mark.parametrize("case", ["point", "preint", "map"])
def test_ray_marcher_matches_reference_shaders(golden, gpu_ctx, case):
    g = golden
    vol = abi.volume_struct(g["hu"], tuple(g["spacing"]))
    tf = abi.tf_struct(abi.PRESETS["bone"])
    r = R.Renderer(gpu_ctx, vol, tf)
    r.set_labels(g["labels"], abi.soft_struct(g["soft"]))
    if case == "map":
        r.set_environment_map(abi.env_struct(g["light_map"]))
    params = abi.FrameParams.from_buffer_copy(g[f"{case}_params"].tobytes())
    assert params.path_tracing.enabled == 0
    W, H = int(g["width"]), int(g["height"])
    r.resize(W, H)
    assert np.array_equal(r.pack_uniforms(params, 1), g[f"{case}_uniforms"])
    r.record(1, params)
    assert r.accumulated_samples() == 0  # the ray marcher accumulates nothing
    ao = _half(r.read_volume(abi.VOLUME_AO))
    shadow = _half(r.read_volume(abi.VOLUME_SHADOW))
    _close(ao, _half(g[f"{case}_ao"]), "occlusion volume")
    _close(shadow, _half(g[f"{case}_shadow"]), "shadow volume")
    hdr, ref = _half(r.read_hdr()), _half(g[f"{case}_hdr"])
    _close(hdr, ref, "image")
    assert abs(hdr[..., :3].mean() - ref[..., :3].mean()) <= 0.01 * ref[..., :3].mean() + 1e-6
    out = r.read_output()
    assert out.shape == (H, W, 4) and out[..., :3].std() > 0
    r.destroy()


def test_ray_marcher_rejects_batched_frames(golden, gpu_ctx):
    g = golden
    vol = abi.volume_struct(g["hu"], tuple(g["spacing"]))
    r = R.Renderer(gpu_ctx, vol, abi.tf_struct(abi.PRESETS["bone"]))
    params = abi.FrameParams.from_buffer_copy(g["point_params"].tobytes())
    r.resize(16, 16)
    with pytest.raises(R.VolptError) as e:
        r.record_frames(1, 4, params)
    assert e.value.status == abi.VV_ERR_ARG
    r.destroy()


@pytest.mark.parametrize("size", [(1, 1), (3, 17), (37, 21), (96, 64)])
@pytest.mark.parametrize("mode", ["hybrid", "isolate", "ghost", "binary"])
def test_lanes_per_ray_give_the_same_image(small_cfg, gpu_ctx, monkeypatch, size, mode):
    """Two and four lanes per ray (k_dvr_masks) against one (k_dvr): every HDR
    value and every byte of the image, at sizes that leave a warp's rays partly
    outside, with ghosts (whose lighting decides their opacity, and so whether
    the surface behind them is the one refined), cuts and binary masks."""
    cfg = small_cfg
    r = R.Renderer(gpu_ctx, cfg["volume"], cfg["tf"])
    try:
        p = scene.frame_params_for(cfg, list(r.center), r.diagonal, clip_sagittal=True)
        soft = mode in ("hybrid", "isolate") or scene.mode_case(mode, p, list(r.center))
        if mode == "isolate":
            scene.mode_case("isolate", p, list(r.center))
        r.set_labels(cfg["labels_vol"], abi.soft_struct(cfg["soft"]) if soft else None)
        p.camera.distance = abi.f32(p.camera.distance * 0.45)
        p.path_tracing.enabled = 0
        r.resize(*size)
        images = []
        for lanes in ("1", "2", "4"):
            monkeypatch.setenv("VV_DVR_LANES", lanes)
            r.reset_view()
            r.record(1, p)
            images.append((r.read_hdr(), r.read_output()))
        for hdr, out in images[1:]:
            assert np.array_equal(hdr, images[0][0]) and np.array_equal(out, images[0][1])
    finally:
        r.destroy()


AXES = {"+x": (90.0, 0.0), "-x": (-90.0, 0.0), "+y": (180.0, 0.0), "-y": (0.0, 0.0), "+z": (0.0, 90.0),
        "-z": (0.0, -90.0)}  # the key light's azimuth and elevation as seen by a camera that looks along +y


@pytest.mark.parametrize("tilt", [0.0, 11.0])
@pytest.mark.parametrize("towards", AXES)
def test_shadow_sweep_with_and_without_room_for_its_factors(gpu_ctx, towards, tilt):
    """The sweep whose factors are taken ahead, slices chained (a renderer with
    label masks has the room), against the sweep of plain launches (one without
    has none): the same volume bit by bit, along each axis both ways. Both
    renderers draw the transfer function alone."""
    rng = np.random.default_rng(5)
    dims = (75, 58, 66)  # 38 x 29 x 33 texels, blocks of 8 x 8 partly outside
    hu = rng.integers(-1000, 1500, dims[::-1]).astype(np.int16)
    cfg = dict(min_spacing=1.0, label_params=abi.label_params_default())
    volume = abi.volume_struct(hu, (1.0, 1.0, 1.0))
    sweeps = []
    for labels in (None, np.zeros(hu.shape, np.uint8)):
        r = R.Renderer(gpu_ctx, volume, abi.tf_struct(abi.PRESETS["bone"]))
        try:
            if labels is not None:
                r.set_labels(labels)
            p = scene.frame_params_for(cfg, list(r.center), r.diagonal)
            p.path_tracing.enabled = 0
            p.camera.pitch = p.camera.yaw = 0.0
            azimuth, elevation = AXES[towards]
            p.lighting.azimuth = abi.to_radians(azimuth + tilt)
            p.lighting.elevation = abi.to_radians(elevation + (tilt if abs(elevation) < 90.0 else -tilt))
            r.resize(16, 16)
            for _ in range(2):  # twice: with the light moved between, so that both are swept
                p.lighting.elevation, other = abi.f32(0.3), p.lighting.elevation
                r.record(1, p)
                p.lighting.elevation = other
                r.record(2, p)
                sweeps.append(r.read_volume(abi.VOLUME_SHADOW))
        finally:
            r.destroy()
    assert _half(sweeps[0]).std() > 0.05
    for s in sweeps[1:]:
        assert np.array_equal(s, sweeps[0])


@pytest.mark.parametrize("size", [(16, 16), (37, 21), (96, 64)])
@pytest.mark.parametrize("mode", [abi.LABEL_HYBRID, abi.LABEL_ISOLATE])
def test_lanes_per_ray_with_labels_up_to_the_volumes_faces(small_cfg, gpu_ctx, monkeypatch, size, mode):
    """Labels that fill the volume to its faces, its silhouette inside the image:
    rays that miss the volume gather nothing, whatever the rays beside them in
    the warp do, with two and four lanes per ray as with one."""
    z, y, x = np.mgrid[0:21, 0:27, 0:30]
    labels = (1 + (x // 5 + y // 4 + z // 6) % 10).astype(np.uint8)
    hu = (200 + 37 * labels.astype(np.int16)).astype(np.int16)
    params = abi.LabelParams.from_buffer_copy(bytes(small_cfg["label_params"]))
    params.mode = mode
    r = R.Renderer(gpu_ctx, abi.volume_struct(hu, (1.0, 1.0, 1.0)), small_cfg["tf"])
    try:
        r.set_labels(labels)
        p = scene.frame_params_for(dict(min_spacing=1.0, label_params=params), list(r.center), r.diagonal)
        p.camera.yaw, p.camera.pitch = abi.f32(0.5), abi.f32(0.3)
        p.path_tracing.enabled = 0
        r.resize(*size)
        images = []
        for lanes in ("1", "2", "4"):
            monkeypatch.setenv("VV_DVR_LANES", lanes)
            r.reset_view()
            r.record(1, p)
            images.append(r.read_hdr())
        clear = _half(images[0])[..., 3] == 1.0  # transmittance: nothing met
        assert 0.1 < clear.mean() < 0.95
        for image in images[1:]:
            assert np.array_equal(image, images[0])
    finally:
        r.destroy()


@pytest.mark.parametrize("skip", [1, 0])
@pytest.mark.parametrize("mode", ["plain", "off", "tint"])
@pytest.mark.parametrize("hu,fmt", [(0, abi.DENSITY_FP16), (0, abi.DENSITY_BF16), (2048, abi.DENSITY_FP16),
                                    (2048, abi.DENSITY_UNORM16)])
def test_occlusion_and_shadow_next_to_an_opacity_edge(gpu_ctx, hu, fmt, mode, skip):
    """A homogeneous volume whose transfer function is opaque up to one HU below
    it: the lookup between the two LUT entries gives an extinction, although the
    bucket maximum of the density, which starts one entry higher, is 0. The
    extinction is constant (the sampler clamps to the volume), so the occlusion
    is min(2 exp(-15 c), 1) everywhere (16 directions of 8 samples, 15 mm) and
    each slice of the sweep lets exp(-2 c) through (half resolution, 1 mm).
    Bars: the occlusion's FP16 ulp and the 8 FP32 adds, 1e-3; a slice's FP16
    rounding, 2^-11 relative, over 12 slices, 1e-2."""
    volume = np.full((24, 24, 24), hu, np.int16)
    tf = abi.tf_struct([(-1024.0, (0.8, 0.7, 0.6), 6.0), (hu - 1.0, (0.8, 0.7, 0.6), 6.0),
                        (float(hu), (0.8, 0.7, 0.6), 0.0), (3071.0, (0.8, 0.7, 0.6), 0.0)])
    lp = abi.label_params_default()
    lp.mode = abi.LABEL_TINT if mode == "tint" else abi.LABEL_OFF
    struct = abi.volume_struct(volume, (1.0, 1.0, 1.0))
    cpu = O.CpuRenderer(struct, tf, volume, density_format=fmt)
    r = R.Renderer(gpu_ctx, struct, tf, abi.precision(density_format=fmt))
    try:
        if mode != "plain":
            r.set_labels(np.zeros(volume.shape, np.uint8))
        p = scene.frame_params_for(dict(min_spacing=1.0, label_params=lp), list(r.center), r.diagonal)
        p.path_tracing.enabled = 0
        p.skip_empty_space = skip
        p.camera.yaw = p.camera.pitch = 0.0
        p.lighting.azimuth, p.lighting.elevation = 0.0, abi.to_radians(90.0)  # towards +z
        r.resize(16, 16)
        r.record(1, p)
        c = float(r.probe_extinction(p, [[11.3, 12.1, 10.6]], smooth=False)[0, 2])  # blue: no chroma
        lp.mode = abi.LABEL_OFF
        cpu.resize(16, 16)
        q = scene.frame_params_for(dict(min_spacing=1.0, label_params=lp), list(r.center), r.diagonal)
        expected, bound = cpu.extinction(q, [[11.3, 12.1, 10.6]], smooth=False)[0, [2, 3]]
        assert c > 0.02 and abs(c - expected) <= 0.05 * expected and bound == 0.0
        ao, shadow = _half(r.read_volume(abi.VOLUME_AO)), _half(r.read_volume(abi.VOLUME_SHADOW))
        assert np.all(np.abs(ao - min(2.0 * np.exp(-15.0 * c), 1.0)) <= 1e-3)
        through = np.exp(-2.0 * c * np.arange(12, 0, -1))[:, None, None]  # z fastest from the light: the last slice first
        assert np.all(np.abs(shadow[..., 3] - through) <= 1e-2 * through + 1e-4)
    finally:
        r.destroy()


@pytest.mark.parametrize("preintegrate", [0, 1])
@pytest.mark.parametrize("size", [(1, 1), (37, 21), (96, 64)])
def test_transfer_function_alone_as_with_labels_that_draw_nothing(small_cfg, gpu_ctx, size, preintegrate):
    """Rays wait for more company with labels than without; which rays are lit
    together changes none of them. Tint over a label volume of zeros draws what
    the transfer function alone does, bit by bit."""
    cfg = small_cfg
    r = R.Renderer(gpu_ctx, cfg["volume"], cfg["tf"])
    try:
        r.set_labels(np.zeros(cfg["labels_vol"].shape, np.uint8))
        p = scene.frame_params_for(cfg, list(r.center), r.diagonal, clip_sagittal=True)
        p.camera.distance = abi.f32(p.camera.distance * 0.45)
        p.path_tracing.enabled = 0
        p.preintegrate = preintegrate
        r.resize(*size)
        images = []
        for mode in (abi.LABEL_OFF, abi.LABEL_TINT):
            p.labels.mode = mode
            r.record(1, p)
            images.append(r.read_hdr())
        assert size == (1, 1) or np.any(images[0][..., :3])
        assert np.array_equal(images[0], images[1])
    finally:
        r.destroy()


def test_lanes_per_ray_light_an_extinction_that_is_not_a_number(small_cfg, gpu_ctx, monkeypatch):
    """A label extinction of NaN shows as NaN pixels, with two and four lanes per
    ray as with one."""
    cfg = small_cfg
    r = R.Renderer(gpu_ctx, cfg["volume"], cfg["tf"])
    try:
        r.set_labels(cfg["labels_vol"], abi.soft_struct(cfg["soft"]))
        p = scene.frame_params_for(cfg, list(r.center), r.diagonal)
        p.camera.distance = abi.f32(p.camera.distance * 0.45)
        p.path_tracing.enabled = 0
        p.labels.extinction = float("nan")
        r.resize(37, 21)
        images = []
        for lanes in ("1", "2", "4"):
            monkeypatch.setenv("VV_DVR_LANES", lanes)
            r.reset_view()
            r.record(1, p)
            images.append(r.read_hdr())
        assert np.isnan(_half(images[0])).any()
        for image in images[1:]:
            assert np.array_equal(np.isnan(_half(image)), np.isnan(_half(images[0])))
    finally:
        r.destroy()
