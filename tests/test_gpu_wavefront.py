"""How the wavefront tracer schedules its paths changes none of them (GPU): the
ordering of the later flights, a pass alone (short queues spread over the chip)
or beside another renderer's, slots refilled or not, background paths that end
with their item, and the prepared grid of flight majorants.

A pass of one frame per pixel stores its sums without atomics, so those images
are compared bit by bit. Frames accumulated by one pass are added with float
atomics in an order the device decides: N positive FP32 terms in any order
differ by at most about N * 2^-23 relative, so 1e-5 holds for the sums of up
to 40 frames here."""
import numpy as np
import pytest

from volview_gb300 import abi, scene
from volview_gb300 import renderer as R

pytestmark = pytest.mark.gpu


def _renderer(cfg, ctx, env=None):
    r = R.Renderer(ctx, cfg["volume"], cfg["tf"])
    r.set_labels(cfg["labels_vol"], abi.soft_struct(cfg["soft"]))
    if env is not None:
        r.set_environment_map(abi.env_struct(env))
    return r


def _params(cfg, r, near=0.5):
    p = scene.frame_params_for(cfg, list(r.center), r.diagonal, clip_sagittal=True)
    p.camera.distance = abi.f32(p.camera.distance * near)
    p.path_tracing.denoiser = abi.DENOISE_OFF
    return p


def _frame(r, p):
    r.reset_view()
    r.record(1, p)
    return r.read_accumulation()


@pytest.mark.parametrize("light", ["studio", "map"])
@pytest.mark.parametrize("size", [(1, 1), (37, 21), (131, 77)])
def test_order_and_company_change_no_path(small_cfg, gpu_ctx, monkeypatch, size, light):
    """131 x 77 paths run through the waves and then the finishing launch, the
    smaller images through the finishing launch alone."""
    cfg = small_cfg
    r = _renderer(cfg, gpu_ctx, scene.synthetic_light_map() if light == "map" else None)
    ctx = R.Context(0)
    other = _renderer(cfg, ctx)
    try:
        p = _params(cfg, r)
        if light == "map":
            p.lighting.environment = abi.ENV_MAP
        r.resize(*size)
        other.resize(96, 64)
        q = _params(cfg, other)
        images = []
        for bin_min, company in ((None, False), ("0", False), (None, True), ("0", True)):
            if bin_min is None:
                monkeypatch.delenv("VV_WF_BIN_MIN", raising=False)
            else:
                monkeypatch.setenv("VV_WF_BIN_MIN", bin_min)
            if company:
                other.reset_view()
                other.record_frames(1, 32, q)
            images.append(_frame(r, p))
            other.synchronize()
        assert size == (1, 1) or np.any(images[0][0][..., :3])
        for image in images[1:]:
            for a, b in zip(image, images[0]):
                assert np.array_equal(a, b)
    finally:
        r.destroy()
        other.destroy()
        ctx.destroy()


@pytest.mark.parametrize("slot_frames", [16, 2])
@pytest.mark.parametrize("near", [0.4, 3.0])
def test_frames_of_one_pass_sum_to_single_frames(small_cfg, gpu_ctx, near, slot_frames):
    """Eight frames in one pass (with slots for all of them, and refilled from
    two frames' worth) against eight single frames, close up and at a distance
    where most paths leave the volume at once."""
    cfg = small_cfg
    r = _renderer(cfg, gpu_ctx)
    try:
        p = _params(cfg, r, near)
        r.resize(83, 59)
        for f in range(8):
            r.record(f + 1, p)
        single = r.read_accumulation()
        r.reset_view()
        r.set_pass_budget(2, slot_frames)
        r.record_frames(1, 8, p)
        for a, b in zip(r.read_accumulation(), single):
            assert np.all(np.abs(a - b) <= 1e-5 * np.abs(b) + 1e-6)
    finally:
        r.destroy()


def test_flight_majorants_follow_their_inputs(small_cfg, gpu_ctx):
    """A renderer whose parameters change between frames gives the images of
    fresh renderers: the flight majorants follow the skipping of empty space,
    the label mode, the label extinction and the tissues' anisotropy."""
    cfg = small_cfg
    kept = _renderer(cfg, gpu_ctx)
    try:
        kept.resize(61, 43)

        def base():
            return _params(cfg, kept)

        def skipping(p):
            p.skip_empty_space = 0

        def mode(p):
            p.labels.mode = abi.LABEL_TINT

        def extinction(p):
            p.labels.extinction = abi.f32(p.labels.extinction * 0.5)

        def anisotropy(p):
            p.lighting.anisotropy = abi.f32(0.9)

        for change in (lambda p: None, skipping, extinction, anisotropy, mode, skipping, lambda p: None):
            p = base()
            change(p)
            image = _frame(kept, p)
            fresh = _renderer(cfg, gpu_ctx)
            try:
                fresh.resize(61, 43)
                for a, b in zip(image, _frame(fresh, p)):
                    assert np.array_equal(a, b)
            finally:
                fresh.destroy()
    finally:
        kept.destroy()


@pytest.mark.parametrize("samples", [1, 3])
@pytest.mark.parametrize("size", [(37, 21), (131, 77), (311, 300)])
def test_the_finishing_launch_changes_no_path(small_cfg, gpu_ctx, monkeypatch, size, samples):
    """Paths handed to the finishing launch at the end, midway and all at once:
    alone in their warps, and, where every warp is full with them (311 x 300), 32
    to a warp."""
    r = _renderer(small_cfg, gpu_ctx)
    try:
        p = _params(small_cfg, r)
        p.path_tracing.samples_per_frame = samples
        r.resize(*size)
        images = []
        for tail in ("0", "1024", "20000", "100000000"):
            monkeypatch.setenv("VV_WF_TAIL", tail)
            images.append(_frame(r, p))
        for image in images[1:]:
            for a, b in zip(image, images[0]):
                assert np.array_equal(a, b)
    finally:
        r.destroy()


@pytest.mark.parametrize("beside", ["renderer", "engine"])
def test_passes_beside_each_other_know_it_and_change_no_path(small_cfg, gpu_ctx, beside):
    """A pass beside several of another renderer's, or of a batch engine's, packs
    its short queues; the next one, by itself, spreads them. Both give the same
    sums bit by bit, and no pass is left counted."""
    r = _renderer(small_cfg, gpu_ctx)
    ctx = R.Context(0)
    other = _renderer(small_cfg, ctx)
    engine = R.BatchEngine(ctx, 3, 16) if beside == "engine" else None
    try:
        p, q = _params(small_cfg, r), _params(small_cfg, other)
        r.resize(131, 77)
        other.resize(960, 720)  # three passes of 64 frames take many times as long as r's one
        images, seen = [], []
        for company in (True, False):
            for k in range(3 if company else 0):
                if engine:
                    engine.record([(other, q, 1 + 64 * k, 64, True)])
                else:
                    other.record_frames(1 + 64 * k, 64, q)
            r.reset_view()
            r.record(1, p)
            seen.append(r.probe_company())
            images.append(r.read_accumulation())
            other.synchronize()
        assert [spread for _, spread in seen] == [False, True]
        assert seen[0][0] >= 1 and seen[1][0] == 0
        for a, b in zip(*images):
            assert np.array_equal(a, b)
    finally:
        if engine:
            engine.synchronize()
            engine.destroy()
        r.destroy()
        other.destroy()
        ctx.destroy()


@pytest.mark.parametrize("kernel", ["wavefront", "persistent"])
def test_majorants_are_counted_once_per_brick_that_a_flight_enters(gpu_ctx, monkeypatch, kernel):
    """One dense brick, clipped away whole: a flight crosses it through many
    tentative collisions, none of which reads a voxel or casts a shadow ray, and
    the one majorant it needs is one event."""
    if kernel != "wavefront":
        monkeypatch.setenv("VV_PT_KERNEL", kernel)
    hu = np.full((8, 8, 8), 1500, np.int16)
    r = R.Renderer(gpu_ctx, abi.volume_struct(hu, (4.0, 4.0, 4.0)), abi.tf_struct(abi.PRESETS["bone"]))
    try:
        p = scene.frame_params_for(dict(min_spacing=4.0, label_params=abi.label_params_default()), list(r.center),
                                   r.diagonal, clip_sagittal=True)
        p.clipping.planes[0].position = abi.f32(r.bounds[0][0] - 1.0)
        p.camera.distance = abi.f32(p.camera.distance * 0.5)
        p.path_tracing.denoiser = abi.DENOISE_OFF
        r.resize(40, 30)
        r.count_events(True)
        r.record(1, p)
        events = r.count_events(False)
        assert events["path"] == 1200 and events["trilinear"] == events["cubic"] == 0
        assert 600 <= events["majorant"] <= 1200
    finally:
        r.destroy()
