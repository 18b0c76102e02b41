"""The resident solver with neighbour terms (3-D windows) on tall tiles, against
the streaming solver: windows whose colours hold several fields, so that a few
gangs share the chip (four NTSC fields: 81 rows, six a warp), and lone fields on
large planes up to the tallest tile that fits beside the neighbour terms (87
rows). The two kernels perform the same operations on every pixel and differ
only in the order of FP64 additions, below the float rounding of alpha and
beta: their planes are equal."""
import numpy as np
import pytest

from hvdg import _cabi, api, synth

pytestmark = pytest.mark.gpu


def _cfg(**kw):
    base = dict(cg_tol=1e-6, temporal_strength=0.5, passes=1, irls_outer=2, cg_iterations=12)
    base.update(kw)
    return api.default_config(**base)


def _fields(g, n):
    return [api.Field(synth.make_field(60 + i, g.standard, 0.7, field_index=i % 4,
                                       geometry=g).samples, g, parity=i % 2) for i in range(n)]


def _wide(w, lines):
    # PAL: NTSC planes this large are past the automatic anisotropy's samples
    g = _cabi.default_geometry(_cabi.STD_PAL)
    a0 = g.active_video_start
    return _cabi.geometry_copy(g, field_width=a0 + w + 20, field_height=lines + 30,
                               active_video_end=a0 + w, first_active_field_line=20,
                               last_active_field_line=20 + lines)


@pytest.mark.parametrize("std,n,kw", [
    (0, 13, {}),                           # colours of four and three fields
    (0, 16, {}),                           # four of four: the default export chunk
    (0, 10, dict(extended_temporal=0)),    # stride three
    (1, 12, {}),                           # PAL, stride five
])
def test_window_of_several_fields_a_colour(std, n, kw):
    fields = _fields(_cabi.default_geometry(std), n)
    cfg = _cfg(fast=1, **kw)
    with api.Context(0) as ctx:
        ctx.set_tuning(16, 0)        # a set tiling selects the streaming solver
        stream = ctx.decode_field_window(fields, cfg)
        it = ctx.last_diag.cg_iterations_run
        ctx.set_tuning(0, 0)
        resident = ctx.decode_field_window(fields, cfg)
        assert ctx.last_diag.cg_iterations_run == it
    for a, b in zip(stream, resident):
        assert np.array_equal(a.luma, b.luma) and np.array_equal(a.chroma, b.chroma)


@pytest.mark.parametrize("w,lines", [
    (1024, 720),     # 80 rows: five a warp
    (1024, 729),     # 81 rows: the sixth row of one warp
    (1280, 576),     # 82 and 83 rows
    (1024, 783),     # 87 rows, the tallest
    (1024, 784),     # past it: the streaming solver takes both calls
])
def test_tall_tiles_of_a_lone_field(w, lines):
    fields = _fields(_wide(w, lines), 3)
    cfg = _cfg(fast=0)
    with api.Context(0) as ctx:
        ctx.set_tuning(16, 0)
        stream = ctx.decode_field_window(fields, cfg)
        it = ctx.last_diag.cg_iterations_run
        ctx.set_tuning(0, 0)
        resident = ctx.decode_field_window(fields, cfg)
        assert ctx.last_diag.cg_iterations_run == it
    for a, b in zip(stream, resident):
        assert np.array_equal(a.luma, b.luma) and np.array_equal(a.chroma, b.chroma)


def test_export_chunk_of_a_sequence():
    """Eight frames in one call (sequence.plan_chunks' default chunk)."""
    frames, _ = synth.make_frames(71, _cabi.STD_NTSC, 8, noise_sigma=1.0, moving=True)
    fp = api.frame_params(_cabi.STD_NTSC)
    cfg = _cfg(fast=1)
    with api.Context(0) as ctx:
        ctx.set_tuning(16, 0)
        stream = ctx.decode_frame_sequence_window(frames, 1, 7, fp, cfg)
        ctx.set_tuning(0, 0)
        resident = ctx.decode_frame_sequence_window(frames, 1, 7, fp, cfg)
    assert len(stream) == len(resident) == 6
    for a, b in zip(stream, resident):
        for key in ("luma", "chroma", "u", "v"):
            assert np.array_equal(a[key], b[key]), key
