"""A batch of planes of many sizes: the resident solver takes them in one launch,
its gangs passing from planes that fill them to planes that leave some of their
CTAs without a tile and back. Equal to the streaming solver plane for plane (the
two differ in the order of FP64 additions only, below the float rounding of
alpha and beta), and to the same planes decoded alone."""
import numpy as np
import pytest

from hvdg import _cabi, api, synth

pytestmark = pytest.mark.gpu


def _geom(std, w, lines):
    g = _cabi.default_geometry(std)
    return _cabi.geometry_copy(g, active_video_end=g.active_video_start + w,
                               last_active_field_line=g.first_active_field_line + lines)


def _fields(sizes):
    fields = []
    for i, (std, w, lines) in enumerate(sizes):
        g = _geom(std, w, lines)
        fields.append(api.Field(
            synth.make_field(20 + i, std, 0.7, field_index=i % 4, geometry=g).samples, g,
            parity=i % 2, irls_outer=1 + i % 3, cg_iterations=(1 + i % 3) * (6 + 5 * (i % 4))))
    return fields


@pytest.mark.parametrize("sizes", [
    [(0, 40 + 23 * i, 17 + 9 * i) for i in range(16)],       # one strip to seven
    [(0, 758 - 7 * i, 240 - 3 * i) for i in range(9)],       # near whole fields
    [(i % 2, 8 + 130 * (i % 5), 16 + 37 * (i % 6)) for i in range(30)],
])
def test_many_sizes_in_one_launch(sizes):
    fields = _fields(sizes)
    cfg = api.default_config(fast=0, cg_tol=1e-6, temporal_strength=-1.0)
    with api.Context(0) as ctx:
        ctx.set_tuning(16, 0)        # a set tiling selects the streaming solver
        stream = ctx.decode_fields(fields, cfg)
        it, n_stream = ctx.last_diag.cg_iterations_run, ctx.last_diag.kernel_launches
        ctx.set_tuning(0, 0)
        got = ctx.decode_fields(fields, cfg)
        assert ctx.last_diag.cg_iterations_run == it
        assert ctx.last_diag.kernel_launches == n_stream    # one solver launch, not one a size
        alone = [ctx.decode_fields([f], cfg)[0] for f in fields]
    for a, b, c in zip(stream, got, alone):
        for key in ("luma", "chroma"):
            assert np.array_equal(getattr(a, key), getattr(b, key)), key
            assert np.array_equal(getattr(b, key), getattr(c, key)), key
