"""The resident solver (k_resident.cu) against the streaming one (k_solver.cu)
and the FP64 oracle, where its tiling can go wrong: planes narrower than a
strip, one column or row past a tile, odd widths, fewer rows than warps,
tall tiles (97 rows), more fields than gangs, mixed sizes in one batch, the
3-D neighbour terms, and a pass that ends early.

The two kernels perform the same operations on every pixel and differ only in
the order of FP64 additions, whose effect is below the float rounding of alpha
and beta: their planes are equal."""
import numpy as np
import pytest

from hvdg import _cabi, api, synth

pytestmark = pytest.mark.gpu


def _geom(std, w=0, lines=0, sub=0.0):
    g = _cabi.default_geometry(std)
    if w:
        g = _cabi.geometry_copy(g, active_video_end=g.active_video_start + w)
    if lines:
        g = _cabi.geometry_copy(g, last_active_field_line=g.first_active_field_line + lines)
    return _cabi.geometry_copy(g, subcarrier_hz=sub) if sub else g


def _fields(g, n, seed=3, outer=0, cg=-1):
    return [api.Field(synth.make_field(seed + i, g.standard, 0.7, field_index=i % 4,
                                       geometry=g).samples, g, parity=i % 2,
                      irls_outer=outer, cg_iterations=cg) for i in range(n)]


def _both(ctx, call):
    ctx.set_tuning(16, 0)        # a set tiling selects the streaming solver
    stream = call()
    it = ctx.last_diag.cg_iterations_run
    ctx.set_tuning(0, 0)
    resident = call()
    assert ctx.last_diag.cg_iterations_run == it
    for a, b in zip(stream, resident):
        assert np.array_equal(a.luma, b.luma) and np.array_equal(a.chroma, b.chroma)
    return resident


@pytest.mark.parametrize("std,w,lines,n,sub", [
    (0, 8, 16, 1, 0.0),        # a sliver
    (0, 64, 16, 1, 0.0),       # one strip, one row per warp
    (1, 65, 17, 3, 0.0),       # a column and a row past it
    (0, 333, 121, 2, 0.0),     # odd width
    (1, 700, 33, 5, 0.0),
    (0, 0, 0, 7, 0.0),         # whole fields, more than the gangs
    (1, 0, 0, 4, 0.0),         # 97-row tiles
    (0, 0, 110, 12, 0.0),      # seven rows a warp, the last one short
    (1, 129, 40, 1, 4.4340e6),  # a declared subcarrier: general phasors
])
def test_planes_equal_streaming(std, w, lines, n, sub):
    g = _geom(std, w, lines, sub)
    cfg = api.default_config(fast=0, cg_tol=1e-6, temporal_strength=-1.0, lambda_c=1.2,
                             structure_coupling=0.4)
    with api.Context(0) as ctx:
        _both(ctx, lambda: ctx.decode_fields(_fields(g, n, outer=3, cg=24), cfg))


def test_mixed_batch_equals_streaming():
    fs = synth.mixed_batch(91, 5, 4, outer_range=(1, 4), cg_per_outer=9)
    fields = [api.Field(f.samples, _cabi.default_geometry(f.standard), parity=f.parity,
                        irls_outer=f.irls_outer, cg_iterations=f.cg_iterations) for f in fs]
    g = _geom(0, 97, 50)
    fields += _fields(g, 3, outer=2, cg=10)
    with api.Context(0) as ctx:
        _both(ctx, lambda: ctx.decode_fields(fields, api.default_config(
            fast=0, cg_tol=1e-6, temporal_strength=-1.0)))


@pytest.mark.parametrize("std,w,lines,fast", [(0, 64, 16, 1), (1, 333, 121, 0), (0, 0, 0, 1),
                                              (1, 0, 0, 1)])
def test_neighbour_terms_equal_streaming(std, w, lines, fast):
    g = _geom(std, w, lines)
    cfg = api.default_config(fast=fast, cg_tol=1e-6, temporal_strength=0.5, passes=1,
                             irls_outer=2, cg_iterations=12, chroma_aniso=0.7)
    with api.Context(0) as ctx:
        _both(ctx, lambda: ctx.decode_field_window(_fields(g, 4), cfg))


def test_early_exits_and_oracle():
    """Automatic tolerances (0.02 slow) end passes early; within the bound the
    other tests hold the decode to."""
    from oracle import hvd_oracle as O
    g = _geom(1, 150, 40)
    cfg = api.default_config(fast=0, temporal_strength=-1.0, irls_outer=3, cg_iterations=120)
    with api.Context(0) as ctx:
        f = _fields(g, 1, seed=11)[0]
        out = _both(ctx, lambda: ctx.decode_fields([f], cfg))[0]
        assert ctx.last_diag.cg_iterations_run < 120
    (y, chi, _), = O.decode_fields_2d([synth.to_ire(f.samples)], [0], g, cfg)
    assert np.abs(out.luma - y).max() < 1e-4 and np.abs(out.chroma - chi).max() < 1e-4
