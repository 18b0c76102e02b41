"""The init's edge-energy blend at the edges of its tiles (56 columns x 7 or 21
rows): against the FP64 oracle within the bound of the full-field init test,
and, plane for plane, a batch that takes the tall tiles against the same fields
alone on the low ones."""
import numpy as np
import pytest

from hvdg import _cabi, api, synth
from oracle import hvd_oracle as O

pytestmark = pytest.mark.gpu


def _geom(std, w, lines):
    g = _cabi.default_geometry(std)
    return _cabi.geometry_copy(g, active_video_end=g.active_video_start + w,
                               last_active_field_line=g.first_active_field_line + lines)


@pytest.mark.parametrize("sym", [0, 1])
@pytest.mark.parametrize("std,w,lines", [(0, 56, 21), (1, 57, 22), (0, 55, 20), (0, 113, 8),
                                         (1, 64, 7), (0, 9, 43), (0, 169, 64)])
def test_blend_vs_oracle(ctx, std, w, lines, sym):
    g = _geom(std, w, lines)
    f = synth.make_field(41 + w, std, 0.5, geometry=g)
    cfg = api.default_config(fast=0, temporal_strength=-1.0, symmetry_variant=sym)
    obs = O.prepare_field(synth.to_ire(f.samples), g, cfg, 0)
    fal, lal = g.first_active_field_line, g.last_active_line
    th = obs.theta[fal:lal].astype(np.float32)
    sw = obs.vswitch[fal:lal].astype(np.int8)
    y, chi = ctx.holographic_init(obs.s.astype(np.float32), th, sw, g, cfg)
    yo, co = O.holographic_init(obs.s, O.make_carrier(th, sw, g), g, symmetry_variant=bool(sym))
    print(np.abs(chi - co).max(), np.abs(y - yo).max())
    assert np.abs(chi - co).max() < 5e-3 and np.abs(y - yo).max() < 5e-3


@pytest.mark.parametrize("std,w,lines", [(0, 330, 121), (1, 281, 106)])
def test_tall_tiles_equal_low_ones(ctx, std, w, lines):
    g = _geom(std, w, lines)
    fs = [api.Field(synth.make_field(7 + i % 3, std, 0.5, geometry=g).samples, g, parity=0)
          for i in range(48)]
    cfg = api.default_config(fast=0, temporal_strength=-1.0, cg_iterations=0)
    alone = [ctx.decode_fields([f], cfg)[0] for f in fs[:3]]
    for i, d in enumerate(ctx.decode_fields(fs, cfg)):
        assert np.array_equal(d.luma, alone[i % 3].luma)
        assert np.array_equal(d.chroma, alone[i % 3].chroma)
