"""The order statistics that a cluster of CTAs selects -- noise sigma, automatic
chroma anisotropy, the integer search's median -- on planes smaller than the
cluster, of odd sizes, and past its registers (the one-CTA kernels), against
the FP64 oracle."""
import numpy as np
import pytest

from hvdg import _cabi, api, synth
from oracle import hvd_oracle as O

pytestmark = pytest.mark.gpu


def _geom(std, w, lines, **kw):
    g = _cabi.default_geometry(std)
    return _cabi.geometry_copy(g, **{**dict(
        active_video_end=g.active_video_start + w,
        last_active_field_line=g.first_active_field_line + lines), **kw})


@pytest.mark.parametrize("std,w,lines", [(0, 48, 16), (1, 131, 40), (0, 700, 33), (0, 758, 240),
                                         (0, 1000, 420)])
def test_noise_sigma_vs_oracle(ctx, std, w, lines):
    """sigma is a quantile of float second differences of samples of at most
    150 IRE over 0.78: a few ulps of 150, 1e-4."""
    kw = {}
    if lines > 242:
        kw = dict(field_width=1160, field_height=450, active_video_start=140,
                  active_video_end=140 + w, first_active_field_line=20,
                  last_active_field_line=20 + lines)
    g = _geom(std, w, lines, **kw)
    cfg = api.default_config(temporal_strength=0.5, passes=1, irls_outer=1, cg_iterations=2, fast=1,
                             coherence_gate=0.0, trajectory_fit=0, nr_anchor=0.0)
    fs = [synth.make_field(91 + i, std, 1.0, field_index=i, parity=i % 2, geometry=g)
          for i in range(3)]
    ctx.decode_field_window([api.Field(f.samples, g, parity=i % 2) for i, f in enumerate(fs)], cfg)
    want = O.mean_median([O.estimate_noise_ire(
        O.prepare_field(synth.to_ire(f.samples), g, cfg, i % 2).s) for i, f in enumerate(fs)])
    print(w, lines, ctx.last_diag.sigma_ire, want)
    assert abs(ctx.last_diag.sigma_ire - want) <= 1e-4


@pytest.mark.parametrize("std,w,lines", [(0, 40, 16), (1, 61, 24), (1, 333, 121)])
def test_anisotropy_vs_oracle(ctx, std, w, lines):
    """The decode with the automatic split against the decode with the oracle's
    split given: 0.05, the bound of the full-field decode."""
    g = _geom(std, w, lines)
    f = synth.make_field(17, std, 0.5, geometry=g)
    cfg = api.default_config(fast=0, cg_tol=1e-6, irls_outer=2, cg_iterations=30,
                             temporal_strength=-1.0)
    obs = O.prepare_field(synth.to_ire(f.samples), g, cfg, 0)
    _, chi0 = O.holographic_init(obs.s, obs.carrier, g)
    an = O.resolve_chroma_aniso(chi0, cfg, std == _cabi.STD_PAL)
    a = ctx.decode_fields([api.Field(f.samples, g, parity=0)], cfg)[0]
    b = ctx.decode_fields([api.Field(f.samples, g, parity=0)],
                          _cabi.config_copy(cfg, chroma_aniso=an))[0]
    assert np.abs(a.luma - b.luma).max() < 0.05 and np.abs(a.chroma - b.chroma).max() < 0.05


@pytest.mark.parametrize("h,w", [(40, 56), (24, 24), (8, 16), (200, 640)])
def test_integer_search_confidence_vs_oracle(ctx, h, w):
    """Blocks of 8: a few tiles, an even and an odd count, 2000 of them."""
    rng = np.random.default_rng(h + w)
    a = (50 + 20 * rng.standard_normal((h, w))).astype(np.float32)
    b = np.roll(a, (1, -2), (0, 1)) + rng.standard_normal((h, w)).astype(np.float32)
    dy, dx, cf = ctx.estimate_motion(a, b, 8, 3, 1)
    oy, ox, oc = O.estimate_motion_sad(a, b, block=8, search=3)
    assert np.abs(dy - oy).max() <= 1e-6 and np.abs(dx - ox).max() <= 1e-6
    assert np.abs(cf - oc).max() <= 1e-6
