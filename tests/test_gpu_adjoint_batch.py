"""Fields that go through the decode adjoint together against the same fields
one call at a time -- a budget, a geometry or a zero cotangent of its own among
them -- and the transposed row pad on planes of few rows, where a row takes
images from both pads, against the FP64 adjoint oracle."""
import numpy as np
import pytest

from hvdg import _cabi, api, synth
from oracle import hvd_adjoint as A
from oracle import hvd_oracle as O

pytestmark = pytest.mark.gpu

CPI = (51200.0 - 16384.0) / 100.0


def _geom(std, w, lines):
    g = _cabi.default_geometry(std)
    return _cabi.geometry_copy(g, active_video_end=g.active_video_start + w,
                               last_active_field_line=g.first_active_field_line + lines)


def _field(seed, g, parity, **kw):
    return api.Field(synth.make_field(seed, g.standard, 0.6, field_index=parity,
                                      geometry=g).samples, g, parity=parity, **kw)


def _cot(rng, g):
    shape = (g.active_lines, g.active_width)
    return (rng.standard_normal(shape).astype(np.float32),
            (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64))


def test_fields_together_equal_fields_alone(ctx):
    """The solves end at 1e-6 of the right-hand side; ten times that bounds
    what another order of the FP64 sums can change."""
    rng = np.random.default_rng(5)
    ga, gb, gc = _geom(0, 130, 40), _geom(1, 97, 33), _geom(0, 130, 41)
    flds = [_field(i, g, i % 2, **kw) for i, (g, kw) in enumerate(
        [(ga, {}), (ga, {}), (ga, {}), (ga, {}), (ga, dict(irls_outer=2)), (ga, {}),
         (gb, {}), (gb, {}), (gc, {}), (ga, {})])]
    cots = [_cot(rng, f.geometry) for f in flds]
    cots[2] = (np.zeros_like(cots[2][0]), np.zeros_like(cots[2][1]))
    cots[9] = (np.zeros_like(cots[9][0]), np.zeros_like(cots[9][1]))
    cfg = api.default_config(irls_outer=3, cg_iterations=30, fast=0, cg_tol=1e-6,
                             temporal_strength=-1.0)
    sb, sc, fw = ctx.decode_fields_adjoint(flds, cfg, [c[0] for c in cots], [c[1] for c in cots],
                                           200, want_forward=True)
    total = dict.fromkeys(sc, 0.0)
    mag = dict.fromkeys(sc, 0.0)
    for i, f in enumerate(flds):
        s1, c1, f1 = ctx.decode_fields_adjoint([f], cfg, [cots[i][0]], [cots[i][1]], 200,
                                               want_forward=True)
        for k in sc:
            total[k] += c1[k]
            mag[k] += abs(c1[k])
        assert np.abs(fw[i].luma - f1[0].luma).max() <= 1e-4
        assert np.abs(fw[i].chroma - f1[0].chroma).max() <= 1e-4
        assert np.linalg.norm(sb[i] - s1[0]) <= 1e-5 * np.linalg.norm(s1[0])
    assert not sb[2].any() and not sb[9].any()
    for k in sc:
        assert abs(sc[k] - total[k]) <= 1e-5 * mag[k]


@pytest.mark.parametrize("lines", [2, 3, 8, 16, 17, 33])
def test_few_rows_vs_fp64_oracle(ctx, lines):
    """The bound of the full-field test (1e-3) against the FP64 adjoint."""
    rng = np.random.default_rng(lines)
    g = _geom(0, 80, lines)
    flds = [_field(70 + i, g, i) for i in range(2)]
    cots = [_cot(rng, g) for _ in flds]
    cfg = api.default_config(irls_outer=2, cg_iterations=200, fast=0, cg_tol=1e-6,
                             temporal_strength=-1.0, chroma_aniso=1.0)
    sb, _, _ = ctx.decode_fields_adjoint(flds, cfg, [c[0] for c in cots], [c[1] for c in cots], 300)
    fal, a0 = g.first_active_field_line, g.active_video_start
    for f, s, (yb, cb) in zip(flds, sb, cots):
        obs = O.prepare_field(synth.to_ire(f.samples), g, cfg)
        _, _, chi0 = A.init_parts(obs.s, obs.carrier, g)
        aniso = O.resolve_chroma_aniso(chi0, cfg, False)
        chis = A.refine_forward_budget(obs.s, obs.carrier, chi0, cfg, aniso)
        want, chi0_bar, _ = A.refine_adjoint(obs.s, obs.carrier, chis, cfg, aniso, yb, cb, 1e-8, 3000)
        want = (want + A.init_adjoint(obs.s, obs.carrier, g, chi0_bar)) / CPI
        got = s[fal:fal + lines, a0:a0 + 80].astype(np.float64)
        rel = np.linalg.norm(got - want) / np.linalg.norm(want)
        print(lines, rel)
        assert rel < 1e-3
