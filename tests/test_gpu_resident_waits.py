"""The resident solver's wait bound holds for one exchange, not for a field: a
batch of more fields than gangs, whose gangs have CTAs without a tile (five NTSC
fields: 49 CTAs a gang, 48 tiles), decodes with a bound that an exchange (a few
us) stays far below and a whole solve (about 5 us a sweep, over 1000 sweeps)
exceeds several times."""
import numpy as np
import pytest

from hvdg import _cabi, api, synth

pytestmark = pytest.mark.gpu


def test_wait_bound_is_per_exchange():
    g = _cabi.default_geometry(_cabi.STD_NTSC)
    fields = [api.Field(synth.make_field(80 + i, g.standard, 0.7, field_index=i).samples, g,
                        parity=i % 2) for i in range(5)]
    cfg = api.default_config(fast=0, cg_tol=1e-9, temporal_strength=-1.0, irls_outer=80,
                             cg_iterations=80 * 80)
    with api.Context(0) as ctx:
        want = ctx.decode_fields(fields, cfg)
        assert ctx.last_diag.cg_iterations_run > 5 * 1000
        ctx.set_device_wait_limit(2000)
        got = ctx.decode_fields(fields, cfg)
    for a, b in zip(got, want):
        assert np.array_equal(a.luma, b.luma) and np.array_equal(a.chroma, b.chroma)


def test_waits_that_run_out_end_every_gang():
    """With a bound of one poll the gangs give up in their first exchanges, and
    their CTAs without a tile with them; the context decodes again afterwards."""
    g = _cabi.default_geometry(_cabi.STD_NTSC)
    fields = [api.Field(synth.make_field(80 + i, g.standard, 0.7, field_index=i).samples, g,
                        parity=i % 2) for i in range(5)]
    cfg = api.default_config(fast=0, cg_tol=1e-6, temporal_strength=-1.0, irls_outer=2,
                             cg_iterations=20)
    with api.Context(0) as ctx:
        want = ctx.decode_fields(fields, cfg)
        ctx.set_device_wait_limit(1)
        with pytest.raises(api.HvdgError) as err:
            ctx.decode_fields(fields, cfg)
        assert err.value.status == _cabi.ERR_DEVICE_TIMEOUT
        ctx.set_device_wait_limit(0)
        again = ctx.decode_fields(fields, cfg)
    for a, b in zip(again, want):
        assert np.array_equal(a.luma, b.luma) and np.array_equal(a.chroma, b.chroma)
