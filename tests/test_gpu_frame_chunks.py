"""Woven frames that go through in chunks, with copies beside the kernels,
against the same frames one call at a time: equal planes, whole chunks and a
short last one, more chunks than events, voted field orders, the streaming
solver (one chunk), and page-locked buffers."""
import numpy as np
import pytest
import torch

from hvdg import _cabi, api, synth

pytestmark = pytest.mark.gpu

KEYS = ("luma", "chroma", "u", "v")


def _equal(got, want):
    for k in KEYS:
        assert np.array_equal(got[k], want[k]), k


def _pin(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


@pytest.mark.parametrize("std,n,kw", [
    (_cabi.STD_NTSC, 2, {}), (_cabi.STD_NTSC, 3, {}), (_cabi.STD_NTSC, 9, {}),
    (_cabi.STD_PAL, 5, {}), (_cabi.STD_NTSC, 5, dict(cg_iterations=0)),
    (_cabi.STD_NTSC, 3, dict(acc=0, monochrome=1)),
])
def test_frames_together_equal_frames_alone(ctx, std, n, kw):
    frames, _ = synth.make_frames(31, std, n, noise_sigma=1.0)
    fp = api.frame_params(std)
    cfg = api.default_config(**{**dict(irls_outer=2, cg_iterations=12, fast=1, cg_tol=1e-6), **kw})
    alone = [ctx.decode_frame_buffer(f, fp, cfg) for f in frames]
    for fs in (frames, [_pin(f) for f in frames]):
        got = ctx.decode_frame_buffers(fs, fp, cfg)
        for g, w in zip(got, alone):
            _equal(g, w)
    with api.Context(0) as c2:
        c2.set_tuning(16, 0)
        for g, w in zip(c2.decode_frame_buffers(frames, fp, cfg), alone):
            _equal(g, w)


@pytest.mark.parametrize("std,n", [(_cabi.STD_NTSC, 1), (_cabi.STD_PAL, 3), (_cabi.STD_NTSC, 35)])
def test_yc_frames_together_equal_frames_alone(ctx, std, n):
    ys, cs, _ = synth.make_yc_frames(83, std, min(n, 3), noise_sigma=0.7)
    fp = api.frame_params(std)
    fp.chroma_dc = 512.0
    cfg = api.default_config()
    alone = [ctx.decode_yc_frame_buffer(y, c, fp, cfg) for y, c in zip(ys, cs)]
    pick = [i % len(ys) for i in range(n)]
    got = ctx.decode_yc_frame_buffers([ys[i] for i in pick], [cs[i] for i in pick], fp, cfg)
    for i, g in zip(pick, got):
        _equal(g, alone[i])
