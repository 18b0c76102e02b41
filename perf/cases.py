"""Performance cases of the Y/C separator: the work its users have it do,
through the public entry points (hvdg.api, hvdg.autograd), over the sizes the
standards, the tests and the benchmark use.

A case is a dict of plain values. `listed()` names the fixed ones, `draw(rng)`
gives another of the same ranges, `prepare(case, seed)` builds what a program
holds before the call, `run(state)` makes one call, `work(case)` counts what
the call cannot do without and `exact(case, seed)` computes a 2-D field decode
in 64 bits with plain torch.

The pictures are synthetic composites: luma blobs and step edges, band-limited
chroma patches on the burst-locked subcarrier, sync, burst and noise, rendered
from the seed on the GPU; moving sequences add translating rectangles.
"""
from __future__ import annotations

import ctypes
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "hvd-cvbs-decoding_b200"))

from hvdg import _cabi, api, autograd  # noqa: E402

DEV = "cuda"
BLANK16, WHITE16 = 16384.0, 51200.0      # 16-bit codes of 0 and 100 IRE
BLANK10, WHITE10 = 240.0, 800.0          # 10-bit frame buffers


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------

def listed():
    return [
        # a short, odd window of a field, as a box of the selective decode or a
        # cropped capture gives: the smallest call, launches and latency
        dict(name="field_crop", kind="fields", n_ntsc=1, n_pal=0, width=333, lines=121,
             dtype="f32", outer_lo=4, outer_hi=4, cg=0, pinned=False),
        # one whole field at a research budget (5 x 30): one call, one field
        dict(name="field_ntsc", kind="fields", n_ntsc=1, n_pal=0, width=0, lines=0,
             dtype="u16", outer_lo=5, outer_hi=5, cg=30, pinned=False),
        # a player's lookahead of PAL fields at the default budget, int16
        # codes from the capture, into page-locked planes
        dict(name="fields8_pal", kind="fields", n_ntsc=0, n_pal=8, width=0, lines=0,
             dtype="s16", outer_lo=4, outer_hi=4, cg=0, pinned=True),
        # the batched decode of mixed fields with uneven budgets, samples and
        # planes resident on the device (the benchmark's headline workload)
        dict(name="batch64_mixed", kind="device", n_ntsc=40, n_pal=24, width=0, lines=0,
             dtype="u16", outer_lo=4, outer_hi=12, cg=50),
        # a moving NTSC window, 3-D terms with integer-SAD motion, long budget
        # in the slow field-by-field sweep
        dict(name="window16_ntsc_sad", kind="window", standard="ntsc", n=16, sad=True, fast=False,
             passes=1, outer=10, cg=50),
        # a moving PAL window at the engine's defaults: float motion, two
        # passes, the second anchored, coherence gate, trajectory fit
        dict(name="window8_pal", kind="window", standard="pal", n=8, sad=False, fast=True,
             passes=2, outer=4, cg=0),
        # the plugin's own call: six NTSC frames in, four core frames out
        dict(name="sequence6_ntsc", kind="sequence", standard="ntsc", n=6, core=4),
        # the plugin's fallback: composite frames woven and decoded in 2-D,
        # page-locked frames and planes
        dict(name="weave8_ntsc", kind="weave", standard="ntsc", n=8),
        # Y/C-native sources (S-Video captures): chroma demodulated, no solve
        dict(name="yc8_pal", kind="yc", standard="pal", n=8),
        # training: decode and its adjoint, gradients of samples and scalars
        dict(name="adjoint8_ntsc", kind="adjoint", standard="ntsc", n=8, outer=10, cg=50),
        # motion between two luma fields, the search the reference ships
        dict(name="motion_pal", kind="motion", standard="pal", sad=False, tile=32, search=16),
        # the same with the exhaustive integer search
        dict(name="motion_ntsc_sad", kind="motion", standard="ntsc", sad=True, tile=16,
             search=16),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["fields", "fields", "device", "device", "window", "sequence", "weave",
                       "yc", "adjoint", "motion"])
    std = rng.choice(["ntsc", "pal"])
    if kind == "fields" and rng.random() < 0.5:   # one plane of any size
        return dict(kind=kind, n_ntsc=1, n_pal=0, width=_log_int(rng, 48, 760),
                    lines=_log_int(rng, 16, 242), dtype=rng.choice(["f32", "u16", "s16"]),
                    outer_lo=4, outer_hi=4, cg=rng.choice([0, 2, 10, 30]), pinned=False)
    if kind in ("fields", "device"):
        n = _log_int(rng, 1, 12 if kind == "fields" else 48)
        n_pal = rng.randint(0, n)
        lo = rng.randint(2, 6)
        d = dict(kind=kind, n_ntsc=n - n_pal, n_pal=n_pal, width=0, lines=0,
                 dtype=rng.choice(["u16", "u16", "s16", "f32"]), outer_lo=lo,
                 outer_hi=lo + rng.randint(0, 6), cg=rng.choice([0, 5, 20, 50]))
        if kind == "fields":
            d["pinned"] = rng.random() < 0.5
        return d
    if kind == "window":
        fast = rng.random() < 0.6
        n = rng.randint(3, 10)
        return dict(kind=kind, standard=std, n=n, sad=rng.random() < 0.4, fast=fast,
                    passes=rng.randint(1, 2) if fast else 1, outer=rng.randint(3, 8),
                    cg=0 if fast else rng.randint(5, 40))
    if kind == "sequence":
        n = rng.randint(3, 7)
        return dict(kind=kind, standard=std, n=n, core=rng.randint(1, n - 2))
    if kind in ("weave", "yc"):
        return dict(kind=kind, standard=std, n=_log_int(rng, 1, 12))
    if kind == "adjoint":
        return dict(kind=kind, standard=std, n=rng.randint(1, 3), outer=rng.randint(2, 6),
                    cg=rng.randint(10, 50))
    tile = rng.choice([16, 24, 32])
    return dict(kind=kind, standard=std, sad=rng.random() < 0.5, tile=tile,
                search=rng.randint(6, 16))


# --------------------------------------------------------------------------
# Synthetic composites on the device
# --------------------------------------------------------------------------

def _std(name: str) -> int:
    return _cabi.STD_PAL if name == "pal" else _cabi.STD_NTSC


def _geometry(standard: int, width: int = 0, lines: int = 0):
    g = api.default_geometry(standard)
    if width:   # an odd window inside the standard's active picture
        g.active_video_end = g.active_video_start + width
    if lines:
        g.last_active_field_line = g.first_active_field_line + lines
    return g


def _last_line(g) -> int:
    return g.last_active_field_line or g.field_height


class _Scene:
    """Picture content on the frame grid, drawn from a seed."""

    def __init__(self, seed: int, g, n_rects: int):
        r = random.Random(seed)
        rows, w = 2 * (_last_line(g) - g.first_active_field_line), \
            g.active_video_end - g.active_video_start
        self.rows, self.w = rows, w
        u = r.uniform
        self.blobs = [(u(0, rows), u(0, w), u(6, 60), u(8, 120), u(-45, 45)) for _ in range(20)]
        self.edges = [(u(0, math.pi), u(-0.4, 0.4), u(-30, 30)) for _ in range(5)]
        self.patches = []
        for _ in range(14):
            r0, c0 = u(-0.1, 0.9) * rows, u(-0.1, 0.9) * w
            self.patches.append((r0, r0 + u(0.15, 0.6) * rows, c0, c0 + u(0.1, 0.5) * w,
                                 u(-40, 40), u(-40, 40)))
        self.rects = []
        for _ in range(n_rects):
            hh, ww = u(0.12, 0.3) * rows, u(0.08, 0.22) * w
            self.rects.append((u(0.1, 0.9) * rows - hh / 2, u(0.1, 0.9) * w - ww / 2, hh, ww,
                               r.randint(-24, 24) / 2.0, r.randint(-12, 12) / 2.0,
                               u(10, 90), u(-40, 40), u(-40, 40)))
        self.theta = u(-math.pi, math.pi)

    def render(self, y, t: float):
        """Luma and the two chroma components at frame rows y (n, 1)."""
        x = torch.arange(self.w, device=DEV, dtype=torch.float64)[None, :]
        luma = torch.full((y.shape[0], self.w), 50.0, device=DEV, dtype=torch.float64)
        for cy, cx, sy, sx, amp in self.blobs:
            luma += (amp * torch.exp(-0.5 * ((y - cy) / sy) ** 2)) * \
                torch.exp(-0.5 * ((x - cx) / sx) ** 2)
        for ang, off, step in self.edges:
            d = math.cos(ang) * (x / self.w - 0.5) + math.sin(ang) * (y / self.rows - 0.5) - off
            luma += step * (d > 0)
        a, b = torch.zeros_like(luma), torch.zeros_like(luma)
        for r0, r1, c0, c1, va, vb in self.patches:
            m = ((y >= r0) & (y < r1)) & ((x >= c0) & (x < c1))
            a, b = torch.where(m, va, a), torch.where(m, vb, b)
        for r0, c0, hh, ww, vx, vy, yv, va, vb in self.rects:
            top, left = r0 + vy * t, c0 + vx * t
            cx = (torch.minimum(x + 1, torch.full_like(x, left + ww)) -
                  torch.clamp(x, min=left)).clamp(0, 1)
            cy = (torch.minimum(y + 1, torch.full_like(y, top + hh)) -
                  torch.clamp(y, min=top)).clamp(0, 1)
            c = cy * cx
            luma = luma * (1 - c) + yv * c
            a, b = a * (1 - c) + va * c, b * (1 - c) + vb * c
        return luma.clamp(0.0, 100.0), a, b


def _lowpass(a, fs: float, hz: float):
    """Gaussian low-pass along the rows, mirrored at the ends."""
    p = torch.cat([a.flip(1), a, a.flip(1)], 1)
    f = torch.fft.rfftfreq(p.shape[1], 1.0 / fs, device=a.device, dtype=torch.float64)
    n = a.shape[1]
    return torch.fft.irfft(torch.fft.rfft(p) * torch.exp(-0.5 * (f / hz) ** 2),
                           n=p.shape[1])[:, n:2 * n]


def _field(scene: _Scene, g, index: int, parity: int, sigma: float, gen):
    """One field in IRE (field_height, field_width): luma part, chroma part
    and noise, float64 on the device."""
    pal = g.standard == _cabi.STD_PAL
    fh, fw, fal = g.field_height, g.field_width, g.first_active_field_line
    n = _last_line(g) - fal
    a0, a1 = g.active_video_start, g.active_video_end
    y = 2.0 * torch.arange(n, device=DEV, dtype=torch.float64)[:, None] + parity
    luma, ca, cb = scene.render(y, index / 2.0)
    ca = _lowpass(ca, g.sample_rate, 1.3e6)
    cb = _lowpass(cb, g.sample_rate, 1.3e6 if pal else 0.5e6)
    if pal:
        u, v = ca, cb
    else:
        s33, c33 = math.sin(math.radians(33.0)), math.cos(math.radians(33.0))
        u, v = -ca * s33 + cb * c33, ca * c33 + cb * s33
    line = torch.arange(fh, device=DEV, dtype=torch.float64)[:, None]
    xs = torch.arange(fw, device=DEV, dtype=torch.float64)[None, :]
    adv = 2 * math.pi * 0.7516 if pal else math.pi
    phi = scene.theta + (0.75 if pal else 1.5) * math.pi * index + adv * line + 0.5 * math.pi * xs
    # Re[(V - iU) c], c = exp(i phi), and -conj on the V-switched PAL lines
    sw = torch.ones_like(line)
    if pal:
        sw = torch.where(torch.remainder(line + index, 2) == 0, 1.0, -1.0).to(torch.float64)
    cr, ci = sw * torch.cos(phi), torch.sin(phi)
    lpart, cpart = torch.zeros((2, fh, fw), device=DEV, dtype=torch.float64)
    lpart[fal:fal + n, a0:a1] = luma
    cpart[fal:fal + n, a0:a1] = v * cr[fal:fal + n, a0:a1] + u * ci[fal:fal + n, a0:a1]
    sync = min(int(round(4.7e-6 * g.sample_rate)), max(0, g.colour_burst_start - 8))
    lpart[:, :sync] = -40.0
    blen = 4 * (10 if pal else 9)
    bs = (g.colour_burst_start + g.colour_burst_end) // 2 - blen // 2
    if pal:   # +-135 degrees
        br = bi = 21.43 * math.sin(math.pi / 4)
    else:     # 180 degrees
        br, bi = 0.0, 20.0
    cpart[:, bs:bs + blen] = (br * cr - bi * ci)[:, bs:bs + blen]
    noise = sigma * torch.randn((fh, fw), device=DEV, dtype=torch.float64, generator=gen)
    return lpart, cpart, noise


def _gen(seed: int):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    return gen


def _codes(ire, dtype: str):
    """Samples as a capture delivers them: (tensor, blanking, white)."""
    if dtype == "f32":
        return ire.to(torch.float32), 0.0, 100.0
    if dtype == "s16":
        c = torch.round(BLANK10 + ire * ((WHITE10 - BLANK10) / 100.0))
        return c.clamp(-32768, 32767).to(torch.int16), BLANK10, WHITE10
    c = torch.round(BLANK16 + ire * ((WHITE16 - BLANK16) / 100.0)).clamp(0, 65535)
    return c.to(torch.int32).to(torch.uint16), BLANK16, WHITE16


def _batch(case, seed: int):
    """Independent fields of the mixed batch: (geometry, parity, samples,
    blanking, white, outers) of each, in a seeded order."""
    r = random.Random(seed)
    stds = [_cabi.STD_NTSC] * case["n_ntsc"] + [_cabi.STD_PAL] * case["n_pal"]
    r.shuffle(stds)
    geoms = {s: _geometry(s, case["width"], case["lines"]) for s in set(stds)}
    gen, out = _gen(seed), []
    for i, s in enumerate(stds):
        g = geoms[s]
        sigma, outer = r.uniform(0.2, 2.0), r.randint(case["outer_lo"], case["outer_hi"])
        parts = _field(_Scene(r.randrange(1 << 30), g, 0), g, i % 4, i % 2, sigma, gen)
        smp, blank, white = _codes(parts[0] + parts[1] + parts[2], case["dtype"])
        out.append((g, i % 2, smp, blank, white, outer))
    return out


def _sequence(standard: int, n: int, seed: int, sigma: float = 0.5):
    g = _geometry(standard)
    scene, gen = _Scene(seed, g, 4), _gen(seed)
    return g, [_field(scene, g, j, j % 2, sigma, gen) for j in range(n)]


def _frame(top, bottom, fp, level):
    """A field-sequential int16 frame buffer of two fields in IRE. PAL frames
    carry two extra samples on each of two lines."""
    f1 = fp.field1_lines
    lines = torch.cat([top[:f1], bottom[:fp.frame_height - f1]])
    codes = torch.round(level + lines * ((WHITE10 - BLANK10) / 100.0))
    codes = codes.clamp(-32768, 32767).to(torch.int16)
    if fp.extra_sample_line_count == 0:
        return codes.reshape(-1)
    at = sorted({fp.extra_sample_lines[i] for i in range(fp.extra_sample_line_count)})
    cut, parts = 0, []
    for ln in at:
        parts += [codes[cut:ln + 1].reshape(-1), codes[ln, -2:]]
        cut = ln + 1
    return torch.cat(parts + [codes[cut:].reshape(-1)])


def _pinned(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p


# --------------------------------------------------------------------------
# prepare / run
# --------------------------------------------------------------------------

def _config(case):
    """2-D decodes: the engine's default budget (cg 0), or `cg` iterations in
    every outer pass, whatever the tolerance."""
    if case["cg"] == 0:
        return api.default_config(temporal_strength=-1.0)
    return api.default_config(temporal_strength=-1.0, fast=0, cg_tol=1e-6)


def _budget(case, outer: int):
    """(irls_outer, cg_iterations) of a field; the default one for cg 0."""
    return (0, -1) if case["cg"] == 0 else (outer, outer * case["cg"])


def _motion_luma(case, seed: int):
    g, parts = _sequence(_std(case["standard"]), 3, seed)
    a0, a1, fal, lal = (g.active_video_start, g.active_video_end, g.first_active_field_line,
                        _last_line(g))
    return [(p[0] + p[2])[fal:lal, a0:a1].to(torch.float32).cpu().numpy().copy()
            for p in (parts[0], parts[2])]


def prepare(case, seed: int):
    kind = case["kind"]
    st = dict(kind=kind, ctx=api.Context(0))
    if kind in ("fields", "device"):
        st["cfg"] = _config(case)
        batch = _batch(case, seed)
        st["batch"] = batch
        if kind == "fields":
            st["fields"], st["out"] = [], [] if case["pinned"] else None
            for g, par, smp, blank, white, outer in batch:
                o, cg = _budget(case, outer)
                host = smp.cpu()
                if case["pinned"]:
                    host = _pinned(host)
                    hw = (g.active_lines, g.active_width)
                    y = torch.zeros(hw, dtype=torch.float32, pin_memory=True)
                    c = torch.zeros(hw, dtype=torch.complex64, pin_memory=True)
                    st["out"].append(api.Decoded(y.numpy(), c.numpy()))
                st["fields"].append(api.Field(host.numpy(), g, par, blank, white, o, cg))
            return st
        n = len(batch)
        px = [g.active_lines * g.active_width for g, *_ in batch]
        st["luma"] = torch.empty(sum(px), dtype=torch.float32, device=DEV)
        st["chroma"] = torch.empty((sum(px), 2), dtype=torch.float32, device=DEV)
        ins, outs, at = (_cabi.FieldIn * n)(), (_cabi.FieldOut * n)(), 0
        types = {torch.uint16: _cabi.SAMPLES_U16, torch.int16: _cabi.SAMPLES_S16,
                 torch.float32: _cabi.SAMPLES_F32_IRE}
        for i, (g, par, smp, blank, white, outer) in enumerate(batch):
            ins[i].samples, ins[i].sample_type = smp.data_ptr(), types[smp.dtype]
            ins[i].parity, ins[i].blanking_level, ins[i].white_level = par, blank, white
            ins[i].geometry = ctypes.pointer(g)
            ins[i].irls_outer, ins[i].cg_iterations = _budget(case, outer)
            outs[i].luma = st["luma"][at:].data_ptr()
            outs[i].chroma = st["chroma"][at:].data_ptr()
            at += px[i]
        st["ins"], st["outs"], st["n"] = ins, outs, n
        return st
    if kind == "window":
        std = _std(case["standard"])
        g, parts = _sequence(std, case["n"], seed)
        kw = dict(temporal_strength=0.5, passes=case["passes"], irls_outer=case["outer"])
        if not case["fast"]:
            kw.update(fast=0, cg_tol=1e-6, cg_iterations=case["outer"] * case["cg"],
                      nr_anchor=0.0, coherence_gate=0.0, trajectory_fit=0)
        if case["sad"]:
            kw.update(me_mode=1, me_block=16, me_range=16)
        st["cfg"] = api.default_config(**kw)
        st["fields"] = []
        for j, p in enumerate(parts):
            smp, blank, white = _codes(p[0] + p[1] + p[2], "u16")
            st["fields"].append(api.Field(smp.cpu().numpy(), g, j % 2, blank, white))
        return st
    if kind in ("sequence", "weave", "yc"):
        std = _std(case["standard"])
        fp = api.frame_params(std)
        _, parts = _sequence(std, 2 * case["n"], seed)
        st["fp"], st["cfg"] = fp, api.default_config()
        if kind == "yc":
            fp.chroma_dc = 512.0
            gen = _gen(seed + 1)
            chroma = [p[1] + 0.5 * torch.randn(p[1].shape, device=DEV, dtype=torch.float64,
                                               generator=gen) for p in parts]
            st["c"] = [_pinned(_frame(chroma[i], chroma[i + 1], fp, 512.0)).numpy()
                       for i in range(0, len(parts), 2)]
            full = [p[0] + p[2] for p in parts]
        else:
            full = [p[0] + p[1] + p[2] for p in parts]
        frames = [_frame(full[i], full[i + 1], fp, BLANK10) for i in range(0, len(full), 2)]
        if kind == "sequence":
            st["frames"] = [f.cpu().numpy() for f in frames]
            st["core"] = ((case["n"] - case["core"]) // 2,
                          (case["n"] - case["core"]) // 2 + case["core"])
            return st
        st["frames"] = [_pinned(f).numpy() for f in frames]
        sz = fp.frame_width * fp.frame_height
        st["out"] = [{k: torch.zeros(sz, dtype=dt, pin_memory=True).numpy()
                      for k, dt in (("luma", torch.int16), ("chroma", torch.int16),
                                    ("u", torch.float64), ("v", torch.float64))}
                     for _ in frames]
        return st
    if kind == "adjoint":
        std = _std(case["standard"])
        g = _geometry(std)
        gen = _gen(seed)
        smp, truth = [], []
        fal, lal = g.first_active_field_line, _last_line(g)
        for i in range(case["n"]):
            p = _field(_Scene(seed + i, g, 0), g, i % 4, i % 2, 0.5, gen)
            smp.append((p[0] + p[1] + p[2]).to(torch.float32))
            truth.append(p[0][fal:lal, g.active_video_start:g.active_video_end].float())
        st["geometry"], st["samples"] = g, torch.stack(smp)
        st["truth"] = torch.stack(truth)
        st["cfg"] = api.default_config(temporal_strength=-1.0, fast=0, cg_tol=1e-6,
                                       irls_outer=case["outer"],
                                       cg_iterations=case["outer"] * case["cg"])
        return st
    if kind == "motion":
        st["pair"] = _motion_luma(case, seed)
        st["args"] = (case["tile"], case["search"], 1 if case["sad"] else 0)
        return st
    raise ValueError(kind)


def run(st):
    kind, ctx = st["kind"], st["ctx"]
    if kind == "fields":
        dec = ctx.decode_fields(st["fields"], st["cfg"], out=st["out"])
        return [d.luma for d in dec], [d.chroma for d in dec]
    if kind == "device":
        ctx.decode_fields_device(st["ins"], st["outs"], st["n"], st["cfg"])
        return st["luma"], st["chroma"]
    if kind == "window":
        dec = ctx.decode_field_window(st["fields"], st["cfg"])
        return [d.luma for d in dec], [d.chroma for d in dec]
    if kind == "sequence":
        return ctx.decode_frame_sequence_window(st["frames"], *st["core"], st["fp"], st["cfg"])
    if kind == "weave":
        return ctx.decode_frame_buffers(st["frames"], st["fp"], st["cfg"], out=st["out"])
    if kind == "yc":
        return ctx.decode_yc_frame_buffers(st["frames"], st["c"], st["fp"], st["cfg"],
                                           out=st["out"])
    if kind == "adjoint":
        # mean-squared error of the decoded luma, plus the chroma energy
        smp = st["samples"].clone().requires_grad_()
        par = [torch.tensor(v, requires_grad=True) for v in (1.0, 0.5, 1.0, 0.25)]
        y, chi = autograd.decode(ctx, smp, st["geometry"], *par, cfg=st["cfg"])
        loss = ((y - st["truth"]) ** 2).mean() + 0.1 * (chi ** 2).mean()
        loss.backward()
        return y, chi, smp.grad, [p.grad for p in par]
    return ctx.estimate_motion(*st["pair"], *st["args"])


# --------------------------------------------------------------------------
# work
# --------------------------------------------------------------------------

# additions and multiplications of one pixel: a CG iteration (direction,
# residual and chi updates 12, carrier 8, luma part 4, differences 6, fluxes 6,
# divergence 18, curvature 14, four inner products 16), an outer pass (weights
# and gradient)
_FLOPS_CG, _FLOPS_OUTER = 84.0, 120.0


def _solve_flops(px: float, outer: float, cg: float) -> float:
    return px * outer * (_FLOPS_OUTER + cg * _FLOPS_CG)


def work(case):
    """Inputs read once, outputs written once; the floating-point work of the
    solve, and of the cyclic convolutions as an FFT of the same size."""
    kind = case["kind"]

    def field(std, width=0, lines=0):
        g = _geometry(std, width, lines)
        return g.field_width * g.field_height, g.active_lines * g.active_width

    init = lambda px: px * 10.0 * math.log2(max(px, 2)) * 3.0  # noqa: E731
    size = {"u16": 2, "s16": 2, "f32": 4}
    if kind in ("fields", "device"):
        by = fl = 0.0
        outer = 0.5 * (case["outer_lo"] + case["outer_hi"]) if case["cg"] else 4
        for std, n in ((_cabi.STD_NTSC, case["n_ntsc"]), (_cabi.STD_PAL, case["n_pal"])):
            raw, px = field(std, case["width"], case["lines"])
            by += n * (raw * size[case["dtype"]] + 12.0 * px)
            fl += n * (init(px) + _solve_flops(px, outer, case["cg"] or 1))
        return dict(bytes=by, flops=fl)
    raw, px = field(_std(case["standard"]))
    if kind == "window":
        n = case["n"]
        fl = n * (init(px) + case["passes"] * _solve_flops(px, case["outer"], case["cg"] or 1))
        return dict(bytes=n * (2.0 * raw + 12.0 * px), flops=fl)
    if kind == "sequence":
        fl = 2 * case["n"] * (init(px) + 2 * _solve_flops(px, 4, 1))
        return dict(bytes=case["n"] * 4.0 * raw + case["core"] * 40.0 * raw, flops=fl)
    if kind in ("weave", "yc"):
        n = case["n"]
        fl = n * (init(2 * px) + (_solve_flops(2 * px, 4, 1) if kind == "weave" else 0.0))
        return dict(bytes=n * (4.0 + 40.0 + (4.0 if kind == "yc" else 0.0)) * raw, flops=fl)
    if kind == "adjoint":
        n = case["n"]
        fl = n * (4 * init(px) + _solve_flops(px, case["outer"], 2 * case["cg"]) +
                  _solve_flops(px, case["outer"], case["cg"]))
        return dict(bytes=n * (4.0 * raw + 12.0 * px + 4.0 * px + 4.0 * raw), flops=fl)
    tiles = px / case["tile"] ** 2
    cand = (2 * case["search"] + 1) ** 2 if case["sad"] else (2 * case["search"] / 4 + 1) ** 2 / 16 + 49
    return dict(bytes=8.0 * px + 12.0 * tiles, flops=2.0 * px * cand)


# --------------------------------------------------------------------------
# exact: the 2-D field decode in 64 bits
# --------------------------------------------------------------------------

def _median(v):
    return float(np.sort(v)[v.size // 2]) if v.size else 0.0


def _lockin(f, g):
    """Per-line carrier phase from the bursts and the V-switch senses."""
    pal = g.standard == _cabi.STD_PAL
    h, n = f.shape[0], g.colour_burst_end - g.colour_burst_start
    xs = np.arange(g.colour_burst_start, g.colour_burst_end)
    seg = f[:, g.colour_burst_start:g.colour_burst_end]
    seg = seg - seg.mean(1, keepdims=True)
    z = (seg * np.exp(-0.5j * math.pi * xs)[None, :]).sum(1) / n
    amp, ang, ys = np.abs(z), np.angle(z), np.arange(h)
    adv = 2 * math.pi * 0.7516 if pal else math.pi
    good = amp > 0.2 * amp.max()
    fg = int(np.argmax(good))
    wrap = lambda a: np.arctan2(np.sin(a), np.cos(a))  # noqa: E731
    sw = np.ones(h)
    if pal:
        best = None
        for s in (1.0, -1.0):
            m = ang[fg] - 0.5 * math.pi + s * 0.25 * math.pi + adv * (ys - fg)
            sy = np.where((ys - fg) % 2 == 0, s, -s)
            dev = wrap(ang - (m + 0.5 * math.pi - sy * 0.25 * math.pi))
            score = float((np.cos(dev) * amp)[good].sum())
            if best is None or score > best[0]:
                best = (score, m, sy)
        model, sw = best[1], best[2]
        d = wrap(ang - 0.5 * math.pi + sw * 0.25 * math.pi - model)
    else:
        model = ang[fg] - 0.5 * math.pi + adv * (ys - fg)
        d = wrap(ang - 0.5 * math.pi - model)

    def smooth(a, lam=25.0):   # (diag(a) + lam L) x = a d, L the 1-D Laplacian
        m = np.diag(a + 2 * lam) - lam * (np.eye(h, k=1) + np.eye(h, k=-1))
        m[0, 0] -= lam
        m[-1, -1] -= lam
        return np.linalg.solve(m, a * d)

    a = np.where(good, np.clip(amp / (_median(amp[good]) + 1e-9), 0.0, 2.0), 0.0)
    x = smooth(a)
    return model + smooth(a * 0.15 / np.maximum(np.abs(d - x), 0.15)), sw


def _dx(a):
    return torch.nn.functional.pad(a[:, 1:] - a[:, :-1], (0, 1))


def _dy(a):
    return torch.nn.functional.pad(a[1:] - a[:-1], (0, 0, 0, 1))


def _dxt(a):   # adjoint of _dx; the last column of `a` is zero
    return torch.nn.functional.pad(a[:, :-1], (1, 0)) - a


def _dyt(a):
    return torch.nn.functional.pad(a[:-1], (0, 0, 1, 0)) - a


def _box(a, r):
    p = torch.nn.functional.pad(a, (r, r, r, r))
    k = 2 * r + 1
    return torch.nn.functional.avg_pool2d(p[None, None], k, 1)[0, 0]


def _init64(s, c, g):
    """Two Gaussian crops of the demodulated spectrum, blended by how little
    edge energy each leaves in the luma."""
    h, w = s.shape
    pad = min(16, h - 1)
    rows = torch.arange(-pad, h + pad, device=s.device)
    rows = torch.remainder(rows, 2 * h - 2)
    rows = torch.where(rows < h, rows, 2 * h - 2 - rows)
    spec = torch.fft.fft2((s * c.conj())[rows])
    fx = torch.fft.fftfreq(w, 1.0 / g.sample_rate, device=s.device, dtype=torch.float64)
    fy = torch.fft.fftfreq(h + 2 * pad, 1.0, device=s.device, dtype=torch.float64)
    num, den = 0.0, 0.0
    for mhz, cph in ((0.8, 120.0), (1.8, 30.0)):
        gx = torch.exp(-0.5 * (fx / (mhz * 1e6)) ** 2)
        gy = torch.exp(-0.5 * (fy / (cph / (2.0 * h))) ** 2)
        chi = 2.0 * torch.fft.ifft2(spec * gy[:, None] * gx[None, :])[pad:pad + h]
        y = s - (chi * c).real
        wt = 1.0 / (_box(_dx(y).abs() + _dy(y).abs(), 3) + 0.5)
        num, den = num + chi * wt, den + wt
    return num / den


def _aniso64(chi, pal: bool) -> float:
    grp = 4 if pal else 2
    n = chi.shape[0] // grp
    p = chi[:n * grp].reshape(n, grp, -1).mean(1)
    ts = torch.arange(1, n, 2, device=chi.device)
    xs = torch.arange(1, chi.shape[1], 3, device=chi.device)

    def p98(v):
        v = torch.sort(v.reshape(-1)).values
        return float(v[v.numel() - 1 - v.numel() // 50]) if v.numel() else 0.0

    px = p98((p[ts][:, xs] - p[ts][:, xs - 1]).abs())
    py = p98((p[ts][:, xs] - p[ts - 1][:, xs]).abs())
    r = py / max(px, 1e-6)
    return min(max(0.7 + 0.9 * (r - 1.3), 0.55), 1.0) if pal else \
        min(max(0.5 + 1.1 * (r - 1.3), 0.5), 1.0)


def _solve64(s, c, chi, pal: bool, outers: int, inner: int, tol: float):
    eps, epsc, k = 0.5, 1.0, 0.25
    mu_h, mu_v = _aniso64(chi, pal), 1.0
    n = s.numel()
    for _ in range(outers):
        yc = s - (chi * c).real
        gx, gy = _dx(yc) ** 2, _dy(yc) ** 2
        wx, wy = eps / torch.sqrt(gx + eps * eps), eps / torch.sqrt(gy + eps * eps)
        wcx = epsc / torch.sqrt(_dx(chi).abs() ** 2 + k * gx + epsc * epsc)
        wcy = epsc / torch.sqrt(_dy(chi).abs() ** 2 + k * gy + epsc * epsc)

        def grad(y, u):
            im = 2.0 * (_dxt(wx * _dx(y)) + _dyt(wy * _dy(y)))
            return -im * c.conj() + 2.0 * (mu_h * _dxt(wcx * _dx(u)) + mu_v * _dyt(wcy * _dy(u)))

        g = grad(yc, chi)
        d = -g
        gg = gg0 = float((g.abs() ** 2).sum())
        for _ in range(inner):
            q = grad(-(d * c).real, d)
            curv = 0.5 * float((q.conj() * d).real.sum())
            if curv <= 1e-12:
                break
            a = -0.5 * float((g.conj() * d).real.sum()) / curv
            chi, g = chi + a * d, g + a * q
            new = float((g.abs() ** 2).sum())
            d, gg = -g + (new / max(gg, 1e-30)) * d, new
            if gg < tol * tol * gg0 or gg < 1e-10 * n:
                break
    return s - (chi * c).real, chi


def exact(case, seed: int):
    if case["kind"] not in ("fields", "device"):
        return None   # motion, weaving and requantisation: no 64-bit restatement here
    luma, chroma = [], []
    for g, _, smp, blank, white, outer in _batch(case, seed):
        ire = (smp.to(torch.int32) if smp.dtype == torch.uint16 else smp).to(torch.float64)
        ire = (ire - blank) / ((white - blank) / 100.0)
        theta, sw = _lockin(ire.cpu().numpy(), g)
        fal, lal = g.first_active_field_line, _last_line(g)
        a0, a1 = g.active_video_start, g.active_video_end
        c = np.exp(1j * (theta[fal:lal, None] + 0.5 * math.pi * np.arange(a0, a1)[None, :]))
        if g.standard == _cabi.STD_PAL:
            c = np.where(sw[fal:lal, None] < 0, -np.conj(c), c)
        c = torch.from_numpy(c).to(DEV)
        s = ire[fal:lal, a0:a1].contiguous()
        chi = _init64(s, c, g)
        pal = g.standard == _cabi.STD_PAL
        if case["cg"] == 0:   # 4 outers, 2 * 2 / 3 iterations over them: one each
            y, chi = _solve64(s, c, chi, pal, 4, 1, 0.10)
        else:
            y, chi = _solve64(s, c, chi, pal, outer, case["cg"], 1e-6)
        luma.append(y)
        chroma.append(chi)
    if case["kind"] == "fields":
        return luma, chroma
    return (torch.cat([y.reshape(-1) for y in luma]),
            torch.cat([torch.view_as_real(x).reshape(-1, 2) for x in chroma]))
