"""The calls whose speed is tracked: what a decoder and an encoder ask of the post-filter library.

listed() names them, draw() gives more of the same ranges, prepare() makes a
call's inputs on the GPU from a seed, run() makes the call through
goav1_b200's public entry points, and work() counts the bytes (and, for the
encoder searches, the arithmetic) that no implementation can do without.

Inputs follow goav1_b200/synth.py's workloads (cosine-gradient texture,
per-8x8 DC offsets, Gaussian noise; quadtree blocks over 64x64 superblocks
with eight segments; switchable restoration units; lag-3 film grain), made
with tensor operations so that a batch of frames takes a fraction of a second.
All outputs are whole numbers (samples, SSE sums, presets, mask bits).
"""

import ctypes as C
import math

import numpy as np
import torch

from goav1_b200 import abi, learned, synth
from goav1_b200.postfilter import PostFilterRunner, cdef_plan_picture

LAYOUTS = {"420": (1, 1), "422": (1, 0), "444": (0, 0)}
LF_CDEF = abi.PF_STAGE_LOOP_FILTER | abi.PF_STAGE_CDEF | abi.PF_STAGE_EXTEND_BORDERS

# The mixed queue: streams of several sizes, depths and layouts served from one batch.
MIXED = ((16, 640, 360, 8, "420"), (16, 1280, 720, 8, "420"), (8, 1920, 1080, 10, "420"), (8, 1280, 720, 8, "444"))


def _chain(name, w, h, bd, ss, frames, full=True, host=False, graphs=False):
    return {"name": name, "kind": "chain", "w": w, "h": h, "bd": bd, "ss": ss, "frames": frames, "full": full,
            "host": host, "graphs": graphs}


def listed():
    return [
        # The smallest call: one CIF frame of a real-time decoder, deblocking and CDEF.
        _chain("cif_frame", 352, 288, 8, "420", 1, full=False),
        # One decoded frame at a time, full chain, frames and side information in HBM.
        _chain("hd_frame", 1920, 1080, 8, "420", 1),
        # The decoder's own call: one frame in page-locked host memory, back when it returns.
        _chain("hd_frame_host", 1920, 1080, 8, "420", 1, host=True),
        # A ragged 10-bit 4:4:4 frame (screen content at an odd window size), captured graphs on.
        _chain("odd_frame_10bit_444", 853, 479, 10, "444", 1, graphs=True),
        # Bulk work: 60 frames of 1080p video in one call.
        _chain("hd_batch", 1920, 1080, 8, "420", 60),
        # The largest: 16 frames of 4K 10-bit video in one call.
        _chain("uhd_batch_10bit", 3840, 2160, 10, "420", 16),
        # A server's queue: 48 frames of four kinds in one call, captured graphs on.
        {"name": "mixed_batch", "kind": "mixed", "copies": 8, "graphs": True},
        # The encoder's CDEF strength search over all 64 luma and chroma strengths.
        {"name": "cdef_search", "kind": "search", "w": 1920, "h": 1080, "level": 1},
        # The same decision steered by the trained network.
        {"name": "cdef_search_learned", "kind": "learned", "w": 1920, "h": 1080},
        # The encoder's restoration unit search with the restored frame as its output.
        {"name": "lr_search", "kind": "lr_search", "w": 1920, "h": 1080},
        # Super-resolved video: 8 frames at denominator 9 (an odd coded width).
        {"name": "superres_batch", "kind": "superres", "w": 1920, "h": 1080, "bd": 8, "ss": "420", "denom": 9,
         "frames": 8},
        # Deblocking masks and levels of one frame from its decoded block records.
        {"name": "lf_build", "kind": "lf_build", "w": 1920, "h": 1080, "ss": "420"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, most):
    """A frame size of up to `most` luma samples, 4:3 to 2.4:1, odd sizes among them."""
    h = _log(rng, 144, 2160)
    w = int(h * rng.uniform(4 / 3, 2.4))
    while w * h > most or w > 3840:
        w, h = int(w * 0.8), int(h * 0.8)
    if rng.random() < 0.5:
        w, h = w & ~7, h & ~7
    return w, h


def draw(rng):
    kind = rng.choice(["chain"] * 5 + ["mixed", "search", "learned", "lr_search", "superres", "lf_build"])
    if kind == "chain":
        w, h = _size(rng, 3840 * 2160)
        host = rng.random() < 0.25
        frames = 1 if rng.random() < 0.4 else _log(rng, 2, 60)
        frames = max(1, min(frames, (8_000_000 if host else 60_000_000) // (w * h)))
        c = _chain("", w, h, rng.choice([8, 8, 10, 12]), rng.choice(["420", "420", "422", "444"]), frames,
                   full=rng.random() < 0.75, host=host, graphs=rng.random() < 0.25)
        del c["name"]
        return c
    if kind == "mixed":
        return {"kind": kind, "copies": rng.randint(1, 7), "graphs": rng.random() < 0.5}
    w, h = _size(rng, 2560 * 1440)
    if kind == "search":
        return {"kind": kind, "w": w, "h": h, "level": rng.randint(1, 8)}
    if kind == "superres":
        return {"kind": kind, "w": w, "h": h, "bd": rng.choice([8, 10]), "ss": rng.choice(["420", "444"]),
                "denom": rng.randint(9, 16), "frames": _log(rng, 1, 8)}
    if kind == "lf_build":
        return {"kind": kind, "w": w, "h": h, "ss": rng.choice(["420", "422", "444"])}
    return {"kind": kind, "w": w, "h": h}


# ---------------------------------------------------------------------------
# Inputs


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _dims(w, h, ss, align=64):
    """(cropped, allocated) plane sizes as (w, h) pairs, as goav1 allocates a frame."""
    sx, sy = ss
    aw, ah = -(-w // align) * align, -(-h // align) * align
    return ([(w, h)] + [((w + sx) >> sx, (h + sy) >> sy)] * 2, [(aw, ah)] + [(aw >> sx, ah >> sy)] * 2)


class Frames:
    """n frames of one geometry in one buffer, each frame's planes back to back."""

    def __init__(self, n, w, h, bd, ss):
        self.n, self.w, self.h, self.bd, self.ss = n, w, h, bd, ss
        self.bps = 1 if bd == 8 else 2
        self.crop, self.alloc = _dims(w, h, ss)
        self.plane_bytes = [a[0] * a[1] * self.bps for a in self.alloc]
        self.frame_bytes = sum(self.plane_bytes)
        self.nbytes = n * self.frame_bytes

    def plane(self, buf, i, p):
        at = i * self.frame_bytes + sum(self.plane_bytes[:p])
        t = buf[at:at + self.plane_bytes[p]]
        return (t if self.bps == 1 else t.view(torch.int16)).view(self.alloc[p][1], self.alloc[p][0])

    def pf(self, buf, i, memory):
        f = abi.pf_frame()
        f.width, f.height, f.bit_depth, f.ss_x, f.ss_y, f.memory = self.w, self.h, self.bd, *self.ss, memory
        at = buf.data_ptr() + i * self.frame_bytes
        for p in range(3):
            q = f.plane[p]
            q.data, q.stride = at, self.alloc[p][0] * self.bps
            q.width, q.height = self.crop[p]
            q.alloc_width, q.alloc_height = self.alloc[p]
            at += self.plane_bytes[p]
        return f


def _texture(rng):
    return [dict(p=rng.uniform(8, 64, 4), f=rng.uniform(0, 2 * np.pi, 2), a=rng.uniform(20, 60),
                 b=rng.uniform(10, 40), c=rng.uniform(10, 30)) for _ in range(3)]


def _content(fr, buf, i, g, tex, mv, dc, noise):
    """One frame's samples: three cosine gradients, DC offsets per 8x8 block, noise."""
    scale, top = 1 << (fr.bd - 8), (1 << fr.bd) - 1
    for p in range(3):
        out = fr.plane(buf, i, p)
        h, w = out.shape
        sx, sy = fr.ss if p else (0, 0)
        t = tex[p]
        ys = (torch.arange(h, device="cuda", dtype=torch.float32) + (mv[1] >> sy))[:, None] * (2 * math.pi)
        xs = (torch.arange(w, device="cuda", dtype=torch.float32) + (mv[0] >> sx))[None, :] * (2 * math.pi)
        v = (128 + t["a"] * torch.cos(xs / t["p"][0] + t["f"][0]) + t["b"] * torch.cos(ys / t["p"][1] + t["f"][1])
             + t["c"] * torch.cos(xs / t["p"][2]) * torch.cos(ys / t["p"][3])) * scale
        if dc:
            d = torch.randint(-dc, dc + 1, ((h + 7) // 8, (w + 7) // 8), generator=g, device="cuda")
            v = v + d.repeat_interleave(8, 0).repeat_interleave(8, 1)[:h, :w]
        if noise:
            v = v + noise * torch.randn((h, w), generator=g, device="cuda")
        out.copy_(v.round_().clamp_(0, top))


def _up(t, s):
    return t.repeat_interleave(s, -2).repeat_interleave(s, -1)


def _blocks(g, n, rows, cols):
    """Random quadtrees over 64x64 superblocks down to 4x4: log2 of each 4x4 cell's block size."""
    lg = torch.full((n, rows, cols), 4, dtype=torch.int32, device="cuda")
    for k in (4, 3, 2, 1):
        s = 1 << k
        split = torch.rand((n, rows // s, cols // s), generator=g, device="cuda") < 0.55
        lg = torch.where((lg == k) & _up(split, s), k - 1, lg)
    return lg


def _at_origin(t, size_y, size_x, gy, gx):
    """The value that each cell's block has at its origin cell."""
    flat = (gy - gy % size_y) * t.shape[2] + (gx - gx % size_x)
    return t.reshape(t.shape[0], -1).gather(1, flat.reshape(t.shape[0], -1).long()).view(t.shape)


def _pack(bits):
    """Little-endian words of the last axis."""
    w = (1 << torch.arange(bits.shape[-1], device="cuda", dtype=torch.int32))
    return (bits.to(torch.int32) * w).sum(-1)


def _edge_words(edge, cls, nclass, regions, lanes):
    """Mask words [n, region, pos, class, half] of one edge direction: `edge` and `cls` hold the cells of the
    128x128 regions as [n, sbh, sbw, pos, bit]."""
    n, npos = edge.shape[0], edge.shape[3]
    out = torch.zeros((n, regions, 32, nclass, 2), dtype=torch.int32, device="cuda")
    for k in range(nclass):
        bits = (edge & (cls == k)).reshape(n, regions, npos, 2, lanes)
        out[:, :, :npos, k] = _pack(bits)
    return out.view(n, regions, -1)


class Side:
    """Side information of n frames of one geometry, as device tensors (one row per frame)."""

    def __init__(self, seed, n, w, h, ss, full=True, lr_width=0, lr_unit=128):
        g = _gen(seed)
        rng = np.random.default_rng([seed & 0x7FFFFFFF, 0x51DE])
        sx, sy = ss
        self.full = full
        self.mi_cols, self.mi_rows = ((w + 7) >> 3) << 1, ((h + 7) >> 3) << 1
        self.sbw, self.sbh = (self.mi_cols + 31) // 32, (self.mi_rows + 31) // 32
        R, K = self.sbh * 32, self.sbw * 32
        regions = self.sbh * self.sbw
        lg = _blocks(g, n, R, K)
        size = 1 << lg
        gy = torch.arange(R, device="cuda", dtype=torch.int32)[None, :, None].expand(n, R, K)
        gx = torch.arange(K, device="cuda", dtype=torch.int32)[None, None, :].expand(n, R, K)
        inside = (gy < self.mi_rows) & (gx < self.mi_cols)

        def per_block():
            return _at_origin(torch.rand((n, R, K), generator=g, device="cuda"), size, size, gy, gx)

        tlog = (per_block() * (lg.clamp(max=3) + 1)).to(torch.int32)
        skip = per_block() < 0.3
        seg = (per_block() * 8).to(torch.int64)

        # Deblocking edges: every transform boundary, its class the smaller of the two sides'.
        def region(t, rh, rw, vertical):
            t = t.reshape(n, self.sbh, rh, self.sbw, rw)
            return t.permute(0, 1, 3, 4, 2) if vertical else t.permute(0, 1, 3, 2, 4)

        cls = tlog.clamp(max=2)
        words = []
        for d in (0, 1):
            pos = gx if d == 0 else gy
            prev = torch.roll(cls, 1, 2 - d)
            edge = ((pos & ((1 << tlog) - 1)) == 0) & (pos > 0) & inside
            words.append(_edge_words(region(edge, 32, 32, d == 0), region(torch.minimum(cls, prev), 32, 32, d == 0), 3,
                                     regions, 16))
        cs = size[:, ::1 << sy, ::1 << sx] >> max(sx, sy)
        cs = cs.clamp(1, 8)
        cgy, cgx = gy[:, :R >> sy, :K >> sx], gx[:, :R >> sy, :K >> sx]
        cin = (cgy < (self.mi_rows + sy) >> sy) & (cgx < (self.mi_cols + sx) >> sx)
        ccls = (cs >= 2).to(torch.int32)
        for d in (0, 1):
            pos = cgx if d == 0 else cgy
            prev = torch.roll(ccls, 1, 2 - d)
            edge = ((pos & (cs - 1)) == 0) & (pos > 0) & cin
            words.append(_edge_words(region(edge, 32 >> sy, 32 >> sx, d == 0),
                                     region(torch.minimum(ccls, prev), 32 >> sy, 32 >> sx, d == 0), 2, regions,
                                     16 >> (sy if d == 0 else sx)))
        self.masks = torch.cat(words, 2).to(torch.int16).contiguous()
        assert self.masks.shape[2] == abi.PF_LF_MASK_WORDS

        # Levels: frame levels plus eight segments' deltas.
        self.level = rng.integers(0, 64, size=(n, 4))
        delta = rng.integers(-15, 16, size=(n, 8, 4))
        base = self.level[:, None, :]
        seg_level = np.clip(base + delta, 0, 63)
        seg_level[:, :, 2:][np.broadcast_to(base[:, :, 2:] == 0, seg_level[:, :, 2:].shape)] = 0
        seg_level[(self.level[:, 0] == 0) & (self.level[:, 1] == 0)] = 0
        lv = torch.from_numpy(seg_level.astype(np.uint8)).cuda()
        cache = torch.zeros((n, self.mi_rows, self.mi_cols, 4), dtype=torch.uint8, device="cuda")
        frame = torch.arange(n, device="cuda")[:, None, None]
        sg = seg[:, :self.mi_rows, :self.mi_cols]
        cache[..., 0] = lv[frame, sg, 0]
        cache[..., 1] = lv[frame, sg, 1]
        cg = seg[:, ::1 << sy, ::1 << sx][:, :(self.mi_rows + sy) >> sy, :(self.mi_cols + sx) >> sx]
        cache[:, :cg.shape[1], :cg.shape[2], 2] = lv[frame, cg, 2]
        cache[:, :cg.shape[1], :cg.shape[2], 3] = lv[frame, cg, 3]
        self.level_cache = cache

        # CDEF: coded 8x8 blocks, presets and the units' indices.
        self.ucols, self.urows = (w + 63) // 64, (h + 63) // 64
        ur, uc = self.urows, self.ucols
        coded = torch.zeros((n, ur * 16, uc * 16), dtype=torch.bool, device="cuda")
        coded[:, :self.mi_rows, :self.mi_cols] = ~skip[:, :self.mi_rows, :self.mi_cols]
        c8 = coded.view(n, ur * 8, 2, uc * 8, 2).any(4).any(2)
        out8 = torch.ones_like(c8)
        out8[:, :self.mi_rows >> 1, :self.mi_cols >> 1] = False
        units = (c8 & ~out8).view(n, ur, 8, uc, 8)
        self.read = units.any(4).any(2).to(torch.uint8).contiguous()
        bits = (c8 | out8).view(n, ur, 8, uc, 8).permute(0, 1, 3, 2, 4)
        self.noskip = _pack(bits).to(torch.uint8).contiguous()
        self.index = torch.randint(0, 8, (n, ur, uc), generator=g, device="cuda").to(torch.uint8)
        pri, sec = rng.integers(0, 16, size=(2, n, 8)), rng.integers(0, 4, size=(2, n, 8))
        self.strength = (pri << 2 | sec).astype(np.uint8)
        self.damping = rng.integers(3, 7, size=n)

        # Restoration units: none, Wiener or self-guided, over the (upscaled) plane.
        self.units, self.unit_size = [], (lr_unit, lr_unit >> 1)
        for p in range(3):
            psx, psy = ss if p else (0, 0)
            us = self.unit_size[1 if p else 0]
            pw, ph = ((lr_width or w) + psx) >> psx, (h + psy) >> psy
            k = max(1, (pw + us // 2) // us) * max(1, (ph + us // 2) // us)
            u = np.zeros((n, k, 10), np.int8)
            u[..., 0] = np.array([abi.PF_LR_NONE, abi.PF_LR_WIENER, abi.PF_LR_SGRPROJ])[rng.integers(0, 3, (n, k))]
            u[..., 1] = rng.integers(0, 16, (n, k))
            u[..., 2], u[..., 3] = rng.integers(-96, 32, (n, k)), rng.integers(-32, 96, (n, k))
            for d in (0, 1):
                u[..., 4 + 3 * d] = 0 if p else rng.integers(-5, 11, (n, k))
                u[..., 5 + 3 * d], u[..., 6 + 3 * d] = rng.integers(-23, 9, (n, k)), rng.integers(-17, 47, (n, k))
            self.units.append(torch.from_numpy(u.view(np.uint8)).cuda())
        self.grain = [self._film_grain(rng) for _ in range(n)]

    @staticmethod
    def _film_grain(rng):
        g = abi.pf_film_grain(apply=1, seed=int(rng.integers(0, 65536)), scaling_shift=int(rng.integers(8, 12)),
                              ar_coeff_lag=3, ar_coeff_shift=int(rng.integers(6, 10)), overlap=1)
        for pts, field, k in ((g.y_points, "num_y_points", 14), (g.cb_points, "num_cb_points", 10),
                              (g.cr_points, "num_cr_points", 10)):
            for i, x in enumerate(np.sort(rng.choice(256, size=k, replace=False))):
                pts[i][0], pts[i][1] = int(x), int(rng.integers(0, 256))
            setattr(g, field, k)
        for co, k in ((g.ar_coeffs_y, 24), (g.ar_coeffs_cb, 25), (g.ar_coeffs_cr, 25)):
            for i, v in enumerate(rng.integers(-128, 128, k)):
                co[i] = int(v)
        g.cb_mult, g.cb_luma_mult, g.cr_mult, g.cr_luma_mult = (int(v) for v in rng.integers(0, 256, 4))
        g.cb_offset, g.cr_offset = (int(v) for v in rng.integers(0, 512, 2))
        return g

    def to_host(self):
        """The arrays in ordinary host memory, as a decoder's own are."""
        for k in ("masks", "level_cache", "index", "read", "noskip"):
            setattr(self, k, getattr(self, k).cpu())
        self.units = [u.cpu() for u in self.units]
        return self

    def pf(self, i, stages=None):
        s = abi.pf_frame_side()
        s.stages = stages if stages is not None else (abi.PF_STAGES_ALL if self.full else LF_CDEF)
        s.side_memory = abi.PF_MEM_DEVICE if self.masks.is_cuda else abi.PF_MEM_HOST
        lf = s.lf
        lf.level_y[0], lf.level_y[1], lf.level_u, lf.level_v = (int(v) for v in self.level[i])
        lf.masks, lf.sb128_w, lf.sb128_h = self.masks[i].data_ptr(), self.sbw, self.sbh
        lf.level_cache, lf.mi_cols, lf.mi_rows = self.level_cache[i].data_ptr(), self.mi_cols, self.mi_rows
        cd = s.cdef
        cd.bits, cd.damping, cd.strength_count = 3, int(self.damping[i]), 8
        for k in range(8):
            cd.y_strength[k], cd.uv_strength[k] = int(self.strength[0, i, k]), int(self.strength[1, i, k])
        cd.index, cd.read, cd.noskip = (t[i].data_ptr() for t in (self.index, self.read, self.noskip))
        cd.index_stride, cd.index_rows = self.ucols, self.urows
        lr = s.lr
        lr.unit_size_y, lr.unit_size_uv = self.unit_size
        for p in range(3):
            lr.type[p] = abi.PF_LR_SWITCHABLE
            lr.units[p], lr.unit_count[p] = self.units[p][i].data_ptr(), self.units[p].shape[1]
        s.fg = self.grain[i]
        return s


def _video(seed, n, w, h, bd, ss, dc=12, noise=4.0, one_texture=True):
    """(Frames, buffer) of n frames: one texture moving from frame to frame, or n textures."""
    fr = Frames(n, w, h, bd, LAYOUTS[ss])
    buf = torch.empty(fr.nbytes, dtype=torch.uint8, device="cuda")
    g, rng = _gen(seed + 1), np.random.default_rng([seed & 0x7FFFFFFF, 0xF00D])
    tex, scale = _texture(rng), 1 << (bd - 8)
    for i in range(n):
        mv = rng.integers(-8, 9, 2) * (i + 1)
        if not one_texture:
            tex = _texture(rng)
        _content(fr, buf, i, g, tex, (int(mv[0]), int(mv[1])), dc * scale, noise * scale)
    return fr, buf


# ---------------------------------------------------------------------------
# Calls

_runners = {}


def _runner(graphs=False, host_batch=False):
    """The runner that each kind of caller keeps: with or without captured graphs, and one of its own for
    batches of host frames (its copy streams and staging belong to it)."""
    key = (graphs, host_batch)
    if key not in _runners:
        r = PostFilterRunner()
        if graphs:
            r.batch_graphs(True)
        _runners[key] = (r, torch.cuda.ExternalStream(r.stream))
    return _runners[key]


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("chain", "mixed"):
        groups = [(case["frames"], case["w"], case["h"], case["bd"], case["ss"])] if kind == "chain" else \
            [(max(1, k * case["copies"] // 8), w, h, bd, ss) for k, w, h, bd, ss in MIXED]
        host = case.get("host", False)
        full = case.get("full", True)
        mem = abi.PF_MEM_HOST if host else abi.PF_MEM_DEVICE
        parts = []
        for i, (n, w, h, bd, ss) in enumerate(groups):
            fr, buf = _video(seed + 101 * i, n, w, h, bd, ss, one_texture=kind == "chain")
            side = Side(seed + 101 * i + 7, n, w, h, LAYOUTS[ss], full, lr_unit=256 if w * h > 4_000_000 else 128)
            parts.append((fr, buf, side.to_host() if host else side))
        total = sum(fr.nbytes for fr, _, _ in parts)
        if host:
            pristine, io, disp = (torch.zeros(total, dtype=torch.uint8, pin_memory=True) for _ in range(3))
        else:
            pristine, io, disp = (torch.zeros(total, dtype=torch.uint8, device="cuda") for _ in range(3))
        items, at = [], 0
        for fr, buf, side in parts:
            pristine[at:at + fr.nbytes].copy_(buf)
            for i in range(fr.n):
                items.append((fr.pf(io[at:], i, mem), side.pf(i), fr.pf(disp[at:], i, mem) if full else None))
            at += fr.nbytes
        r, stream = _runner(case["graphs"], host and len(items) > 1)
        st.update(runner=r, stream=stream, pristine=pristine, io=io, disp=disp if full else None, items=items,
                  keep=[p[2] for p in parts], host=host, arr=r.batch_items(items))
        return st
    w, h = case["w"], case["h"]
    r, stream = _runner()
    st.update(runner=r, stream=stream)
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 0x5EA7])
    if kind in ("search", "learned", "lr_search"):
        # The source without noise; the reconstruction with blocky distortion,
        # deblocked before the CDEF search as an encoder does.
        sigma = float(rng.choice([2.0, 4.0, 8.0]))
        fr, src = _video(seed, 1, w, h, 8, "420", dc=0, noise=0)
        _, rec = _video(seed, 1, w, h, 8, "420", dc=6 if kind == "lr_search" else 12, noise=sigma)
        side = Side(seed + 7, 1, w, h, (1, 1))
        if kind != "lr_search":
            torch.cuda.synchronize()
            r.apply(fr.pf(rec, 0, abi.PF_MEM_DEVICE), side.pf(0, abi.PF_STAGE_LOOP_FILTER))
            r.sync()
        st.update(bufs=(src, rec), src=fr.pf(src, 0, abi.PF_MEM_DEVICE), rec=fr.pf(rec, 0, abi.PF_MEM_DEVICE),
                  noskip=np.ascontiguousarray(side.noskip[0].cpu().numpy()),
                  qindex=int(rng.choice(learned.QINDEX_CHOICES)))
        if kind == "search":
            st["ctrls"] = cdef_plan_picture(case["level"], islice=True, not_highest_layer=True).ctrls
            st["level"] = case["level"]
        elif kind == "learned":
            st["model"] = learned.load_model()
        else:
            st["out"] = torch.zeros(fr.nbytes, dtype=torch.uint8, device="cuda")
            st["restored"] = fr.pf(st["out"], 0, abi.PF_MEM_DEVICE)
        return st
    if kind == "superres":
        n, ss = case["frames"], LAYOUTS[case["ss"]]
        cw = (8 * w + case["denom"] // 2) // case["denom"]
        fr, pristine = _video(seed, n, cw, h, case["bd"], case["ss"])
        up = Frames(n, w, h, case["bd"], ss)
        side = Side(seed + 7, n, cw, h, ss, lr_width=w)
        io = pristine.clone()
        uio, disp = (torch.zeros(up.nbytes, dtype=torch.uint8, device="cuda") for _ in range(2))
        dev = abi.PF_MEM_DEVICE
        st.update(pristine=pristine, io=io, up=uio, disp=disp, keep=side,
                  items=[(fr.pf(io, i, dev), side.pf(i), up.pf(uio, i, dev), up.pf(disp, i, dev)) for i in range(n)])
        return st
    st.update(_lf_map(case, seed))
    return st


def _lf_map(case, seed):
    """A block record map: quadtree nodes kept whole or halved either way, intra blocks with the transform
    reduced up to two steps, inter blocks skipped or with a split transform tree."""
    w, h, ss = case["w"], case["h"], LAYOUTS[case["ss"]]
    cols, rows = ((w + 7) >> 3) << 1, ((h + 7) >> 3) << 1
    R, K = -(-rows // 32) * 32, -(-cols // 32) * 32
    g = _gen(seed)
    bdims, txd, maxtx = synth.av1_tables()
    lg = _blocks(g, 1, R, K)
    s = 1 << lg
    gy = torch.arange(R, device="cuda", dtype=torch.int32)[None, :, None].expand(1, R, K)
    gx = torch.arange(K, device="cuda", dtype=torch.int32)[None, None, :].expand(1, R, K)

    def rand():
        return torch.rand((1, R, K), generator=g, device="cuda")

    shape = (_at_origin(rand(), s, s, gy, gx) * 3).to(torch.int32) * (lg > 0)
    bh, bw = torch.where(shape == 1, s >> 1, s), torch.where(shape == 2, s >> 1, s)
    oy, ox = gy - gy % bh, gx - gx % bw
    size_of = torch.zeros((33, 33), dtype=torch.int64, device="cuda")
    for i, (bw4, bh4) in enumerate(bdims):
        if bw4 <= 32 and bh4 <= 32:
            size_of[bh4, bw4] = i
    bs = size_of[bh.long(), bw.long()]
    tmax = torch.tensor([m[0] for m in maxtx], device="cuda")
    tuv = torch.tensor([m[3 if ss[0] == 0 else (1 if ss[1] else 2)] for m in maxtx], device="cuda")
    tsub = torch.tensor([t[4] if i else 0 for i, t in enumerate(txd)], device="cuda")

    def per_block(k):
        return (_at_origin(rand(), bh, bw, gy, gx) * k).to(torch.int64)

    intra = per_block(10) < 3
    skip = ~intra & (per_block(10) < 3)
    tx = tmax[bs]
    steps = per_block(3)
    for k in (1, 2):
        tx = torch.where(intra & (steps >= k), tsub[tx], tx)
    split = ~intra & ~skip & (tx > 0) & (per_block(10) < 6)
    zero = torch.zeros_like(bs)
    fields = [(0, 2, ox), (2, 2, oy), (4, 2, (ox + bw).clamp(max=cols)), (6, 2, (oy + bh).clamp(max=rows)), (8, 1, bs),
              (9, 1, zero + 1), (10, 1, intra), (11, 1, skip), (12, 1, tx), (13, 1, tuv[bs]), (14, 1, zero + 1),
              (15, 1, per_block(8)), (16, 1, torch.where(intra, zero, 1 + per_block(7))),
              (17, 1, torch.where(intra, zero, per_block(2))), (18, 1, per_block(25) - 12)]
    fields += [(19 + k, 1, per_block(25) - 12) for k in range(4)]
    fields += [(24, 2, torch.where(split, 1 + per_block(65535), zero)), (26, 2, torch.where(split, per_block(65536), zero))]
    rec = torch.zeros((R, K, 32), dtype=torch.uint8, device="cuda")
    for at, size, v in fields:
        v = v[0].to(torch.int64)
        for b in range(size):
            rec[:, :, at + b] = ((v >> (8 * b)) & 255).to(torch.uint8)
    return {"records": rec[:rows, :cols].contiguous(), "levels": synth.make_lf_levels(seed & 0x7FFFFFFF, "deltas"),
            "ss": ss}


def _search_outputs(res, mse, idx):
    return {"bits": int(res.bits), "y": np.ctypeslib.as_array(res.y_strength).copy(),
            "uv": np.ctypeslib.as_array(res.uv_strength).copy(), "cost": int(res.cost), "mse": mse.view(np.int64),
            "index": idx}


def run(state):
    r, kind = state["runner"], state["kind"]
    if kind in ("chain", "mixed"):
        # The decoder's reconstruction arrives in the frames, which the call filters in place.
        if state["host"]:
            state["io"].copy_(state["pristine"])
        else:
            with torch.cuda.stream(state["stream"]):
                state["io"].copy_(state["pristine"], non_blocking=True)
        if len(state["items"]) == 1:
            r.apply(*state["items"][0])
        else:
            r.apply_batch(state["arr"])
        return [state["io"]] + ([state["disp"]] if state["disp"] is not None else [])
    if kind == "superres":
        with torch.cuda.stream(state["stream"]):
            state["io"].copy_(state["pristine"], non_blocking=True)
        r.apply_batch_superres(state["items"])
        return [state["io"], state["up"], state["disp"]]
    if kind == "search":
        if state["level"] == 1:
            return _search_outputs(*r.cdef_search(state["src"], state["rec"], state["noskip"], state["qindex"],
                                                  learned.LAMBDA))
        return _search_outputs(*r.cdef_search_ex(state["src"], state["rec"], state["noskip"], state["qindex"],
                                                 learned.LAMBDA, state["ctrls"]))
    if kind == "learned":
        return _search_outputs(*r.cdef_search_learned(state["src"], state["rec"], state["noskip"], state["qindex"],
                                                      learned.LAMBDA, state["model"], want_stats=False)[:3])
    if kind == "lr_search":
        units = r.lr_search(state["src"], state["rec"], state["restored"])
        return [np.frombuffer(units, np.uint8), state["out"]]
    return list(r.lf_build(state["records"], state["levels"], *state["ss"]))


def work(case):
    kind = case["kind"]
    if kind == "mixed":
        parts = [_chain("", w, h, bd, ss, max(1, k * case["copies"] // 8)) for k, w, h, bd, ss in MIXED]
        return {"bytes": sum(work(p)["bytes"] for p in parts), "flops": 0}
    px = case["w"] * case["h"]
    if kind == "lf_build":
        # A 32-byte record read and 4 level bytes and about 1.25 mask bytes written per 4x4 cell.
        return {"bytes": px / 16 * 37.25, "flops": 0}
    if kind in ("search", "learned"):
        # Source and reconstruction once; a trial is 12 taps (difference, constrain, weighted sum), the range
        # clamp and the squared error of each sample: about 90 operations.
        n = cdef_plan_picture(case["level"], islice=True, not_highest_layer=True).ctrls if kind == "search" else None
        luma = 64 if n is None else n.count / n.subsampling
        chroma = 64 if n is None else sum(1 for i in range(n.count) if n.uv[i] >= 0)
        if kind == "learned":
            luma = chroma = 3
        return {"bytes": 3 * px, "flops": px * 90 * (luma + 0.5 * chroma)}
    if kind == "lr_search":
        # Two luma planes read and one written; four self-guided filters of about 60 operations a sample.
        return {"bytes": 3 * px, "flops": px * 4 * 60}
    ss = LAYOUTS[case["ss"]]
    samples = 1 + 2 / (1 << (ss[0] + ss[1]))
    bps = 1 if case["bd"] == 8 else 2
    if kind == "superres":
        scale = 8 / case["denom"]
        # The coded frame in and out, the upscaled and the display frame out.
        return {"bytes": case["frames"] * px * (samples * bps * (2 * scale + 2) + 0.33), "flops": 0}
    # The frame in, the reference (and the display) out, the side information in.
    return {"bytes": case["frames"] * px * (samples * bps * (3 if case["full"] else 2) + 0.33), "flops": 0}


def exact(case, seed):
    """Every output is a whole number that has to be equal: none has a value in 64 bits beside it."""
    return None
