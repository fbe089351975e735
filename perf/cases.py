"""The decoder's workloads as timed cases: what its users decode, through the
calls they make.

A case is a dict of plain values.  Its geometry (sizes, samplings, qualities,
restart intervals) is fixed by the case; the picture content comes from the
seed, so another seed gives other files of the same shapes.  ``prepare`` makes
the JPEG files in host memory (pinned, where a program would read them into
pinned memory) and the decoder objects a program keeps; ``run`` is one pass
from those files to decoded pixels through the public calls.

Kinds:

* ``reader``  -- ``Reader.open_bytes`` then ``pixels``: one file to host
  pixels (the drop-in path, baseline or progressive)
* ``batch``   -- ``Batch.stage`` / ``run`` / ``wait``: files in pinned memory
  to pixels on the device (a training or transcoding input pipeline)
* ``host``    -- ``Batch.decode``: a list of files to host arrays
* ``server``  -- ``Server.submit`` / ``wait`` / ``device_tensor`` / ``release``
* ``plane``   -- ``cjIDCTPlane`` on a decoded component (the iDCT by itself)
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cudajpeg_b200 as cj
from cudajpeg_b200 import serve
from cudajpeg_b200 import workloads as W

DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ---------------------------------------------------------------- cases

def _reader(name, w, h, mode, q, ri=0, progressive=False):
    return {"name": name, "kind": "reader", "w": w, "h": h, "mode": mode, "q": q, "ri": ri,
            "progressive": progressive}


def _batch(name, kind, n, lo, hi, step, modes, qlo, qhi, restarts, out, idct, plan):
    """n images, sides log-uniform in [lo, hi] in multiples of `step`, modes
    with the given weights, qualities in [qlo, qhi], a share `restarts` of
    them with a restart interval; `plan` seeds the geometry."""
    return {"name": name, "kind": kind, "n": n, "lo": lo, "hi": hi, "step": step, "modes": modes,
            "qlo": qlo, "qhi": qhi, "restarts": restarts, "out": out, "idct": idct, "plan": plan}


MIX = "420:6,422:2,444:1,gray:1"


def listed():
    return [
        # one thumbnail or avatar: the smallest call, all latency
        _reader("reader_thumb", 120, 90, "420", 85),
        # one web-sized photo (the single-image configuration)
        _reader("reader_1024x768", 1024, 768, "420", 75),
        # one large scan or satellite tile (the large-image configuration)
        _reader("reader_4096", 4096, 4096, "420", 90),
        # one 24-megapixel camera file: 4:2:2, a restart marker per MCU row
        _reader("reader_camera", 6000, 4000, "422", 92, 375),
        # one progressive web photo, default scan script of the IJG encoder
        _reader("reader_progressive", 1024, 768, "420", 80, 0, True),
        # the mixed batch of the batch configuration, tensor-core iDCT,
        # pixels left on the device: the largest call
        _batch("batch_mixed_1024", "batch", 1024, 64, 2048, 8, MIX, 50, 95, 0.3, "rgb", "tc", 4),
        # many thumbnails: per-image work counts
        _batch("batch_thumbs_512", "batch", 512, 64, 256, 8, MIX, 70, 90, 0.0, "rgb", "int", 12),
        # motion JPEG: 1080p frames to NV12 for a video pipeline
        _batch("batch_mjpeg_nv12", "batch", 48, 1080, 1920, 0, "420:1", 80, 80, 1.0, "nv12", "int", 13),
        # display-quality chroma: fancy upsampling of odd-sized photos
        _batch("batch_fancy_24", "batch", 24, 500, 1600, 1, "420:3,422:1", 75, 95, 0.0, "fancy", "tc", 14),
        # a list of files to host arrays, the shortest program
        _batch("host_decode_40", "host", 40, 33, 1023, 1, MIX, 50, 95, 0.3, "rgb", "int", 15),
        # a burst of requests to the decode server
        _batch("server_24", "server", 24, 200, 1000, 1, MIX, 60, 95, 0.3, "rgb", "int", 16),
        # the tensor-core plane iDCT by itself (the precision configuration)
        {"name": "plane_8192", "kind": "plane", "w": 8192, "h": 8192, "mode": "gray", "q": 95, "form": "tc"},
    ]


def draw(rng):
    def logint(lo, hi, step=1):
        return max(step, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)

    kind = rng.choice(["reader", "reader", "progressive", "batch", "batch", "odd", "host", "server", "plane"])
    mode = rng.choice(["420", "420", "422", "444", "gray"])
    if kind in ("reader", "progressive"):
        prog = kind == "progressive"
        w, h = logint(64, 2048 if prog else 6000), logint(64, 1536 if prog else 4000)
        ri = rng.choice([0, 0, rng.randint(1, 400)])
        return _anon(_reader("", w, h, mode, rng.randint(50, 95), 0 if prog else ri, prog))
    if kind == "plane":
        return {"kind": "plane", "w": 8 * logint(16, 768), "h": 8 * logint(16, 512), "mode": mode,
                "q": rng.randint(50, 95), "form": rng.choice(["tc", "int", "f32"])}
    fmt = rng.choice(["rgb", "rgb", "nv12", "planar", "fancy"])
    idct = rng.choice(["int", "tc"])
    restarts = rng.choice([0.0, 0.3, 1.0])
    plan = rng.randint(100, 1 << 20)
    qlo = rng.randint(40, 85)
    lo = logint(40, 400)
    hi = min(2048, lo * rng.randint(1, 6) + 1)
    if kind == "batch":  # sizes in whole blocks, up to a thousand images
        n = min(logint(65, 1024), max(65, 200_000_000 // (hi * hi)))
        return _anon(_batch("", "batch", n, lo, hi, 8, MIX, qlo, 95, restarts,
                            fmt if fmt in ("rgb", "nv12") else "rgb", idct, plan))
    n = logint(1, 60)
    if kind == "odd":
        return _anon(_batch("", "batch", n, lo, hi, 1, MIX, qlo, 95, restarts, fmt, idct, plan))
    return _anon(_batch("", kind, n, lo, hi, 1, MIX, qlo, 95, restarts, "rgb", "int", plan))


def _anon(c):
    c.pop("name")
    return c


def _images(case):
    """(w, h, mode, quality, restart interval) of every image of a case."""
    if case["kind"] in ("reader", "plane"):
        return [(case["w"], case["h"], case["mode"], case["q"], case.get("ri", 0))]
    if case["step"] == 0:  # frames of one size, a restart marker per MCU row
        return [(case["hi"], case["lo"], "420", case["qlo"], -(-case["hi"] // 16))] * case["n"]
    rng = np.random.default_rng(case["plan"])
    names, weights = zip(*(p.split(":") for p in case["modes"].split(",")))
    p = np.array([float(x) for x in weights])
    out = []
    for _ in range(case["n"]):
        w, h = (max(case["step"], int(round(math.exp(v) / case["step"])) * case["step"])
                for v in rng.uniform(math.log(case["lo"]), math.log(case["hi"]), 2))
        mode = str(rng.choice(names, p=p / p.sum()))
        q = int(rng.integers(case["qlo"], case["qhi"] + 1))
        ri = int(rng.integers(16, 65)) if rng.random() < case["restarts"] else 0
        out.append((w, h, mode, q, ri))
    return out


# ---------------------------------------------------------------- files

def _picture(gen, w, h, ch, noise):
    """Smooth sinusoid and gradient fields plus noise, as the repository's
    ``smooth_content``, made on the device: uint8 [h, w, ch]."""
    u = torch.rand(ch, 6, generator=gen, device=DEV)
    x = torch.arange(w, device=DEV, dtype=torch.float32) / w
    y = torch.arange(h, device=DEV, dtype=torch.float32) / h
    fx = torch.sin((0.5 + 3.5 * u[:, 0:1]) * 2 * math.pi * x + 2 * math.pi * u[:, 2:3])
    fy = torch.cos((0.5 + 3.5 * u[:, 1:2]) * 2 * math.pi * y + 2 * math.pi * u[:, 3:4])
    f = 128 + 70 * fy[:, :, None] * fx[:, None, :]
    f += ((120 * u[:, 4:5] - 60) * (x - 0.5))[:, None, :] + ((120 * u[:, 5:6] - 60) * (y - 0.5))[:, :, None]
    f += noise * torch.randn(ch, h, w, generator=gen, device=DEV)
    return f.clamp_(0, 255).to(torch.uint8).permute(1, 2, 0).contiguous().cpu().numpy()


def _texture(gen, w, h, noise):
    """The large-image content: eight oriented waves and luma noise."""
    u = torch.rand(8, 3, generator=gen, device=DEV)
    x = torch.arange(w, device=DEV, dtype=torch.float32)[None, :]
    y = torch.arange(h, device=DEV, dtype=torch.float32)[:, None]
    f = torch.full((h, w), 128.0, device=DEV)
    for k in range(8):
        th, wave = math.pi * u[k, 0], (2 + 38 * u[k, 1]) * 2 * math.pi / max(w, h)
        f += 11 * torch.sin(wave * (torch.cos(th) * x + torch.sin(th) * y) + 2 * math.pi * u[k, 2])
    f += noise * (2 * torch.rand(h, w, generator=gen, device=DEV) - 1)
    t = 60 * torch.rand(3, 1, 1, generator=gen, device=DEV) - 30
    f = f[None] + t * (x[None] / w - 0.5)
    return f.clamp_(0, 255).to(torch.uint8).permute(1, 2, 0).contiguous().cpu().numpy()


def _files(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(1_000_003 * int(seed) + 17)
    files = []
    for w, h, mode, q, ri in _images(case):
        ch = 1 if mode == "gray" else 3
        if ch == 3 and w * h >= 1 << 24:
            arr = _texture(gen, w, h, 5.0)
        else:
            arr = _picture(gen, w, h, ch, 8.0)
        if ch == 1:
            arr = arr[..., 0]
        files.append(_progressive(arr, mode, q) if case.get("progressive") else W.encode(arr, mode, q, ri))
    return files


# ---- a progressive encoder (ITU T.81 Annex G), as the package writes only
# baseline files.  The scan script is the IJG encoder's default one; the
# Huffman tables are made per scan from the symbol counts.

ZIGZAG = np.array(sorted(range(64), key=lambda n: (n // 8 + n % 8,
                                                   n // 8 if (n // 8 + n % 8) % 2 else n % 8)))


def _coefficients(arr, mode, dqt):
    """Quantised zig-zag coefficients per component: int64 [rows, cols, 64],
    rows and cols padded to whole MCUs."""
    a = arr.astype(np.float64)
    if a.ndim == 2:
        planes, sy, sx = [a], 1, 1
    else:
        r, g, b = a[..., 0], a[..., 1], a[..., 2]
        planes = [0.299 * r + 0.587 * g + 0.114 * b, 128 - 0.168736 * r - 0.331264 * g + 0.5 * b,
                  128 + 0.5 * r - 0.418688 * g - 0.081312 * b]
        sx, sy = {"420": (2, 2), "422": (2, 1), "444": (1, 1)}[mode]
    h, w = planes[0].shape
    mh, mw = -(-h // (8 * sy)), -(-w // (8 * sx))
    n = np.arange(8)
    basis = np.where(n[:, None] == 0, math.sqrt(0.125), 0.5) * np.cos((2 * n[None, :] + 1) * n[:, None] * math.pi / 16)
    out = []
    for c, p in enumerate(planes):
        p = np.pad(p, ((0, mh * 8 * sy - h), (0, mw * 8 * sx - w)), mode="edge")
        if c:
            p = p.reshape(p.shape[0] // sy, sy, p.shape[1] // sx, sx).mean((1, 3))
        blocks = p.reshape(p.shape[0] // 8, 8, p.shape[1] // 8, 8).transpose(0, 2, 1, 3) - 128
        f = (basis @ blocks @ basis.T).reshape(*blocks.shape[:2], 64)[..., ZIGZAG]
        out.append(np.rint(f / dqt[min(c, 1)]).astype(np.int64))
    return out, sx, sy


def _bit_length(v):
    return np.frexp(np.abs(v).astype(np.float64))[1].astype(np.int64)


class _Stream:
    """Tokens of one scan: each a symbol of a Huffman table or none, then raw
    bits, ordered by an int64 key."""

    def __init__(self):
        self.parts = []

    def add(self, key, table, symbol, value, bits):
        key = np.asarray(key, np.int64)
        self.parts.append([np.broadcast_to(np.asarray(x, np.int64), key.shape)
                           for x in (key, table, symbol, value, bits)])

    def encode(self, ac):
        """The scan's DHT segments and its stuffed entropy-coded bytes."""
        key, table, symbol, value, bits = (np.concatenate(x) for x in zip(*self.parts))
        order = np.argsort(key, kind="stable")
        table, symbol, value, bits = table[order], symbol[order], value[order], bits[order]
        code, length, dht = np.zeros(len(order), np.int64), np.zeros(len(order), np.int64), b""
        for t in (0, 1):
            use = (table == t) & (symbol >= 0)
            if not use.any():
                continue
            count = np.bincount(symbol[use], minlength=256)
            syms = sorted(np.flatnonzero(count), key=lambda s: -count[s])
            # Shannon lengths, at most 16 bits, with room for the all-ones code
            size = [min(16, max(1, math.ceil(-math.log2(0.97 * count[s] / count.sum())))) for s in syms]
            codes, sizes, nxt = np.zeros(256, np.int64), np.zeros(256, np.int64), 0
            for k, s in enumerate(syms):
                nxt = (nxt + 1) << (size[k] - size[k - 1]) if k else 0
                codes[s], sizes[s] = nxt, size[k]
            code[use], length[use] = codes[symbol[use]], sizes[symbol[use]]
            body = bytes([16 * ac + t]) + bytes(size.count(k) for k in range(1, 17)) + bytes(int(s) for s in syms)
            dht += b"\xff\xc4" + (len(body) + 2).to_bytes(2, "big") + body
        value = (code << bits) | value
        bits = bits + length
        n = int(bits.sum())
        at = np.arange(n) - np.repeat(np.cumsum(bits) - bits, bits)
        stream = (np.repeat(value, bits) >> (np.repeat(bits, bits) - 1 - at)) & 1
        stream = np.concatenate([stream, np.ones(-n % 8, np.int64)])
        return dht, np.packbits(stream.astype(np.uint8)).tobytes().replace(b"\xff", b"\xff\x00")


def _eob_runs(stream, table, last, se, empty, base):
    """Add the end-of-band symbols: a run starts at each block that ends in an
    EOB and does not continue the previous block's run."""
    eob = last < se
    start = eob & ~(empty & np.concatenate([[False], eob[:-1]]))
    at = np.flatnonzero(start)
    # the blocks of a run: its first, then the empty blocks after it
    runs = np.bincount(np.cumsum(start)[eob] - 1, minlength=len(at)) if len(at) else np.zeros(0, np.int64)
    if len(runs) and runs.max() > 0x7FFF:
        raise ValueError("end-of-band run too long")
    size = _bit_length(runs) - 1
    stream.add(base[at], table, size << 4, runs - (1 << size), size)


def _ac_scan(coef, ss, se, ah, al, table):
    """One AC scan of a component's blocks [n, 64] (raster order)."""
    n, width = len(coef), se - ss + 1
    a = np.abs(coef[:, ss:se + 1])
    mag, neg = a >> al, coef[:, ss:se + 1] < 0
    k = np.arange(width)
    s = _Stream()
    new = mag == 1 if ah else mag > 0
    hist = (a >> ah) > 0 if ah else np.zeros_like(new)
    last = np.where(new.any(1), width - 1 - np.argmax(new[:, ::-1], 1), -1)
    # zero-history coefficients since the previous newly nonzero one
    zeros = np.cumsum(~(new | hist), 1)
    prev = np.maximum.accumulate(np.where(new, k, -1), 1)
    prev = np.concatenate([np.full((n, 1), -1), prev[:, :-1]], 1)
    at_prev = np.where(prev >= 0, np.take_along_axis(zeros, np.maximum(prev, 0), 1), 0)
    run = zeros - at_prev
    group = np.cumsum(new, 1) - new  # newly nonzero coefficients before this one

    # a token's place: block, newly nonzero coefficients before it, ZRLs of
    # that run before it (4: after the last one), symbols before bits, position
    def key(b, g, z, kind, pos):
        return ((b * 65 + g) * 5 + z) * 130 + kind * 65 + pos

    b, i = np.nonzero(new)
    r, g = run[b, i], group[b, i]
    sizes = _bit_length(mag[b, i])
    if ah:
        value = 1 - neg[b, i].astype(np.int64)
    else:
        value = np.where(neg[b, i], (1 << sizes) - 1 - mag[b, i], mag[b, i])
    s.add(key(b, g, r // 16, 0, 1), table, (r % 16) * 16 + sizes, value, sizes)
    for z in range(4):
        m = r // 16 > z
        s.add(key(b[m], g[m], z, 0, 0), table, 0xF0, 0, 0)
    if ah:  # correction bits
        b, i = np.nonzero(hist)
        tail = group[b, i] == new.sum(1)[b]  # after the block's last newly nonzero one
        z = np.where(tail, 4, run[b, i] // 16)
        s.add(key(b, group[b, i], z, 1, i), 2, -1, (a[b, i] >> al) & 1, 1)
    _eob_runs(s, table, last, width - 1, ~new.any(1), key(np.arange(n), new.sum(1), 4, 0, 2))
    return s.encode(1)


def _dc_scan(coefs, sx, sy, ah, al):
    """The interleaved DC scan of all components."""
    s = _Stream()
    nc = len(coefs)
    mh, mw = coefs[-1].shape[:2]
    bpm = sx * sy + nc - 1
    for c, co in enumerate(coefs):
        vy, vx = (sy, sx) if c == 0 else (1, 1)
        dc = co[..., 0] >> al
        dc = dc.reshape(mh, vy, mw, vx).transpose(0, 2, 1, 3).reshape(-1)
        per = vx * vy
        at = np.arange(len(dc))
        key = at // per * bpm + at % per + (sx * sy + c - 1 if c else 0)
        if ah:
            s.add(key, 2, -1, dc & 1, 1)
            continue
        diff = np.diff(dc, prepend=0)
        size = _bit_length(diff)
        s.add(key, min(c, 1), size, np.where(diff < 0, diff + (1 << size) - 1, diff), size)
    return s.encode(0)


def _progressive(arr, mode, q):
    """`arr` as a progressive JPEG (the IJG encoder's default scan script)."""
    head = W.encode(arr[:16, :16], mode, q)  # its quantisation tables and frame header
    dqt, sof, pos, tables = b"", b"", 2, []
    while head[pos + 1] != 0xDA:
        n = int.from_bytes(head[pos + 2:pos + 4], "big") + 2
        seg = head[pos:pos + n]
        if seg[1] == 0xDB:
            dqt += seg
            tables += [np.frombuffer(seg[4 + 65 * k + 1:4 + 65 * (k + 1)], np.uint8).astype(np.float64)
                       for k in range(len(seg[4:]) // 65)]
        elif seg[1] == 0xC0:
            sof = b"\xff\xc2" + seg[2:5] + arr.shape[0].to_bytes(2, "big") + arr.shape[1].to_bytes(2, "big") + seg[9:]
        pos += n
    coefs, sx, sy = _coefficients(arr, mode, tables if len(tables) > 1 else tables * 2)
    nc = len(coefs)
    h, w = arr.shape[:2]

    def blocks(c):  # a component's own blocks, without the MCU padding
        ch, cw = (h, w) if c == 0 else (-(-h // sy), -(-w // sx))
        return coefs[c][:-(-ch // 8), :-(-cw // 8)].reshape(-1, 64)

    script = [(None, 0, 0, 0, 1), (0, 1, 5, 0, 2), (2, 1, 63, 0, 1), (1, 1, 63, 0, 1), (0, 6, 63, 0, 2),
              (0, 1, 63, 2, 1), (None, 0, 0, 1, 0), (2, 1, 63, 1, 0), (1, 1, 63, 1, 0), (0, 1, 63, 1, 0)]
    out = b"\xff\xd8" + dqt + sof
    for c, ss, se, ah, al in script:
        if c is not None and c >= nc:
            continue
        if c is None:
            dht, data = _dc_scan(coefs, sx, sy, ah, al)
            comps = [(k + 1, 0x11 if k else 0x00) for k in range(nc)]
        else:
            dht, data = _ac_scan(blocks(c), ss, se, ah, al, min(c, 1))
            comps = [(c + 1, 0x11 if c else 0x00)]
        sos = bytes([len(comps)]) + b"".join(bytes(x) for x in comps) + bytes([ss, se, 16 * ah + al])
        out += dht + b"\xff\xda" + (len(sos) + 2).to_bytes(2, "big") + sos + data
    return out + b"\xff\xd9"


# ---------------------------------------------------------------- passes

FORMAT = {"rgb": cj.OUTPUT_RGB, "planar": cj.OUTPUT_PLANAR, "nv12": cj.OUTPUT_NV12, "fancy": cj.OUTPUT_RGB_FANCY}
FORM = {"int": cj.IDCT_INT, "tc": cj.IDCT_TC, "f32": cj.IDCT_F32}


class _DeviceBytes:
    """Device memory of a decoded batch as one byte range."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (ptr, False), "version": 2}


class _HostView(np.ndarray):
    """A host view of a decoder's output buffer."""


def _held(out, owner):
    """`out`, a view of its decoder's memory, keeps that decoder open."""
    out = out.view(_HostView) if isinstance(out, np.ndarray) else out
    out.owner = owner
    return out


def _pinned(data):
    t = torch.empty(len(data), dtype=torch.uint8, pin_memory=torch.cuda.is_available())
    t.numpy()[:] = np.frombuffer(data, np.uint8)
    return t


def prepare(case, seed):
    files = _files(case, seed)
    kind = case["kind"]
    state = {"kind": kind, "n": len(files)}
    if kind == "reader":
        state["reader"] = cj.Reader()
        state["file"] = _pinned(files[0])
    elif kind == "plane":
        r = state["reader"] = cj.Reader()
        r.open_bytes(files[0])
        state["geom"] = r.plane_geometry(0)
        state["mode"] = FORM[case["form"]]
        state["plane"] = torch.zeros((state["geom"]["rows"], state["geom"]["stride"]), dtype=torch.uint8, device=DEV)
    elif kind == "server":
        state["server"] = serve.Server()
        state["files"] = files
    else:
        b = state["batch"] = cj.Batch()
        b.set_output(FORMAT[case["out"]], FORM[case["idct"]])
        state["files"] = files
        blob, state["offsets"], state["sizes"] = b.pack(files)
        state["blob"] = _pinned(blob)
    return state


def run(state):
    kind = state["kind"]
    if kind == "reader":
        f, r = state["file"], state["reader"]
        r.open_bytes((f.data_ptr(), f.numel()))
        return _held(r.pixels(copy=False), r)
    if kind == "plane":
        state["reader"].plane_launch(state["geom"], state["plane"].data_ptr(), state["mode"],
                                     torch.cuda.current_stream().cuda_stream)
        return state["plane"]
    if kind == "server":
        s = state["server"]
        tickets = [s.submit(f) for f in state["files"]]
        for t in tickets:
            s.wait(t)
        # the results' memory is the server's until release: take copies
        out = [s.device_tensor(t).clone() for t in tickets]
        torch.cuda.current_stream().synchronize()
        for t in tickets:
            s.release(t)
        return out
    b = state["batch"]
    if kind == "host":
        return b.decode(state["files"])[0]
    b.stage(state["blob"].data_ptr(), state["offsets"], state["sizes"])
    b.run()
    b.wait()
    if state["n"] <= 60:
        return [_held(b.device_tensor(k), b) for k in range(state["n"])]
    # sizes in whole blocks: the outputs lie back to back
    return _held(torch.as_tensor(_DeviceBytes(b.lib.cjBatchDeviceImage(b.ptr, 0), b.stats()["output_bytes"]),
                                 device=DEV), b)


def work(case):
    """Each file read once and each output byte written once; the arithmetic
    of the iDCT (two 8x8x8 products per block) as operations."""
    files = _files(case, 0)
    out = blocks = 0
    for w, h, mode, _, _ in _images(case):
        sx, sy = {"420": (2, 2), "422": (2, 1), "444": (1, 1), "gray": (1, 1)}[mode]
        cw, ch = -(-w // sx), -(-h // sy)
        nb = -(-w // (8 * sx)) * -(-h // (8 * sy)) * sx * sy
        if mode == "gray":
            out, blocks = out + w * h, blocks + nb
            continue
        if case["kind"] == "plane":
            out, blocks = out + nb * 64, blocks + nb
        else:
            planes = w * h + 2 * cw * ch
            out += planes if case.get("out") in ("nv12", "planar") else 3 * w * h
            blocks += nb + 2 * (nb // (sx * sy))
    read = blocks * 128 if case["kind"] == "plane" else sum(len(f) for f in files)
    return {"bytes": read + out, "flops": blocks * 2 * 2 * 512}


def exact(case, seed):
    """Every output is bytes (pixels): there is nothing to compare in 64 bits."""
    return None
