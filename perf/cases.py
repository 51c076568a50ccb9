"""Performance cases of the imaging framework: what a user's program has it do.

Every case is a call (or the few calls that make up one unit of a user's
work) through the public entry points: the engine (``q_psdm_b200.engine``),
the C ABI that the table generator and the transforms are called through
(``q_psdm_b200._lib``), and the surrogate network (``q_psdm_b200.surrogate``).
Geometries are those of the benchmark configurations (image, spread, trace
length, t* bins, apertures), with seeded positions, data and noise; the
tables are v(z) = v0 + k z traveltimes and t* of a depth-dependent Q.

``exact`` restates each path in 64 bits with torch alone.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from q_psdm_b200 import _lib
from q_psdm_b200 import engine as E
from q_psdm_b200 import surrogate as S
from q_psdm_b200.tables import DESC_DTYPE, LineTables

DEV = "cuda"
DX = 10.0                       # image cell (m) in x, y and z
ORIGIN = (500000.0, 4000000.0)  # survey origin (m), as absolute coordinates have it
SCALED = 0.01                   # SU coordinates in cm (scalco = -100)
DT = 0.002
F3, F4 = 130.0, 140.0
NBINS = 16


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one receiver line of 32 traces of 1000 samples through the real FFT:
        # the smallest call of the library, as a caller's own trace processing makes it
        dict(name="fft_r2c_small", kind="fft", inverse=False, n=1008, batch=32),
        # the inverse transforms of the 16 t* panels of 1024 traces of 3000 samples
        dict(name="fft_c2r_panels", kind="fft", inverse=True, n=6006, batch=16384),
        # drop-in (compat) mode, the small configuration: one gather of 32 x 32
        # receivers from host SU records into one 128 x 100 line, the image read back
        dict(name="compat_small", kind="image", mode="compat", host=True, nxi=128, nzi=100,
             lines=1, nt=1000, shots=1, nrx=32, nry=32, half_x=40, half_y=30, q=60.0,
             v0=2000.0, k=0.6, fpeak=25.0, dtstar=0.0015, g=600.0, table=40, tz=40, reach_x=1000,
             reach_y=500, panels="fp32", kahan=False, uneven=False, dips="constant"),
        # drop-in mode at scale: one gather of 96 x 96 receivers into one 512 x 400 line
        dict(name="compat_gather", kind="image", mode="compat", host=False, nxi=512, nzi=400,
             lines=1, nt=2000, shots=1, nrx=96, nry=96, half_x=200, half_y=100, q=80.0,
             v0=1800.0, k=0.5, fpeak=30.0, dtstar=0.002, g=600.0, table=160, tz=80, reach_x=2500,
             reach_y=1500, panels="fp32", kahan=False, uneven=False, dips="constant"),
        # the plain physics form (FP32 panels, the engine's default form): one
        # gather into one 512 x 400 line
        dict(name="plain_gather", kind="image", mode="plain", host=False, nxi=512, nzi=400,
             lines=1, nt=2000, shots=1, nrx=96, nry=96, half_x=200, half_y=100, q=80.0,
             v0=1800.0, k=0.5, fpeak=30.0, dtstar=0.002, g=600.0, table=160, tz=80, reach_x=2500,
             reach_y=1500, panels="fp32", kahan=False, uneven=False, dips="constant"),
        # the batched form on the small configuration: one gather from host
        # records, the image read back; launches and latency count
        dict(name="batched_small", kind="image", mode="batched", host=True, nxi=128, nzi=100,
             lines=1, nt=1000, shots=1, nrx=32, nry=32, half_x=40, half_y=30, q=60.0,
             v0=2000.0, k=0.6, fpeak=25.0, dtstar=0.0015, g=600.0, table=40, tz=40, reach_x=1000,
             reach_y=500, panels="fp16", kahan=False, uneven=False, dips="constant"),
        # the batched form at scale: two gathers into a brick of four 512 x 400 lines
        dict(name="batched_brick", kind="image", mode="batched", host=False, nxi=512, nzi=400,
             lines=4, nt=2000, shots=2, nrx=96, nry=96, half_x=200, half_y=100, q=80.0,
             v0=1800.0, k=0.5, fpeak=30.0, dtstar=0.002, g=600.0, table=160, tz=80, reach_x=2500,
             reach_y=1500, panels="fp16", kahan=False, uneven=False, dips="constant"),
        # gathers of uneven trace counts and apertures (500 to 12000 traces, 1 to
        # 4 km) into two 768 x 500 lines, compensated sums, dip limits that vary
        dict(name="batched_uneven", kind="image", mode="batched", host=False, nxi=768, nzi=500,
             lines=2, nt=2500, shots=4, nrx=128, nry=128, half_x=400, half_y=200, q=80.0,
             v0=1800.0, k=0.5, fpeak=25.0, dtstar=0.0025, g=600.0, table=160, tz=80, reach_x=2500,
             reach_y=1500, panels="fp16", kahan=True, uneven=True, dips="varied"),
        # the combined form: three gathers of 100 x 100 receivers into a brick of
        # eight 1024 x 600 lines, 40 dB gain limit
        dict(name="batched_large", kind="image", mode="batched", host=False, nxi=1024, nzi=600,
             lines=8, nt=3000, shots=3, nrx=100, nry=100, half_x=200, half_y=100, q=100.0,
             v0=1800.0, k=0.5, fpeak=25.0, dtstar=0.005, g=100.0, table=160, tz=80, reach_x=2500,
             reach_y=1500, panels="fp16", kahan=False, uneven=False, dips="constant"),
        # table generation: a batch of sources on the local grids of a line's
        # tables (+-2.5 km x +-1.5 km, 6 km deep, 50 m nodes)
        dict(name="eikonal_sources", kind="eikonal", nx=111, ny=65, nz=123, h=50.0, sources=32),
        # the surrogate's training: 16 mini-batches of 8192 samples
        dict(name="mlp_train", kind="mlp_train", batch=8192, steps=16),
        # the surrogate's use: gate errors and the dense tables of one 512-cdp line
        # (two tables of 5 million coarse and 17 million fine values)
        dict(name="surrogate_tables", kind="surrogate", nxi=512, nodes=52, coarse=320, fine=160,
             reach_x=2500, reach_y=1500),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fft", "compat", "plain", "batched", "batched", "eikonal", "mlp_train",
                       "surrogate"])
    if kind == "fft":
        n = _npfar(log(200, 12000))
        return dict(kind="fft", inverse=rng.random() < 0.5, n=n,
                    batch=log(1, max(2, 100_000_000 // n)))
    if kind == "eikonal":
        return dict(kind="eikonal", nx=rng.randint(40, 120), ny=rng.randint(30, 90),
                    nz=rng.randint(40, 125), h=rng.choice([20.0, 40.0, 50.0]),
                    sources=log(2, 32))
    if kind == "mlp_train":
        return dict(kind="mlp_train", batch=log(300, 16384), steps=rng.randint(2, 16))
    if kind == "surrogate":
        coarse = rng.choice([200, 320])
        return dict(kind="surrogate", nxi=rng.randint(64, 512), nodes=rng.randint(20, 60),
                    coarse=coarse, fine=coarse // 2, reach_x=rng.randint(800, 2500),
                    reach_y=rng.randint(500, 1500))
    while True:
        nxi, nzi = log(100, 1024), log(60, 600)
        c = dict(kind="image", mode=kind, host=False, nxi=nxi, nzi=nzi,
                 lines=rng.randint(1, 8) if kind == "batched" else rng.randint(1, 2),
                 # drop-in mode images the sample at 2 s: traces reach it
                 nt=log(1000 if kind == "compat" else 600, 3000), shots=rng.randint(1, 4),
                 nrx=log(20, 110), nry=log(10, 110),
                 half_x=min(log(30, 250), nxi), half_y=log(20, 120), q=float(rng.randint(40, 150)),
                 v0=1800.0, k=0.5, fpeak=25.0, dtstar=rng.choice([0.002, 0.003, 0.005]),
                 g=rng.choice([100.0, 600.0]), table=160, tz=80,
                 reach_x=rng.choice([1500, 2500]), reach_y=rng.choice([1000, 1500]),
                 panels="fp16" if kind == "batched" and rng.random() < 0.8 else "fp32",
                 kahan=kind != "compat" and rng.random() < 0.25,
                 uneven=kind == "batched" and rng.random() < 0.3,
                 dips=rng.choice(["constant", "constant", "varied"]))
        c["host"] = c["nrx"] * c["nry"] * c["shots"] <= 3000 and rng.random() < 0.5
        pairs = _pairs(c)
        if 1e5 <= pairs <= {"compat": 2e9, "plain": 1e9, "batched": 1.2e10}[kind]:
            return c


def _npfar(nmin):
    lengths = sorted(a * b * c for a in (1, 2, 4, 8, 16) for b in (1, 3, 9)
                     for c in (x * y * z * w for x in (1, 5) for y in (1, 7) for z in (1, 11)
                               for w in (1, 13)))
    m = (nmin + 1) // 2
    return 2 * next(v for v in lengths if v >= m)


# ---------------------------------------------------------------------------
# imaging: geometry, data, tables
# ---------------------------------------------------------------------------
def _geometry(c, seed):
    """Integer SU coordinates (cm) [ntr][4] and apertures [ntr][2] of the gathers."""
    rng = np.random.default_rng([int(seed), 17])
    wx = c["nxi"] * DX
    ny_line = 0.5 * (c["lines"] - 1) * DX
    # receiver spread over the image in x, and as deep a strip in y as wide
    dr = wx / c["nrx"]
    gx = dr * (0.5 + np.arange(c["nrx"])) + rng.uniform(-0.2, 0.2) * dr
    dry = min(dr, 2.4 * c["half_y"] * DX / c["nry"]) if c["nry"] < c["nrx"] else wx / c["nry"]
    gy = dry * (np.arange(c["nry"]) - 0.5 * (c["nry"] - 1)) + rng.uniform(-0.2, 0.2) * dry
    gxy = np.stack([a.ravel() for a in np.meshgrid(gx, gy, indexing="xy")], 1)
    out, ap = [], []
    for i in range(c["shots"]):
        sx = wx * (i + 1) / (c["shots"] + 1) + rng.uniform(-0.5, 0.5) * DX
        sy = ny_line + rng.uniform(-0.25, 0.25) * min(c["half_y"] * DX, c["reach_y"])
        r = gxy
        hx, hy = c["half_x"], c["half_y"]
        if c["uneven"]:
            # the n receivers nearest to the shot; sizes and apertures spread
            # over their range by shot, so that the work does not depend on the seed
            f = (i + 0.5) / c["shots"]
            n = int((0.03 + 0.7 * f) * len(gxy))
            d2 = ((gxy - (sx, sy)) ** 2).sum(1)
            r = gxy[np.sort(np.argsort(d2, kind="stable")[:max(n, 1)])]
            hx = max(4, int(c["half_x"] * (1.0 - 0.75 * f)))
            hy = max(4, int(c["half_y"] * (1.0 - 0.75 * f)))
        h = np.empty((len(r), 4))
        h[:, 0], h[:, 1], h[:, 2:] = sx, sy, r
        out.append(h)
        ap.append(np.broadcast_to(np.array([hx, hy]), (len(r), 2)))
    h = np.concatenate(out)
    h[:, 0::2] += ORIGIN[0]
    h[:, 1::2] += ORIGIN[1]
    return np.rint(h / SCALED).astype(np.int32), np.concatenate(ap).astype(np.int32)


def _gate(c, hdr, ap, line):
    """(accepted, first column, last column) of every trace for one line."""
    s = hdr.astype(np.float64) * SCALED
    cdpx = np.trunc(((s[:, 0] + s[:, 2]) * 0.5 - ORIGIN[0]) / DX + 0.5).astype(np.int64)
    cdpy = np.trunc(((s[:, 1] + s[:, 3]) * 0.5 - (ORIGIN[1] + line * DX)) / DX + 0.5)
    x1, y1 = ORIGIN[0] + c["nxi"] * DX + 2000.0, ORIGIN[1] + 2048 * DX + 3000.0
    box = ((s[:, 0::2] >= ORIGIN[0] - 2000.0) & (s[:, 0::2] <= x1)).all(1) \
        & ((s[:, 1::2] >= ORIGIN[1] - 22000.0) & (s[:, 1::2] <= y1)).all(1)
    hx, hy = np.minimum(ap[:, 0], c["half_x"]), np.minimum(ap[:, 1], c["half_y"])
    lo, hi = np.maximum(cdpx - hx, 0), np.minimum(cdpx + hx - 1, c["nxi"] - 1)
    return box & (cdpy <= hy) & (cdpy >= -hy) & (hi >= lo), lo, hi


def _pairs(c):
    """Point-traces of a pass (seed 0), without the tables' coverage."""
    hdr, ap = _geometry(c, 0)
    n = 0
    for line in range(c["lines"]):
        ok, lo, hi = _gate(c, hdr, ap, line)
        n += int((hi - lo + 1)[ok].sum()) * c["nzi"]
    return n


def _time(r, z, v0, k):
    arg = 1.0 + k * k * (r * r + z * z) / (2.0 * v0 * (v0 + k * z))
    return torch.acosh(torch.clamp(arg, min=1.0)) / k


def _inv_q(z, q):
    """t* / T of the tables at depth z."""
    return (1.0 + 0.3 * torch.sin(z / 700.0)) / q


def _sizes(c):
    nodes = int((c["nzi"] - 1) * DX // c["tz"]) + 2
    nxs = 2 * -(-c["reach_x"] // c["table"]) + 1
    nys = 2 * -(-c["reach_y"] // c["table"]) + 1
    return -(-c["nxi"] // 16), nodes, nxs, nys


def _tables(c):
    """A line's tables in the engine's layout, [cell][iys][ixs][ixl][node], on the GPU."""
    nxg, nodes, nxs, nys = _sizes(c)
    f8 = dict(dtype=torch.float64, device=DEV)
    xs = (torch.arange(nxs, **f8) - 0.5 * (nxs - 1)) * c["table"]
    ys = (torch.arange(nys, **f8) - 0.5 * (nys - 1)) * c["table"]
    xl = (torch.arange(16, **f8) - 7.5) * DX
    z = torch.arange(nodes, **f8) * c["tz"]
    r = torch.hypot(xs[None, :, None, None] - xl[None, None, :, None], ys[:, None, None, None])
    t = _time(r, z, c["v0"], c["k"])
    q = t * _inv_q(z, c["q"])
    # v(z): every cell has the same values around its own middle
    t, q = (a.float().reshape(1, -1).expand(nxg, -1).contiguous().reshape(-1) for a in (t, q))
    desc = np.zeros(nxg, DESC_DTYPE)
    for i in range(nxg):
        desc[i] = (i * nys * nxs * 16 * nodes, nys, nxs, c["table"], c["table"])
    return t, q, desc


def _engine_tables(c, t, q, desc):
    nxg, nodes, _, _ = _sizes(c)
    d = desc.view(np.uint8).reshape(-1, 16).copy()
    return dict(nxg=nxg, nzg=1, nxi1=16, nzi1=nodes, cdp1=1, cdp2=c["nxi"], ttt_desc=d,
                qqq_desc=d, ttt=t, qqq=q)


def _dips(c):
    """The four dip-limit fields [nxi][nzi]: the reference's constants, or smooth
    limits between about 5 and 15 degrees."""
    contract = math.radians(3.0)
    if c["dips"] == "constant":
        lo, hi = math.tan(-math.radians(10.0) + contract), math.tan(math.radians(10.0) - contract)
        f = np.empty((4, c["nxi"], c["nzi"]), np.float32)
        f[0::2], f[1::2] = lo, hi
        return f
    x = np.arange(c["nxi"])[:, None] / 90.0
    z = np.arange(c["nzi"])[None, :] / 70.0
    a = np.radians(10.0 + 5.0 * np.sin(x + 0.5 * z))
    b = np.radians(9.0 + 4.0 * np.cos(0.7 * x - z))
    return np.tan(np.stack([-a, b, -b, a])).astype(np.float32)


def _traces(c, hdr, seed):
    """Samples [ntr][nt] (float32, GPU): a flat reflector and three diffractors,
    Ricker wavelets attenuated by exp(-pi f t*), noise at 20 dB."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    n, nf = c["nt"], c["nt"] // 2 + 1
    s = torch.from_numpy(hdr.astype(np.float64) * SCALED - np.array(ORIGIN * 2)).to(DEV)
    depth = (c["nzi"] - 1) * DX
    wx = c["nxi"] * DX
    mid = 0.5 * (s[:, :2] + s[:, 2:])
    events = [(mid[:, 0], mid[:, 1], 0.55 * depth, 1.0)] + [
        (wx * a + 0 * mid[:, 0], 0 * mid[:, 0], depth * b, 0.5)
        for a, b in ((0.3, 0.3), (0.5, 0.5), (0.7, 0.8))]
    f = torch.arange(nf, device=DEV, dtype=torch.float32) / (n * DT)
    w = (f / c["fpeak"]) ** 2 * torch.exp(-(f / c["fpeak"]) ** 2) * (2.0 / c["fpeak"] / DT)
    out = torch.empty((len(hdr), n), dtype=torch.float32, device=DEV)
    for a in range(0, len(hdr), 8192):
        b = min(len(hdr), a + 8192)
        spec = torch.zeros((b - a, nf), dtype=torch.complex64, device=DEV)
        for ex, ey, ez, amp in events:
            z = torch.tensor(ez, dtype=torch.float64, device=DEV)
            t = sum(_time(torch.hypot(s[a:b, i] - ex[a:b], s[a:b, i + 1] - ey[a:b]), z, c["v0"],
                          c["k"]) for i in (0, 2))
            q = (t * _inv_q(z, c["q"])).float()
            # the phase in cycles, reduced in double precision before the sine
            cyc = torch.remainder(t[:, None] * f.double(), 1.0).float()
            spec += torch.polar(amp * w * torch.exp(-math.pi * f * q[:, None]),
                                -2.0 * math.pi * cyc)
        tr = torch.fft.irfft(spec, n=n, dim=1)
        rms = tr.square().mean(1, keepdim=True).sqrt() + 1e-30
        out[a:b] = tr + 0.1 * rms * torch.randn(tr.shape, generator=g, device=DEV)
    return out


def _records(hdr, traces):
    """Big-endian SU records (uint8 [ntr][240 + 4 nt], GPU)."""
    ntr, nt = traces.shape
    rec = torch.zeros((ntr, 240 + 4 * nt), dtype=torch.uint8, device=DEV)
    h = np.zeros((ntr, 240), np.uint8)

    def put(off, vals, dt):
        a = np.broadcast_to(np.asarray(vals), (ntr,)).astype(dt)
        h[:, off:off + a.dtype.itemsize] = a.reshape(-1, 1).view(np.uint8)
    put(70, -100, ">i2")
    for i, off in enumerate((72, 76, 80, 84)):
        put(off, hdr[:, i], ">i4")
    put(114, nt, ">u2")
    put(116, int(round(DT * 1e6)), ">u2")
    rec[:, :240] = torch.from_numpy(h).to(DEV)
    rec[:, 240:] = traces.contiguous().view(torch.uint8).reshape(ntr, nt, 4).flip(2) \
        .reshape(ntr, 4 * nt)
    return rec


class _DeviceImage:
    """The engine's image buffer, for torch, zero-copy; keeps the engine alive."""

    def __init__(self, eng, shape):
        self.eng = eng
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", version=3,
                                             data=(eng.image_device_ptr(), False))


def _prepare_image(c, seed):
    hdr, ap = _geometry(c, seed)
    rec = _records(hdr, _traces(c, hdr, seed))
    kw = dict(nxi=c["nxi"], nzi=c["nzi"], ntl=c["nt"], dt=DT, dxi=DX, dyi=DX, dzi=DX,
              scaled=SCALED, fxv=ORIGIN[0], fyv=ORIGIN[1] - 21000.0, nxv=c["nxi"], nyv=4348,
              fc=c["fpeak"], threshold=c["g"], max_batch=len(hdr))
    if c["mode"] != "compat":
        kw.update(mode=1, panel_dtype=2 if c["panels"] == "fp16" else 0, nbins=NBINS,
                  dtstar=c["dtstar"], dzii=float(c["tz"]), kahan=int(c["kahan"]),
                  form=int(c["mode"] == "batched"))
    p = E.static_params(**kw)
    eng = E.Engine(p)
    tab = _engine_tables(c, *_tables(c)) if c["mode"] != "compat" else None
    dips = _dips(c)
    torch.cuda.synchronize()  # the tables are complete before the engine copies them
    eng.set_lines([dict(fxi=ORIGIN[0], cyi=ORIGIN[1] + i * DX, dips=dips, tables=tab)
                   for i in range(c["lines"])])
    off = E.offset_params(p, 0, c["nxi"], aznx1=c["half_x"], aznx2=c["half_x"],
                          azny1=c["half_y"], azny2=c["half_y"])
    st = dict(eng=eng, off=off, ntr=len(hdr), uneven=c["uneven"], host=c["host"])
    if c["host"]:
        st["rec"], st["ap"] = rec.cpu().numpy(), np.ascontiguousarray(ap)
    else:
        st["rec"], st["ap"] = rec, torch.from_numpy(np.ascontiguousarray(ap)).to(DEV)
        eng.begin_offset(off)
        st["img"] = torch.as_tensor(_DeviceImage(eng, eng.image_shape()), device=DEV)
    return st


def _run_image(st):
    """One offset group: the image cleared, the gathers submitted, the image."""
    eng = st["eng"]
    eng.begin_offset(st["off"])
    if st["host"]:
        if st["uneven"]:
            eng.submit_gathers(st["rec"], st["ap"])
        else:
            eng.submit(st["rec"])
        img = eng.get_image()
        return [img] if img.ndim == 2 else list(img)
    if st["uneven"]:
        eng.submit_gathers_device(st["rec"].data_ptr(), st["ap"].data_ptr(), st["ntr"])
    else:
        eng.submit_device(st["rec"].data_ptr(), st["ntr"])
    return list(st["img"])


def _nsb(nt):
    dt = float(np.float32(DT))
    pre, suf = int(0.48 / dt), int(0.36 / dt)
    t11 = float(np.float32(nt - 1) * np.float32(DT))
    f = np.float32
    span = f(f(f(t11) - f(0)) - f(pre) * f(DT)) - f(suf) * f(DT)
    return _npfar(int(float(span) / 2.0 / dt) + pre + suf)


def _panels64(c, tr):
    """t*-binned compensated panels [ntr][16][nffti] in float64."""
    nt = tr.shape[1]
    nfft, nffti = _npfar(nt), _npfar(2 * nt)
    j = torch.arange(nt, device=DEV, dtype=torch.float64)
    t = j * DT
    gain = torch.where(t < 0.1, torch.full_like(t, 0.01), t * t)
    tap = 0.5 - 0.5 * torch.cos(math.pi * torch.arange(200, device=DEV, dtype=torch.float64) / 200)
    gain[:200] *= tap
    gain[-200:] *= tap.flip(0)
    X = torch.fft.rfft(tr.double() * gain, n=nfft)
    nk = nfft // 2 + 1
    df = 1.0 / (nfft * DT)
    f = torch.arange(nk, device=DEV, dtype=torch.float64) * df
    n3, n4 = int(F3 / df + 0.5), int(F4 / df + 0.5)
    k = torch.arange(nk, device=DEV, dtype=torch.float64)
    w = 2.0 * math.pi * df
    ww = torch.where(k < n3, k * w, n3 * w * torch.cos((k - n3) / (n4 - n3) * math.pi * 0.5) ** 2)
    ww = torch.where(k < n4, ww, torch.zeros_like(ww))
    G, lnG = c["g"], math.log(c["g"])
    ts = torch.arange(NBINS, device=DEV, dtype=torch.float64)[:, None] * float(np.float32(c["dtstar"]))
    x = math.pi * f * ts
    a = torch.where(x <= lnG, torch.exp(x.clamp(max=lnG)), torch.where(
        x <= lnG + 0.2, G * (1 - lnG - 2.5 * lnG * lnG) + G * (1 + 5 * lnG) * x - 2.5 * G * x * x,
        torch.full_like(x, 1.1 * G)))
    ph = -2.0 * f * ts * torch.log(f.clamp(min=1e-300) / c["fpeak"])
    F = torch.polar(ww * a, ph) * (-1j) / nfft
    F[:, 0] = 0
    Y = torch.zeros((len(tr), NBINS, nffti // 2 + 1), dtype=torch.complex128, device=DEV)
    Y[:, :, :nk] = X[:, None, :] * F
    return torch.fft.irfft(Y, n=nffti) * nffti


def _exact_line(c, hdr, ap, tr, tab, line):
    """The image of one line in float64."""
    f8 = dict(dtype=torch.float64, device=DEV)
    nxi, nzi = c["nxi"], c["nzi"]
    ok, lo, hi = _gate(c, hdr, ap, line)
    sel = np.nonzero(ok)[0]
    img = torch.zeros((nxi, nzi), **f8)
    if not len(sel):
        return img
    rel = hdr.astype(np.float64) * SCALED - np.array(
        [ORIGIN[0], ORIGIN[1] + line * DX] * 2)
    rel = torch.from_numpy(rel.astype(np.float32).astype(np.float64)).to(DEV)
    lo, hi = (torch.from_numpy(a).to(DEV) for a in (lo, hi))
    W = int((hi - lo + 1)[sel].max())
    dips = torch.from_numpy(_dips(c)).to(DEV).double()
    tz = math.radians(8.0)
    sign = torch.tensor([-1.0, 1.0, -1.0, 1.0], **f8)[:, None, None]
    dipc = dips + sign * tz * (1.0 + dips * dips)
    z = torch.arange(nzi, **f8) * DX
    nffti = _npfar(2 * c["nt"])
    dt1 = _npfar(c["nt"]) * DT / nffti
    compat = c["mode"] == "compat"
    if not compat:
        nxg, nodes, nxs, nys = _sizes(c)
        t32, q32, _ = tab
        TQ = torch.stack([t32, q32], -1).reshape(nxg, nys, nxs, 16, nodes, 2)
        fz = z / c["tz"]
        zi = fz.long()
        wz = (fz - zi)[:, None]
        zj = (zi + 1).clamp(max=nodes - 1)
        wz = torch.where((zi + 1 < nodes)[:, None], wz, torch.zeros_like(wz))

        def look(p, cols):
            """(T, t*) [n][W][nzi][2] and coverage [n][W] of surface points p [n][2]."""
            cell = cols // 16
            xc = (cell * 16 + 7.5) * DX
            fx = (p[:, 0:1] - xc) / c["table"] + 0.5 * (nxs - 1)
            fy = (p[:, 1:2] / c["table"] + 0.5 * (nys - 1)).expand_as(fx)
            cov = (fx >= 0) & (fx <= nxs - 1) & (fy >= 0) & (fy <= nys - 1)
            ix = fx.long().clamp(0, nxs - 2)
            iy = fy.long().clamp(0, nys - 2)
            wx, wy = (fx - ix)[..., None, None], (fy - iy)[..., None, None]
            g = lambda dy, dx: TQ[cell, iy + dy, ix + dx, cols % 16].double()  # noqa: E731
            v = (1 - wy) * ((1 - wx) * g(0, 0) + wx * g(0, 1)) \
                + wy * ((1 - wx) * g(1, 0) + wx * g(1, 1))
            v = (1 - wz) * v[:, :, zi] + wz * v[:, :, zj]
            return v, cov
    step = max(1, int(2.0e7 // (W * nzi)))
    for a in range(0, len(sel), step):
        idx = torch.from_numpy(sel[a:a + step]).to(DEV)
        cols = lo[idx][:, None] + torch.arange(W, device=DEV)
        live = cols <= hi[idx][:, None]
        cols = cols.clamp(max=nxi - 1)
        p = rel[idx]
        x = cols * DX
        dsx, dgx = p[:, 0:1] - x, p[:, 2:3] - x
        ds = torch.sqrt((dsx ** 2 + p[:, 1:2] ** 2)[..., None] + z * z)
        dg = torch.sqrt((dgx ** 2 + p[:, 3:4] ** 2)[..., None] + z * z)
        uz = z / ds + z / dg
        tanx = (dsx[..., None] / ds + dgx[..., None] / dg) / uz
        tany = (p[:, 1, None, None] / ds + p[:, 3, None, None] / dg) / uz
        d, e = dips[:, cols], dipc[:, cols]
        m = live[..., None] & (tanx > e[0]) & (tanx < e[1]) & (tany > e[2]) & (tany < e[3])
        w = torch.ones_like(tanx)
        for v, i in ((tanx, 0), (tany, 2)):
            w = torch.where(v < d[i], w * (v - e[i]) / (d[i] - e[i]), w)
            w = torch.where(v > d[i + 1], w * (e[i + 1] - v) / (e[i + 1] - d[i + 1]), w)
        r = (ds / dg) ** 3
        if compat:
            val = 25.0 * w * (r + 1.0 / r)
        else:
            pan = _panels64(c, tr[idx])
            S_, cs = look(p[:, :2], cols)
            G_, cg = look(p[:, 2:], cols)
            t = S_[..., 0] + G_[..., 0]
            ft = t / dt1
            it = ft.long()
            m = m & (cs & cg)[..., None] & (it > 0) & (it + 1 < nffti)
            it = it.clamp(0, nffti - 2)
            fb = ((S_[..., 1] + G_[..., 1]) / c["dtstar"]).clamp(0, NBINS - 1)
            b = fb.long().clamp(max=NBINS - 2)
            wt, wb = ft - it, fb - b
            at = b * nffti + it
            flat = pan.reshape(len(idx), -1)
            get = lambda o: torch.gather(flat, 1, (at + o).reshape(len(idx), -1)).reshape(at.shape)  # noqa: E731
            p0 = get(0) * (1 - wt) + get(1) * wt
            p1 = get(nffti) * (1 - wt) + get(nffti + 1) * wt
            r = r * G_[..., 0] / S_[..., 0]
            v = torch.where(t > 0.1, 100.0 / (t * t), torch.full_like(t, 10000.0))
            val = w * (r + 1.0 / r) * v * (p0 * (1 - wb) + p1 * wb)
        img.index_add_(0, cols.reshape(-1), torch.where(m, val, torch.zeros_like(val))
                       .reshape(-1, nzi))
    return img


def _exact_image(c, seed):
    pairs = _pairs(c)
    if pairs > 6e10:
        return None
    hdr, ap = _geometry(c, seed)
    tr = _traces(c, hdr, seed)
    tab = _tables(c) if c["mode"] != "compat" else None
    # as many lines as take a few seconds; the others have no value here
    n = max(1, min(c["lines"], int(6e9 // max(1, pairs // c["lines"]))))
    scale = float(_nsb(c["nt"])) if c["host"] else 1.0
    return [_exact_line(c, hdr, ap, tr, tab, i) / scale if i < n else None
            for i in range(c["lines"])]


# ---------------------------------------------------------------------------
# transforms
# ---------------------------------------------------------------------------
def _fft_input(c, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    x = torch.randn((c["batch"], c["n"]), generator=g, device=DEV)
    if not c["inverse"]:
        return x
    return torch.view_as_real(torch.fft.rfft(x)).contiguous()


def _prepare_fft(c, seed):
    x = _fft_input(c, seed)
    m = c["n"] // 2 + 1
    shape = (c["batch"], c["n"]) if c["inverse"] else (c["batch"], m, 2)
    return dict(x=x, y=torch.empty(shape, dtype=torch.float32, device=DEV), c=c,
                call=_lib.lib().qpsdm_fft_c2r if c["inverse"] else _lib.lib().qpsdm_fft_r2c)


def _run_fft(st):
    c = st["c"]
    _lib.check(st["call"](st["x"].data_ptr(), c["n"], c["batch"], st["y"].data_ptr(), None),
               what="fft")
    return st["y"]


def _exact_fft(c, seed):
    x = _fft_input(c, seed).double()
    if c["inverse"]:
        return torch.fft.irfft(torch.view_as_complex(x), n=c["n"]) * c["n"]
    return torch.view_as_real(torch.fft.rfft(x))


# ---------------------------------------------------------------------------
# table generation: traveltime and t* of a batch of surface sources
# ---------------------------------------------------------------------------
def _eikonal_input(c, seed):
    """A v0 + kz z model with a slow cloud of low Q, and sources on its surface."""
    rng = np.random.default_rng([int(seed), 23])
    h, hm = c["h"], c["h"]
    nx, ny, nz = c["nx"] + 24, c["ny"] + 16, c["nz"]
    ax = [torch.arange(n, dtype=torch.float32, device=DEV) * hm for n in (nz, ny, nx)]
    Z, Y, X = torch.meshgrid(*ax, indexing="ij")
    ext = [(nx - 1) * hm, (ny - 1) * hm, (nz - 1) * hm]
    cen = rng.uniform(0.35, 0.65, 3) * ext
    rad = rng.uniform(0.15, 0.25, 3) * ext
    rho2 = ((X - cen[0]) / rad[0]) ** 2 + ((Y - cen[1]) / rad[1]) ** 2 + ((Z - cen[2]) / rad[2]) ** 2
    w = torch.exp(-rho2)
    vel = ((1800.0 + 0.5 * Z) * (1.0 - 0.2 * w)).contiguous()
    invq = (0.01 + 0.04 * w).contiguous()
    src = np.zeros((c["sources"], 4), np.float32)
    # on a 0.5 m lattice, anywhere above the model's middle: every coordinate exact
    gx, gy = (c["nx"] - 1) * h, (c["ny"] - 1) * h
    src[:, 0] = np.rint(2.0 * (rng.uniform(0, 23 * h, c["sources"]) + 0.5 * gx)) * 0.5
    src[:, 1] = np.rint(2.0 * (rng.uniform(0, 15 * h, c["sources"]) + 0.5 * gy)) * 0.5
    src[:, 2] = src[:, 0] - 0.5 * gx
    src[:, 3] = src[:, 1] - 0.5 * gy
    return vel, invq, (nx, ny, nz, hm), torch.from_numpy(src).to(DEV)


def _prepare_eikonal(c, seed):
    vel, invq, (nx, ny, nz, hm), src = _eikonal_input(c, seed)
    n = c["nx"] * c["ny"] * c["nz"] * c["sources"]
    f4 = dict(dtype=torch.float32, device=DEV)
    return dict(vel=vel, invq=invq, model=_lib.EikModel(nx, ny, nz, hm, 0.0, 0.0, 1800.0, 0.5),
                src=src, grid=_lib.EikGrid(c["nx"], c["ny"], c["nz"], c["h"]), c=c,
                work=torch.empty(4 * n + 4, **f4),
                T=torch.empty((c["sources"], c["nz"], c["ny"], c["nx"]), **f4),
                S=torch.empty((c["sources"], c["nz"], c["ny"], c["nx"]), **f4))


def _run_eikonal(st):
    c = st["c"]
    rc = _lib.lib().qpsdm_eikonal_solve(
        st["vel"].data_ptr(), st["invq"].data_ptr(), C.byref(st["model"]), st["src"].data_ptr(),
        c["sources"], C.byref(st["grid"]), 3.0 * c["h"], 4 * (c["nx"] + c["ny"] + c["nz"]),
        st["work"].data_ptr(), st["T"].data_ptr(), st["S"].data_ptr(), None)
    _lib.check(rc, what="eikonal_solve")
    return [st["T"], st["S"]]


def _trilinear(g, hm, x, y, z):
    out = 0.0
    w, i = [], []
    for a, n in ((x, g.shape[2]), (y, g.shape[1]), (z, g.shape[0])):
        f = (a / hm).clamp(0.0, n - 1.0)
        j = f.long().clamp(max=n - 2)
        w.append(f - j)
        i.append(j)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                out = out + g[i[2] + dz, i[1] + dy, i[0] + dx] \
                    * (w[0] if dx else 1 - w[0]) * (w[1] if dy else 1 - w[1]) \
                    * (w[2] if dz else 1 - w[2])
    return out


def _exact_eikonal(c, seed):
    """The fixed point of the first-order upwind scheme, relaxed in float64."""
    vel, invq, (_, _, _, hm), src = _eikonal_input(c, seed)
    vel, invq, src, h = vel.double(), invq.double(), src.double(), c["h"]
    T_out, S_out = [], []
    inf = 1e30
    f8 = dict(dtype=torch.float64, device=DEV)
    per = max(1, int(6e7 // (c["nx"] * c["ny"] * c["nz"])))
    for a in range(0, c["sources"], per):
        s = src[a:a + per][:, :, None, None, None]
        x = s[:, 2] + torch.arange(c["nx"], **f8)[None, None, None, :] * h
        y = s[:, 3] + torch.arange(c["ny"], **f8)[None, None, :, None] * h
        z = torch.arange(c["nz"], **f8)[None, :, None, None] * h
        x, y, z = torch.broadcast_tensors(x, y, z)
        v = _trilinear(vel, hm, x, y, z)
        q = _trilinear(invq, hm, x, y, z)
        r2 = (x - s[:, 0]) ** 2 + (y - s[:, 1]) ** 2
        start = r2 + z * z <= (3.0 * h) ** 2
        t0 = _time(torch.sqrt(r2), z, 1800.0, 0.5)
        qs = _trilinear(invq, hm, s[:, 0], s[:, 1], 0 * s[:, 0])
        T = torch.where(start, t0, torch.full_like(t0, inf))
        St = torch.where(start, t0 * qs, torch.zeros_like(t0))
        f = h / v
        qf = q / (v * v)

        def near(A, d, fill):
            lo = torch.full_like(A, fill)
            hi = torch.full_like(A, fill)
            n = A.shape[d]
            lo.narrow(d, 1, n - 1).copy_(A.narrow(d, 0, n - 1))
            hi.narrow(d, 0, n - 1).copy_(A.narrow(d, 1, n - 1))
            return lo, hi
        for it in range(4 * (c["nx"] + c["ny"] + c["nz"])):
            m = [torch.minimum(*near(T, d, inf)) for d in (3, 2, 1)]
            t0_ = torch.minimum(torch.minimum(m[0], m[1]), m[2])
            t2_ = torch.maximum(torch.maximum(m[0], m[1]), m[2])
            t1_ = torch.minimum(torch.maximum(m[0], m[1]),
                                torch.maximum(torch.minimum(m[0], m[1]), m[2]))
            t = t0_ + f
            two = 0.5 * (t0_ + t1_ + torch.sqrt((2 * f * f - (t0_ - t1_) ** 2).clamp(min=0)))
            use2 = (t > t1_) & (t1_ < inf)
            t = torch.where(use2, two, t)
            s3 = t0_ + t1_ + t2_
            three = (s3 + torch.sqrt((s3 * s3 - 3 * (t0_ * t0_ + t1_ * t1_ + t2_ * t2_ - f * f))
                                     .clamp(min=0))) / 3
            t = torch.where(use2 & (t > t2_) & (t2_ < inf), three, t)
            new = torch.where(start | (t0_ >= inf), T, torch.minimum(T, t))
            if it % 16 == 15 and not bool((new < T * (1 - 1e-13)).any()):
                T = new
                break
            T = new
        num_w, den = [], 0.0
        for d in (3, 2, 1):
            lo, hi = near(T, d, inf)
            best = torch.minimum(lo, hi)
            wgt = torch.where(best < T, (T - best) / (h * h), torch.zeros_like(T))
            num_w.append((d, lo <= hi, wgt))
            den = den + wgt
        free = ~start & (den > 0)
        for it in range(4 * (c["nx"] + c["ny"] + c["nz"])):
            num = qf
            for d, low, wgt in num_w:
                lo, hi = near(St, d, 0.0)
                num = num + wgt * torch.where(low, lo, hi)
            new = torch.where(free, num / den.clamp(min=1e-300), St)
            if it % 16 == 15 and not bool(((new - St).abs() > 1e-13 * new.abs()).any()):
                St = new
                break
            St = new
        T_out.append(T)
        S_out.append(St)
    return [torch.cat(T_out), torch.cat(S_out)]


# ---------------------------------------------------------------------------
# the surrogate network
# ---------------------------------------------------------------------------
HID = 128


def _weights(seed, out_scale):
    """Parameters in the library's order, and as (W, b) pairs."""
    rng = np.random.default_rng([int(seed), 31])
    dims = [(HID, 16, 5), (HID, HID, HID), (HID, HID, HID), (HID, HID, HID), (16, HID, HID)]
    flat, mats = [], []
    for i, (o, k, live) in enumerate(dims):
        w = np.zeros((o, k), np.float32)
        rows = 2 if i == 4 else o
        gain = out_scale / math.sqrt(live) if i == 4 else math.sqrt(2.0 / live)
        w[:rows, :live] = rng.standard_normal((rows, live)) * gain
        flat += [w.ravel(), np.zeros(o, np.float32)]
        mats.append((torch.from_numpy(w[:rows, :live].astype(np.float64)).to(DEV),
                     torch.zeros(rows, dtype=torch.float64, device=DEV)))
    return np.concatenate(flat), mats


def _net64(mats, x, shift, scale):
    h = (x.double() - shift) * scale
    for w, b in mats[:-1]:
        h = torch.nn.functional.silu(h @ w.T + b)
    return h @ mats[-1][0].T + mats[-1][1]


SHIFT = np.array([4000.0, 2000.0, 4000.0, 2000.0, 2500.0], np.float32)
SCALE = (1.0 / np.array([4000.0, 2000.0, 4000.0, 2000.0, 2500.0])).astype(np.float32)
W_OUT = (1.0, 25.0)
LR = 5e-4


def _samples(c, seed, steps):
    """Mini-batches (x [steps][batch][5], t [steps][batch][2]) of smooth corrections."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    x = torch.rand((steps, c["batch"], 5), generator=g, device=DEV)
    x = x * torch.from_numpy(2.0 / SCALE).to(DEV)
    u = (x - torch.from_numpy(SHIFT).to(DEV)) * torch.from_numpy(SCALE).to(DEV)
    r = torch.hypot(u[..., 0] - u[..., 2], u[..., 1] - u[..., 3])
    t = torch.stack([2.0 * torch.sin(2.0 * u[..., 2] + r) * (1.0 + u[..., 4]),
                     0.2 * torch.cos(1.5 * u[..., 0] - u[..., 4]) * (1.0 + r)], -1)
    return x.contiguous(), t.contiguous()


def _prepare_mlp_train(c, seed):
    net = S.Mlp(params=_weights(seed, 0.1)[0])
    net.set_scaling(SHIFT, SCALE, W_OUT)
    x, t = _samples(c, seed, c["steps"] + 8)
    for i in range(8):  # a run in progress: the optimiser's moments are not those of a first step
        net.train_step(x[i], t[i], 1e-9)
    return dict(net=net, x=x[8:], t=t[8:], steps=c["steps"])


def _run_mlp_train(st):
    net = st["net"]
    for i in range(st["steps"]):
        net.train_step(st["x"][i], st["t"][i], LR)
    return net.params()


def _exact_mlp_train(c, seed):
    mats = _weights(seed, 0.1)[1]
    x, t = _samples(c, seed, c["steps"] + 8)
    shift, scale = (torch.from_numpy(a).to(DEV).double() for a in (SHIFT, SCALE))
    wo = torch.tensor(W_OUT, dtype=torch.float64, device=DEV)
    par = [p.requires_grad_() for m in mats for p in m]
    mom = [(torch.zeros_like(p), torch.zeros_like(p)) for p in par]
    for i in range(c["steps"] + 8):
        lr = 1e-9 if i < 8 else LR
        y = _net64(mats, x[i], shift, scale)
        loss = (wo * (y - t[i].double()) ** 2).sum() / c["batch"]
        grads = torch.autograd.grad(loss, par)
        with torch.no_grad():
            for p, g, (m, v) in zip(par, grads, mom):
                m.mul_(0.9).add_(g, alpha=0.1)
                v.mul_(0.999).addcmul_(g, g, value=0.001)
                p -= lr * (m / (1 - 0.9 ** (i + 1))) / ((v / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
    out = []
    for i, (w, b) in enumerate(mats):
        full = torch.zeros((16 if i == 4 else HID, 16 if i == 0 else HID), dtype=torch.float64,
                           device=DEV)
        full[:w.shape[0], :w.shape[1]] = w.detach()
        fb = torch.zeros(full.shape[0], dtype=torch.float64, device=DEV)
        fb[:len(b)] = b.detach()
        out += [full.reshape(-1), fb]
    return torch.cat(out)


def _sur_geometry(c, spacing):
    nxg = -(-c["nxi"] // 16)
    nxs = 2 * -(-c["reach_x"] // spacing) + 1
    nys = 2 * -(-c["reach_y"] // spacing) + 1
    return nxg, nxs, nys


def _features(c, spacing):
    """(px, py, x, y, z) of every table value [cell][iys][ixs][16][nodes], float64."""
    nxg, nxs, nys = _sur_geometry(c, spacing)
    f8 = dict(dtype=torch.float64, device=DEV)
    cell = torch.arange(nxg, **f8)
    xc = (cell * 16 + 7.5) * DX
    px = xc[:, None] + (torch.arange(nxs, **f8) - 0.5 * (nxs - 1)) * spacing
    py = LINE_Y + (torch.arange(nys, **f8) - 0.5 * (nys - 1)) * spacing
    x = (cell[:, None] * 16 + torch.arange(16, **f8)) * DX
    z = torch.arange(c["nodes"], **f8) * 80.0
    return px, py, x, z


LINE_Y = 2000.0
BG = S.Background(1800.0, 0.5, 80.0)


def _corrections(px, py, x, z, amp):
    """Smooth corrections (ms) of T and t* as an eikonal model gives them: near
    the network's where amp is small, beyond the gate around one patch."""
    u, v = (px - x) / 2500.0, (py - LINE_Y) / 1500.0
    bump = torch.exp(-((x - 1500.0) / 600.0) ** 2 - ((z - 1200.0) / 500.0) ** 2)
    t = 0.3 * torch.sin(u + 0.5 * v) * torch.cos(z / 1500.0) + amp * bump * (1.0 + 0.5 * u)
    return t, 0.02 * t


def _grid5(c, spacing):
    px, py, x, z = _features(c, spacing)
    return torch.broadcast_tensors(px[:, None, :, None, None], py[None, :, None, None, None],
                                   x[:, None, None, :, None], z)


def _coarse_tables(c, seed):
    amp = 3.0 + np.random.default_rng([int(seed), 41]).uniform(-0.5, 0.5)
    PX, PY, X, Z = _grid5(c, c["coarse"])
    tb = _time(torch.hypot(PX - X, PY - LINE_Y), Z, BG.v0, BG.kz)
    t, q = _corrections(PX, PY, X, Z, amp)
    return (tb + 1e-3 * t).float().reshape(-1), (tb / BG.q_ref + 1e-3 * q).float().reshape(-1)


def _prepare_surrogate(c, seed):
    net = S.Mlp(params=_weights(seed, 0.2)[0])
    net.set_scaling(SHIFT, SCALE, W_OUT)
    t, q = _coarse_tables(c, seed)
    nxg, nxs, nys = _sur_geometry(c, c["coarse"])
    desc = np.zeros(nxg, DESC_DTYPE)
    for i in range(nxg):
        desc[i] = (i * nys * nxs * 16 * c["nodes"], nys, nxs, c["coarse"], c["coarse"])
    # the data live on the GPU, as the table generator leaves them
    tab = LineTables(1, c["nxi"], DX, 8.0, nxg, 1, 16, c["nodes"], 80.0, desc,
                     np.zeros(0, np.float32), np.zeros(0, np.float32), dict(ttt=t, qqq=q))
    return dict(sur=S.Surrogate(net, BG, []), tab=tab, c=c)


def _run_surrogate(st):
    c, tab = st["c"], st["tab"]
    err = S.gate_errors(st["sur"], [tab], [LINE_Y])
    dense, _ = S.dense_tables_device(st["sur"], tab, tab.dev["ttt"], tab.dev["qqq"], err, fci=1,
                                     line_y=LINE_Y, surf_dx=c["fine"], surf_dy=c["fine"],
                                     half_x=float(c["reach_x"]), half_y=float(c["reach_y"]))
    return [err, dense["ttt"], dense["qqq"]]


def _exact_surrogate(c, seed):
    mats = _weights(seed, 0.2)[1]
    shift, scale = (torch.from_numpy(a).to(DEV).double() for a in (SHIFT, SCALE))

    def net(spacing):
        PX, PY, X, Z = _grid5(c, spacing)
        shape = torch.broadcast_shapes(PX.shape, Z.shape)
        out = torch.empty(shape + (2,), dtype=torch.float64, device=DEV)
        for i in range(shape[0]):
            F = torch.stack([a[i].reshape(-1) for a in (PX, PY, X, 0 * X + LINE_Y, Z)], -1).float()
            tb = _time(torch.hypot(PX[i] - X[i], PY[i] - LINE_Y), Z[i], BG.v0, BG.kz)
            y = _net64(mats, F, shift, scale).reshape(shape[1:] + (2,))
            out[i, ..., 0] = tb + 1e-3 * y[..., 0]
            out[i, ..., 1] = tb / BG.q_ref + 1e-3 * y[..., 1]
        return out
    nxg, nxs, nys = _sur_geometry(c, c["coarse"])
    t, q = (a.double().reshape(nxg, nys, nxs, 16, c["nodes"]) for a in _coarse_tables(c, seed))
    err = (net(c["coarse"])[..., 0] - t).abs().amax((3, 4)) * 1e3
    fine = net(c["fine"])
    _, fxs, fys = _sur_geometry(c, c["fine"])
    f8 = dict(dtype=torch.float64, device=DEV)
    fx = ((torch.arange(fxs, **f8) - 0.5 * (fxs - 1)) * c["fine"] / c["coarse"]
          + 0.5 * (nxs - 1)).clamp(0, nxs - 1)
    fy = ((torch.arange(fys, **f8) - 0.5 * (fys - 1)) * c["fine"] / c["coarse"]
          + 0.5 * (nys - 1)).clamp(0, nys - 1)
    ix, iy = fx.long().clamp(max=nxs - 2), fy.long().clamp(max=nys - 2)
    wx, wy = (fx - ix)[None, None, :, None, None], (fy - iy)[None, :, None, None, None]
    at = lambda a, dy, dx: a[:, iy + dy][:, :, ix + dx]  # noqa: E731
    worst = torch.stack([at(err, dy, dx) for dy in (0, 1) for dx in (0, 1)]).amax(0)
    out = [err.reshape(-1)]
    for k, tab in enumerate((t, q)):
        bil = (1 - wy) * ((1 - wx) * at(tab, 0, 0) + wx * at(tab, 0, 1)) \
            + wy * ((1 - wx) * at(tab, 1, 0) + wx * at(tab, 1, 1))
        out.append(torch.where((worst > 2.0)[..., None, None], bil, fine[..., k]).reshape(-1))
    return out


# ---------------------------------------------------------------------------
def prepare(case, seed):
    return case["kind"], {"image": _prepare_image, "fft": _prepare_fft,
                          "eikonal": _prepare_eikonal, "mlp_train": _prepare_mlp_train,
                          "surrogate": _prepare_surrogate}[case["kind"]](case, seed)


def run(state):
    kind, st = state
    return {"image": _run_image, "fft": _run_fft, "eikonal": _run_eikonal,
            "mlp_train": _run_mlp_train, "surrogate": _run_surrogate}[kind](st)


def exact(case, seed):
    return {"image": _exact_image, "fft": _exact_fft, "eikonal": _exact_eikonal,
            "mlp_train": _exact_mlp_train,
            "surrogate": _exact_surrogate}[case["kind"]](case, seed)


def work(case):
    c = case
    if c["kind"] == "fft":
        n, b = c["n"], c["batch"]
        return dict(bytes=4.0 * b * (2 * n + 2), flops=2.5 * b * n * math.log2(n))
    if c["kind"] == "eikonal":
        n = c["nx"] * c["ny"] * c["nz"] * c["sources"]
        model = (c["nx"] + 24) * (c["ny"] + 16) * c["nz"]
        # one traveltime and one t* update a node, both fields written once
        return dict(bytes=8.0 * n + 8.0 * model, flops=80.0 * n)
    if c["kind"] == "mlp_train":
        # forward, and two gradients of each layer
        n = c["batch"] * c["steps"]
        return dict(bytes=28.0 * n + 4.0 * 53776 * 6 * c["steps"], flops=3.0 * 100096 * n)
    if c["kind"] == "surrogate":
        n = [int(np.prod(_sur_geometry(c, s))) * 16 * c["nodes"] for s in (c["coarse"], c["fine"])]
        return dict(bytes=8.0 * (n[0] + n[1]), flops=100096.0 * (n[0] + n[1]))
    hdr, _ = _geometry(c, 0)
    pts = c["lines"] * c["nxi"] * c["nzi"]
    b = len(hdr) * (240.0 + 4 * c["nt"]) + 20.0 * pts
    if c["mode"] != "compat":
        nxg, nodes, nxs, nys = _sizes(c)
        b += 8.0 * c["lines"] * nxg * nys * nxs * 16 * nodes
    nffti = _npfar(2 * c["nt"])
    fft = len(hdr) * 2.5 * nffti * math.log2(nffti) * (0.5 if c["mode"] == "compat" else NBINS + 0.5)
    return dict(bytes=b, flops=_pairs(c) * (35.0 if c["mode"] == "compat" else 64.0) + fft)
