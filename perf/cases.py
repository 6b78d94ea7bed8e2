"""The work a user of the film library has it do, as cases to be timed.

A case is one call sequence through the public entry points (canvaz_film.film,
canvaz_film.deposit, canvaz_film.camera over the C ABI of
include/canvaz_film.h) on canvases made on the GPU from a seed:

  frame    one frame of a canvas stepped alone: a fixed dt (cf_encode_frame),
           dt chosen on the device (cf_step_adaptive), or the program's own
           loop (cf_choose_substeps, cf_update_params, cf_encode_frame)
  batch    one frame of many uneven canvases (cf_batch_step)
  deposit  a frame's strokes binned, copied and laid (cf_upload_deposits,
           cf_lay_deposits)
  lit      the renderer's fragment shader over the film (cf_render_lit)
  relief   the top-down view (cf_render_relief)
  resolve  the display epilogue (cf_resolve)

Canvases are the kinds of canvaz_film.synth (Gaussian blobs, tilted drip
polylines, thick pours), with the same distributions, rasterised with torch so
that making them is quick.  The states a pass steps go on from where the last
pass left them, as a simulation does.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(_ROOT, "paint-sim-3d_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(_ROOT, "paint-sim-3d_gb300"))

from canvaz_film import camera, capi, deposit, synth  # noqa: E402
from canvaz_film.film import Batch, Film  # noqa: E402

PREC = {"ref": capi.CF_PREC_REFERENCE, "fp32": capi.CF_PREC_FP32, "bf16": capi.CF_PREC_BF16}
H_MIN = 1.5e-5  # wet from this height on
CELLS_PER_BLOB = 33_500  # 500 blobs on 4096 x 4096
CELLS_PER_LINE = 21_000  # 200 polylines on 2048 x 2048
CELLS_PER_POUR = 14_000  # 300 pours on 2048 x 2048


def listed():
    return [
        # the smallest canvas that is stepped: a thumbnail or a test swatch
        dict(name="swatch64", kind="frame", field="drips", w=64, h=64, count=6, prec="ref", drive="adaptive", awake=True,
             whole=False),
        # a preview canvas whose whole state is read back after the frame (undo, save)
        dict(name="blobs512_state", kind="frame", field="blobs", w=512, h=512, count=20, prec="fp32", drive="fixed",
             awake=True, whole=True),
        # an odd size, whose rows start on no 16-byte boundary, in the small storage
        dict(name="ragged1021_bf16", kind="frame", field="drips", w=1021, h=765, count=40, prec="bf16", drive="adaptive",
             awake=True, whole=False),
        # the program's default canvas, precision and loop: 1.2 x 0.8 m at 1 mm, implicit steps,
        # several substeps a frame, tiles that fall asleep
        dict(name="app1200x800", kind="frame", field="pours", w=1200, h=800, count=68, prec="ref", drive="app",
             awake=False, whole=False),
        # a steep canvas of drips, dt chosen on the device
        dict(name="drips2048", kind="frame", field="drips", w=2048, h=2048, count=200, prec="fp32", drive="adaptive",
             awake=True, whole=False),
        # the largest canvas: a blob field over a cured ground, in both storages in use
        dict(name="blobs4096", kind="frame", field="blobs", w=4096, h=4096, count=500, prec="fp32", drive="fixed",
             awake=True, whole=False),
        dict(name="blobs4096_bf16", kind="frame", field="blobs", w=4096, h=4096, count=500, prec="bf16", drive="fixed",
             awake=True, whole=False),
        # thick runny paint: every frame takes implicit steps (dt chosen on the device)
        dict(name="pours2048", kind="frame", field="pours", w=2048, h=2048, count=300, prec="fp32", drive="adaptive",
             awake=True, whole=False),
        # uneven canvases served together
        dict(name="batch16", kind="batch", films=16, lo=256, hi=1024, prec="fp32"),
        # a stroke-heavy frame's paint laid on a wet canvas
        dict(name="strokes2048", kind="deposit", w=2048, h=2048, strokes=1024, prec="fp32"),
        # the picture the program shows: the fragment shader at full HD
        dict(name="lit1080p", kind="lit", w=2048, h=2048, vw=1920, vh=1080),
        # the display epilogue with every stage on
        dict(name="resolve2048", kind="resolve", w=2048, h=2048, bloom=0.6, grain=0.03, vignette=0.3, sharpen=0.25),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["batch", "deposit", "lit", "relief", "resolve"])
    if kind == "frame":
        field = rng.choice(["blobs", "blobs", "drips", "drips", "pours"])
        side = _side(rng, 64, 1100 if field == "pours" else 3600)
        a = math.sqrt(rng.uniform(0.5, 2.0))
        w, h = max(48, int(side * a)), max(48, int(side / a))
        per = {"blobs": CELLS_PER_BLOB, "drips": CELLS_PER_LINE, "pours": CELLS_PER_POUR}[field]
        count = max(3, int(w * h / per * rng.uniform(0.5, 2.0)))
        drive = rng.choice(["adaptive", "app"]) if field == "pours" else rng.choice(["fixed", "adaptive"])
        return dict(kind=kind, field=field, w=w, h=h, count=count, prec=rng.choice(["ref", "fp32", "bf16"]), drive=drive,
                    awake=drive != "app", whole=rng.random() < 0.25)
    if kind == "batch":
        lo = _side(rng, 64, 400)
        return dict(kind=kind, films=rng.randint(3, 24), lo=lo, hi=int(lo * rng.uniform(1.5, 3.0)),
                    prec=rng.choice(["ref", "fp32", "bf16"]))
    side = _side(rng, 300, 2048)
    w, h = side, max(64, int(side * rng.uniform(0.6, 1.0)))
    if kind == "deposit":
        return dict(kind=kind, w=w, h=h, strokes=_side(rng, 4, 1024), prec=rng.choice(["ref", "fp32", "bf16"]))
    vw = _side(rng, 160, 1920)
    if kind == "resolve":
        return dict(kind=kind, w=w, h=h, bloom=rng.choice([0.0, rng.uniform(0.1, 1.0)]), grain=rng.uniform(0.0, 0.05),
                    vignette=rng.uniform(0.0, 0.5), sharpen=rng.choice([0.0, rng.uniform(0.1, 0.5)]))
    return dict(kind=kind, w=w, h=h, vw=vw, vh=max(90, int(vw * rng.uniform(0.5, 0.8))))


# ---- canvases ----------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Raster:
    """The height and the height-weighted pigment mix of shapes added one by
    one, and the index of the tallest at each cell."""

    def __init__(self, w, h, pigs):
        d = _dev()
        self.hh = torch.zeros(h, w, dtype=torch.float32, device=d)
        self.best = torch.zeros(h, w, dtype=torch.float32, device=d)
        self.arg = torch.zeros(h, w, dtype=torch.int64, device=d)
        self.num = torch.zeros(h, w, 12, dtype=torch.float32, device=d)
        self.pigs = torch.as_tensor(pigs, dtype=torch.float32, device=d)

    def add(self, k, x0, y0, prof):
        sl = (slice(y0, y0 + prof.shape[0]), slice(x0, x0 + prof.shape[1]))
        self.hh[sl] += prof
        self.num[sl] += prof[:, :, None] * self.pigs[k]
        take = prof > self.best[sl]
        self.best[sl] = torch.where(take, prof, self.best[sl])
        self.arg[sl] = torch.where(take, torch.full_like(self.arg[sl], k), self.arg[sl])


def _window(cx0, cx1, cy0, cy1, w, h):
    return max(int(cx0), 0), min(int(cx1) + 1, w), max(int(cy0), 0), min(int(cy1) + 1, h)


def _rasterise(field, w, h, count, rng):
    if field == "drips":
        pigs = rng.dirichlet(np.full(12, 0.5), count)
        R = _Raster(w, h, pigs)
        sub = (torch.arange(4, device=R.hh.device, dtype=torch.float32) - 1.5) * 0.25
        for k in range(count):
            n, r, h0 = int(rng.integers(2, 7)), rng.uniform(1.0, 4.0), rng.uniform(0.2, 3.0) * 1e-3
            ang, ln = rng.uniform(0, 2 * np.pi, n), rng.uniform(10, 120, n)
            pts = np.concatenate([rng.uniform([0, 0], [w, h])[None], np.stack([ln * np.cos(ang), ln * np.sin(ang)], 1)])
            pts = np.cumsum(pts, 0)
            x0, x1, y0, y1 = _window(pts[:, 0].min() - r - 1, pts[:, 0].max() + r + 1, pts[:, 1].min() - r - 1,
                                     pts[:, 1].max() + r + 1, w, h)
            if x0 >= x1 or y0 >= y1:
                continue
            d = R.hh.device
            px = (torch.arange(x0, x1, device=d, dtype=torch.float32) + 0.5)[None, None, None, :] + sub[None, :, None, None]
            py = (torch.arange(y0, y1, device=d, dtype=torch.float32) + 0.5)[None, None, :, None] + sub[:, None, None, None]
            dist = None
            for s in range(n):
                (ax, ay), (bx, by) = pts[s], pts[s + 1]
                vx, vy = bx - ax, by - ay
                t = (((px - ax) * vx + (py - ay) * vy) / max(vx * vx + vy * vy, 1e-30)).clamp(0.0, 1.0)
                q = torch.sqrt((px - (ax + t * vx)) ** 2 + (py - (ay + t * vy)) ** 2)
                dist = q if dist is None else torch.minimum(dist, q)
            x = dist / r
            R.add(k, x0, y0, torch.where(x < 1.0, h0 * (1.0 - x * x), torch.zeros_like(x)).mean((0, 1)))
        tau, mu = rng.uniform(0.0, 20.0, count), np.exp(rng.uniform(np.log(0.5), np.log(50.0), count))
        return R, tau, mu, rng.uniform(0.6, 1.0, count)
    pour = field == "pours"
    cx, cy = rng.uniform(0, w, count), rng.uniform(0, h, count)
    sg = rng.uniform(8.0 if pour else 5.0, 40.0, count)
    pk = rng.uniform(3.0, 5.0, count) * 1e-3 if pour else rng.uniform(0.1, 2.0, count) * 1e-3
    R = _Raster(w, h, rng.dirichlet(np.full(12, 0.5), count))
    for k in range(count):
        r = 4.0 * sg[k]
        x0, x1, y0, y1 = _window(cx[k] - r, cx[k] + r, cy[k] - r, cy[k] + r, w, h)
        if x0 >= x1 or y0 >= y1:
            continue
        d = R.hh.device
        gx = torch.exp(-((torch.arange(x0, x1, device=d, dtype=torch.float32) + 0.5 - cx[k]) ** 2) / (2 * sg[k] ** 2))
        gy = torch.exp(-((torch.arange(y0, y1, device=d, dtype=torch.float32) + 0.5 - cy[k]) ** 2) / (2 * sg[k] ** 2))
        R.add(k, x0, y0, pk[k] * gy[:, None] * gx[None, :])
    if pour:
        return R, rng.uniform(0.0, 0.3, count), np.exp(rng.uniform(np.log(0.05), np.log(0.2), count)), np.zeros(count)
    tau, mu = rng.uniform(0.0, 20.0, count), np.exp(rng.uniform(np.log(0.5), np.log(50.0), count))
    return R, tau, mu, rng.uniform(0.6, 1.0, count)


def _stored(v, prec):
    """Values the film's pigment storage holds exactly."""
    t = torch.as_tensor(v, dtype=torch.float32, device=_dev())
    return t if prec == "fp32" else (t.half() if prec == "ref" else t.bfloat16()).float()


def _canvas(field, w, h, count, prec, awake, seed):
    """State planes on the device (the layout of cf_state_view), the colour
    tables and the settings of one canvas."""
    rng = np.random.Generator(np.random.PCG64([seed, w, h, count]))
    R, tau, mu, nn = _rasterise(field, w, h, count, rng)
    n, d = w * h, R.hh.device
    hv = torch.where(R.hh >= H_MIN, R.hh, torch.zeros_like(R.hh)).reshape(n)
    wet = hv > 0
    a = R.arg.reshape(n)
    # slot 14 holds ln mu + 10, except that the bf16 storage keeps mu itself
    ln14 = torch.log(_stored(mu, prec).double()).float() + 10.0 if prec == "bf16" else _stored(np.log(mu) + 10.0, prec)
    tau, nn = _stored(tau, prec), _stored(nn, prec)
    pig = torch.zeros(n, 64, dtype=torch.float32, device=d)
    pig[:, :12] = torch.where(wet[:, None], R.num.reshape(n, 12) / R.hh.reshape(n, 1).clamp_min(1e-30), 0.0)
    for slot, v in ((13, tau), (14, ln14), (15, nn)):
        pig[:, slot] = torch.where(wet, v[a], 0.0)
    del R
    strata_h = torch.zeros(n, 4, dtype=torch.float32, device=d)
    strata_h[:, 0] = hv
    mu_c = torch.exp(ln14.double() - 10.0).float()
    planes = {
        "h": hv, "m": torch.full((n,), 5e-5 if field == "blobs" else 0.0, dtype=torch.float32, device=d),
        "rheo": torch.stack([torch.where(wet, mu_c[a], 1.0), torch.where(wet, tau[a], 0.0)], 1).contiguous(),
        "strata_h": strata_h, "strata_pig": pig, "strata_cure": torch.zeros(n, 4, dtype=torch.float32, device=d),
        "sub_refl": torch.as_tensor(synth.substrate(field != "blobs")).to(d).half().repeat(n, 1),
        "lay": torch.zeros(n, dtype=torch.int32, device=d),
    }
    s = dict(width_m=w * 1e-3, height_m=h * 1e-3, rho=1300.0, sigma=0.03, weave_um=0.0, raw_canvas=int(field != "blobs"),
             min_substeps=4 if field == "pours" and not awake else 1, implicit_hydro=int(field == "pours"),
             all_active=int(awake))
    if field == "drips":
        s.update(tilt_deg=60.0, tilt_dir_deg=90.0)
    tables = (synth.reference_tables() if field == "pours"
              else (synth.random_tables(rng), synth.reference_tables()[1]))
    return planes, tables, capi.Settings.default(**s)


def _view(planes, pig_format=capi.CF_PIG_F32):
    v = capi.StateView(pig_format=pig_format, device=1)
    for k, t in planes.items():
        setattr(v, k, t.data_ptr())
    return v


def _film(field, w, h, count, prec, awake, seed):
    planes, tables, st = _canvas(field, w, h, count, prec, awake, seed)
    f = Film(st, w, h, PREC[prec])
    f.set_tables(*tables)
    torch.cuda.synchronize()
    f._check(f.L.cf_write_state(f.p, C.byref(_view(planes))), "cf_write_state")
    return f, st


class _ColorPlane:
    """A film's colour plane where it lies; a tensor made of it keeps the film,
    which owns the memory, alive."""

    def __init__(self, film):
        self.film = film
        ptr, shape, typestr = film.color_device_ptr(), (film.n, 4), "<f2"
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


class _Readback:
    """Where a program keeps what it reads of a film after a frame: the colour
    plane in place, h, and with `whole` all eight state planes."""

    def __init__(self, f, prec, whole):
        n, d = f.n, "cuda"
        self.film = f
        self.out = {"h": torch.zeros(n, device=d)}
        if whole:
            self.out.update(m=torch.zeros(n, device=d), rheo=torch.zeros(n, 2, device=d),
                            strata_h=torch.zeros(n, 4, device=d), strata_cure=torch.zeros(n, 4, device=d),
                            sub_refl=torch.zeros(n, 16, dtype=torch.float16, device=d),
                            lay=torch.zeros(n, dtype=torch.int32, device=d),
                            strata_pig=torch.zeros(n, 64, device=d,
                                                   dtype=torch.float32 if prec == "fp32" else
                                                   torch.float16 if prec == "ref" else torch.bfloat16))
        self.view = _view(self.out, capi.PREC_TO_PIG[PREC[prec]])
        self.color = torch.as_tensor(_ColorPlane(f), device=d)

    def __call__(self):
        f = self.film
        f._check(f.L.cf_read_state_async(f.p, C.byref(self.view), None), "cf_read_state_async")
        return dict(self.out, color=self.color)


# ---- the kinds ---------------------------------------------------------------
def _frame_prepare(c, seed):
    f, _ = _film(c["field"], c["w"], c["h"], c["count"], c["prec"], c["awake"], seed)
    if c["drive"] == "fixed":
        f.update_params(1e-3, 1)
    return {"film": f, "read": _Readback(f, c["prec"], c["whole"])}


def _frame_run(s):
    f, drive = s["film"], s["case"]["drive"]
    if drive == "fixed":
        f.encode_frame(1)
    elif drive == "adaptive":
        f.step_adaptive(1.0 / 60.0)
    else:
        n = f.choose_substeps(1.0 / 60.0)
        f.update_params(1.0 / 60.0, n)
        f.encode_frame(n)
    return s["read"]()


def _batch_sizes(c):
    """Sides spread evenly over the logarithm of the range, multiples of 16 as
    canvases are cut; every fifth one not."""
    n = c["films"]
    out = []
    for k in range(n):
        side = c["lo"] * (c["hi"] / c["lo"]) ** (k / max(n - 1, 1))
        out.append(int(side) + 1 if k % 5 == 4 else max(48, int(round(side / 16.0)) * 16))
    return out


def _batch_count(side):
    return max(3, int(side * side / 14_000))


def _batch_prepare(c, seed):
    b, reads = Batch(), []
    for k, side in enumerate(_batch_sizes(c)):
        f, _ = _film("blobs", side, side, _batch_count(side), c["prec"], True, seed * 64 + k)
        f.update_params(1e-3, 1)
        b.add(f)
        reads.append(_Readback(f, c["prec"], False))
    return {"batch": b, "reads": reads}


def _batch_run(s):
    s["batch"].step(1, 1)
    return [r() for r in s["reads"]]


def _strokes(c, seed):
    """Brush strokes and dabs: radius 1.5-6 cells, 0-40 cells long."""
    rng = np.random.Generator(np.random.PCG64([seed, c["strokes"], c["w"]]))
    n, dx = c["strokes"], 1e-3
    a = rng.uniform(0.01, 0.99, (n, 2)) * [c["w"] * dx, c["h"] * dx]
    ang, ln, r = rng.uniform(0, 2 * np.pi, n), rng.uniform(0, 40, n) * dx, rng.uniform(1.5, 6.0, n) * dx
    b = a + ln[:, None] * np.stack([np.cos(ang), np.sin(ang)], 1)
    pig = np.zeros((n, 16))
    pig[:, :12] = rng.dirichlet(np.full(12, 0.5), n)
    pig[:, 13] = rng.uniform(0.5, 2.0, n)
    method = rng.integers(1, 7, n)
    out = np.zeros(n, deposit.DEPOSIT_DTYPE)
    for k in range(n):
        make = deposit.capsule if k % 3 == 0 else deposit.stroke
        d = make(a[k], b[k], float(r[k]), float(np.pi * r[k] * r[k] * (ln[k] + r[k]) * 0.3), deposit.pack_pig(pig[k]), dx)
        d["kind"] |= int(method[k]) << deposit.METHOD_SHIFT
        out[k] = d
    return out


def _deposit_prepare(c, seed):
    count = max(3, c["w"] * c["h"] // CELLS_PER_BLOB)
    f, _ = _film("blobs", c["w"], c["h"], count, c["prec"], True, seed)
    return {"film": f, "read": _Readback(f, c["prec"], False), "strokes": _strokes(c, seed)}


def _deposit_run(s):
    f = s["film"]
    f.upload_deposits(s["strokes"])
    f.lay_deposits()
    return s["read"]()


def _seen_film(c, seed):
    """A drip canvas a few frames into its run, and the top of its relief."""
    count = max(4, c["w"] * c["h"] // CELLS_PER_LINE)
    f, st = _film("drips", c["w"], c["h"], count, "fp32", True, seed)
    for _ in range(5):
        f.step_adaptive(1.0 / 60.0)
    r = _Readback(f, "fp32", False)
    return f, st, float(r()["h"].max()) + 0.5e-3


def _lit_prepare(c, seed):
    f, st, top = _seen_film(c, seed)
    cam = camera.render_cam(c["w"], c["h"], float(st.width_m), float(st.height_m), top, yaw=0.6 + 0.02 * (seed % 16),
                            aspect=c["vw"] / c["vh"])
    return {"film": f, "cam": cam, "out": torch.zeros(c["vh"], c["vw"], 4, device="cuda")}


def _lit_run(s):
    s["film"].render_lit(s["cam"], s["case"]["vw"], s["case"]["vh"], s["out"].data_ptr())
    return s["out"]


def _relief_prepare(c, seed):
    f, st, _ = _seen_film(c, seed)
    return {"film": f, "pixel": 0.75e-3 * (1.0 + 0.01 * (seed % 7)),
            "out": torch.zeros(c["vh"], c["vw"], 4, dtype=torch.uint8, device="cuda")}


def _relief_run(s):
    s["film"].render_relief(s["out"].data_ptr(), 0.01, 0.01, s["pixel"], s["case"]["vw"], s["case"]["vh"])
    return s["out"]


def _resolve_prepare(c, seed):
    f, _, _ = _seen_film(c, seed)
    return {"film": f, "out": torch.zeros(c["h"], c["w"], 4, dtype=torch.uint8, device="cuda")}


def _resolve_run(s):
    c = s["case"]
    s["film"].resolve(s["out"].data_ptr(), exposure_ev=0.3, bloom=c["bloom"], grain=c["grain"], vignette=c["vignette"],
                      sharpen=c["sharpen"])
    return s["out"]


_KINDS = {"frame": (_frame_prepare, _frame_run), "batch": (_batch_prepare, _batch_run),
          "deposit": (_deposit_prepare, _deposit_run), "lit": (_lit_prepare, _lit_run),
          "relief": (_relief_prepare, _relief_run), "resolve": (_resolve_prepare, _resolve_run)}


def prepare(case, seed):
    return dict(_KINDS[case["kind"]][0](case, seed), case=case)


def run(state):
    return _KINDS[state["case"]["kind"]][1](state)


# ---- what a pass cannot do without --------------------------------------------
def _wet_cells(field, w, h, count):
    """Expected number of wet cells: the mean footprint of a shape, overlapping
    at random."""
    if field == "drips":  # 4 segments of 65 cells, 5 wide
        area = count * 4 * 65 * 5
    else:
        lo, ln = (8.0, 5.6) if field == "pours" else (5.0, 4.05)  # ln(peak / H_MIN) at the mean
        area = count * 2 * math.pi * ln * (40.0 ** 3 - lo ** 3) / (3 * (40.0 - lo))
    return w * h * (1.0 - math.exp(-area / (w * h)))


def _frame_work(field, w, h, count, prec, drive, whole):
    """Every cell's h and colour; of a wet cell also m, the rheology written,
    the front offset, the strata's thicknesses and cure read and written, the
    top pigments and the substrate read.  The implicit steps add, per iteration
    of a wet cell, the mobilities, three vectors read and two written."""
    wet = _wet_cells(field, w, h, count)
    pb = 4 if prec == "fp32" else 2
    rb = 2 if prec == "bf16" else 4
    b = w * h * (4 + 4 + 8) + wet * (4 + 3 * rb + 8 + 32 + 32 + 16 * pb + 32)
    fl = wet * 4 * 80.0  # four faces, about 80 operations each
    if field == "pours":
        b += wet * 40 * (16 + 5 * 4)
        fl += wet * 40 * 30.0
    if whole:
        b += w * h * (4 + 4 + 8 + 16 + 64 * pb + 16 + 32 + 4)
    return b, fl


def work(case):
    c = case
    kind = c["kind"]
    if kind == "frame":
        b, fl = _frame_work(c["field"], c["w"], c["h"], c["count"], c["prec"], c["drive"], c["whole"])
    elif kind == "batch":
        each = [_frame_work("blobs", s, s, _batch_count(s), c["prec"], "fixed", False) for s in _batch_sizes(c)]
        b, fl = sum(x[0] for x in each), sum(x[1] for x in each)
    elif kind == "deposit":
        # painted cells (the mean stroke covers 2 r l + pi r^2), each read and written once, and the h read back
        painted = c["w"] * c["h"] * (1.0 - math.exp(-c["strokes"] * 200.0 / (c["w"] * c["h"])))
        per = 4 + 16 + 16 + 64 * (4 if c["prec"] == "fp32" else 2)
        b, fl = painted * (2 * per + 8) + 8 * c["w"] * c["h"], painted * 16 * 40.0
    elif kind == "resolve":
        b = c["w"] * c["h"] * 12
        fl = c["w"] * c["h"] * (100.0 + (32 * 30.0 if c["bloom"] else 0.0))
    else:
        # h, m, colour (and the detail texel) once, the picture once
        b = c["w"] * c["h"] * (24 if kind == "lit" else 16) + c["vw"] * c["vh"] * (16 if kind == "lit" else 4)
        fl = c["vw"] * c["vh"] * (4000.0 if kind == "lit" else 500.0)
    return {"bytes": b, "flops": fl}


# ---- 64-bit values ------------------------------------------------------------
def _f(x):
    return float(np.float32(x))


def _first_frame(field, w, h, count, prec, drive, seed):
    """h and the rheology after one explicit frame of one substep from a state
    just written, in 64 bits.  No front offsets exist yet, so the contact-line
    terms vanish: nothing wets a dry cell, and the hold level is the one far
    from a front."""
    planes, _, st = _canvas(field, w, h, count, prec, True, seed)
    D = torch.float64
    hh = planes["h"].to(D).reshape(h, w)
    m = planes["m"].to(D).reshape(h, w)
    slot = planes["strata_pig"].to(D)
    mu0, tau0, n0 = (torch.exp(slot[:, 14] - 10.0), slot[:, 13], slot[:, 15])
    if prec == "bf16":
        mu0 = mu0.float().bfloat16().to(D)
    wet = hh > 0
    dx = _f(st.width_m) / w
    tilt, tdir = math.radians(_f(st.tilt_deg)), math.radians(_f(st.tilt_dir_deg))
    g = _f(st.gravity)
    gx, gy, gz = g * math.sin(tilt) * math.cos(tdir), g * math.sin(tilt) * math.sin(tdir), max(g * math.cos(tilt), 0.0)
    gxy = math.hypot(gx, gy)
    rho, sigma = _f(st.rho), _f(st.sigma)
    theta = math.radians(_f(st.contact_angle_deg))
    dt = _f(1e-3)
    if drive == "adaptive":  # the step from the written state's tallest cell and least viscosity
        tall = hh > 4.0 * _f(st.h_min)
        hm = max(float(hh.max()) if bool(tall.any()) else 0.0, 1e-5)
        mm = float(planes["rheo"][:, 0].to(D).reshape(h, w)[tall].min()) if bool(tall.any()) else 1.0
        mm = max(mm, 1e-3)
        dt = _f(1.0 / 60.0)
        speed = min(rho * gxy * hm * hm / mm, _f(st.v_cap))
        if speed > 1e-6:
            dt = min(dt, 0.5 * dx / speed)
        mob = hm ** 3 / (3.0 * mm)
        hyd = rho * gz * min(mob, _f(st.m_cap_hydro))
        if hyd > 0:
            dt = min(dt, 0.2 * dx * dx / hyd)
        cap = 32.0 * sigma * min(mob, _f(st.m_cap))
        if cap > 0:
            dt = min(dt, dx ** 4 / cap)
    m_cap = max(min(_f(st.m_cap), 0.5 * dx ** 4 / (32.0 * sigma * dt)), 1e-14)
    m_hyd = min(0.1 * dx * dx / (dt * rho * max(gz, 0.1)), _f(st.m_cap_hydro))

    # rheology: one stratum, its viscosity and yield stress raised by the cure
    cure = min(_f(st.cure_rate) * dt, 1.0)
    one = lambda v, dry: torch.where(wet, v.reshape(h, w), torch.full_like(hh, dry))  # noqa: E731
    mu = one(mu0 * math.exp(_f(st.lnmu_cure) * cure * cure), 1.0)
    tau = one(tau0 + _f(st.tau_cure) * cure * cure, 0.0)
    n_ = one(torch.where(n0 > 0, n0, torch.full_like(n0, _f(st.n_index))), _f(st.n_index))
    rheo = torch.stack([mu, tau], -1).reshape(-1, 2)
    if prec == "bf16":
        mu, tau, n_ = (v.float().bfloat16().to(D) for v in (mu, tau, n_))

    lc = math.sqrt(sigma / (rho * max(gz, 0.1)))
    hold = 2.0 * lc * math.sin(0.5 * theta) * (1.0 - math.exp(-(math.sqrt(2.0 * 64 * 64) - 0.5) * dx / lc))

    jj, ii = torch.arange(h, device=hh.device), torch.arange(w, device=hh.device)

    def fold(r, size):
        r = torch.where(r < 0, -r - 1, r)
        return torch.where(r >= size, 2 * size - r - 1, r).clamp(0, size - 1)

    def at(v, di, dj):  # the value at (i + di, j + dj), mirrored at the edges
        return v[fold(jj + dj, h)][:, fold(ii + di, w)]

    def out_at(v, di, dj):  # ..., zero outside
        x, y = ii + di, jj + dj
        inside = ((y >= 0) & (y < h))[:, None] & ((x >= 0) & (x < w))[None, :]
        return torch.where(inside, at(v, di, dj), torch.zeros_like(v))

    u = hh + m - torch.where(wet, torch.full_like(hh, hold), torch.zeros_like(hh))
    wa_, wd_ = _f(0.6666667), _f(0.16666667)
    lap = (wa_ * (at(u, -1, 0) + at(u, 1, 0) + at(u, 0, -1) + at(u, 0, 1)) +
           wd_ * (at(u, -1, -1) + at(u, 1, -1) + at(u, -1, 1) + at(u, 1, 1)) - 4.0 * (wa_ + wd_) * u) / dx / dx
    pi_a = 3.0 * sigma * (1.0 - math.cos(theta)) / _f(st.h_star)
    pc = -sigma * lap + pi_a * (1.0 - hh / _f(st.h_star)).clamp_min(0.0) ** 2
    ph = rho * gz * u

    def flux_of(grad, depth, mu, ty, n):  # Herschel-Bulkley
        y = (depth - ty / grad.clamp_min(1e-300)).clamp_min(0.0)
        go = (grad >= 1e-9) & (depth > 0) & (y > 0)
        y1 = torch.where(go, y, torch.ones_like(y))
        g1 = torch.where(go, grad, torch.ones_like(y))
        up = torch.where((n - 1.0).abs() < 1e-4, 0.5 * g1 / mu * y1 * y1,
                         n / (n + 1.0) * (g1 / mu) ** (1.0 / n) * y1 ** ((n + 1.0) / n))
        return torch.where(go, up * (depth - n * y1 / (2.0 * n + 1.0)), torch.zeros_like(y))

    plug = torch.zeros_like(hh)
    gb = rho * gxy
    if gb >= 1e-6:
        q = torch.where(wet, flux_of(torch.full_like(hh, gb), hh, mu.clamp_min(1e-4), tau, n_), torch.zeros_like(hh))
        stiff = (wet & (tau > 0)).to(D)
        win = torch.nn.functional.avg_pool2d(torch.stack([q, hh, stiff])[None], 7, 1, 3, divisor_override=1)[0]
        plug = torch.where(wet & (win[2] > 0.5), win[0] / win[1].clamp_min(1e-300), torch.zeros_like(hh))

    s2 = _f(0.70710678)
    gm = (rho * gx, rho * gy)
    thr = [((out_at(hh, a, b) > 2.0 * hh + _f(st.h_min)).to(D)) for a, b in ((-1, 0), (1, 0), (0, -1), (0, 1))]
    feed = sum(thr).clamp_min(1.0)
    flux = []
    for k, (di, dj) in enumerate(((1, 0), (0, 1), (1, 1), (1, -1))):
        x, y = ii + di, jj + dj
        inside = ((y >= 0) & (y < h))[:, None] & (x < w)[None, :]
        hb = torch.where(inside, at(hh, di, dj), torch.zeros_like(hh))
        live = inside & wet & (hb > 0)
        b_ = lambda v: at(v, di, dj)  # noqa: E731

        def pw(a, c, fb):  # the capillary part of a dry cell is the given cell's
            return torch.where(at(hh, a, c) > 0, at(pc, a, c), fb)

        if k < 2:
            ti, tj = (0, 1) if k == 0 else (1, 0)
            nc, nh = -(b_(pc) - pc) / dx, -(b_(ph) - ph) / dx
            tc = -(pw(ti, tj, pc) + pw(di + ti, dj + tj, b_(pc)) - pw(-ti, -tj, pc) - pw(di - ti, dj - tj, b_(pc))) * 0.25 / dx
            th = -(at(ph, ti, tj) + at(ph, di + ti, dj + tj) - at(ph, -ti, -tj) - at(ph, di - ti, dj - tj)) * 0.25 / dx
            tl = gm if k == 0 else (gm[1], gm[0])
            wgt = wa_
        else:
            nc, nh = -(b_(pc) - pc) / dx * s2, -(b_(ph) - ph) / dx * s2
            tc = -(pw(1, 0, pc) - pw(0, dj, b_(pc))) / dx * s2
            th = -(at(ph, 1, 0) - at(ph, 0, dj)) / dx * s2
            tl = ((gm[0] + gm[1]) * s2, (gm[0] - gm[1]) * s2)
            tl = tl if k == 2 else (tl[1], tl[0])
            wgt = _f(0.23570226)
        hf = 0.5 * (hh + hb)
        hf1 = torch.where(live, hf, torch.ones_like(hf))
        wa = torch.where(live, hh / (hh + hb).clamp_min(1e-300), torch.zeros_like(hf))
        ty = wa * tau + (1.0 - wa) * b_(tau)
        nf = torch.where(n_ == b_(n_), n_, wa * n_ + (1.0 - wa) * b_(n_))
        muf = torch.exp(wa * torch.log(mu.clamp_min(1e-4)) + (1.0 - wa) * torch.log(b_(mu).clamp_min(1e-4)))
        thin = torch.minimum(hh, hb) / hf1
        yx, yy = nc * thin ** 3, tc * thin ** 3
        gl = torch.sqrt(yx * yx + yy * yy)
        sc = torch.where((ty > 0) & (gl > sigma / 1e-6), sigma / 1e-6 / gl.clamp_min(1e-300), torch.ones_like(gl))
        ggx, ggy = yx * sc + nh + tl[0], yy * sc + th + tl[1]
        grad = torch.sqrt(ggx * ggx + ggy * ggy)
        depth = torch.where(ty > 0, torch.where(ggx >= 0, hh, hb), hf)
        q = flux_of(grad, depth, muf, ty, nf)
        meff = torch.where(q > 0, q / grad.clamp_min(1e-9), torch.zeros_like(q))
        gl = math.hypot(*tl)
        mt = (plug * hh if tl[0] >= 0 else b_(plug * hh)) / gl if gl >= 1e-6 else torch.zeros_like(q)
        mt = torch.where(ty > 0, mt, meff)
        qn = mt * tl[0] + meff.clamp_max(m_hyd) * nh + meff.clamp_max(m_cap) * nc * thin ** _f(st.fcap_exp)
        qn = torch.minimum(torch.maximum(qn, -2.0 * hf), 2.0 * hf)
        steep = torch.minimum(hh, hb) < 0.5 * torch.maximum(hh, hb)
        if k < 2:
            qn = torch.where(steep, qn / torch.where(hb > hh, feed, b_(feed)) ** _f(0.7), qn)
        else:
            qn = torch.where(steep, torch.zeros_like(qn), qn)
        flux.append(torch.where(live & ((meff > 0) | (mt > 0)), qn * wgt, torch.zeros_like(qn)))
    back = [out_at(flux[0], -1, 0), out_at(flux[1], 0, -1), out_at(flux[2], -1, -1), out_at(flux[3], -1, 1)]
    out = sum(f.clamp_min(0.0) for f in flux) + sum((-f).clamp_min(0.0) for f in back)
    al = torch.where(out > 0, (0.5 * hh * dx / (dt * out.clamp_min(1e-300))).clamp_max(1.0), torch.ones_like(out))
    div = torch.zeros_like(hh)
    for f, r, (di, dj) in zip(flux, back, ((1, 0), (0, 1), (1, 1), (1, -1))):
        div += torch.where(f < 0, f * at(al, di, dj), f * al)
        div -= torch.where(r < 0, r * al, r * at(al, -di, -dj))
    hn = (hh - dt * div / dx).clamp_min(0.0)
    hn = torch.where((hn < hh) & (hn < 1e-9), torch.zeros_like(hn), hn)
    return hn.reshape(-1), rheo


def _laid(c, seed):
    """h after the strokes: each cell's mean of 4 x 4 samples of every stroke's
    profile, added."""
    count = max(3, c["w"] * c["h"] // CELLS_PER_BLOB)
    hh = _canvas("blobs", c["w"], c["h"], count, c["prec"], True, seed)[0]["h"].double().reshape(c["h"], c["w"])
    dx = _f(_f(c["w"] * 1e-3) / c["w"])
    d = hh.device
    sub = ((torch.arange(4, device=d, dtype=torch.float64) - 1.5) * 0.25)
    for s in _strokes(c, seed):
        (x0, y0), (x1, y1) = s["p0"].astype(float), s["p1"].astype(float)
        r0, r1, h0, kind = float(s["r0"]), float(s["r1"]), float(s["h0"]), int(s["kind"])
        rb = max(r0, r1) + dx
        a0, a1, b0, b1 = _window((min(x0, x1) - rb) / dx, (max(x0, x1) + rb) / dx, (min(y0, y1) - rb) / dx,
                                 (max(y0, y1) + rb) / dx, c["w"], c["h"])
        if a0 >= a1 or b0 >= b1:
            continue
        px = ((torch.arange(a0, a1, device=d) + 0.5)[None, None, None, :] + sub[None, :, None, None]) * dx
        py = ((torch.arange(b0, b1, device=d) + 0.5)[None, None, :, None] + sub[:, None, None, None]) * dx
        qx, qy, ex, ey = px - x0, py - y0, px - x1, py - y1
        l = math.hypot(x1 - x0, y1 - y0)
        if l <= 0.0:
            x = torch.sqrt(qx * qx + qy * qy) / r0
            v = torch.where(x < 1.0, h0 * (1.0 - x * x), torch.zeros_like(x))
        else:
            ux, uy = (x1 - x0) / l, (y1 - y0) / l
            u = qx * ux + qy * uy
            ok = (u >= -r0) & (u <= l + r1)
            dist = (qx * uy - qy * ux).abs()
            if kind & deposit.CAP_START:
                dist = torch.where(u < 0, torch.sqrt(qx * qx + qy * qy), dist)
            else:
                ok &= qx * float(s["n0"][0]) + qy * float(s["n0"][1]) >= 0
            if kind & deposit.CAP_END:
                dist = torch.where(u > l, torch.sqrt(ex * ex + ey * ey), dist)
            else:
                ok &= ex * float(s["n1"][0]) + ey * float(s["n1"][1]) < 0
            rt = r0 + (r1 - r0) * (u / l).clamp(0.0, 1.0)
            x = dist / rt
            v = torch.where(ok & (x < 1.0), h0 * (rt / r0) * (1.0 - x * x), torch.zeros_like(x))
        hh[b0:b1, a0:a1] += v.mean((0, 1))
    return hh.reshape(-1)


def exact(case, seed):
    """h (and the rheology) in 64 bits where a pass is one explicit substep or
    a laying of strokes; a frame of several substeps or implicit steps, the
    colours (held as half floats) and the pictures have none here."""
    c = case
    if c["kind"] == "frame" and c["field"] != "pours":
        hn, rheo = _first_frame(c["field"], c["w"], c["h"], c["count"], c["prec"], c["drive"], seed)
        out = {"h": hn, "color": None}
        if c["whole"]:
            out.update(rheo=rheo, m=None, strata_h=None, strata_cure=None, sub_refl=None, lay=None, strata_pig=None)
        return out
    if c["kind"] == "batch":
        return [{"h": _first_frame("blobs", s, s, _batch_count(s), c["prec"], "fixed", seed * 64 + k)[0], "color": None}
                for k, s in enumerate(_batch_sizes(c))]
    if c["kind"] == "deposit":
        return {"h": _laid(c, seed), "color": None}
    return None
