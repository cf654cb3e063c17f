"""The work that users of this framework have it do, as timed cases.

Five kinds of call, through the C ABI (include/smip_gpu.h) or the Python
layer over it:

* ``acc``   -- a stack of frames into the accumulators, and the four results of
  it: shifts, shift-and-add sum, power spectrum, packed bispectrum.  Frames lie
  in device memory, in page-locked or in ordinary host memory; the bispectrum
  comes back into a page-locked buffer that the program keeps.
* ``fft``   -- spectra computed elsewhere into the bispectrum accumulator.
* ``reco``  -- phase recovery from a bispectrum that the stack holds.
* ``job``   -- a whole job: frames in, image and phase map out.  The program
  keeps its results in single precision, as an image file does.
* ``shift`` -- one frame's shift without any allocation (an acquisition loop).

Frames are speckle images: an object seen through a random Kolmogorov screen
with image motion, photon and read noise, quantised to the frame type
(floating frames: bias subtracted, so that some pixels are below zero).
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "speckle-stacker_gb300"))

import smip_gb300 as G  # noqa: E402

CODES = {"u8": G.U8, "u16": G.U16, "f32": G.F32, "f64": G.F64}
NUMPY = {"u8": np.uint8, "u16": np.uint16, "f32": np.float32, "f64": np.float64}


# --------------------------------------------------------------------- cases
def listed():
    return [
        # an acquisition loop asks for each frame's shift as it arrives: the smallest call
        {"name": "shift_64", "kind": "shift", "w": 64, "h": 64},
        # the smallest of a queue of jobs: 50 small frames straight from a reader's memory
        {"name": "acc_64_u8", "kind": "acc", "w": 64, "h": 64, "d": 16, "n": 50, "dtype": "u8", "source": "host"},
        # a whole small job, frames to image: 40 frames of a binary star
        {"name": "job_128_u8", "kind": "job", "w": 128, "h": 128, "d": 32, "r": 64, "n": 40, "dtype": "u8"},
        # a crop of no special size at the command line's default depth
        {"name": "acc_100_u8", "kind": "acc", "w": 100, "h": 100, "d": 20, "n": 200, "dtype": "u8", "source": "pinned"},
        # calibrated (bias-subtracted) frames are floating; both axes odd
        {"name": "acc_99x75_f32", "kind": "acc", "w": 99, "h": 75, "d": 14, "n": 150, "dtype": "f32", "source": "device"},
        # a camera's own frame size
        {"name": "acc_640x480_u16", "kind": "acc", "w": 640, "h": 480, "d": 20, "n": 200, "dtype": "u16", "source": "device"},
        # the ordinary large job, frames resident on the device
        {"name": "acc_256_u16", "kind": "acc", "w": 256, "h": 256, "d": 32, "n": 2000, "dtype": "u16", "source": "device"},
        # a large extended object, the deepest bispectrum in ordinary use; frames from page-locked memory
        {"name": "acc_512_u16", "kind": "acc", "w": 512, "h": 512, "d": 48, "n": 500, "dtype": "u16", "source": "pinned"},
        # a program with its own transforms hands over spectra
        {"name": "fft_256", "kind": "fft", "w": 256, "h": 256, "d": 32, "n": 64},
        # phase recovery of the small, the ordinary and the large object
        {"name": "reco_128", "kind": "reco", "w": 128, "h": 128, "d": 24, "r": 48},
        {"name": "reco_256", "kind": "reco", "w": 256, "h": 256, "d": 32, "r": 128},
        {"name": "reco_512", "kind": "reco", "w": 512, "h": 512, "d": 48, "r": 200},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["acc", "acc", "acc", "reco", "reco", "job", "fft", "shift"])
    if kind == "shift":  # powers of two up to 256 a side
        return {"kind": kind, "w": rng.choice([16, 32, 64, 128, 256]), "h": rng.choice([16, 32, 64, 128, 256])}
    if rng.random() < 0.5:  # powers of two
        w = rng.choice([64, 128, 256, 512])
        h = w if rng.random() < 0.7 else rng.choice([64, 128, 256, 512])
    else:
        w = _log(rng, 48, 640)
        h = w if rng.random() < 0.4 else _log(rng, 48, 512)
    d = rng.randint(8, max(9, min(48, min(w, h) // 2)))
    c = {"kind": kind, "w": w, "h": h, "d": d}
    if kind in ("reco", "job"):  # within the largest listed walk's number of points and pairs
        top = min(min(w, h) / 2, 200, 128 if kind == "job" else 200)
        c["r"] = min(_log(rng, 16, max(17, top)), int(math.sqrt(200 * 200 * 49 * 49) / (d // 2 * 2 + 1)))
    if kind in ("acc", "job", "fft"):
        most = 1.0e12 / (14.0 * triples(w, h, d))
        pixels = 3.0e8 if kind != "fft" else 1.0e8
        c["n"] = max(4, min(_log(rng, 16, 2000 if kind == "acc" else 400), int(most), int(pixels / (w * h))))
    if kind in ("acc", "job"):
        c["dtype"] = rng.choice(["u8", "u16", "u16", "f32", "f64"])
    if kind == "acc":
        c["source"] = rng.choice(["device", "pinned", "host"])
    return c


# ---------------------------------------------------------------------- work
def triples(w, h, d):
    """Products F(u) F(v) conj F(u+v) of one frame."""
    e = d // 2
    rows = sum(w // 2 + 1 - a for a in range(e + 1))
    cols = sum(h - abs(l) for l in range(-e, e + 1))
    return rows * cols


def visits(r):
    """About how many points the spiral of radius r passes."""
    return math.pi * r * r


def work(case):
    w, h = case["w"], case["h"]
    px, kind = w * h, case["kind"]
    fft = 2.5 * px * math.log2(px)  # one real transform
    if kind == "shift":
        return {"bytes": 16 * px + 8, "flops": 3 * fft + 3 * px}
    d = case["d"] // 2 * 2
    out = 8 * G.bispec_base_size(w, h, d)
    if kind == "reco":
        pairs = visits(case["r"]) * (d + 1) ** 2
        return {"bytes": out + 25 * px, "flops": 18 * pairs}
    n = case["n"]
    acc = 14 * triples(w, h, d) * n
    if kind == "fft":
        return {"bytes": 16 * px * n + out, "flops": acc}
    frames = n * px * np.dtype(NUMPY[case["dtype"]]).itemsize
    # per frame: transform, |F|^2, correlation product and inverse, sum
    acc += n * (2 * fft + 6 * px)
    if kind == "acc":
        return {"bytes": frames + out + 16 * px + 8 * n, "flops": acc}
    pairs = visits(case["r"]) * (d + 1) ** 2
    return {"bytes": frames + 50 * px, "flops": acc + 18 * pairs + 2 * fft}


# -------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def speckle(w, h, n, dtype, seed):
    """n frames (n, h, w) of one object on the device, as the frame type."""
    g = _gen(seed)
    dev = "cuda"
    yy = torch.arange(h, device=dev, dtype=torch.float32)[:, None]
    xx = torch.arange(w, device=dev, dtype=torch.float32)[None, :]
    obj = torch.zeros(h, w, device=dev)
    for x, y, s, flux in torch.rand(12, 4, generator=g, device=dev).tolist():
        x, y = w * (0.4 + 0.2 * x), h * (0.4 + 0.2 * y)
        s = 0.8 + 2.2 * s
        obj += (0.1 + 0.9 * flux) / s**2 * torch.exp(-((xx - x) ** 2 + (yy - y) ** 2) / (2 * s * s))
    obj_ft = torch.fft.fft2(obj)
    fy = torch.fft.fftfreq(h, device=dev)[:, None]
    fx = torch.fft.fftfreq(w, device=dev)[None, :]
    f2 = fx * fx + fy * fy
    f2[0, 0] = 1.0
    r0 = min(w, h) / 2 / 12.0  # pupil diameter / r0 = 12
    amp = torch.sqrt(0.023 * r0 ** (-5 / 3) * f2 ** (-11 / 6)) / math.sqrt(w * h)
    amp[0, 0] = 0.0
    pupil = ((2 * (xx - (w - 1) / 2) / w) ** 2 + (2 * (yy - (h - 1) / 2) / h) ** 2 <= 0.25).float()
    full = {"u8": 255.0, "u16": 65535.0, "f32": 20000.0, "f64": 20000.0}[dtype]
    out = torch.empty(n, h, w, device=dev, dtype={"u8": torch.uint8, "u16": torch.int16, "f32": torch.float32, "f64": torch.float64}[dtype])
    scale = None
    step = max(1, (1 << 25) // (w * h))
    for a in range(0, n, step):
        k = min(step, n - a)
        z = torch.randn(k, h, w, 2, generator=g, device=dev)
        screen = torch.fft.fft2(torch.view_as_complex(z) * amp).real
        psf = torch.fft.fft2(pupil * torch.exp(1j * screen)).abs() ** 2
        psf /= psf.sum((1, 2), keepdim=True)
        move = torch.randint(-3, 4, (k, 2), generator=g, device=dev).float()
        tilt = torch.exp(-2j * math.pi * (move[:, 0, None, None] * fx + move[:, 1, None, None] * fy))
        img = torch.fft.ifft2(torch.fft.fft2(psf) * obj_ft * tilt).real.clamp_(min=0)
        if scale is None:
            scale = 0.5 * full / img.amax((1, 2)).mean()
        img = torch.poisson(img * scale, generator=g) + 2.0 * torch.randn(k, h, w, generator=g, device=dev)
        if dtype in ("f32", "f64"):
            out[a:a + k] = img
        else:
            img = torch.round(img + 0.04 * full).clamp_(0, full).to(torch.int32)
            out[a:a + k] = img.to(out.dtype)  # 16 bits: the same bits, signed
    return out.view(torch.uint16) if dtype == "u16" else out


def spectra_of(frames, dtype=torch.complex128):
    """Fc[f][a][c] = F_f(-a, c - h/2) for a <= w/2, from real frames (n, h, w)."""
    n, h, w = frames.shape
    real = torch.float64 if dtype == torch.complex128 else torch.float32
    a = torch.arange(w // 2 + 1, device="cuda")
    c = torch.arange(h, device="cuda") - h // 2
    out = torch.empty(n, w // 2 + 1, h, device="cuda", dtype=dtype)
    step = max(1, (1 << 25) // (w * h))
    for k in range(0, n, step):
        x = frames[k:k + step]
        x = (x.view(torch.int16).to(torch.int32) & 0xFFFF) if x.dtype == torch.uint16 else x
        f = torch.fft.rfft2(x.to(real))  # F(x >= 0): F(-a, y) = conj F(a, -y)
        out[k:k + step] = f[:, (-c) % h, :].conj()[:, :, a].transpose(1, 2)
    return out


def packed_bispectrum(fc, h, d):
    """Mean of F(u) F(v) conj F(u+v) over the frames of fc, in the packed order."""
    n, hw, _ = fc.shape
    e = d // 2
    bs1 = h // 2 * 2 + 1
    out = torch.zeros(hw, bs1, e + 1, 2 * e + 1, device="cuda", dtype=fc.dtype)
    at = (torch.arange(h, device="cuda") - h // 2) % bs1
    buf = torch.empty_like(fc)
    wc = fc.conj().resolve_conj()
    for a2 in range(e + 1):
        rows = hw - a2
        for l in range(-e, e + 1):
            c0, c1 = max(0, -l), min(h, h - l)
            t = buf.view(-1)[: n * rows * (c1 - c0)].view(n, rows, c1 - c0)
            torch.mul(fc[:, :rows, c0:c1], wc[:, a2:, c0 + l:c1 + l], out=t)
            v = fc[:, a2, l + h // 2]
            out[:rows, at[c0:c1], a2, l % (2 * e + 1)] = torch.matmul(v, t.view(n, -1)).view(rows, c1 - c0) / n
    return out.view(-1)


# ------------------------------------------------------------- C ABI handles
_lib = C.CDLL(G.LIB_PATH)
_lib.smip_last_error.restype = C.c_char_p
_vp, _long = C.c_void_p, C.c_long
for _name, _args in {
    "smip_stack_create": [C.POINTER(_vp), C.c_int, _long, _long, _long, _vp, _long],
    "smip_stack_destroy": [_vp],
    "smip_stack_reset": [_vp],
    "smip_stack_push_frames": [_vp, _vp, C.c_int, _long, _long, C.c_int],
    "smip_stack_accumulate_fft": [_vp, _vp, _long, C.c_int],
    "smip_stack_shifts": [_vp, _vp, _long, _long],
    "smip_stack_sum": [_vp, _vp],
    "smip_stack_power": [_vp, _vp],
    "smip_stack_bispectrum": [_vp, _vp],
}.items():
    getattr(_lib, _name).argtypes = _args


def _ok(rc):
    if rc:
        raise RuntimeError(_lib.smip_last_error().decode())


class Handle:
    """A stack of the C ABI."""

    def __init__(self, w, h, d):
        self.h = _vp()
        _ok(_lib.smip_stack_create(C.byref(self.h), 0, w, h, d, None, 0))

    def __del__(self):
        if self.h:
            _lib.smip_stack_destroy(self.h)
            self.h = None


# ------------------------------------------------------------------- prepare
def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind == "shift":
        frames = speckle(w, h, 2, "f64", seed)
        return {"case": case, "frames": frames, "shift": torch.zeros(2, dtype=torch.int32, device="cuda")}
    d = case["d"]
    size = G.bispec_base_size(w, h, d)
    if kind == "reco":
        fc = spectra_of(speckle(w, h, 8, "u16", seed), torch.complex64)
        st = G.Stack(w, h, d)
        st.set_bispectrum(_host(packed_bispectrum(fc, h, d)))
        st.prepare_reco(case["r"])
        return {"case": case, "stack": st}
    if kind == "fft":
        f = speckle(w, h, case["n"], "f32", seed)
        return {"case": case, "spectra": torch.fft.fft2(f.double()), "stack": Handle(w, h, d),
                "bispectrum": torch.empty(2 * size, dtype=torch.float32, pin_memory=True)}
    frames = speckle(w, h, case["n"], case["dtype"], seed)
    if kind == "job":
        st = G.Stack(w, h, d)
        st.prepare_reco(case["r"])
        return {"case": case, "stack": st, "frames": _host(frames)}
    if case["source"] == "host":
        frames = _host(frames)
    elif case["source"] == "pinned":
        frames = frames.cpu().pin_memory()
    return {"case": case, "stack": Handle(w, h, d), "frames": frames,
            "shifts": np.zeros((case["n"], 2), np.int32), "sum": np.zeros((h, w)), "power": np.zeros((h, w)),
            "bispectrum": torch.empty(2 * size, dtype=torch.float32, pin_memory=True)}


# ----------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "shift":
        f = state["frames"]
        G.xcorr_displacement_noalloc(f[0].data_ptr(), f[1].data_ptr(), case["w"], case["h"], state["shift"].data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
        return state["shift"]
    st = state["stack"]
    if kind == "reco":
        phases, flags, cons = st.reconstruct_phases(case["r"])
        return {"phases": phases, "flags": flags, "consistency": cons}
    if kind == "job":
        st.reset()
        st.push_frames(state["frames"])
        image, phases, flags, cons = st.finish(case["r"])
        return {"image": image.astype(np.complex64), "phases": phases.astype(np.complex64), "flags": flags,
                "consistency": cons.astype(np.float32), "shifts": st.shifts(), "sum": st.sum(), "power": st.power()}
    _ok(_lib.smip_stack_reset(st.h))
    b = state["bispectrum"]
    if kind == "fft":
        _ok(_lib.smip_stack_accumulate_fft(st.h, state["spectra"].data_ptr(), case["n"], 1))
        _ok(_lib.smip_stack_bispectrum(st.h, b.data_ptr()))
        return {"bispectrum": b}
    f = state["frames"]
    at = f.ctypes.data if isinstance(f, np.ndarray) else f.data_ptr()
    _ok(_lib.smip_stack_push_frames(st.h, at, CODES[case["dtype"]], case["n"], 0, int(case["source"] == "device")))
    _ok(_lib.smip_stack_shifts(st.h, state["shifts"].ctypes.data, 0, case["n"]))
    _ok(_lib.smip_stack_sum(st.h, state["sum"].ctypes.data))
    _ok(_lib.smip_stack_power(st.h, state["power"].ctypes.data))
    _ok(_lib.smip_stack_bispectrum(st.h, b.data_ptr()))
    return {"shifts": state["shifts"], "sum": state["sum"], "power": state["power"], "bispectrum": b}


# --------------------------------------------------------------------- exact
def _real(t):
    """complex128 as interleaved doubles, the layout of the C ABI's buffers."""
    return torch.view_as_real(t).reshape(-1)


def _accumulated(frames):
    """(sum / n, power, spectra) of a stack in 64 bits."""
    n, h, w = frames.shape
    fc = spectra_of(frames)
    p = torch.zeros(h, w, device="cuda", dtype=torch.float64)
    total = torch.zeros(h, w, device="cuda", dtype=torch.float64)
    ref = None
    for k in range(n):
        x = frames[k]
        x = ((x.view(torch.int16).to(torch.int32) & 0xFFFF) if x.dtype == torch.uint16 else x).double()
        f = torch.fft.fft2(x)
        p += f.abs() ** 2
        if ref is None:
            ref = f.conj()
            total += x
            continue
        m = int(torch.argmax(torch.fft.ifft2(ref * f).real.reshape(-1)))
        sx, sy = m % w, m // w
        sx -= w if sx >= (w + 1) // 2 else 0
        sy -= h if sy >= (h + 1) // 2 else 0
        # sum(x, y) += |frame(x + sx, y + sy)| inside the frame
        y0, y1, x0, x1 = max(0, -sy), min(h, h - sy), max(0, -sx), min(w, w - sx)
        total[y0:y1, x0:x1] += x[y0 + sy:y1 + sy, x0 + sx:x1 + sx].abs()
    return total / n, p / (n * w * h), fc


def _offsets(w, h, d, ux, uy, vx, vy):
    """Packed offset and conjugation of B(u, v) by the library's index rule."""
    e = d // 2
    sizes = (w // 2 * 2 + 1, h // 2 * 2 + 1, 2 * e + 1)
    u0, u1, u2, u3 = ux, uy, vx, vy
    both_neg = (u0 <= 0) & (u2 <= 0)
    both_pos = (u0 > 0) & (u2 > 0)
    pos0 = (u0 > 0) & ~both_pos
    s = u0 + u2 > 0
    t = u1 + u3
    conj = both_pos | (~both_neg & ~both_pos & ~s)

    def pick(neg, pos, p_s, p_n, n_s, n_n):
        r = torch.where(s, n_s, n_n)
        r = torch.where(pos0, torch.where(s, p_s, p_n), r)
        r = torch.where(both_pos, pos, r)
        return torch.where(both_neg, neg, r)

    a0 = pick(u0, -u0, -u0 - u2, -u0, u0, u0 + u2)
    a1 = pick(u1, -u1, -t, -u1, u1, t)
    a2 = pick(u2, -u2, u2, u2 + u0, -u2 - u0, -u2)
    a3 = pick(u3, -u3, u3, t, -t, -u3)
    swap = (a2.abs() > e) | (a3.abs() > e)
    a0, a2 = torch.where(swap, a2, a0), torch.where(swap, a0, a2)
    a1, a3 = torch.where(swap, a3, a1), torch.where(swap, a1, a3)
    a0, a2 = -a0, -a2
    a0, a1 = torch.where(a0 < 0, a0 + sizes[0], a0), torch.where(a1 < 0, a1 + sizes[1], a1)
    a2, a3 = torch.where(a2 < 0, a2 + sizes[2], a2), torch.where(a3 < 0, a3 + sizes[2], a3)
    base1, base2 = sizes[1], e + 1
    return ((a0 * base1 + a1) * base2 + a2) * sizes[2] + a3, conj


def _spiral(r_max):
    out, r, phi, i, j = [], 0.0, 0.0, 0, 0
    while r <= r_max:
        ii, jj = i, j
        step = math.inf if r == 0.0 else 1.0 / (2.0 * math.pi * r)
        while (ii, jj) == (i, j):
            phi += step
            if phi > 2.0 * math.pi:
                phi = 0.0
                r += 1.0
            ii, jj = int(r * math.cos(phi)), int(r * math.sin(phi))
        i, j = ii, jj
        out.append((i, j))
    return out


def _walk(b, w, h, d, r):
    """The spiral phase recovery in 64 bits: phases, flags, consistency (h, w)."""
    e = d // 2
    side = 2 * e + 1
    vx = torch.arange(-e, e + 1, device="cuda").repeat(side)
    vy = torch.arange(-e, e + 1, device="cuda").repeat_interleave(side)
    lo, hi = (-(w // 2), -(h // 2)), (w - 1 - w // 2, h - 1 - h // 2)
    pts = []
    for q in _spiral(r):  # a point that gets no phase may be passed again
        if lo[0] <= q[0] <= hi[0] and lo[1] <= q[1] <= hi[1] and abs(q[0]) + abs(q[1]) > 1:
            pts.append(q)
    phases = np.zeros(w * h, np.complex128)
    flags = np.zeros(w * h, bool)
    cons = np.zeros(w * h)
    for x, y, im in ((0, 0, 0.0), (1, 0, 0.0), (0, 1, 0.0), (-1, 0, -0.0), (0, -1, -0.0)):
        p = x % w + y % h * w
        phases[p], flags[p], cons[p] = complex(1.0, im), True, 1.0
    pv = ((vx % w) + (vy % h) * w).cpu().numpy()
    b = b.to(torch.complex128)
    for k in range(0, len(pts), 4096):
        part = torch.tensor(pts[k:k + 4096], device="cuda")
        ux, uy = part[:, :1] - vx, part[:, 1:] - vy
        ins = (ux >= lo[0]) & (ux <= hi[0]) & (uy >= lo[1]) & (uy <= hi[1])
        off, conj = _offsets(w, h, d, ux, uy, vx.expand_as(ux), vy.expand_as(uy))
        x = b[torch.where(ins, off, 0).clamp(0, b.numel() - 1)]
        x = torch.where(conj, x.conj(), x)
        m = x.abs()
        use = (ins & (m > 2.220446049250313e-16)).cpu().numpy()
        unit = torch.where(m > 0, x / m, 0).conj().cpu().numpy()
        pu = ((ux % w) + (uy % h) * w).cpu().numpy()
        for q, (px, py) in enumerate(pts[k:k + 4096]):
            p = px % w + py % h * w
            if flags[p]:
                continue
            ok = use[q] & flags[pu[q]] & flags[pv]
            n = np.count_nonzero(ok)
            if not n:
                continue
            t = phases[pu[q][ok]] * phases[pv[ok]] * unit[q][ok]
            t = t / np.abs(t)
            mean = t.sum() / n
            cons[p] = abs(mean)
            phases[p] = mean / cons[p] if cons[p] > 2.220446049250313e-16 else 0.0
            flags[p] = True
    return phases.reshape(h, w), flags.reshape(h, w).astype(np.uint8), cons.reshape(h, w)


def exact(case, seed):
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind == "shift":
        return None
    d = case["d"] // 2 * 2
    if kind in ("reco", "job") and visits(case["r"]) * ((d + 1) ** 2 + 2000) > 2.2e8:
        return None
    if kind == "reco":
        fc = spectra_of(speckle(w, h, 8, "u16", seed), torch.complex64)
        b = packed_bispectrum(fc, h, d)
        phases, _, cons = _walk(b, w, h, d, case["r"])
        return {"phases": phases, "flags": None, "consistency": cons}
    if kind == "fft":
        f = speckle(w, h, case["n"], "f32", seed)
        return {"bispectrum": _real(packed_bispectrum(spectra_of(f), h, d))}
    total, power, fc = _accumulated(speckle(w, h, case["n"], case["dtype"], seed))
    b = packed_bispectrum(fc, h, d)
    if kind == "acc":
        return {"shifts": None, "sum": total, "power": power, "bispectrum": _real(b)}
    phases, _, cons = _walk(b, w, h, d, case["r"])
    x = np.where(np.arange(w) < w - w // 2, np.arange(w), np.arange(w) - w)
    y = np.where(np.arange(h) < h - h // 2, np.arange(h), np.arange(h) - h)
    a = math.pi / case["r"]  # Hann window of aperture 2 r
    win = (0.5 + 0.5 * np.cos(a * y))[:, None] * (0.5 + 0.5 * np.cos(a * x))[None, :]
    image = np.fft.ifft2(np.sqrt(power.cpu().numpy()) * phases * win)
    return {"image": image / np.abs(image).max(), "phases": phases, "flags": None, "consistency": cons,
            "shifts": None, "sum": total, "power": power}
