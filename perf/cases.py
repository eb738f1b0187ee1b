"""The work that users of fastfft_b200 have it do, as cases that can be timed and checked.

Every case is one pass through the public calls of FourierTransformer on buffers and plans that
a program keeps: plain transforms with padding and cropping (2D, any-length 2D, 3D, complex
input), the one-template correlation, and the batched correlation with its outputs (windows,
fused peak search, fused maximum projection) in each storage type of image and templates.

A case is a dict of plain values; "family" selects the calls:
  transform   FwdFFT of an ix x iy image padded to nx x ny (op "forward"), or that and the InvFFT
              of its spectrum keeping wx x wy (op "round_trip"); real or complex input
  volume      FwdFFT of an ix x iy x iz volume padded to nx x ny x nz, and the InvFFT of another
              volume's spectrum keeping its wx x wy x wz window at the centre (or the origin)
  single      FwdImageInvFFT of one template against an image spectrum, window wx x wy
  many        one batched correlation of `count` templates against an image spectrum; out is
              "windows", "peaks" (best score and position per template) or "mip" (best score and
              template per window pixel); sizes "" (all tx x ty) or a list of edge lengths that
              the templates' sizes are drawn from
"""
from __future__ import annotations

import math
import random

import torch

import fastfft_b200 as F
from fastfft_b200 import KernelFunction as KF

REAL = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
# image spectrum storage that goes with a template storage
IMAGE = {"float32": "complex64", "float16": "complex32", "bfloat16": "complex_bf16"}


def listed():
    return [
        # A small picture padded into a larger transform and brought back: four short kernels,
        # bound by calls and launches (particle images, and every first try of the library).
        dict(name="pad_64_to_512", family="transform", op="round_trip", dtype="float32", ix=64, iy=64,
             nx=512, ny=512, wx=512, wy=512),
        # The spectrum of a micrograph, made once for each image that is searched.
        dict(name="image_spectrum_4096", family="transform", op="forward", dtype="float32", ix=4096, iy=4096,
             nx=4096, ny=4096, wx=4096, wy=4096),
        # A detector image that is no power of two, padded to the next lengths 3 * 2^k and
        # 5 * 2^k and cropped again (filtering, resampling).
        dict(name="pad_crop_1536x1280", family="transform", op="round_trip", dtype="float32", ix=1100, iy=901,
             nx=1536, ny=1280, wx=1000, wy=777),
        # Lengths that a user cannot choose: any other size, odd ones among them.
        dict(name="any_length_1000x945", family="transform", op="round_trip", dtype="float32", ix=811, iy=743,
             nx=1000, ny=945, wx=601, wy=600),
        # Complex images (already demodulated or Fourier-filtered data).
        dict(name="complex_512", family="transform", op="round_trip", dtype="complex64", ix=300, iy=260,
             nx=512, ny=512, wx=256, wy=256),
        # A particle volume padded for interpolation, and the central part of an inverse.
        dict(name="volume_64_256_128", family="volume", dtype="float32", ix=64, iy=64, iz=64, nx=256, ny=256,
             nz=256, wx=128, wy=128, wz=128, centre=True),
        # The reference's own call: one template at a time against a micrograph.
        dict(name="single_384_4096_1024", family="single", dtype="float32", tx=384, ty=384, nx=4096, ny=4096,
             wx=1024, wy=1024),
        # The template search on one micrograph, all windows wanted: the throughput workload.
        dict(name="search_384_4096_1024", family="many", dtype="float32", out="windows", count=64, sizes="",
             tx=384, ty=384, nx=4096, ny=4096, wx=1024, wy=1024, per_launch=64),
        # The same search where only the best score per pixel over all templates is kept.
        dict(name="search_mip_384_2048_700", family="many", dtype="float32", out="mip", count=48, sizes="",
             tx=384, ty=384, nx=2048, ny=2048, wx=700, wy=700, per_launch=0),
        # Templates of uneven sizes in one call.
        dict(name="uneven_4096_512", family="many", dtype="float32", out="windows", count=256,
             sizes="128,192,256,384", tx=384, ty=384, nx=4096, ny=4096, wx=512, wy=512, per_launch=32),
        # 16-bit storage of templates and image spectrum, only the peaks wanted.
        dict(name="peaks_bf16_300_3072_900", family="many", dtype="bfloat16", out="peaks", count=40, sizes="",
             tx=300, ty=300, nx=3072, ny=3072, wx=900, wy=900, per_launch=0),
        # A handful of small templates on a small image: short kernels, partly filled launches.
        dict(name="small_batch_96_1024_256", family="many", dtype="float32", out="windows", count=12, sizes="",
             tx=96, ty=96, nx=1024, ny=1024, wx=256, wy=256, per_launch=0),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _part(rng, n, lo=8):
    """A part of a length n: all of it at times, else any number, odd ones among them."""
    return n if rng.random() < 0.15 else _log(rng, max(lo, n // 12), n)


def draw(rng):
    kind = rng.choice(["transform", "transform", "any", "complex", "volume", "single", "many", "many", "many"])
    if kind in ("transform", "any", "complex"):
        if kind == "any":
            nx, ny = _log(rng, 40, 1500), _log(rng, 40, 1500)
        elif kind == "complex":
            nx, ny = 1 << rng.randint(6, 11), 1 << rng.randint(6, 11)
        else:
            lens = [64, 128, 256, 512, 1024, 2048, 4096, 384, 768, 1536, 3072, 640, 1280, 2560, 896, 1792]
            nx, ny = rng.choice(lens), rng.choice(lens)
        op = "forward" if rng.random() < 0.4 else "round_trip"
        dtype = "complex64" if kind == "complex" else rng.choice(["float32", "float32", "float16", "bfloat16"])
        return dict(family="transform", op=op, dtype=dtype, ix=_part(rng, nx), iy=_part(rng, ny), nx=nx, ny=ny,
                    wx=_part(rng, nx), wy=_part(rng, ny))
    if kind == "volume":
        n = [rng.choice([32, 64, 128, 256]) for _ in range(3)]
        i = [_part(rng, v, 16) for v in n]
        w = [_part(rng, v, 16) for v in n]
        return dict(family="volume", dtype="float32", ix=i[0], iy=i[1], iz=i[2], nx=n[0], ny=n[1], nz=n[2],
                    wx=w[0], wy=w[1], wz=w[2], centre=rng.random() < 0.5)
    n = rng.choice([512, 1024, 2048, 4096, 1536, 3072])
    dtype = rng.choice(["float32", "float32", "float16", "bfloat16"])
    t, w = _log(rng, 32, min(500, n // 4)), _log(rng, 64, min(1100, n // 2))
    u, v = min(n // 4, max(32, t + rng.randint(-9, 9))), min(n // 2, max(64, w + rng.randint(-40, 40)))
    if kind == "single":
        return dict(family="single", dtype=dtype, tx=t, ty=u, nx=n, ny=n, wx=w, wy=v)
    # (a projection over few templates could keep negative scores, see _keys)
    out = rng.choice(["windows", "windows", "peaks", "mip"])
    sizes = ""
    if rng.random() < 0.35:
        sizes = ",".join(str(x) for x in sorted(rng.randint(16, min(t, u)) for _ in range(4)))
    return dict(family="many", dtype=dtype, out=out, count=rng.randint(32 if out == "mip" else 2, 48), sizes=sizes, tx=t, ty=u, nx=n,
                ny=n, wx=w, wy=v, per_launch=rng.choice([0, 0, 32, 64]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _pitch(x):
    """FFTW pitch of a real row of x values."""
    return 2 * (x // 2 + 1)


def _randn(seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.randn(*shape, generator=g, device="cuda")


def _padded(x, dtype):
    """Values [..., y, x] as the FFTW-padded rows that the library reads, stored as dtype."""
    p = torch.zeros(*x.shape[:-1], _pitch(x.shape[-1]), dtype=dtype, device="cuda")
    p[..., : x.shape[-1]] = x.to(dtype)
    return p


def _blobs(seed, ny, nx):
    """N(0, 1) noise with Gaussian blobs (sigma 8, amplitude 5), as a micrograph with particles."""
    img = _randn(seed, ny, nx)
    r = random.Random(seed)
    y = torch.arange(ny, device="cuda", dtype=torch.float32)
    x = torch.arange(nx, device="cuda", dtype=torch.float32)
    gy, gx = [], []
    for _ in range(20):
        gy.append(torch.exp(-((y - r.uniform(0, ny)) ** 2) / 128.0))
        gx.append(torch.exp(-((x - r.uniform(0, nx)) ** 2) / 128.0))
    return img + 5.0 * torch.stack(gy).T @ torch.stack(gx)


def _image_spectrum(case, seed):
    """The image's half spectrum as [kx][ky], normalised by 1 / sqrt(nx ny): (complex128 values
    of what is stored, the stored buffer)."""
    nx, ny = case["nx"], case["ny"]
    s = torch.fft.rfft2(_blobs(seed + 7919, ny, nx).double()).T.contiguous() / math.sqrt(nx * ny)
    if case["dtype"] == "float32":
        buf = s.to(torch.complex64)
        return buf.to(torch.complex128), buf
    buf = torch.view_as_real(s).to(REAL[case["dtype"]])
    return torch.view_as_complex(buf.double()), buf


def _sizes(case):
    """(x, y) of each template."""
    if not case["sizes"]:
        return [(case["tx"], case["ty"])] * case["count"]
    edges = [int(v) for v in case["sizes"].split(",")]
    r = random.Random(case["count"])
    return [(e, e) for e in (r.choice(edges) for _ in range(case["count"]))]


def _templates(case, seed):
    flat = _randn(seed, sum(x * y for x, y in _sizes(case)))
    out, at = [], 0
    for x, y in _sizes(case):
        out.append(flat[at: at + x * y].reshape(y, x))
        at += x * y
    return out


def _signal(case, seed):
    """The input of a plain transform as its values [z,] y, x."""
    shape = [case[k] for k in ("iz", "iy", "ix") if k in case]
    if case["dtype"] == "complex64":
        return torch.view_as_complex(_randn(seed, *shape, 2))
    return _randn(seed, *shape).to(REAL[case["dtype"]])


def _volume_spectrum(case, seed):
    """The spectrum [kz][kx][ky] of a whole random volume, as stored."""
    x = _randn(seed + 104729, case["nz"], case["ny"], case["nx"]).double()
    return torch.fft.rfftn(x).transpose(-1, -2).contiguous().to(torch.complex64)


def _origin(case):
    if not case.get("centre"):
        return 0, 0, 0
    return tuple((case["n" + a] - case["w" + a]) // 2 for a in "xyz")


# ---------------------------------------------------------------------------
# A case's state and its pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    family, dtype = case["family"], case["dtype"]
    s = {"case": case}
    if family in ("transform", "volume"):
        three = family == "volume"
        z = (case["iz"], case["nz"], case["wz"]) if three else (1, 1, 1)
        ft = F.FourierTransformer(input_dtype=dtype, image_dtype="complex64", rank=3 if three else 2)
        if three:
            ft.SetInverseOutputOrigin(*_origin(case))
        ft.SetForwardFFTPlan(case["ix"], case["iy"], z[0], case["nx"], case["ny"], z[1])
        ft.SetInverseFFTPlan(case["nx"], case["ny"], z[1], case["wx"], case["wy"], z[2])
        x = _signal(case, seed)
        kx = case["nx"] if dtype == "complex64" else case["nx"] // 2 + 1
        lead = [case["nz"]] if three else []
        s["spectrum"] = torch.zeros(*lead, kx, case["ny"], dtype=torch.complex64, device="cuda")
        if dtype == "complex64":
            s["input"] = x.contiguous()
            out = torch.zeros(case["wy"], case["wx"], dtype=torch.complex64, device="cuda")
            s["out"], s["window"] = out, out
        else:
            ft.SetOutputDtype("float32")
            s["input"] = _padded(x, REAL[dtype])
            if three:
                s["other"] = _volume_spectrum(case, seed)
            lead = [case["wz"]] if three else []
            s["out"] = torch.zeros(*lead, case["wy"], _pitch(case["wx"]), device="cuda")
            s["window"] = s["out"][..., : case["wx"]]
        s["ft"] = ft
        return s
    ft = F.FourierTransformer(input_dtype=dtype, image_dtype=IMAGE[dtype])
    ft.SetOutputDtype("float32")
    if case.get("per_launch"):
        ft.SetTemplatesPerLaunch(case["per_launch"])
    ft.SetForwardFFTPlan(case["tx"], case["ty"], 1, case["nx"], case["ny"], 1)
    ft.SetInverseFFTPlan(case["nx"], case["ny"], 1, case["wx"], case["wy"], 1)
    s["ft"] = ft
    _, s["image"] = _image_spectrum(case, seed)
    s["op"] = KF.conj_mul()
    if family == "single":
        s["input"] = _padded(_randn(seed, case["ty"], case["tx"]), REAL[dtype])
        s["out"] = torch.zeros(case["wy"], _pitch(case["wx"]), device="cuda")
        return s
    s["inputs"] = [_padded(t, REAL[dtype]) for t in _templates(case, seed)]
    s["sizes"] = _sizes(case) if case["sizes"] else None
    if case["out"] == "windows":
        s["out"] = torch.zeros(case["count"], case["wy"], _pitch(case["wx"]), device="cuda")
        s["outs"] = list(s["out"])
    elif case["out"] == "peaks":
        s["keys"] = torch.zeros(case["count"], dtype=torch.int64, device="cuda")
    else:
        s["keys"] = torch.zeros(case["wy"], case["wx"], dtype=torch.int64, device="cuda")
    return s


def _keys(keys):
    """Packed keys as their two words, without a copy: the complement of the index, and the
    score (whose ordered bits read as minus the score where it is positive, as a best score over
    a window or over many templates is)."""
    return {"index": keys.view(torch.int32)[..., 0::2], "minus_score": keys.view(torch.float32)[..., 1::2]}


def run(s):
    case, ft = s["case"], s["ft"]
    if case["family"] in ("transform", "volume"):
        ft.FwdFFT(s["input"], s["spectrum"])
        if case.get("op") == "forward":
            return s["spectrum"]
        ft.InvFFT(s["other"] if case["family"] == "volume" else s["spectrum"], s["out"])
        return {"spectrum": s["spectrum"], "window": s["window"]}
    if case["family"] == "single":
        ft.FwdImageInvFFT(s["input"], s["image"], s["out"], None, s["op"], None)
        return s["out"][:, : case["wx"]]
    if case["out"] == "windows":
        if s["sizes"] is None:
            ft.FwdImageInvFFTMany(s["inputs"], s["image"], s["outs"], None, s["op"], None)
        else:
            ft.FwdImageInvFFTManySized(s["inputs"], s["sizes"], s["image"], s["outs"], None, s["op"], None)
        return s["out"][..., : case["wx"]]
    if case["out"] == "peaks":
        ft.FwdImageInvFFTManyPeaks(s["inputs"], s["image"], s["keys"], sizes=s["sizes"], intra_op=s["op"])
    else:
        s["keys"].zero_()
        ft.FwdImageInvFFTManyMip(s["inputs"], s["image"], s["keys"], sizes=s["sizes"], intra_op=s["op"])
    return _keys(s["keys"])


# ---------------------------------------------------------------------------
# What a pass cannot do without, and how far another correct pass may be off
# ---------------------------------------------------------------------------
def _fft_flops(*lengths, real=True):
    n = math.prod(lengths)
    return (2.5 if real else 5.0) * n * math.log2(n)


def work(case):
    size = {"float32": 4, "float16": 2, "bfloat16": 2, "complex64": 8}[case["dtype"]]
    if case["family"] in ("transform", "volume"):
        n = [case[k] for k in ("nz", "ny", "nx") if k in case]
        i = math.prod(case[k] for k in ("iz", "iy", "ix") if k in case)
        w = math.prod(case[k] for k in ("wz", "wy", "wx") if k in case)
        real = case["dtype"] != "complex64"
        spec = 8 * math.prod(n[:-1]) * (n[-1] // 2 + 1 if real else n[-1])
        fwd = {"bytes": i * size + spec, "flops": _fft_flops(*n, real=real)}
        if case.get("op") == "forward":
            return fwd
        return {"bytes": fwd["bytes"] + spec + w * (4 if real else 8), "flops": 2 * fwd["flops"]}
    # the lags kept need the image up to template + window - 1, the image comes as its whole spectrum
    sizes = [(case["tx"], case["ty"])] if case["family"] == "single" else _sizes(case)
    flops = sum(2 * _fft_flops(x + case["wx"] - 1, y + case["wy"] - 1) for x, y in sizes)
    window = case["wx"] * case["wy"]
    out = {"windows": 4 * window * len(sizes), "peaks": 8 * len(sizes), "mip": 16 * window}[case.get("out", "windows")]
    image = 2 * size * case["ny"] * (case["nx"] // 2 + 1)
    return {"bytes": sum(x * y for x, y in sizes) * size + image + out, "flops": flops}


def tolerance(case):
    # 32-bit sums throughout, also where the inputs are stored in 16 bits (exact() takes the stored
    # values).  Measured against exact(): 2e-7 (short transforms) to 7e-7 (chirp-z lengths,
    # correlations) in the 2-norm.
    t = {"rel": 3e-6, "max": 3e-5}
    if case.get("out") == "mip":
        t["differ"] = 1e-4     # pixels whose two best templates agree to rounding
    return t


def exact(case, seed):
    """run()'s outputs for the same inputs from torch.fft in 64 bits."""
    if case["family"] in ("transform", "volume"):
        x = _signal(case, seed)
        x = x.to(torch.complex128) if case["dtype"] == "complex64" else x.double()
        n = [case[k] for k in ("nz", "ny", "nx") if k in case]
        dims = list(range(len(n)))
        if case["dtype"] == "complex64":
            spec = torch.fft.fftn(x, s=n, dim=dims)
        else:
            spec = torch.fft.rfftn(x, s=n, dim=dims)
        spec = spec.transpose(-1, -2).contiguous()
        if case.get("op") == "forward":
            return spec
        if case["family"] == "volume":
            other = _volume_spectrum(case, seed).to(torch.complex128).transpose(-1, -2).contiguous()
            full = torch.fft.irfftn(other, s=n)
        else:
            full = torch.zeros(*n, dtype=x.dtype, device="cuda")
            full[tuple(slice(0, v) for v in x.shape)] = x
        ox, oy, oz = _origin(case)
        at = [slice(o, o + case["w" + a]) for a, o in (("z", oz), ("y", oy), ("x", ox)) if "w" + a in case]
        return {"spectrum": spec, "window": full[tuple(at)].contiguous() * math.prod(n)}
    nx, ny, wx, wy = case["nx"], case["ny"], case["wx"], case["wy"]
    image, _ = _image_spectrum(case, seed)
    image = image.T.contiguous()
    one = case["family"] == "single"
    ts = [_randn(seed, case["ty"], case["tx"])] if one else _templates(case, seed)
    wins, best = [], None
    for k, t in enumerate(ts):
        t = t.to(REAL[case["dtype"]]).double()
        c = torch.fft.irfft2(torch.fft.rfft2(t, s=(ny, nx)).conj() * image, s=(ny, nx))[:wy, :wx] * (nx * ny)
        if one:
            return c.contiguous()
        if case["out"] == "windows":
            wins.append(c.contiguous())
        elif case["out"] == "peaks":
            at = int(c.reshape(-1).argmax())
            wins.append((c.reshape(-1)[at], at))
        else:
            if best is None:
                best, arg = c.clone(), torch.zeros_like(c, dtype=torch.int32)
            else:
                arg[c > best] = k
                best = torch.maximum(best, c)
    if case["out"] == "windows":
        return torch.stack(wins)
    if case["out"] == "peaks":
        index = torch.tensor([w[1] for w in wins], dtype=torch.int32, device="cuda")
        return {"index": ~index, "minus_score": -torch.stack([w[0] for w in wins])}
    return {"index": ~arg, "minus_score": -best}
