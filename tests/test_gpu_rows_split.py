"""Row passes on the split block FFT (lengths 384 and 1536) through the plain 2D transforms, against
an FP64 FFT: odd row counts (a last pair with one row, blocks partly empty), the pruned and the
general input head, window origins, 16-bit storage; and through the correlation with its fused peak
search and projection, window origins and scales among them."""
import numpy as np
import pytest

from _util import RTOL_L2_FP32, RTOL_MAX_FP32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ix,iy,wx,wy,ox,oy", [
    (384, 64, 90, 37, 200, 33, 0, 0),
    (384, 384, 384, 384, 384, 384, 0, 0),
    (384, 128, 97, 128, 383, 127, 1, 1),
    (1536, 64, 384, 9, 1024, 61, 0, 0),
    (1536, 128, 385, 127, 1000, 128, 300, 0),
    (1536, 64, 1535, 64, 1, 64, 1535, 0),
])
@pytest.mark.parametrize("dtype", ["float32", "float16"])
def test_round_trip(torch_cuda, nx, ny, ix, iy, wx, wy, ox, oy, dtype):
    import torch

    import fastfft_b200 as F
    from oracle import fastfft_oracle as O

    rng = np.random.default_rng(nx + ix)
    t = torch.from_numpy(rng.standard_normal((iy, ix)).astype(np.float32)).to(getattr(torch, dtype))
    ft = F.FourierTransformer(input_dtype=dtype)
    ft.SetOutputDtype("float32")
    ft.SetInverseOutputOrigin(ox, oy)
    ft.SetForwardFFTPlan(ix, iy, 1, nx, ny, 1)
    ft.SetInverseFFTPlan(nx, ny, 1, wx, wy, 1)
    x = torch.zeros(iy, 2 * (ix // 2 + 1), dtype=t.dtype)
    x[:, :ix] = t
    spec = torch.zeros(nx // 2 + 1, ny, dtype=torch.complex64, device="cuda")
    ft.FwdFFT(x.cuda(), spec)
    ref = np.fft.rfft2(t.double().numpy(), s=(ny, nx)).T
    assert O.rel_l2(spec.cpu().numpy(), ref) <= RTOL_L2_FP32
    full = np.fft.rfft2(rng.standard_normal((ny, nx))).T.astype(np.complex64)
    out = torch.zeros(wy, 2 * (wx // 2 + 1), device="cuda")
    ft.InvFFT(torch.from_numpy(np.ascontiguousarray(full)).cuda(), out)
    back = np.fft.irfft2(full.astype(np.complex128).T, s=(ny, nx)) * nx * ny
    ref = back[oy: oy + wy, ox: ox + wx]
    got = out.cpu().numpy()[:, :wx]
    assert O.rel_l2(got, ref) <= RTOL_L2_FP32
    assert np.abs(got - ref).max() <= RTOL_MAX_FP32 * np.abs(back).max()


# (row length, column length, template, window, origin, plan): the first two correlate at the reduced
# row length, the others at the plan's own
FUSED = [
    (384, 128, (97, 50), (255, 61), (0, 0), (1024, 256)),
    (1536, 128, (500, 40), (1001, 87), (0, 0), (2048, 256)),
    (384, 128, (90, 41), (250, 51), (3, 5), (384, 128)),
    (1536, 64, (300, 20), (1230, 33), (305, 1), (1536, 64)),
]


@pytest.mark.parametrize("mx,my,tmpl,win,org,plan", FUSED)
@pytest.mark.parametrize("dtype", ["float32", "float16"])
def test_fused_peaks_and_projection(torch_cuda, mx, my, tmpl, win, org, plan, dtype):
    """Scaled windows against an FP64 correlation; the peak search and the projection, with and
    without windows, against the float32 windows exactly (their keys hold the values before a
    16-bit rounding)."""
    import torch

    import fastfft_b200 as F
    from fastfft_b200 import KernelFunction as KF
    from oracle import fastfft_oracle as O

    (tx, ty), (wx, wy), (ox, oy), (nx, ny) = tmpl, win, org, plan
    rng = np.random.default_rng(mx + ox)
    spec = (np.fft.rfft2(rng.standard_normal((ny, nx))) / np.sqrt(nx * ny)).astype(np.complex64)
    d_spec = torch.from_numpy(np.ascontiguousarray(spec.T)).cuda()
    ts = [torch.from_numpy(rng.standard_normal((ty, tx)).astype(np.float32)).to(getattr(torch, dtype)) for _ in range(3)]
    ins = []
    for t in ts:
        x = torch.zeros(ty, 2 * (tx // 2 + 1), dtype=t.dtype)
        x[:, :tx] = t
        ins.append(x.cuda())
    ft = F.FourierTransformer(input_dtype=dtype)
    ft.SetInverseOutputOrigin(ox, oy)
    ft.SetForwardFFTPlan(tx, ty, 1, nx, ny, 1)
    ft.SetInverseFFTPlan(nx, ny, 1, wx, wy, 1)
    assert ft.CorrelationSize() == (mx, my)
    ops = (KF.scale(0.5), KF.conj_mul_then_scale(0.25), KF.scale(3.0 / 1024))
    pitch = 2 * (wx // 2 + 1)
    windows, results = {}, []
    for out_dtype in ("float32", "float16"):
        ft.SetOutputDtype(out_dtype)
        outs, outs2 = ([torch.zeros(wy, pitch, dtype=getattr(torch, out_dtype), device="cuda") for _ in ts]
                       for _ in range(2))
        ft.FwdImageInvFFTMany(ins, d_spec, outs, *ops)
        windows[out_dtype] = np.stack([o.cpu().numpy()[:, :wx] for o in outs])
        for write in (outs2, None):
            peaks = torch.zeros(len(ts), dtype=torch.int64, device="cuda")
            mip = torch.zeros(wx * wy, dtype=torch.int64, device="cuda")
            ft.FwdImageInvFFTManyPeaks(ins, d_spec, peaks, None, write, *ops)
            if write:
                assert all(torch.equal(a, b) for a, b in zip(outs, outs2))
                for o in outs2:
                    o.zero_()
            ft.FwdImageInvFFTManyMip(ins, d_spec, mip, None, write, 7, *ops)
            if write:
                assert all(torch.equal(a, b) for a, b in zip(outs, outs2))
            results.append((F.decode_peaks(peaks), F.decode_peaks(mip)))
    for t, got in zip(ts, windows["float32"]):
        corr = np.fft.irfft2(np.conj(np.fft.rfft2(t.double().numpy(), s=(ny, nx))) * spec.astype(np.complex128),
                             s=(ny, nx)) * (0.5 * 0.25 * 3.0 / 1024 * nx * ny)
        ref = corr[oy: oy + wy, ox: ox + wx]
        assert O.rel_l2(got, ref) <= RTOL_L2_FP32
        assert np.abs(got - ref).max() <= RTOL_MAX_FP32 * np.abs(corr).max()
    assert np.array_equal(windows["float16"], windows["float32"].astype(np.float16))
    flat = windows["float32"].reshape(len(ts), -1)
    for (vals, idx), (mvals, midx) in results:
        assert np.array_equal(idx, flat.argmax(1)) and np.array_equal(vals, flat.max(1))
        assert np.array_equal(midx, flat.argmax(0) + 7) and np.array_equal(mvals, flat.max(0))
