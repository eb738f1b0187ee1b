"""Row passes on the split block FFT (lengths 384 and 1536) through the plain 2D transforms and the
fused outputs, against the FP64 oracle: odd row counts (a last pair with one row, blocks partly
empty), the pruned and the general input head, window origins, 16-bit storage."""
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
