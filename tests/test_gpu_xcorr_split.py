"""The batched column pass on the split block FFT at each of its lengths, against the FP64 oracle:
odd and full input heads (the pruned and the general first step), windows that end inside a
thread's slots, and launches of 1 to 17 templates (few, single and paired forms, a last pair and
a last group that are partly empty), which must agree bit for bit."""
import numpy as np
import pytest

from _util import RTOL_L2_FP32, RTOL_MAX_FP32

pytestmark = pytest.mark.gpu

# (column length, transform size, template, window): template + window - 1 reaches the length
CASES = [
    (256, 512, (61, 59), (128, 131)),
    (384, 1024, (97, 95), (256, 255)),
    (384, 512, (128, 300), (250, 85)),
    (512, 1024, (128, 129), (300, 384)),
    (768, 1024, (192, 191), (500, 512)),
    (768, 2048, (256, 513), (511, 250)),
    (1024, 2048, (256, 255), (700, 700)),
    (1024, 2048, (400, 801), (600, 200)),
    (1536, 2048, (384, 384), (1024, 1023)),
    (1536, 2048, (300, 901), (900, 600)),
    (2048, 3072, (512, 513), (1200, 1300)),
]


@pytest.mark.parametrize("m,n,tmpl,win", CASES)
def test_split_lengths(torch_cuda, m, n, tmpl, win):
    import torch

    import fastfft_b200 as F
    from oracle import fastfft_oracle as O

    rng = np.random.default_rng(m + tmpl[1])
    spec = O.fwd(O.real_to_padded(rng.standard_normal((n, n)), (n, n, 1), dtype=np.float64), (n, n, 1), (n, n, 1))
    spec = (spec / n).astype(np.complex64)
    count = 17
    ts = [rng.standard_normal((tmpl[1], tmpl[0])).astype(np.float32) for _ in range(count)]
    fin, iout = (*tmpl, 1), (*win, 1)
    plan = O.Plan(fin, (n, n, 1), (n, n, 1), iout)
    ft = F.FourierTransformer()
    ft.SetForwardFFTPlan(*fin, n, n, 1)
    ft.SetInverseFFTPlan(n, n, 1, *iout)
    assert ft.CorrelationSize()[1] == m
    d_in = [torch.from_numpy(O.real_to_padded(t, fin)).cuda() for t in ts]
    d_img = torch.from_numpy(spec.view(np.float32).reshape(-1).copy()).cuda()
    size = ft.ReturnInvOutputMemorySize()
    results = []
    for per_launch in (17, 3, 1):
        ft.SetTemplatesPerLaunch(per_launch)
        outs = [torch.zeros(size, device="cuda") for _ in ts]
        ft.FwdImageInvFFTMany(d_in, d_img, outs, None, F.KernelFunction.conj_mul_then_scale(0.5), None)
        ft.Wait()
        results.append([O.real_from_padded(o.cpu().numpy(), iout) for o in outs])
    for k in (0, 16):
        ref = 0.5 * O.real_from_padded(
            O.fwd_image_inv(O.real_to_padded(ts[k], fin), spec, plan, out_dtype=np.float64), iout)
        assert O.rel_l2(results[0][k], ref) <= RTOL_L2_FP32
        assert O.rel_max(results[0][k], ref) <= RTOL_MAX_FP32
    for other in results[1:]:
        for a, b in zip(results[0], other):
            assert np.array_equal(a, b)
