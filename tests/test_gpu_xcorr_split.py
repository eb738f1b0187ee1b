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
    # the last template heights whose pairs fit three blocks on an SM, and the first that do not
    (1536, 2048, (60, 448), (100, 1089)),
    (1536, 2048, (60, 449), (100, 1088)),
    (2048, 3072, (60, 1600), (100, 449)),
    (2048, 3072, (60, 1601), (100, 448)),
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


@pytest.mark.parametrize("m,ny,tall,short,wy", [(1536, 2048, 448, 1, 1089), (2048, 3072, 1000, 489, 1049)])
def test_pairs_of_unequal_height(torch_cuda, m, ny, tall, short, wy):
    """17 templates of different heights in one launch of the paired form: windows against the
    oracle, and bit for bit as launches of one template give them."""
    import torch

    import fastfft_b200 as F
    from oracle import fastfft_oracle as O

    rng = np.random.default_rng(m + 1)
    nx, tx, wx = 512, 60, 61
    fout, iout = (nx, ny, 1), (wx, wy, 1)
    spec = O.fwd(O.real_to_padded(rng.standard_normal((ny, nx)), fout, dtype=np.float64), fout, fout)
    spec = (spec / np.sqrt(nx * ny)).astype(np.complex64)
    heights = [tall, short, short, tall, tall - 1, short + 1] + [int(h) for h in rng.integers(short, tall + 1, 11)]
    sizes = [(tx - k % 3, h) for k, h in enumerate(heights)]
    ts = [rng.standard_normal((y, x)).astype(np.float32) for x, y in sizes]
    ins = [torch.from_numpy(O.real_to_padded(t, (x, y, 1))).cuda() for t, (x, y) in zip(ts, sizes)]
    d_spec = torch.from_numpy(spec.view(np.float32).reshape(-1).copy()).cuda()
    ft = F.FourierTransformer()
    ft.SetForwardFFTPlan(tx, tall, 1, *fout)
    ft.SetInverseFFTPlan(*fout, *iout)
    assert ft.CorrelationSize()[1] == m
    results = []
    for per_launch in (17, 1):
        ft.SetTemplatesPerLaunch(per_launch)
        outs = [torch.zeros(ft.ReturnInvOutputMemorySize(), device="cuda") for _ in ts]
        before = ft.LaunchCount()
        ft.FwdImageInvFFTManySized(ins, sizes, d_spec, outs)
        assert ft.LaunchCount() - before == 4 + 3 * (17 // per_launch)   # one class: one preparation
        results.append([O.real_from_padded(o.cpu().numpy(), iout) for o in outs])
    for t, (x, y), got, alone in zip(ts, sizes, *results):
        plan = O.Plan((x, y, 1), fout, fout, iout)
        ref = O.real_from_padded(
            O.fwd_image_inv(O.real_to_padded(t, (x, y, 1)), spec, plan, out_dtype=np.float64), iout)
        assert O.rel_l2(got, ref) <= RTOL_L2_FP32, (x, y)
        assert O.rel_max(got, ref) <= RTOL_MAX_FP32, (x, y)
        assert np.array_equal(got, alone), (x, y)


# (class, transform height, plan's template height, template height of the class, window height):
# the plan's templates are taller than the whole class is long
TALL_PLANS = [
    (256, 1024, 384, 100, 100),
    (384, 1024, 450, 150, 180),
    (512, 2048, 600, 200, 250),
    (768, 2048, 800, 250, 500),
    (1024, 3072, 1100, 300, 600),
    (1536, 4096, 1600, 500, 1000),
]


@pytest.mark.parametrize("groups", [1, 2])
@pytest.mark.parametrize("m,ny,tall,small,wy", TALL_PLANS)
def test_plan_taller_than_a_class(torch_cuda, m, ny, tall, small, wy, groups):
    """Uneven batches whose shorter templates correlate at a length below the plan's template
    height, one or two groups in flight: windows against the oracle; peaks and projection against
    those windows."""
    import torch

    import fastfft_b200 as F
    from oracle import fastfft_oracle as O

    rng = np.random.default_rng(m)
    nx, tx, wx = 512, 60, 61
    fout, iout = (nx, ny, 1), (wx, wy, 1)
    assert m // 2 < small + wy - 1 <= m < tall
    spec = O.fwd(O.real_to_padded(rng.standard_normal((ny, nx)), fout, dtype=np.float64), fout, fout)
    spec = (spec / np.sqrt(nx * ny)).astype(np.complex64)
    ft = F.FourierTransformer()
    ft.SetTemplatesPerLaunch(16 if groups == 1 else 2)
    ft.SetPipelinedGroups(groups)
    ft.SetForwardFFTPlan(tx, tall, 1, *fout)
    ft.SetInverseFFTPlan(*fout, *iout)
    assert ft.PipelinedGroups() == groups
    sizes = [(tx, small), (tx, tall), (41, small - 3), (tx, small), (23, small), (tx - 1, tall - 1)]
    ts = [rng.standard_normal((y, x)).astype(np.float32) for x, y in sizes]
    ins = [torch.from_numpy(O.real_to_padded(t, (x, y, 1))).cuda() for t, (x, y) in zip(ts, sizes)]
    d_spec = torch.from_numpy(spec.view(np.float32).reshape(-1).copy()).cuda()
    size = ft.ReturnInvOutputMemorySize()
    outs, outs2 = ([torch.zeros(size, device="cuda") for _ in ts] for _ in range(2))
    peaks = torch.zeros(len(ts), dtype=torch.int64, device="cuda")
    mip = torch.zeros(wx * wy, dtype=torch.int64, device="cuda")
    ft.FwdImageInvFFTManySized(ins, sizes, d_spec, outs)
    ft.FwdImageInvFFTManyPeaks(ins, d_spec, peaks, sizes=sizes, outputs=outs2)
    ft.FwdImageInvFFTManyMip(ins, d_spec, mip, sizes=sizes)
    wins = np.stack([O.real_from_padded(o.cpu().numpy(), iout)[0] for o in outs])
    for t, (x, y), got in zip(ts, sizes, wins):
        plan = O.Plan((x, y, 1), fout, fout, iout)
        ref = O.real_from_padded(
            O.fwd_image_inv(O.real_to_padded(t, (x, y, 1)), spec, plan, out_dtype=np.float64), iout)[0]
        assert O.rel_l2(got, ref) <= RTOL_L2_FP32, (x, y)
        assert O.rel_max(got, ref) <= RTOL_MAX_FP32, (x, y)
    for a, b in zip(outs, outs2):
        assert torch.equal(a, b)
    vals, idx = F.decode_peaks(peaks)
    flat = wins.reshape(len(ts), -1)
    assert np.array_equal(idx, flat.argmax(1)) and np.array_equal(vals, flat.max(1))
    vals, idx = F.decode_peaks(mip)
    assert np.array_equal(idx, flat.argmax(0)) and np.array_equal(vals, flat.max(0))
