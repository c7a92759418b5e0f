"""The Fourier filter of small arrays in shared memory: one- and two-stage axes, every radix,
odd inner axes, axes of length one, self-mirrored planes, batches below and above a wave, and
shapes that take cuFFT (odd first axis, a prime above 16, too large for shared memory), against
numpy in double precision.

Tolerance: the transforms round in FP32, about 2e-7 of the array's size each; 1e-5 of the largest
value holds with room to spare."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("shape,batch", [
    ((32, 32, 32), 3), ((32, 32, 32), 200), ((36, 36, 36), 2),
    ((36, 36, 36), 70), ((12, 12, 12), 700),
    ((2, 1, 1), 2), ((2, 3, 2), 5), ((14, 1, 9), 4), ((24, 22, 26), 3), ((20, 21, 25), 2),
    ((30, 33, 15), 2), ((10, 200, 11), 2), ((512, 3, 4), 2), ((4, 6, 256), 2), ((28, 28, 28), 149),
    ((33, 32, 32), 2), ((34, 34, 34), 2), ((48, 48, 48), 2)])
def test_fft_filter_matches_numpy(shape, batch):
    import torch

    from pytme_b200.refine import _FilterPlan

    rng = np.random.default_rng(sum(shape) + batch)
    x = rng.standard_normal((batch,) + shape).astype(np.float32)
    half = shape[:2] + (shape[2] // 2 + 1,)
    filt = rng.random(half).astype(np.float32)
    # even under k -> -k in the planes that are their own mirror, as filters are
    mirror = filt[np.ix_(-np.arange(half[0]) % half[0], -np.arange(half[1]) % half[1])]
    for k in {0, shape[2] // 2 if shape[2] % 2 == 0 else 0}:
        filt[..., k] = 0.5 * (filt[..., k] + mirror[..., k])
    plan = _FilterPlan(shape, batch)
    got = torch.as_tensor(x).cuda()
    spectrum = torch.empty((batch,) + half, dtype=torch.complex64, device="cuda")
    plan.apply(got, spectrum, torch.as_tensor(filt).cuda())
    want = np.fft.irfftn(np.fft.rfftn(x.astype(np.float64), axes=(1, 2, 3)) * filt,
                         s=shape, axes=(1, 2, 3))
    assert np.abs(got.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()
