"""GPU per-frame PSNR / SSIM (sci_frame_metrics) against the oracle's
restatement of scikit-image 0.16's compare_psnr / compare_ssim."""
import numpy as np
import pytest
import torch

from oracle import reference_port as port
from sci_algorithms_gb300.metrics import frame_psnr_ssim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 7, 7), (3, 9, 13), (2, 64, 80), (4, 130, 257)])
def test_frame_metrics_match_scikit_image_restatement(B, H, W):
    rng = np.random.default_rng(B * 100 + H)
    a = rng.random((B, H, W)).astype(np.float32)
    b = np.clip(a + 0.05 * rng.standard_normal(a.shape), 0, 1).astype(np.float32)
    psnr, ssim = frame_psnr_ssim(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda())
    for f in range(B):
        ra = a[f].astype(np.float64)
        rb = b[f].astype(np.float64)
        assert abs(psnr[f] - port.compare_psnr(ra, rb, data_range=1.)) < 1e-9
        assert abs(ssim[f] - port.compare_ssim(ra, rb, data_range=1.)) < 1e-6


def test_frame_metrics_smooth_and_identical_frames():
    """Smooth frames (small local variance next to a large mean: where
    E[x^2] - E[x]^2 cancels) and identical frames (SSIM 1, PSNR inf)."""
    y, x = np.mgrid[0:96, 0:128] / 128.0
    a = (0.6 + 0.01 * np.sin(7 * x) * np.cos(5 * y))[None].astype(np.float32)
    b = (a + 1e-3 * np.cos(3 * x + y)[None]).astype(np.float32)
    psnr, ssim = frame_psnr_ssim(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda())
    assert abs(ssim[0] - port.compare_ssim(a[0].astype(np.float64), b[0].astype(np.float64),
                                           data_range=1.)) < 1e-6
    p2, s2 = frame_psnr_ssim(torch.from_numpy(a).cuda(), torch.from_numpy(a).cuda())
    assert p2[0] == float("inf") and abs(s2[0] - 1.0) < 1e-12
    with pytest.raises(ValueError):
        frame_psnr_ssim(torch.zeros(1, 6, 9).cuda(), torch.zeros(1, 6, 9).cuda())


def _check(a, b, data_range=1.0):
    """Both metrics of device frames a, b against the oracle.  PSNR: the
    squared errors are exact up to 2^-45, so 1e-11 dB.  SSIM: a window's 1 -
    SSIM is a quotient of float32 sums, at most ~20 roundings deep (2^-24
    each) beside the rounding of x + y, whose effect on the variance is below
    3e-6 of the denominator: 5e-6 of 1 - SSIM in all."""
    psnr, ssim = frame_psnr_ssim(a, b, data_range)
    na, nb = a.cpu().numpy().astype(np.float64), b.cpu().numpy().astype(np.float64)
    for f in range(a.shape[0]):
        p = port.compare_psnr(na[f], nb[f], data_range=data_range)
        assert psnr[f] == p or abs(psnr[f] - p) < 1e-11
        s = port.compare_ssim(na[f], nb[f], data_range=data_range)
        assert abs(ssim[f] - s) <= 5e-6 * (1 - s) + 1e-12, (f, ssim[f], s)


def _pair(B, H, W, noise=0.05, seed=0):
    rng = np.random.default_rng(seed + 1000 * H + W)
    a = rng.random((B, H, W)).astype(np.float32)
    b = np.clip(a + noise * rng.standard_normal(a.shape), 0, 1).astype(np.float32)
    return torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()


# bands of 128 columns, 120 owned; chunks of at least 8 rows, taken in pairs
@pytest.mark.parametrize("W", [7, 8, 11, 127, 128, 129, 131, 132, 247, 248, 249, 252, 367, 368, 370])
@pytest.mark.parametrize("H", [7, 8, 15, 17, 26])
def test_frame_metrics_band_and_chunk_edges(H, W):
    _check(*_pair(2, H, W))


@pytest.mark.parametrize("B,H,W", [(1, 700, 130), (700, 9, 20), (3, 513, 516)])
def test_frame_metrics_tall_and_many_frames(B, H, W):
    _check(*_pair(B, H, W, noise=0.01))


def test_frame_metrics_unaligned_and_scaled_frames():
    a, b = _pair(3, 31, 140)
    store = torch.zeros(2, a.numel() + 1, device="cuda")
    ua, ub = (s[1:].view(a.shape) for s in store)
    ua.copy_(a)
    ub.copy_(b)
    _check(ua, ub)
    for scale in (255.0, 1e-6, 3e7):
        _check(a * scale, b * scale, scale)
    # differences whose squares float32 does not hold
    c = a * 1e-3
    _check(c, torch.nextafter(c, torch.ones_like(c)))
    c = a * 1e-9
    _check(c, torch.nextafter(c, torch.ones_like(c)))
    _check(a, a + 1e-14 * (b > 0.5) + 1e-13 * (a < 1e-3))


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_frame_metrics_bad_pixel_stays_in_its_frame(bad):
    a, b = _pair(3, 40, 150)
    b[1, 20, 70] = bad
    out = torch.empty((2, 3), dtype=torch.float64, device="cuda")
    from sci_algorithms_gb300._lib import call
    call("sci_frame_metrics", a.data_ptr(), b.data_ptr(), 3, 40, 150, 1.0, out[0].data_ptr(),
         out[1].data_ptr(), torch.cuda.current_stream().cuda_stream)
    se, ss = out.cpu().tolist()
    assert (se[1] == float("inf")) if bad == float("inf") else np.isnan(se[1])
    assert np.isnan(ss[1])
    assert np.isfinite([se[0], se[2], ss[0], ss[2]]).all()
    keep = [0, 2]
    _check(a[keep].contiguous(), b[keep].contiguous())


# Frames far outside [0, data_range]: window means and moments are float32 of
# the frames as they are (finite up to 1e18 and more), quotients and squared
# errors do not depend on the range.  The tolerance is _check's, with the
# denominators' 1 - SSIM up to 2.
@pytest.mark.parametrize("size,data_range", [(1e18, 1.0), (1.0, 1e-18), (1e17, 0.25),
                                             (1e10, 1e-12), (1e-18, 1e18), (1e-3, 1e37),
                                             (1e18, 1e36), (1e-30, 1e-36)])
def test_frame_metrics_far_outside_the_data_range(size, data_range):
    a, b = _pair(2, 41, 150, noise=0.2)
    _check(a * size, b * size, data_range)
    # one frame of the stack, one window of the frame
    c, d = a.clone(), b.clone()
    c[1] *= size
    d[1] *= size
    _check(c, d, data_range)


def test_frame_psnr_of_values_near_the_float32_limit():
    a, b = _pair(1, 20, 30)
    for size, data_range in ((3e38, 1e-12), (1e30, 1e-25), (1e-37, 1.0), (1e-30, 1e38)):
        psnr, _ = frame_psnr_ssim(a * size, b * size, data_range)
        na, nb = ((t * size).cpu().numpy()[0].astype(np.float64) for t in (a, b))
        assert abs(psnr[0] - port.compare_psnr(na, nb, data_range=data_range)) < 1e-11
