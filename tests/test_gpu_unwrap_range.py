"""The unwrap's segmented prefilter on maps with one value far above the others
(float32 reaches 1e36 and more): its ringing falls by 0.27 a pixel and stays above
its neighbours for tens of pixels, segments away, as in scipy's unsegmented
recursions.  Samples of both are float32 roundings of FP64 values that agree to
FP64 rounding of what they are sums of, so a ring's mean may be off by an ulp of
its samples' mean magnitude (2.5e-7, as for the samples of ordinary maps)."""
import numpy as np
import pytest

from oracle import phasing_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [128, 143, 512, 2100, 4500])  # four, two and one column a CTA
@pytest.mark.parametrize("peak", [1e18, 1e36])
def test_unwrap_of_wide_ranges(N, peak):
    import torch
    from als_speckle_b200._lib import call, ptr, stream_ptr
    c, r_out, cols = N // 2, (N - 1) // 2, 301
    places = [(c, c), (0, c), (N - 1, 1), (c - 40, N - 1)] if N < 1000 else [(c, c)]
    for r, k in places:
        m = 0.5 + np.random.default_rng(N).random((N, N)).astype(np.float32)
        m[r, k] = peak
        a = torch.from_numpy(m).cuda()
        work = torch.empty((N, N), dtype=torch.float64, device="cuda")
        mean = torch.empty(r_out, dtype=torch.float32, device="cuda")
        call("sp_unwrap", ptr(a), N, 0, r_out, float(c), float(c), cols, ptr(work), None, ptr(mean),
             stream_ptr())
        want = O.unwrap(m, 0, r_out, (c, c), columns=cols).astype(np.float64)
        off = np.abs(mean.cpu().numpy() - want.mean(axis=1))
        assert (off <= 2.5e-7 * np.abs(want).mean(axis=1)).all(), (r, k, np.argmax(off > 0))
