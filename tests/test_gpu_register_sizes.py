"""Registration's line kernels and matrix products over their sizes: every
transform size's line layout, odd and non-square crops, and every number of
32-column groups of the fine grid (M = ceil(1.5 U) from 2 to 255), against the
FP64 oracle.  Shifts lie on the 1/U grid and there is no noise, so FP32 and
FP64 pick the same grid point (neighbouring points differ by > 1e-5 of the
peak, FP32 sums by ~1e-6); aligned frames to 1e-5, as for the registration of
crops in a larger transform."""
import numpy as np
import pytest

from oracle import phasing_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,U,frames", [
    (7, 5, 1, 3), (16, 11, 3, 5), (30, 32, 21, 9), (33, 64, 22, 4), (100, 128, 64, 3), (250, 181, 85, 3),
    (256, 64, 86, 2), (60, 50, 128, 4), (60, 50, 149, 4), (60, 50, 170, 17), (513, 300, 16, 2),
    (1100, 30, 4, 2), (2049, 20, 2, 1)])
def test_register_sizes_vs_oracle(rows, cols, U, frames):
    from als_speckle_b200.phasing import align_frames_subpixel
    rng = np.random.default_rng(rows * cols + U)
    N = max(8, 1 << (max(rows, cols) - 1).bit_length())
    base = np.zeros((rows, cols), np.complex128)
    br, bc = max(2, rows // 2), max(2, cols // 2)
    r0, c0 = (rows - br) // 2, (cols - bc) // 2
    base[r0:r0 + br, c0:c0 + bc] = rng.random((br, bc)) * np.exp(1j * rng.uniform(-1, 1, (br, bc)))
    data = []
    for _ in range(frames):
        dy, dx = rng.integers(-U, U + 1, 2) / U
        data.append(O.fourier_shift(base, dy, dx, N=N) * np.exp(1j * rng.uniform(-np.pi, np.pi)))
    data = np.stack(data).astype(np.complex64)
    ref = base.astype(np.complex64)
    aligned, d = align_frames_subpixel(data, align_to=ref, upsample=U, return_type="both")
    wd, wal = O.register_subpixel(data.astype(np.complex128), ref.astype(np.complex128), N=N, upsample=U)
    # the same grid points (as numerators over U: n/U and d0 + p/U round differently)
    assert np.array_equal(np.rint(d[:, :2] * U), np.rint(wd[:, :2] * U))
    assert np.max(np.abs(np.angle(np.exp(1j * (d[:, 2] - wd[:, 2]))))) < 1e-4
    assert np.linalg.norm(aligned - wal) / np.linalg.norm(wal) < 1e-5
