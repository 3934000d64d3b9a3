"""The tensor-core contraction at 128 columns, where the A operand lies in shared memory up to a depth of 80 and in
tensor memory beyond: both sides of the line, one stage of K, ragged rows, columns and depths, and more tiles than
SMs, so that both accumulators, and the only one, are used again.  Against fp64, at the bound of the other
contraction tests, 1e-5 of the largest value of C."""
import ctypes

import numpy as np
import pytest
import torch

from fbcunn_b200 import capi

pytestmark = pytest.mark.gpu
TOL = 1e-5

# bins, m, n, k
SIZES = [(2, 1, 65, 1), (2, 128, 128, 8), (3, 129, 70, 9), (2, 130, 128, 79), (2, 129, 130, 80), (2, 129, 130, 81),
         (160, 130, 66, 17), (160, 130, 66, 84), (400, 40, 100, 80)]


@pytest.mark.parametrize("mn_a,mn_b", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_both_places_of_the_a_operand(size, mn_a, mn_b):
    bins, m, n, k = size
    rng = np.random.default_rng(m + n + k)

    def draw(rows):
        return (rng.standard_normal((bins, rows, k)) + 1j * rng.standard_normal((bins, rows, k))).astype(np.complex64)

    def stored(x, mn):  # rows padded to a multiple of four with zeros
        x = x.transpose(0, 2, 1) if mn else x
        out = np.zeros(x.shape[:2] + ((x.shape[2] + 3) // 4 * 4,), np.complex64)
        out[:, :, :x.shape[2]] = x
        return torch.from_numpy(out).cuda()

    a, b = draw(m), draw(n)
    da, db = stored(a, mn_a), stored(b, mn_b)
    c = torch.full((bins, m, (n + 3) // 4 * 4), float("nan"), dtype=torch.complex64, device="cuda")
    capi.check(capi.lib().fbfftconv_transpose_mm(
        ctypes.c_void_p(da.data_ptr()), ctypes.c_void_p(db.data_ptr()), ctypes.c_void_p(c.data_ptr()), bins, m, n, k,
        ctypes.c_float(0.5), 2 * mn_a, 1 + 2 * mn_b, 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = c.cpu().numpy()
    ref = 0.5 * np.einsum("bmk,bnk->bmn", a.astype(np.complex128), b.astype(np.complex128).conj(), optimize=True)
    assert np.abs(got[:, :, :n] - ref).max() <= TOL * np.abs(ref).max()
    assert np.all(got[:, :, n:] == 0)
    assert capi.lib().fbfftconv_tensor_core_status(0) == 0
