"""The Cartesian operator's transforms at the sizes where their kernels change
form, against the float64 oracle.

Tolerance: an output value is a sum of H W products formed in fp32 through
register FFTs (at most about 16 roundings deep, each 6e-8 relative, adding as
independent errors) and sums of at most 64 terms; 2e-6 relative L2 is five
times what these give.  The dense forms (heights or widths without a factor
for the FFTs) sum the whole axis, and the split form's accumulator truncates:
1e-5, as the operator tests hold them."""

import numpy as np
import pytest

from oracle.cartesian import CartesianOperator as OCart

REL_FFT, REL_DENSE = 2e-6, 1e-5


def _rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def _cplx(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def _check(W, H, C, T, rows, centered, tol, dft=None):
    import avionic_b200 as av
    rng = np.random.default_rng(W * 1009 + H * 31 + C)
    mask = np.zeros((T, H, W), np.float32)
    for t in range(T):
        n = rows if t != 1 else max(0, rows - 1)  # frames of unequal counts, an empty one with rows == 1
        mask[t, rng.choice(H, size=n, replace=False)] = 1
    mask *= rng.uniform(0.5, 1.5, mask.shape).astype(np.float32)
    op = av.CartesianOperator(W, H, C, T, mask=av.to_device(mask), centered=centered)
    if dft is not None:
        op.dft_mode = dft
    oop = OCart(W, H, C, T, mask=mask, centered=centered)
    x, b1, k = _cplx(rng, (T, H, W)), _cplx(rng, (C, H, W)), _cplx(rng, (T, C, H, W))
    kg = op.backward(av.to_device(x), av.to_device(b1)).cpu().numpy()
    assert _rel(kg, oop.backward(x.astype(complex), b1.astype(complex))) < tol
    kd = av.to_device(k)
    ig = op.forward(kd, av.to_device(b1)).cpu().numpy()
    assert _rel(ig, oop.forward(k.astype(complex), b1.astype(complex))) < tol


# every register FFT length along y with a short and a long class sum, one to
# all rows, column tiles that end inside the image, odd and single coils
Y_CASES = [(16 * 2, 3, 2), (16 * 20, 53, 4), (15, 15, 1), (15 * 7, 30, 3), (14 * 3, 9, 5), (13, 1, 2), (13 * 11, 40, 3),
           (12 * 16 // 12 * 12, 16, 16), (11 * 5, 20, 7), (10 * 13, 44, 2), (9 * 9, 48, 3), (8 * 17, 49, 2),
           (7 * 23, 25, 3), (6 * 37, 60, 2), (5 * 61, 19, 9), (4 * 53, 106, 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("centered", [False, True])
@pytest.mark.parametrize("H,rows,C", Y_CASES)
def test_y_transform_matches_oracle(H, rows, C, centered):
    _check(20 + H % 13, H, C, 3, rows, centered, REL_DENSE if (20 + H % 13) in (23, 29, 31) else REL_FFT)


@pytest.mark.gpu
@pytest.mark.parametrize("dft", [0, 1])
@pytest.mark.parametrize("H,rows", [(34, 7), (37, 20), (4 * 29, 30)])
def test_heights_without_a_register_fft(H, rows, dft):
    _check(24, H, 3, 3, rows, True, REL_DENSE, dft)
