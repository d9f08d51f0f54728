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


# two-step row FFTs: the shortest and longest of each first length, odd widths (8-byte row copies), row counts
# around the rows of a pass; 22, 62 and 251 have none (rows_kernel, dense)
X_CASES = [(64, 5), (99, 17), (100, 16), (121, 1), (144, 12), (143, 8), (196, 24), (225, 33), (128, 9), (256, 7),
           (160, 40), (320, 13), (22, 6), (62, 5), (251, 3)]


@pytest.mark.gpu
@pytest.mark.parametrize("centered", [False, True])
@pytest.mark.parametrize("W,rows", X_CASES)
def test_row_transform_matches_oracle(W, rows, centered):
    _check(W, 48, 3, 3, rows, centered, REL_DENSE if W in (62, 251) else REL_FFT)


@pytest.mark.gpu
@pytest.mark.parametrize("W,centered", [(64, False), (99, True), (160, True), (22, False)])
def test_reconstruction_through_the_row_transform(W, centered):
    """The z update inside the row kernel, with a weighted mask: 30 TV iterations against the oracle (fp32
    iterates stay within a few 1e-6 of float64 this early; 1e-5)."""
    import torch

    import avionic_b200 as av
    from avionic_b200 import synth
    from oracle import solvers as so
    prob = synth.small(W, H=40, W=W, T=3, C=3, binary=False)
    T, C, H, _ = prob["kdata"].shape
    op = av.CartesianOperator(W, H, C, T, mask=av.to_device(prob["mask"]), centered=centered)
    s = av.Solver("TV", op)
    p = s.params
    p.maxIt = 30
    s.params = p
    x = torch.zeros((T, H, W), dtype=torch.complex64, device="cuda")
    s.run(av.to_device(prob["kdata"]), x, av.to_device(prob["b1"]))
    oop = OCart(W, H, C, T, mask=prob["mask"], centered=centered)
    q = so.init_params("TV")
    q.lam = oop.adapt_lambda(*q.adapt_kd)
    q.maxIt = 30
    xo = so.tv(prob["kdata"].astype(complex), np.zeros((T, H, W), complex), prob["b1"].astype(complex), oop, q)
    assert _rel(x.cpu().numpy(), xo) < 1e-5


# grid splits at the ends of each first length, uneven image sides, single and several coils, window widths of 3, 4
# and 5 points, sectors that do not divide the grid; 70 x 66 (grids 140, 132) against 61 (grid 126 x 98) and a width
# whose grid has no split (107 -> 220 and 324: the Stockham passes)
R_CASES = [(64, 64, 1, 1.5, 3.0), (72, 65, 3, 1.5, 3.0), (104, 90, 2, 2.0, 3.0), (128, 120, 4, 1.5, 2.0),
           (70, 66, 2, 2.0, 4.0), (160, 85, 2, 2.0, 3.0), (107, 162, 1, 2.0, 3.0), (61, 65, 5, 2.0, 2.5)]


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,C,osf,J", R_CASES)
def test_radial_operator_matches_oracle(W, H, C, osf, J):
    """Both directions against the float64 gridding.  The samples include the grid's edges (+-1/2), where windows
    wrap.  2e-6: transforms as above, plus Kaiser-Bessel weights of fp32 table accuracy (a few 1e-7)."""
    import torch

    import avionic_b200 as av
    from oracle.radial import RadialOperator as ORad
    from oracle.radial import golden_angle_radial
    rng = np.random.default_rng(W * 100 + H)
    T, spokes, nfe = 2, 5, 2 * max(W, H) // 4 * 2
    traj, dens = golden_angle_radial(nfe, spokes, T)
    traj = traj.astype(np.float32)
    traj[:, 0, :4], traj[:, 1, :4] = (0.5, -0.5, 0.0, -1e-8), (-0.5, 0.5, -1e-8, 0.0)
    dens = dens.astype(np.float32)
    x, b1 = _cplx(rng, (T, H, W)), _cplx(rng, (C, H, W))
    k = _cplx(rng, (T, C, spokes * nfe))
    op = av.RadialOperator(W, H, C, T, av.to_device(traj), av.to_device(dens), spokes, J, 8.0, osf)
    oop = ORad(W, H, C, T, traj, dens, J, 8.0, osf)
    kg = op.backward(av.to_device(x), av.to_device(b1)).cpu().numpy()
    assert _rel(kg, oop.backward(x.astype(complex), b1.astype(complex))) < REL_FFT
    ig = op.forward(av.to_device(k), av.to_device(b1), out=torch.empty((T, H, W), dtype=torch.complex64,
                                                                     device="cuda")).cpu().numpy()
    assert _rel(ig, oop.forward(k.astype(complex), b1.astype(complex))) < REL_FFT


# one CTA of the cluster holds 1 to 6 pixels a thread, uneven blocks of rows, an image of fewer rows than CTAs
# (the per-iteration kernels), one too large for a cluster
@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(40, 7), (33, 18), (64, 64), (128, 100), (160, 130), (200, 190), (330, 320)])
@pytest.mark.parametrize("C", [1, 3])
def test_coil_loops_match_oracle(W, H, C):
    """UTGV2Recon, B1Recon and the H1 solve (fewer iterations than the defaults) against float64.  The loops are
    contractions of fp32 values: 60 iterations add at most 60 roundings of 6e-8 coherently; 1e-5."""
    import avionic_b200 as av
    from oracle import coils as oc
    rng = np.random.default_rng(W + H + C)
    yy, xx = np.meshgrid(np.linspace(-1, 1, H), np.linspace(-1, 1, W), indexing="ij")
    img = (np.exp(-3 * (yy ** 2 + xx ** 2)) + 0.2) * np.exp(1j * (xx + 0.5 * yy))
    maps = np.stack([np.exp(-((yy - np.sin(c)) ** 2 + (xx - np.cos(c)) ** 2)) * np.exp(1j * c * xx) for c in range(C)])
    crec = (maps * img + 0.01 * _cplx(rng, (C, H, W))).astype(np.complex64)
    u = img.astype(np.complex64)
    p = av.coil_default_params()
    p.uNrIt = 60
    q = oc.default_params()
    q["uNrIt"] = 60
    x1 = av.coil_utgv2(av.to_device(maps), av.to_device(crec), list(range(C)), av.to_device(u), params=p)
    xo = oc.utgv2_recon(maps.astype(np.complex64).astype(complex), crec.astype(complex), u.astype(complex),
                        list(range(C)), q)
    assert _rel(x1.cpu().numpy(), xo) < 1e-5
    b = av.coil_b1_recon(av.to_device(u), av.to_device(crec), C, 60, 2.0).cpu().numpy()
    assert _rel(b, oc.b1_recon(u.astype(complex), crec.astype(complex), C, 60, 2.0, q)) < 1e-5
    h = av.coil_b1_from_u_h1(av.to_device(u), av.to_device(crec)).cpu().numpy()
    assert _rel(h, oc.b1_from_u_h1(u.astype(complex), crec.astype(complex), q)) < 1e-5


# whole two-step column transforms (many sampled rows and enough columns for the grid), all rows, width tails, frames
# without rows; at 2.5 n1 rows and just below, where the class sums take over
@pytest.mark.gpu
@pytest.mark.parametrize("centered", [False, True])
@pytest.mark.parametrize("W,H,T,C,rows", [(250, 96, 12, 2, 96), (203, 98, 12, 1, 35), (203, 98, 12, 1, 34),
                                          (160, 128, 20, 3, 64), (167, 162, 13, 2, 50), (250, 200, 9, 2, 60)])
def test_column_transform_matches_oracle(W, H, T, C, rows, centered):
    _check(W, H, C, T, rows, centered, REL_DENSE if W in (203, 167) else REL_FFT)


# short rows
@pytest.mark.gpu
@pytest.mark.parametrize("centered", [False, True])
@pytest.mark.parametrize("W,rows", [(20, 5), (25, 17), (26, 16), (32, 3), (40, 8), (63, 13), (99, 9), (112, 20)])
def test_short_row_transform_matches_oracle(W, rows, centered):
    _check(W, 36, 3, 3, rows, centered, REL_FFT)


# gridding by half sectors: several items a warp (64 x 64, 67 and 90 frames) or shared long lists, lists longer than a batch and empty ones, every
# coil count's instance and a second pass over the coils, grids that the sectors do not divide, windows of 3 to 5 points;
# the same tolerance as for the operator
@pytest.mark.gpu
@pytest.mark.parametrize("W,H,C,T,spokes,osf,J", [(64, 64, 1, 90, 1, 1.5, 3.0), (64, 60, 3, 1, 40, 2.0, 2.0),
                                                  (21, 30, 5, 2, 9, 2.0, 3.0), (66, 64, 8, 2, 7, 1.5, 4.0),
                                                  (45, 45, 12, 3, 1, 1.5, 3.0), (33, 50, 13, 2, 6, 2.0, 3.5),
                                                  (64, 64, 17, 1, 30, 1.5, 3.0), (64, 64, 5, 67, 1, 1.5, 3.0),
                                                  (64, 64, 17, 67, 1, 1.5, 3.0)])
def test_gridding_matches_oracle(W, H, C, T, spokes, osf, J):
    import torch

    import avionic_b200 as av
    from oracle.radial import RadialOperator as ORad
    from oracle.radial import golden_angle_radial
    rng = np.random.default_rng(W * 100 + C)
    nfe = 2 * max(W, H) // 4 * 2
    traj, dens = golden_angle_radial(nfe, spokes, T)
    traj, dens = traj.astype(np.float32), dens.astype(np.float32)
    b1, k = _cplx(rng, (C, H, W)), _cplx(rng, (T, C, spokes * nfe))
    op = av.RadialOperator(W, H, C, T, av.to_device(traj), av.to_device(dens), spokes, J, 8.0, osf)
    ig = op.forward(av.to_device(k), av.to_device(b1), out=torch.empty((T, H, W), dtype=torch.complex64,
                                                                     device="cuda")).cpu().numpy()
    oop = ORad(W, H, C, T, traj, dens, J, 8.0, osf)
    assert _rel(ig, oop.forward(k.astype(complex), b1.astype(complex))) < REL_FFT


# row lengths whose threads do not fill whole warps (first lengths 5, 11, 13 and 15), at each number of rows a pass
@pytest.mark.gpu
@pytest.mark.parametrize("kc", [8, 12, 16])
@pytest.mark.parametrize("W", [20, 99, 104, 150])
def test_row_sums_match_oracle(W, kc):
    """The sums of the step rule and of the gap, which the row kernel adds up over a block: 21 ICTGV2 iterations
    (its step rule lowers sigma and tau early; the stop test evaluates the gap at the 21st).  A sum of squares of
    values good to 2e-6 is good to 4e-6, and sigma and tau are roots of ratios of such sums: 1e-5; the gap adds
    eight sums without cancellation this early: 2e-5."""
    import torch

    import avionic_b200 as av
    from avionic_b200 import synth
    from oracle import solvers as so
    prob = synth.small(W, H=28, W=W, T=3, C=3)
    T, C, H, _ = prob["kdata"].shape
    op = av.CartesianOperator(W, H, C, T, mask=av.to_device(prob["mask"]), centered=False)
    s = av.Solver("ICTGV2", op)
    p = s.params
    p.maxIt, p.stopPDGap = 21, 1e-30
    s.params = p
    s.set_tuning(False, 0, 0)
    s.set_kspace_schedule(kc, False)
    x = torch.zeros((T, H, W), dtype=torch.complex64, device="cuda")
    s.run(av.to_device(prob["kdata"]), x, av.to_device(prob["b1"]))
    oop = OCart(W, H, C, T, mask=prob["mask"], centered=False)
    q = so.init_params("ICTGV2")
    q.lam = oop.adapt_lambda(*q.adapt_kd)
    q.maxIt, q.stopPDGap = 21, 1e-30
    tr = {}
    so.run("ICTGV2", prob["kdata"].astype(complex), np.zeros((T, H, W), complex), prob["b1"].astype(complex), oop, q, tr)
    st = s.stats()
    assert tr["steps"][-1][0] < 0.99 * q.sigma  # the rule has acted
    assert abs(st.sigma - tr["steps"][-1][0]) < 1e-5 * st.sigma
    assert abs(st.tau - tr["steps"][-1][1]) < 1e-5 * st.tau
    assert abs(st.last_gap - tr["PDGap"][-1]) < 2e-5 * tr["PDGap"][-1]


# gridding with several half sectors a warp (9472 sectors and frames or more): the benchmark's 12 coils with the most a
# warp takes and a last block that is not full, windows of 3 and 5 points
@pytest.mark.gpu
@pytest.mark.parametrize("W,H,C,T,osf,J", [(66, 64, 12, 251, 1.5, 3.0), (64, 64, 3, 70, 1.5, 2.0),
                                           (64, 64, 9, 70, 1.5, 4.0)])
def test_gridding_of_many_sectors_matches_oracle(W, H, C, T, osf, J):
    test_gridding_matches_oracle(W, H, C, T, 1, osf, J)
