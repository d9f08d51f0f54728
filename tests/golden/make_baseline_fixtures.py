"""Images and gaps of iterations that amplify rounding (see
tests/test_baseline_iterations.py), as the library on the path gives them.

  python tests/golden/make_baseline_fixtures.py OUT.npz

The stored file was written by the build whose operators were the dense and
split y-transforms and the Stockham row and grid passes for every method."""

import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

# method, W, H, iterations, debug step; split (at most 48 sampled rows a frame) or fp32 y-transforms; mask of 0 and 1 or
# with weights of 0.5 to 1.5
CARTESIAN = [("TGV2", 48, 40, 50, 0, "split", "binary"), ("TGV2", 40, 36, 45, 0, "fp32", "binary"),
             ("TGV2", 96, 24, 51, 0, "split", "binary"), ("ICTV", 40, 36, 30, 0, "split", "binary"),
             ("ICTV", 64, 30, 60, 0, "fp32", "binary"), ("TV", 96, 48, 300, 20, "split", "binary"),
             ("TVTEMP", 48, 40, 60, 0, "split", "weighted")]
RADIAL = [("TGV2", 44, 40, 50), ("ICTV", 48, 44, 20)]


def name(case):
    return "_".join(str(v) for v in case)


def cartesian(av, case):
    """The image, or the gap history where there is a debug step."""
    from avionic_b200 import synth
    method, W, H, iters, step, dft, weights = case
    prob = synth.small(H, H=H, W=W, T=4, C=4, binary=weights == "binary")
    op = av.CartesianOperator(W, H, 4, 4, mask=av.to_device(prob["mask"]), centered=False)
    op.dft_mode = av.DFT_SPLIT_BF16X3 if dft == "split" else av.DFT_FP32
    s = av.Solver(method, op)
    s.set_tuning(False, 0, 0)
    s.set_debug(step > 0, max(step, 1))
    p = s.params
    p.maxIt = iters
    s.params = p
    x = av.to_device(np.repeat(synth.time_average_u0(prob["kdata"], prob["mask"], prob["b1"])[None], 4, axis=0))
    s.run(av.to_device(prob["kdata"]), x, av.to_device(prob["b1"]))
    return s.export()["PDGap"].real if step else x.cpu().numpy()


def radial(av, case):
    import torch
    from avionic_b200 import synth
    method, W, H, iters = case
    rng = np.random.default_rng(W)
    T, C, spokes, nfe = 3, 5, 9, 2 * max(W, H)
    x = torch.from_numpy(synth.phantom_ellipses(H, W, T, rng, period=T)).to("cuda", torch.complex64)
    b1 = torch.from_numpy(synth.coil_maps(H, W, C, rng)).to("cuda", torch.complex64)
    traj, dens = synth.golden_angle_radial(nfe, spokes, T)
    op = av.RadialOperator(W, H, C, T, av.to_device(traj.astype(np.float32)), av.to_device(dens.astype(np.float32)),
                           spokes, 3.0, 8.0, 1.5)
    td = torch.from_numpy(traj.astype(np.float32)).cuda()
    k = torch.stack([synth.nudft_gpu((b1 * x[t]).to(torch.complex128), td[t]).to(torch.complex64) for t in range(T)])
    k = (k / (W * H) ** 0.5 * torch.from_numpy(np.sqrt(dens).astype(np.float32)).cuda()[:, None]).contiguous()
    s = av.Solver(method, op)
    s.set_tuning(False, 0, 0)
    p = s.params
    p.maxIt = iters
    s.params = p
    u = torch.zeros_like(x)
    s.run(k, u, b1)
    return u.cpu().numpy()


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    import avionic_b200 as av
    out = {}
    for c in CARTESIAN:
        out[name(c)] = cartesian(av, c)
    for c in RADIAL:
        out["radial_" + name(c)] = radial(av, c)
    np.savez_compressed(sys.argv[1], **out)
