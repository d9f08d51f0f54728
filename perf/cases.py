"""Performance cases: the work a user of this framework has it do, through its
public entry points.

Kinds of case:

* ``recon``   Cartesian reconstruction (CartesianOperator + Solver.run): any of
  the five methods, line masks at acceleration R (binary or weighted), centred
  or uncentred transform, optionally with the gap history of the debug export;
* ``radial``  radial reconstruction (RadialOperator + Solver.run);
* ``host``    reconstruct_host: host buffers in and out, the CLI's path;
* ``stream``  a batch of mixed requests through BatchEngine;
* ``coils``   H1 coil-sensitivity estimation from Cartesian or radial data;
* ``apply``   one operator round trip, image -> k-space -> image, as a program
  with a solver of its own applies it.

Inputs are seeded phantoms, coil maps, masks and trajectories of the benchmark
problems' kinds; ``exact`` restates each kind in float64 torch.
"""

import ctypes
import math
import random

import numpy as np
import torch

import avionic_b200 as av
from avionic_b200 import synth

PROTOCOL_SEED = 11  # sampling masks and trajectories belong to the scan protocol, not to the subject
C8 = 8              # bytes of a complex64 value
COMPONENTS = {"TV": (1, 3), "TVTEMP": (1, 1), "TGV2": (4, 9), "ICTV": (2, 6), "ICTGV2": (8, 18)}


def listed():
    return [
        # the smallest reconstruction a program asks for (a preview, a unit of a larger search): launches and latency
        dict(name="tgv2_24x20", kind="recon", method="TGV2", W=20, H=24, T=6, C=4, R=4, iters=50, centered=False,
             weighted=False, gap=0),
        # the plain TV reconstruction of a short 2D+t scan, whose fields fit in cache
        dict(name="tv_128", kind="recon", method="TV", W=128, H=128, T=20, C=8, R=8, iters=500, centered=False,
             weighted=False, gap=0),
        # cardiac cine at high acceleration, the default configuration's 500 iterations
        dict(name="ictgv2_cine_192", kind="recon", method="ICTGV2", W=192, H=192, T=30, C=16, R=12, iters=500,
             centered=False, weighted=False, gap=0),
        # the largest matrix, frame and coil counts of the batched set, at its lowest acceleration
        dict(name="tgv2_320_r6", kind="recon", method="TGV2", W=320, H=320, T=48, C=32, R=6, iters=100,
             centered=False, weighted=False, gap=0),
        # ragged sizes (rectangular matrix, a prime height, odd frames and coils), centred transform, density-weighted
        # mask, with the debug export's gap history
        dict(name="ictv_ragged_gap", kind="recon", method="ICTV", W=150, H=131, T=13, C=7, R=4, iters=200,
             centered=True, weighted=True, gap=10),
        # parallel imaging at low acceleration: half of the lines sampled
        dict(name="tvtemp_r2", kind="recon", method="TVTEMP", W=160, H=128, T=24, C=12, R=2, iters=200,
             centered=False, weighted=False, gap=0),
        # golden-angle radial dynamic imaging, the radial benchmark's geometry
        dict(name="radial_tgv2_128", kind="radial", method="TGV2", W=128, H=128, T=40, C=12, spokes=21, readout=256,
             osf=1.5, iters=250),
        # a smaller radial scan with the default configuration's grid oversampling of 2 and uneven sizes
        dict(name="radial_tv_104", kind="radial", method="TV", W=104, H=90, T=23, C=5, spokes=13, readout=208,
             osf=2.0, iters=200),
        # coil maps before a radial reconstruction
        dict(name="coils_radial_128", kind="coils", W=128, H=128, T=40, C=12, spokes=21, readout=256, R=0),
        # operator round trip of the cine problem, centred as a default-constructed operator is
        dict(name="apply_cine_192", kind="apply", W=192, H=192, T=30, C=16, R=12, spokes=0, readout=0, osf=0.0,
             centered=True),
        # the served mix: methods, sizes and operators of the request stream, the stop test's gap every 20 iterations
        dict(name="serve_mix", kind="stream", n=6, mix=22, iters=100),
        # host buffers to host buffers, one protocol's scans one after another
        dict(name="host_tgv2_160", kind="host", method="TGV2", W=160, H=160, T=24, C=10, R=8, iters=200,
             centered=False, weighted=False, gap=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges (work no larger than the largest listed case's of its kind)."""
    while True:
        case = _draw(rng)
        if work(case)["bytes"] <= max(work(c)["bytes"] for c in listed() if c["kind"] == case["kind"]):
            return case


def _draw(rng):
    kind = rng.choice(["recon"] * 5 + ["radial"] * 2 + ["apply"] * 2 + ["coils", "stream", "host"])
    if kind == "stream":
        return dict(kind="stream", n=rng.randint(2, 6), mix=rng.randrange(1000), iters=rng.randrange(20, 101, 20))
    T, C = _log_int(rng, 4, 48), _log_int(rng, 3, 32)
    if kind in ("radial", "coils") or (kind == "apply" and rng.random() < 0.4):
        W, H = _log_int(rng, 64, 160), _log_int(rng, 64, 160)
        T, C = max(T, 8), min(C, 16)
        geometry = dict(spokes=rng.randint(8, 34), readout=2 * max(W, H))
        osf = rng.choice([1.5, 2.0])
        if kind == "coils":
            C = min(C, 12)
            if rng.random() < 0.5:  # Cartesian data; the time average needs image sides with factors up to 13
                W, H = (rng.choice([64, 90, 96, 110, 128, 130, 154, 160]) for _ in range(2))
                return dict(kind="coils", W=W, H=H, T=T, C=C, spokes=0, readout=0, R=rng.randint(3, 12))
            return dict(kind="coils", W=W, H=H, T=T, C=C, R=0, **geometry)
        if kind == "apply":
            return dict(kind="apply", W=W, H=H, T=T, C=C, R=0, osf=osf, centered=False, **geometry)
        return dict(kind=kind, method=rng.choice(["TV", "TGV2", "ICTGV2"]), W=W, H=H, T=T, C=C, osf=osf,
                    iters=_log_int(rng, 40, 250), **geometry)
    W, H = _log_int(rng, 20, 320), _log_int(rng, 20, 320)
    if rng.random() < 0.5:
        W = H = rng.choice(list(synth.MATRICES))
    R = rng.randint(2, 16)
    centered = rng.random() < 0.3
    if kind == "apply":
        return dict(kind=kind, W=W, H=H, T=T, C=C, R=R, spokes=0, readout=0, osf=0.0, centered=centered)
    case = dict(kind=kind, method=rng.choice(["TV", "TVTEMP", "TGV2", "TGV2", "ICTV", "ICTGV2"]), W=W, H=H, T=T, C=C,
                R=R, iters=_log_int(rng, 30, 500), centered=False, weighted=False, gap=0)
    if kind == "recon":
        case.update(centered=centered, weighted=rng.random() < 0.2, gap=20 if rng.random() < 0.3 else 0)
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _dev(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)


def _subject(case, seed):
    """Phantom (T,H,W) and coil maps (C,H,W), complex64 on the GPU."""
    rng = np.random.default_rng(seed)
    make = synth.phantom_ellipses if case.get("method") in ("TV", "TVTEMP") else synth.phantom_cine
    x = make(case["H"], case["W"], case["T"], rng, period=30)
    return _dev(x, torch.complex64), _dev(synth.coil_maps(case["H"], case["W"], case["C"], rng), torch.complex64)


def _add_noise(k, seed, rel):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    sd = rel * float(k.abs().max()) / math.sqrt(2.0)
    for t in range(k.shape[0]):
        k[t] += torch.complex(*(sd * torch.randn(k.shape[1:], generator=g, device="cuda") for _ in range(2)))
    return k


def _f_img_to_k(v, centered):
    """The operators' unitary image -> k-space transform (e^{+2 pi i} kernel)."""
    if centered:
        v = torch.fft.ifftshift(v, dim=(-2, -1))
    v = torch.fft.ifft2(v, norm="ortho")
    return torch.fft.fftshift(v, dim=(-2, -1)) if centered else v


def _f_k_to_img(k, centered):
    if centered:
        k = torch.fft.ifftshift(k, dim=(-2, -1))
    k = torch.fft.fft2(k, norm="ortho")
    return torch.fft.fftshift(k, dim=(-2, -1)) if centered else k


def _cartesian_inputs(case, seed):
    T, H, W = case["T"], case["H"], case["W"]
    x, b1 = _subject(case, seed)
    mask = synth.mask_variable_density(H, W, T, case["R"], np.random.default_rng(PROTOCOL_SEED))
    if case.get("weighted"):
        mask = mask * np.random.default_rng(PROTOCOL_SEED + 1).uniform(0.5, 1.5, mask.shape).astype(np.float32)
    mask = _dev(mask, torch.float32)
    centered = case.get("centered", False)
    if centered:
        mask = torch.roll(mask, (H // 2,), (1,)).contiguous()
    k = torch.empty((T, case["C"], H, W), dtype=torch.complex64, device="cuda")
    for t in range(T):
        k[t] = _f_img_to_k(b1 * x[t], centered)
    k = _add_noise(k, seed, 1e-3) * mask[:, None]
    # start image: coil-combined time average, one frame
    u0 = (b1.conj() * _f_k_to_img(k.sum(0) / mask.sum(0).clamp(min=1.0), centered)).sum(0)
    return dict(k=k, mask=mask, b1=b1, u0=u0, x0=u0[None].repeat(T, 1, 1).contiguous(), truth=x)


def _radial_inputs(case, seed):
    T, C = case["T"], case["C"]
    x, b1 = _subject(case, seed)
    traj, dens = synth.golden_angle_radial(case["readout"], case["spokes"], T)
    traj, dens = _dev(traj, torch.float32), _dev(dens, torch.float32)
    k = torch.empty((T, C, traj.shape[2]), dtype=torch.complex64, device="cuda")
    for t in range(T):
        k[t] = synth.nudft_gpu((b1 * x[t]).to(torch.complex128), traj[t]) / math.sqrt(case["W"] * case["H"])
    k = (_add_noise(k, seed, 2e-3) * dens.sqrt()[:, None]).contiguous()
    return dict(k=k, traj=traj, dens=dens, b1=b1, x0=torch.zeros_like(x), truth=x)


def _requests(case):
    """Sizes of a stream's requests: the served mix (methods 50/30/20 %, 70 % Cartesian, 30 % radial)."""
    r = random.Random(case["mix"])
    out = []
    for i in range(case["n"]):
        method = r.choices(["TV", "TGV2", "ICTGV2"], [5, 3, 2])[0]
        if r.random() < 0.7:
            m = r.choice(list(synth.MATRICES))
            out.append(dict(kind="recon", method=method, W=m, H=m, T=r.randint(8, 48), C=r.randint(4, 32),
                            R=r.randint(6, 16), iters=case["iters"]))
        else:
            out.append(dict(kind="radial", method=method, W=128, H=128, T=r.randint(20, 60), C=12,
                            spokes=r.randint(13, 34), readout=256, osf=1.5, iters=case["iters"]))
    return out


def _inputs(case, seed):
    return _radial_inputs(case, seed) if case.get("spokes") else _cartesian_inputs(case, seed)


def _operator(case, d):
    if case.get("spokes"):
        return av.RadialOperator(case["W"], case["H"], case["C"], case["T"], d["traj"], d["dens"], case["spokes"], 3.0,
                                 8.0, case["osf"])
    return av.CartesianOperator(case["W"], case["H"], case["C"], case["T"], mask=d["mask"],
                                centered=bool(case.get("centered")))


def _params(case):
    p = av.default_params(av.METHODS[case["method"]])
    p.maxIt = case["iters"]
    return p


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "stream":
        s["engine"] = av.BatchEngine(workers=4)
        s["reqs"], s["x"], s["x0"] = [], [], []
        for i, c in enumerate(_requests(case)):
            d = _inputs(c, seed + 1000 * i)
            x = torch.empty_like(d["x0"])
            p = _params(c)
            p.stopPDGap = 1e-12  # evaluated every 20 iterations; never met within these iteration counts
            if c["kind"] == "radial":
                q = av.radial_request(c["method"], d["k"], x, d["b1"], d["traj"], d["dens"], c["spokes"], c["readout"],
                                      params=p, osf=c["osf"], tag=i)
            else:
                q = av.cartesian_request(c["method"], d["k"], x, d["b1"], mask=d["mask"], params=p, tag=i)
            s["reqs"].append((q, d))
            s["x"].append(x)
            s["x0"].append(d["x0"])
        return s
    d = _inputs(case, seed)
    if kind == "host":
        s["args"] = [d[n].cpu().pin_memory().numpy() for n in ("k", "mask", "b1", "u0")]
        s["params"] = _params(case)
        return s
    s.update(d)
    if kind == "coils":
        shape = (case["C"], case["H"], case["W"])
        s["u"] = torch.empty(shape, dtype=torch.complex64, device="cuda")
        s["maps"] = torch.empty_like(s["u"])
        return s
    s["op"] = _operator(case, d)
    if kind == "apply":
        s["x0"] = d["truth"]
        s["kout"], s["img"] = torch.empty_like(d["k"]), torch.empty_like(d["truth"])
        return s
    s["solver"] = av.Solver(case["method"], s["op"], _params(case))
    if case.get("gap"):
        s["solver"].set_debug(True, case["gap"])
    s["params"] = s["solver"].params  # every pass starts from these step sizes (a run adapts them)
    s["x"] = torch.empty_like(d["x0"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "stream":
        for x, x0 in zip(s["x"], s["x0"]):
            x.copy_(x0)
        torch.cuda.current_stream().synchronize()  # the engine's streams are its own
        for q, _ in s["reqs"]:
            s["engine"].submit(q)
        done = []
        while len(done) < len(s["reqs"]):
            done += s["engine"].poll(wait_ms=-1)
        for c in done:
            av.check(c.status)
        return s["x"]
    if kind == "host":
        k, mask, b1, u0 = s["args"]
        x, _ = av.reconstruct_host(case["method"], k, mask, b1, u0, params=s["params"])
        return dict(x=x)
    if kind == "coils":
        W, H, C, T = case["W"], case["H"], case["C"], case["T"]
        if not case["spokes"]:
            u, b1 = av.coil_construction(s["k"], s["mask"])
            return dict(u=u, b1=b1)
        av.check(av.lib.avx_coil_construction_radial(
            W, H, C, T, s["k"].shape[2], ctypes.byref(av.coil_default_params()), av._cptr(s["traj"]),
            av._cptr(s["dens"]), av._cptr(s["k"]), av._cptr(s["u"]), av._cptr(s["maps"])))
        return dict(u=s["u"], b1=s["maps"])
    if kind == "apply":
        return dict(k=s["op"].backward(s["x0"], s["b1"], out=s["kout"]),
                    img=s["op"].forward(s["k"], s["b1"], out=s["img"]))
    s["x"].copy_(s["x0"])
    s["solver"].params = s["params"]
    s["solver"].run(s["k"], s["x"], s["b1"])
    out = dict(x=s["x"])
    if case.get("gap"):
        st = s["solver"].stats()
        out.update(gap=st.last_gap, sigma=st.sigma, tau=st.tau)
    return out


# ---------------------------------------------------------------------------
# work: every state and input array of an iteration read or written once
# ---------------------------------------------------------------------------

def _grid(d, osf):
    n = 2 * math.ceil(osf * d / 2.0)
    while True:
        m = n
        for p in (2, 3, 5, 7, 11, 13):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 2


def _round_trip(case):
    """(values of k-space, flops of one operator application and one adjoint)."""
    W, H, T, C = case["W"], case["H"], case["T"], case["C"]
    if case.get("spokes"):
        S = case["spokes"] * case["readout"]
        osf = case.get("osf") or 2.0
        g = _grid(W, osf) * _grid(H, osf)
        return C * T * S, 2.0 * C * T * (5.0 * g * math.log2(g) + 8.0 * W * H + 64.0 * S)
    rows = max(1, round(H / case["R"]))
    col = min(8.0 * rows * H, 5.0 * H * math.log2(H))  # one column onto the sampled rows
    return C * T * rows * W, 2.0 * C * T * (W * col + rows * 5.0 * W * math.log2(W) + 8.0 * W * H)


def _recon_work(case):
    P, D = COMPONENTS[case["method"]]
    N = case["W"] * case["H"] * case["T"]
    K, fl = _round_trip(case)
    maps = case["W"] * case["H"] * case["C"]
    return (case["iters"] * C8 * (4.0 * P * N + 2.0 * D * N + 3.0 * K + maps),
            case["iters"] * (fl + 30.0 * N * (P + D)))


def work(case):
    kind = case["kind"]
    if kind == "stream":
        each = [_recon_work(c) for c in _requests(case)]
        return dict(bytes=sum(b for b, _ in each), flops=sum(f for _, f in each))
    N = case["W"] * case["H"]
    if kind == "coils":
        # C UTGV2 runs (100 iterations, 12 fields), C - 1 single-coil B1 runs (500, 4 fields), one of C coils (1000)
        C = case["C"]
        k = C * case["T"] * (case["spokes"] * case["readout"] if case["spokes"] else N)
        fields = C * 100 * (2 * 12 + 2) + (C - 1) * 500 * (2 * 4 + 2) + 1000 * C * (2 * 4 + 2)
        return dict(bytes=C8 * (k + 2.0 * C * N + float(fields) * N), flops=8.0 * fields * N)
    if kind == "apply":
        K, fl = _round_trip(case)
        dense = K if case["spokes"] else N * case["T"] * case["C"]  # Cartesian k-space is dense on both sides
        return dict(bytes=C8 * (2.0 * N * case["T"] + 2.0 * N * case["C"] + K + 2.0 * dense), flops=fl)
    b, f = _recon_work(case)
    if kind == "host":
        b += C8 * (N * case["C"] * case["T"] + N * case["C"] + N * case["T"])
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------
# the same results in float64
# ---------------------------------------------------------------------------

class _Cart:
    def __init__(self, case, d):
        self.mask, self.centered = d["mask"].double()[:, None], bool(case.get("centered"))
        self.subfac = d["mask"].numel() / float((d["mask"].double() ** 2).sum())

    def to_k(self, x, b1):
        k = torch.empty((x.shape[0],) + b1.shape, dtype=torch.complex128, device=x.device)
        for t in range(x.shape[0]):
            k[t] = _f_img_to_k(b1 * x[t], self.centered)
        return k.mul_(self.mask)

    def to_img(self, z, b1):
        z.mul_(self.mask)  # in place, as the reference's ForwardOperation masks its input
        out = torch.empty((z.shape[0],) + b1.shape[1:], dtype=torch.complex128, device=z.device)
        for t in range(z.shape[0]):
            out[t] = (b1.conj() * _f_k_to_img(z[t], self.centered)).sum(0)
        return out


class _Radial:
    """Tapered Kaiser-Bessel gridding (width 3, Beatty's shape parameter, Gauss-Legendre deapodisation)."""

    def __init__(self, W, H, traj, dens, osf, spokes):
        J = 3.0
        self.W, self.H, self.Gx, self.Gy = W, H, _grid(W, osf), _grid(H, osf)
        self.subfac = W / (spokes * math.pi / 2.0)
        beta = math.pi * math.sqrt((J / osf) ** 2 * (osf - 0.5) ** 2 - 0.8)

        def kb(u):
            a = (1.0 - (2.0 * u / J) ** 2).clamp(min=0.0)
            w = (torch.special.i0(beta * a.sqrt()) - 1.0) / (float(np.i0(beta)) - 1.0)
            return torch.where(u.abs() < J / 2.0, w, torch.zeros_like(w))

        xg, wg = np.polynomial.legendre.leggauss(64)
        t = torch.from_numpy(xg * J / 2.0).cuda()
        wt = torch.from_numpy(wg * J / 2.0).cuda() * kb(t)

        def psi(d, G):
            p = torch.arange(d, device="cuda", dtype=torch.float64) - d // 2
            return (wt * torch.cos(2.0 * math.pi * t * p[:, None] / G)).sum(1)

        self.ipsi = 1.0 / (psi(H, self.Gy)[:, None] * psi(W, self.Gx)[None])
        self.iy = (torch.arange(H, device="cuda") - H // 2) % self.Gy
        self.ix = (torch.arange(W, device="cuda") - W // 2) % self.Gx
        offs = torch.arange(4, device="cuda")

        def window(kappa, G):
            g = torch.floor(kappa - J / 2.0).long()[..., None] + offs
            return g % G, kb(kappa[..., None] - g)

        ax, wx = window(traj[:, 0].double() * self.Gx, self.Gx)
        ay, wy = window(traj[:, 1].double() * self.Gy, self.Gy)
        T, S = dens.shape
        self.idx = (ay[..., :, None] * self.Gx + ax[..., None, :]).reshape(T, S * 16)
        scale = dens.double().sqrt() / math.sqrt(W * H)
        self.w = ((wy[..., :, None] * wx[..., None, :]).reshape(T, S, 16) * scale[..., None]).reshape(T, S * 16)

    def to_k(self, x, b1):
        T, C = x.shape[0], b1.shape[0]
        out = torch.empty((T, C, self.w.shape[1] // 16), dtype=torch.complex128, device=x.device)
        for t in range(T):
            v = torch.zeros((C, self.Gy, self.Gx), dtype=torch.complex128, device=x.device)
            v[:, self.iy[:, None], self.ix[None]] = b1 * x[t] * self.ipsi
            v = torch.fft.fft2(v).reshape(C, -1)
            out[t] = (v[:, self.idx[t]] * self.w[t]).reshape(C, -1, 16).sum(2)
        return out

    def to_img(self, z, b1):
        T, C = z.shape[0], b1.shape[0]
        out = torch.empty((T, self.H, self.W), dtype=torch.complex128, device=z.device)
        for t in range(T):
            out[t] = (b1.conj() * self.images(t, z[t])).sum(0)
        return out

    def images(self, t, z):
        """Coil images (C,H,W) of one frame's samples (C,S)."""
        C = z.shape[0]
        v = torch.zeros((C, self.Gy * self.Gx, 2), dtype=torch.float64, device=z.device)
        q = (z[:, :, None] * self.w[t].reshape(1, -1, 16)).reshape(C, -1)
        v.index_add_(1, self.idx[t], torch.view_as_real(q))
        g = torch.fft.ifft2(torch.view_as_complex(v).reshape(C, self.Gy, self.Gx)) * (self.Gx * self.Gy)
        return g[:, self.iy[:, None], self.ix[None]] * self.ipsi


def _fwd(u, a):  # D+ along axis a, zero at the last index
    r = torch.zeros_like(u)
    n = u.shape[a]
    r.narrow(a, 0, n - 1).copy_(u.narrow(a, 1, n - 1) - u.narrow(a, 0, n - 1))
    return r


def _fwd_t(u, a):  # (D+)^T
    r = torch.zeros_like(u)
    n = u.shape[a]
    r.narrow(a, 1, n - 1).add_(u.narrow(a, 0, n - 1))
    r.narrow(a, 0, n - 1).sub_(u.narrow(a, 0, n - 1))
    return r


def _grad(u, w):
    return [_fwd(u, 2) / w[0], _fwd(u, 1) / w[1], _fwd(u, 0) / w[2]]


def _div(y, w):
    return -(_fwd_t(y[0], 2) / w[0] + _fwd_t(y[1], 1) / w[1] + _fwd_t(y[2], 0) / w[2])


def _symgrad(v, w):  # the backward difference is -(D+)^T; the yt entry scales its y part by 1 / (2 dx)
    b = lambda u, a: -_fwd_t(u, a)  # noqa: E731
    return [b(v[0], 2) / w[0], b(v[1], 1) / w[1], b(v[2], 0) / w[2],
            b(v[0], 1) / (2 * w[1]) + b(v[1], 2) / (2 * w[0]), b(v[0], 0) / (2 * w[2]) + b(v[2], 2) / (2 * w[0]),
            b(v[1], 0) / (2 * w[2]) + b(v[2], 1) / (2 * w[0])]


def _symdiv(e, w):
    return [_fwd(e[0], 2) / w[0] + _fwd(e[3], 1) / w[1] + _fwd(e[4], 0) / w[2],
            _fwd(e[3], 2) / w[0] + _fwd(e[1], 1) / w[1] + _fwd(e[5], 0) / w[2],
            _fwd(e[4], 2) / w[0] + _fwd(e[5], 1) / w[1] + _fwd(e[2], 0) / w[2]]


def _abs2(v):
    return v.real ** 2 + v.imag ** 2


def _mag(y):  # norm of a 1-, 3- or 6-component field; off-diagonal entries count twice
    return sum(_abs2(c) * (2.0 if i > 2 else 1.0) for i, c in enumerate(y)).sqrt()


def _prox(y, scale):
    d = (scale * _mag(y)).clamp(min=1.0)
    return [c / d for c in y]


def _weights(tsw):
    """Time-space weights (ds, ds, dt) from the complete elliptic integral of the second kind."""
    r = 1.0 / tsw
    q = r if r <= 1.0 else 1.0 / r
    xg, wg = np.polynomial.legendre.leggauss(200)
    th = (xg + 1.0) * math.pi / 4.0
    ell = float(np.sum(wg * np.sqrt(1.0 - (1.0 - q * q) * np.sin(th) ** 2)) * math.pi / 4.0)
    big = math.pi / (2.0 * ell)
    w1, w2 = (q * big, big) if r <= 1.0 else (big, q * big)
    return (1.0 / w1, 1.0 / w1, 1.0 / w2)


def _solve(case, op, d):
    """The primal-dual loop of any method; returns (x, last gap, sigma, tau)."""
    method = case["method"]
    p = _params(case)
    lam = op.subfac * p.adaptK + p.adaptD
    second, second_order = method in ("ICTV", "ICTGV2"), method in ("TGV2", "ICTGV2")
    w = [(1.0, 1.0, float(p.dt)) if method == "TVTEMP" else _weights(p.timeSpaceWeight)]
    a0 = a1 = 1.0
    if method not in ("TV", "TVTEMP"):
        a0, a1 = float(p.alpha0), float(p.alpha1)
    share = [1.0]
    if second:
        w.append(_weights(p.timeSpaceWeight2))
        m = min(float(p.alpha), 1.0 - float(p.alpha))
        share = [float(p.alpha) / m, (1.0 - float(p.alpha)) / m]
    b1 = d["b1"].to(torch.complex128)
    data = d["k"].to(torch.complex128)
    x = [d["x0"].to(torch.complex128)] + [torch.zeros_like(d["x0"], dtype=torch.complex128)] * (len(share) - 1)
    v = [[torch.zeros_like(x[0]) for _ in range(3)] for _ in share] if second_order else [None] * len(share)
    y = [[torch.zeros_like(x[0]) for _ in range(3)] for _ in share]
    q = [[torch.zeros_like(x[0]) for _ in range(6)] for _ in share] if second_order else None
    z = torch.zeros_like(data)
    xb, vb = list(x), [None if c is None else list(c) for c in v]
    sigma, tau, gap = float(p.sigma), float(p.tau), None

    def k_reg(x, v, i):
        u = x[0] - x[1] if second and i == 0 else x[i]
        if method == "TVTEMP":
            return [_fwd(u, 0) / w[0][2]]
        g = _grad(u, w[i])
        return [g[c] - v[i][c] for c in range(3)] if second_order else g

    def div(i):
        return -_fwd_t(y[0][0], 0) / w[0][2] if method == "TVTEMP" else _div(y[i], w[i])

    for k in range(case["iters"]):
        for i in range(len(share)):
            y[i] = _prox([a + sigma * b for a, b in zip(y[i], k_reg(xb, vb, i))], 1.0 / (a1 * share[i]))
            if second_order:
                q[i] = _prox([a + sigma * b for a, b in zip(q[i], _symgrad(vb[i], w[i]))], 1.0 / (a0 * share[i]))
        z.add_(op.to_k(xb[0], b1), alpha=sigma).sub_(data, alpha=sigma).mul_(1.0 / (1.0 + sigma / lam))
        dv = [div(i) for i in range(len(share))]
        xn = [x[0] + tau * (dv[0] - op.to_img(z, b1))] + [x[1] + tau * (dv[1] - dv[0]) for _ in share[1:]]
        xb = [2.0 * a - b for a, b in zip(xn, x)]
        if second_order:
            for i in range(len(share)):
                sd = _symdiv(q[i], w[i])
                vn = [v[i][c] + tau * (y[i][c] + sd[c]) for c in range(3)]
                vb[i] = [2.0 * a - b for a, b in zip(vn, v[i])]
                v[i] = vn
        x = xn
        if k < 10 or k % 50 == 0:
            e = [a - b for a, b in zip(xb, x)]
            ev = [[a - b for a, b in zip(vb[i], v[i])] if second_order else None for i in range(len(share))]
            kx = float(_abs2(op.to_k(e[0], b1)).sum())
            if method != "ICTV":
                for i in range(len(share)):
                    kx += float((_mag(k_reg(e, ev, i)) ** 2).sum())
                    kx += float((_mag(_symgrad(ev[i], w[i])) ** 2).sum()) if second_order else 0.0
            nx = sum(float(_abs2(c).sum()) for c in e + [c for g in ev if g for c in g])
            r = math.sqrt(nx / kx)
            if sigma * tau > r * r:
                if 0.95 * 0.95 * sigma * tau < r * r:
                    sigma, tau = 0.95 * sigma, 0.95 * tau
                else:
                    sigma, tau = r * float(p.sigmaTauRatio), r / float(p.sigmaTauRatio)
        if case.get("gap") and k % case["gap"] == 0:
            f = _abs2(op.to_k(x[0], b1) - data).sum() * 0.5 * lam
            f = f + (data.conj() * z).real.sum() + _abs2(z).sum() / (2.0 * lam)
            dv = [div(i) for i in range(len(share))]
            f = f + (op.to_img(z, b1) - dv[0]).abs().sum()
            if second:
                f = f + (dv[0] - dv[1]).abs().sum()
            for i in range(len(share)):
                if second_order:
                    f = f + sum((a + b).abs().sum() for a, b in zip(_symdiv(q[i], w[i]), y[i]))
                    f = f + share[i] * a0 * _mag(_symgrad(v[i], w[i])).sum()
                f = f + share[i] * a1 * _mag(_grad(x[0], w[0]) if method == "TVTEMP" else k_reg(x, v, i)).sum()
            gap = abs(float(f)) / x[0].numel()
    return x[0], gap, sigma, tau


def _h1_maps(u, crec, mu):
    """|b1| of the H1 system (mu |u|^2 - periodic Laplace) b = mu u |crec_c|, by conjugate gradients."""
    m = mu * _abs2(u) + 4.0

    def apply(v):
        return m * v - v.roll(1, 1) - v.roll(-1, 1) - v.roll(1, 2) - v.roll(-1, 2)

    r = (u.conj() * mu * crec.abs()).clone()
    x, p = torch.zeros_like(r), r.clone()
    dot = lambda a, b: (a.conj() * b).real.sum((1, 2), keepdim=True)  # noqa: E731
    rr = rr0 = dot(r, r)
    for it in range(20000):
        if it % 50 == 0 and bool((rr <= 1e-27 * rr0).all()):
            break
        q = apply(p)
        a = rr / dot(p, q).clamp(min=1e-300)
        x, r = x + a * p, r - a * q
        rn = dot(r, r)
        p = r + (rn / rr.clamp(min=1e-300)) * p
        rr = rn
    return (x / _abs2(x).sum(0).sqrt()).abs()


def _utgv2(b, crec, x1, p):
    one = (1.0, 1.0, 1.0)
    sig, tau = float(p.uSigma), float(p.uTau)
    lw, ib = (b.conj() * crec).sum(0)[None], 1.0 / (1.0 + tau * _abs2(b).sum(0))[None]
    z = torch.zeros_like(x1)[None]
    x, xb = x1[None], x1[None]
    v, vb, y, e = [z, z], [z, z], [z, z], [z, z, z]
    for _ in range(p.uNrIt):
        g = _grad(xb, one)
        s = _symgrad([vb[0], vb[1], z], one)
        y = _prox([y[i] + sig * (g[i] - vb[i]) for i in range(2)], 1.0 / (float(p.uAlpha1) * float(p.uReg)))
        e = [e[0] + sig * s[0], e[1] + sig * s[1], e[2] + sig * s[3]]
        n = (_abs2(e[0]) + _abs2(e[1]) + 2.0 * _abs2(e[2])).sqrt()
        e = [c / (n / (float(p.uAlpha0) * float(p.uReg))).clamp(min=1.0) for c in e]
        xn = (x + tau * (_div([y[0], y[1], z], one) + lw)) * ib
        sd = _symdiv([e[0], e[1], z, e[2], z, z], one)
        vn = [v[i] + tau * (y[i] + sd[i]) for i in range(2)]
        xb, vb = 2.0 * xn - x, [2.0 * vn[i] - v[i] for i in range(2)]
        x, v = xn, vn
    return x[0]


def _b1(u, crec, iters, mu, p):
    sig, tau = float(p.b1Sigma), float(p.b1Tau)
    u = u / u.abs().max()
    lw, iu = u.conj() * crec, 1.0 / (1.0 + tau * _abs2(u))
    x = torch.zeros_like(crec)
    xb, y = x, [x, x]
    for _ in range(iters):
        y = [(y[i] + sig * _fwd(xb, 2 - i)) / (1.0 + sig / mu) for i in range(2)]
        xn = (x + tau * (lw - _fwd_t(y[0], 2) - _fwd_t(y[1], 1))) * iu
        xb, x = 2.0 * xn - x, xn
    return x / _abs2(x).sum(0).sqrt()


def _coils(case, d):
    p = av.coil_default_params()
    k = d["k"].to(torch.complex128)
    C, H, W = case["C"], case["H"], case["W"]
    if case["spokes"]:
        T, S = d["dens"].shape
        op = _Radial(W, H, d["traj"].permute(1, 0, 2).reshape(1, 2, T * S), d["dens"].reshape(1, T * S), 2.0, 1)
        crec = torch.cat([op.images(0, k[:, c].reshape(1, T * S)) for c in range(C)])
    else:
        crec = _f_k_to_img(k.sum(0) / d["mask"].double().sum(0).clamp(min=1.0), False)
    u0 = _abs2(crec).sum(0).sqrt().to(torch.complex128)
    absb1 = _h1_maps(u0, crec, float(p.uH1mu)).to(torch.complex128)
    inds = [int(torch.argmax(crec.abs().sum((1, 2))))]
    u = [_utgv2(absb1[inds], crec[inds], torch.zeros_like(u0), p)]
    maps = {inds[0]: absb1[inds[0]]}
    w = torch.zeros_like(u0)
    for _ in range(1, C):
        last = inds[-1]
        w = (w * w + _abs2(absb1[last])).sqrt()
        s = (crec[last].abs() * crec.abs()).sum((1, 2))
        s[inds] = -1.0
        c = int(torch.argmax(s))
        inds.append(c)
        x = _b1(absb1[c] * u[-1] * w, (crec[c] * w)[None], p.b1NrIt, float(p.b1Reg), p)[0]
        maps[c] = absb1[c] * x / x.abs()
        u.append(_utgv2(torch.stack([maps[i] for i in inds]), crec[inds], u[-1], p))
    return dict(u=torch.stack(u), b1=_b1(u[-1], crec, p.b1FinalNrIt, float(p.b1FinalReg), p))


def exact(case, seed):
    kind = case["kind"]
    if kind == "stream":
        if work(case)["bytes"] > 1.2e12:
            return None  # over the time that a value in 64 bits may take
        return [_exact_recon(c, seed + 1000 * i)[0] for i, c in enumerate(_requests(case))]
    if kind == "coils":
        return _coils(case, _inputs(case, seed))
    if kind == "apply":
        d = _inputs(case, seed)
        op = _exact_operator(case, d)
        b1 = d["b1"].to(torch.complex128)
        return dict(k=op.to_k(d["truth"].to(torch.complex128), b1), img=op.to_img(d["k"].to(torch.complex128), b1))
    x, gap, sigma, tau = _exact_recon(case, seed)
    if kind == "host":
        return dict(x=x.cpu().numpy())
    return dict(x=x, gap=gap, sigma=sigma, tau=tau) if case.get("gap") else dict(x=x)


def _exact_operator(case, d):
    if case.get("spokes"):
        return _Radial(case["W"], case["H"], d["traj"], d["dens"], case["osf"], case["spokes"])
    return _Cart(case, d)


def _exact_recon(case, seed):
    d = _inputs(case, seed)
    return _solve(case, _exact_operator(case, d), d)
