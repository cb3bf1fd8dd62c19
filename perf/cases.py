"""What a user of lamino_b200 has it do, as timed cases.

Each case is one call (or one whole reconstruction) through the public Python
entry points, on device tensors, at the sizes of this repository's workloads:

* requests of the batched / served mix: recon 64 - 256 wide, 8 - 32 thick, two
  datasets of 60 - 240 angles (gamma 0 and a tilt of 20 - 50 degrees);
* the README-size reconstruction: recon 511 x 51 x 511, padded to
  721 x 71 x 721, four gammas x 361 angles, detectors padded to 1233 x 1233;
* the forward tool, which pads the volume and the detector by sqrt(2).

The MBIR drivers pad the volume by 1.4142 and (MBIR2 / 3) the projections by
2.4142 per side; the operator cases carry the padded sizes that the drivers
hand to the operators.  `draw` gives ragged sizes over the same ranges.

Volumes are (3, n1, n2, n3) with n2 the thickness.
"""
import math

import numpy as np
import torch

import lamino_b200 as L

DEV = "cuda" if torch.cuda.is_available() else "cpu"
PAD = np.float32(1.4142)


def _npad(n, f):
    return 2 * (int(np.float32(n) * np.float32(f)) // 2)


def _vol(h, t):
    """Padded volume (n1, n2, n3) of a recon h wide and t thick."""
    f = PAD - np.float32(1)
    return h + _npad(h, f), t + _npad(t, f), h + _npad(h, f)


def _dims(c):
    return c["n1"], c["n2"], c["n3"]


def _op_case(kind, h, t, rows, cols, angles, gammas, **kw):
    n1, n2, n3 = _vol(h, t)
    return dict(kind=kind, n1=n1, n2=n2, n3=n3, rows=rows, cols=cols, angles=angles, gammas=gammas, **kw)


def _pad_det(n):
    return n + _npad(n, PAD)


def listed():
    return [
        # the normal operator inside the solvers: one CG / NAG step's matrix
        # product.  Smallest request of the mix (launches count), an ordinary
        # one, and the README size (the repository's headline figure).
        dict(_op_case("apply", 64, 8, 154, 154, 60, "0,35", precision="fp32"), name="apply_request_small"),
        dict(_op_case("apply", 192, 24, 462, 462, 150, "0,35", precision="fp32"), name="apply_request"),
        dict(_op_case("apply", 511, 51, 1233, 1233, 361, "0,45,90,135", precision="fp32"), name="apply_readme"),
        # the forward tool: simulate a tilted dataset (detector padded by sqrt 2 only)
        dict(_op_case("forward", 256, 32, 362, 362, 181, "35"), name="forward_tool"),
        # the setup of a reconstruction: back-projection of one dataset
        dict(_op_case("adjoint", 64, 8, 154, 154, 60, "0"), name="adjoint_request_small"),
        dict(_op_case("adjoint", 511, 51, 1233, 1233, 361, "45"), name="adjoint_readme"),
        # the normal operator in NUFFT form (op_kind "nufft", gradient, residual)
        dict(_op_case("sysmat", 128, 12, 309, 309, 91, "0,45"), name="sysmat_two_tilts"),
        # the FINUFFT-level boundary: complex type 2 and type 1 on one dataset
        dict(_op_case("nufft", 128, 16, 200, 181, 90, "30"), name="nufft_type2_type1"),
        # once per CG iteration at the README size
        dict(kind="ramp", n1=721, n2=71, n3=721, name="ramp_readme"),
        # prior gradient of one component in a NAG step, largest request of the mix
        dict(kind="qggmrf", n1=362, n2=44, n3=362, sigma=1000.0, p=1.2, name="qggmrf_request"),
        # whole reconstructions: split-Bregman TV (the README's method) on a
        # small recon, few outer iterations; and one request of the mix (NAG + qGGMRF)
        dict(kind="mbir", method=2, h=128, t=16, rows=128, cols=128, angles=90, gammas="0,45,90,135", iters=6,
             name="mbir2_small"),
        dict(kind="mbir", method=3, h=192, t=24, rows=192, cols=192, angles=150, gammas="0,35", iters=40,
             name="mbir3_request"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "forward", "adjoint", "adjoint", "sysmat", "nufft", "ramp", "qggmrf", "mbir"])
    h, t = _log_int(rng, 40, 300), _log_int(rng, 6, 36)
    tilt = rng.choice([0.0, round(rng.uniform(20, 50), 2), round(rng.uniform(0, 180), 2)])
    angles = rng.randint(40, 240)
    if kind == "apply":
        h, t = _log_int(rng, 40, 480), _log_int(rng, 6, 50)
        gammas = rng.choice(["0,%g" % tilt, "0,45,90,135"])
        return _op_case("apply", h, t, _pad_det(h), _pad_det(h + rng.randint(-8, 8)), angles, gammas,
                        precision=rng.choice(["fp32"] * 7 + ["fp16"]))
    if kind == "forward":
        f = math.sqrt(2) - 1
        return _op_case("forward", h, t, h + _npad(h, f), h + rng.randint(-9, 9) + _npad(h, f), angles, "%g" % tilt)
    if kind == "adjoint":
        return _op_case("adjoint", h, t, _pad_det(h), _pad_det(h + rng.randint(-9, 9)), angles, "%g" % tilt)
    if kind == "sysmat":
        h = _log_int(rng, 40, 140)
        return _op_case("sysmat", h, t, _pad_det(h), _pad_det(h + rng.randint(-9, 9)), angles, "0,%g" % tilt)
    if kind == "nufft":
        return _op_case("nufft", h, t, h + rng.randint(-9, 60), h + rng.randint(-9, 60), angles, "%g" % tilt)
    if kind == "ramp":
        h, t = _log_int(rng, 40, 500), _log_int(rng, 6, 50)
        n1, n2, n3 = _vol(h, t)
        return dict(kind="ramp", n1=n1, n2=n2, n3=n3 + rng.randint(-3, 3))
    if kind == "qggmrf":
        n1, n2, n3 = _vol(h, t)
        return dict(kind="qggmrf", n1=n1, n2=n2, n3=n3 + rng.randint(-3, 3),
                    sigma=rng.choice([1.0, 100.0, 1000.0]), p=rng.choice([1.1, 1.2, 1.5]))
    h, t = _log_int(rng, 48, 160), _log_int(rng, 8, 24)
    method = rng.choice([1, 2, 3])
    return dict(kind="mbir", method=method, h=h, t=t, rows=h, cols=h + rng.randint(-4, 4), angles=rng.randint(40, 120),
                gammas="0,%g" % tilt, iters=rng.randint(4, 12))


# ---------------------------------------------------------------------------
# inputs: blobs of magnetization, whose projections are known in closed form
# ---------------------------------------------------------------------------

def _gammas(c):
    return [math.radians(float(v)) for v in c["gammas"].split(",")]


def _angles(c, seed):
    rng = np.random.default_rng(seed)
    return [rng.uniform(0, 2 * np.pi, c["angles"]).astype(np.float32) for _ in c["gammas"].split(",")]


def _blobs(dims, seed, n=48):
    """Centres (x, y, z) = (n3, n2, n1) axes, widths and moments of the blobs."""
    rng = np.random.default_rng(seed + 77)
    half = np.array([dims[2], dims[1], dims[0]], float) / 2
    r0 = rng.uniform(-0.55, 0.55, (n, 3)) * half
    sig = np.exp(rng.uniform(math.log(1.2), math.log(max(2.0, min(half) / 3)), n))
    mu = rng.standard_normal((n, 3))
    t = lambda a: torch.tensor(a, dtype=torch.float32, device=DEV)  # noqa: E731
    return t(r0), t(sig), t(mu)


def _volume(dims, seed, comps=3):
    """Unit vectors from the blobs' field, zero outside the central 70 % laterally."""
    r0, sig, mu = _blobs(dims, seed)
    e = []
    for ax, n in enumerate((dims[2], dims[1], dims[0])):
        k = torch.arange(n, device=DEV, dtype=torch.float32) - n // 2
        e.append(torch.exp(-0.5 * ((k[None] - r0[:, ax, None]) / (2 * sig[:, None])) ** 2))
    f = torch.stack([torch.einsum("bz,by,bx->zyx", e[2] * mu[:, c, None], e[1], e[0]) for c in range(comps)])
    f = f / (torch.linalg.vector_norm(f, dim=0, keepdim=True) + 1e-6)
    a1, a3 = round(dims[0] * 0.15), round(dims[2] * 0.15)
    mask = torch.zeros(dims, device=DEV)
    mask[a1:dims[0] - a1, :, a3:dims[2] - a3] = 1
    return (f * mask).contiguous()


def _projections(dims, theta, gamma, rows, cols, seed):
    """Projections (np, rows, cols) of the blobs plus 1 % Gaussian noise."""
    r0, sig, mu = _blobs(dims, seed)
    th = torch.tensor(theta, device=DEV)
    cg, sg = math.cos(gamma), math.sin(gamma)
    st, ct = torch.sin(th), torch.cos(th)
    u = r0[:, 0] * cg - r0[:, 2] * sg
    v = ct[:, None] * (r0[:, 0] * sg + r0[:, 2] * cg)[None] - st[:, None] * r0[:, 1][None]
    amp = st[:, None] * (sg * mu[:, 0] + cg * mu[:, 2])[None] + ct[:, None] * mu[:, 1][None]
    col = torch.arange(cols, device=DEV) - cols // 2
    row = torch.arange(rows, device=DEV) - rows // 2
    ec = torch.exp(-0.5 * ((col[None] - u[:, None]) / sig[:, None]) ** 2)
    out = torch.empty((len(theta), rows, cols), device=DEV)
    for p in range(len(theta)):
        er = torch.exp(-0.5 * ((row[None] - v[p, :, None]) / sig[:, None]) ** 2)
        torch.matmul((er * (amp[p] * sig)[:, None]).T, ec, out=out[p])
    g = torch.Generator(device=DEV).manual_seed(seed + 5)
    return out.add_(torch.randn(out.shape, device=DEV, generator=g), alpha=0.01 * float(out.std()))


def _padded_projections(c, theta, gamma, seed):
    """A dataset in the middle of a zero-padded detector, as the drivers pad it."""
    rows, cols = c["rows"], c["cols"]
    r, k = int(rows / 2.4142), int(cols / 2.4142)
    out = torch.zeros((c["angles"], rows, cols), device=DEV)
    a, b = (rows - r) // 2, (cols - k) // 2
    out[:, a:a + r, b:b + k] = _projections(_dims(c), theta, gamma, r, k, seed)
    return out


def _complex(shape, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(tuple(shape) + (2,), device=DEV, generator=g).view(torch.complex64).squeeze(-1)


def _inputs(c, seed):
    """The arrays of a case, from the seed alone."""
    kind = c["kind"]
    if kind in ("apply", "sysmat", "forward"):
        return {"x": _volume(_dims(c), seed)}
    if kind == "adjoint":
        return {"proj": _padded_projections(c, _angles(c, seed)[0], _gammas(c)[0], seed)}
    if kind == "nufft":
        v = _volume(_dims(c), seed, comps=2)
        return {"modes": torch.complex(v[0], v[1]), "c": _complex((c["angles"], c["rows"], c["cols"]), seed)}
    if kind == "ramp":
        g = torch.Generator(device=DEV).manual_seed(seed)
        return {"r": _volume(_dims(c), seed) + 0.1 * torch.randn((3,) + _dims(c), device=DEV, generator=g)}
    if kind == "qggmrf":
        g = torch.Generator(device=DEV).manual_seed(seed)
        x = _volume(_dims(c), seed, comps=1)[0] + 0.02 * torch.randn(_dims(c), device=DEV, generator=g)
        return {"x": x, "g": torch.randn(_dims(c), device=DEV, generator=g)}
    dims = (c["h"], c["t"], c["h"])
    return {"datasets": [(_projections(dims, th, gm, c["rows"], c["cols"], seed), th, np.float32(gm))
                         for th, gm in zip(_angles(c, seed), _gammas(c))]}


# ---------------------------------------------------------------------------
# what a program keeps, and one pass
# ---------------------------------------------------------------------------

def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case)
    if case["kind"] in ("apply", "forward", "adjoint", "sysmat", "nufft"):
        s["grids"] = [L.PolarGrid(th, case["rows"], case["cols"], gm)
                      for th, gm in zip(_angles(case, seed), _gammas(case))]
    if case["kind"] == "apply":
        s["op"] = L.ToeplitzNormal(s["grids"], _dims(case), case["precision"])
        s["y"] = torch.empty_like(s["x"])
    elif case["kind"] in ("forward", "adjoint", "sysmat", "nufft"):
        s["plan"] = L.NufftPlan(_dims(case))
    elif case["kind"] == "mbir":
        # tolerances of zero: the iteration count is the case's
        if case["method"] == 3:  # mu = 0: Lipschitz constant from power iterations
            s["params"] = L.ReconParams(maxIters=case["iters"], sigma=1000.0, p=1.2, mu=0.0, tol=0.0, xtol=0.0)
        else:
            s["params"] = L.ReconParams(maxIters=case["iters"], innerIters=3, lam=0.1, mu=10.0, tol=0.0, xtol=0.0)
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "apply":
        return s["op"](s["x"], out=s["y"])
    if kind == "forward":
        return L.forward(s["x"], s["grids"][0], plan=s["plan"])
    if kind == "adjoint":
        return L.adjoint(s["proj"], s["grids"][0], _dims(c), plan=s["plan"])
    if kind == "sysmat":
        return L.sysmat(s["x"], s["grids"], plan=s["plan"])
    if kind == "nufft":
        return {"c": L.nufft3d2(s["modes"], s["grids"][0], plan=s["plan"]),
                "modes": L.nufft3d1(s["c"], s["grids"][0], _dims(c), plan=s["plan"])}
    if kind == "ramp":
        return L.opt.ramp_precond(s["r"])
    if kind == "qggmrf":
        return L.opt.qggmrf(s["g"].clone(), s["x"], c["sigma"], c["p"])
    return {1: L.MBIR1, 2: L.MBIR2, 3: L.MBIR3}[c["method"]](s["datasets"], (c["h"], c["t"], c["h"]), s["params"])


def _fft_flops(points, length):
    return 5.0 * points * math.log2(max(2.0, float(length)))


def work(case):
    """Inputs and outputs once; the transforms on twice the volume's extent (the
    linear convolution / the non-uniform transform) and on the projections."""
    c, kind = case, case["kind"]
    if kind == "mbir":
        h, t = c["h"], c["t"]
        n1, n2, n3 = _vol(h, t)
        sets = len(c["gammas"].split(","))
        V = n1 * n2 * n3
        applies = {1: c["iters"] + 1, 2: 4 * c["iters"], 3: 2 * c["iters"] + 30}[c["method"]]
        pts = sets * c["angles"] * _pad_det(c["rows"]) * _pad_det(c["cols"])
        return {"bytes": applies * (6 * V * 4 + 24 * V * 4) + sets * c["angles"] * c["rows"] * c["cols"] * 4 + 12 * h * t * h,
                "flops": applies * 6 * _fft_flops(4 * V, 8 * V) + _fft_flops(pts, pts / c["angles"] / sets)}
    V = c["n1"] * c["n2"] * c["n3"]
    if kind == "apply":  # x, y and the six spectra of the kernel
        S = 4 * c["n1"] * c["n2"] * (c["n3"] + 1)
        return {"bytes": 24 * V + 6 * S * (2 if c["precision"] == "fp16" else 4), "flops": 6 * _fft_flops(4 * V, 8 * V)}
    if kind == "ramp":
        return {"bytes": 24 * V, "flops": 6 * _fft_flops(V / 2, c["n2"] * c["n3"])}
    if kind == "qggmrf":
        return {"bytes": 20 * V, "flops": 26 * 20 * V}
    sets = len(c["gammas"].split(","))
    pts = c["angles"] * c["rows"] * c["cols"]
    if kind == "sysmat":
        return {"bytes": 24 * V, "flops": 6 * _fft_flops(4 * V, 8 * V)}
    if kind == "nufft":
        return {"bytes": 2 * (8 * V + 8 * pts), "flops": 2 * _fft_flops(8 * V, 8 * V)}
    return {"bytes": 12 * V + 4 * pts,
            "flops": 3 * _fft_flops(4 * V, 8 * V) + _fft_flops(pts / 2, c["rows"] * c["cols"])}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

F64, C128 = torch.float64, torch.complex128
MOST_FLOPS = 1.5e14  # of the exact transforms below: a few seconds


def _modes(n):
    return torch.arange(n, device=DEV, dtype=F64) - n // 2


def _grid(n):
    """Detector frequencies (k + 1/2) 2 pi / n - pi."""
    return (torch.arange(n, device=DEV, dtype=F64) + 0.5) * (2 * math.pi / n) - math.pi


def _cis(a):
    return torch.polar(torch.ones_like(a), a)


def _plane_terms(dims, theta, gamma, rows, cols):
    """Factors of e^{i k.q}, q = X a + Y b(theta), per (angle, row) and per column."""
    n1, n2, n3 = dims
    cg, sg = math.cos(gamma), math.sin(gamma)
    th = torch.tensor(np.asarray(theta, np.float64), device=DEV)
    Y, X = _grid(rows), _grid(cols)
    T = (torch.cos(th)[:, None] * Y[None]).reshape(-1)   # along (sin g, cos g) in (x, z)
    y = (-torch.sin(th)[:, None] * Y[None]).reshape(-1)
    kap = _modes(n3)[None, :] * sg + _modes(n1)[:, None] * cg  # (n1, n3)
    E3 = _cis(_modes(n3)[:, None] * (X * cg)[None])       # (n3, cols)
    E1 = _cis(-_modes(n1)[:, None] * (X * sg)[None])      # (n1, cols)
    return T, y, kap, E1, E3


def _too_much(dims, points):
    return 8.0 * dims[0] * dims[2] * points > MOST_FLOPS


def _type2(modes, dims, theta, gamma, rows, cols):
    """sum_k modes e^{-i k.q}: (len(modes), angles, rows, cols)."""
    T, y, kap, E1, E3 = _plane_terms(dims, theta, gamma, rows, cols)
    n1, n2, n3 = dims
    E1, E3 = E1.conj(), E3.conj().resolve_conj()
    M = [m.to(C128).permute(1, 0, 2).reshape(n2, n1 * n3) for m in modes]
    out = torch.empty((len(modes), T.numel(), cols), dtype=C128, device=DEV)
    step = max(1, int(4e7 / (n1 * max(n3, cols))))
    for a in range(0, T.numel(), step):
        t, yy = T[a:a + step], y[a:a + step]
        ph = _cis(-t[:, None, None] * kap[None])
        e2 = _cis(-yy[:, None] * _modes(n2)[None])
        for i, m in enumerate(M):
            H = (e2 @ m).view(-1, n1, n3) * ph
            out[i, a:a + step] = ((H.reshape(-1, n3) @ E3).view(-1, n1, cols) * E1[None]).sum(1)
    return out.view(len(modes), len(theta), rows, cols)


def _type1(c, dims, theta, gamma, rows, cols, weights):
    """sum_q weights[i](angle) c(q) e^{+i k.q}: (len(weights), n1, n2, n3)."""
    T, y, kap, E1, E3 = _plane_terms(dims, theta, gamma, rows, cols)
    n1, n2, n3 = dims
    c = c.reshape(-1, cols)
    W = [w.repeat_interleave(rows) for w in weights]
    out = torch.zeros((len(weights), n2, n1 * n3), dtype=C128, device=DEV)
    step = max(1, int(4e7 / (n1 * max(n3, cols))))
    for a in range(0, T.numel(), step):
        t, yy = T[a:a + step], y[a:a + step]
        Z = (c[a:a + step, None, :] * E1[None]).reshape(-1, cols) @ E3.T
        Z = (Z.view(-1, n1, n3) * _cis(t[:, None, None] * kap[None])).view(-1, n1 * n3)
        e2 = _cis(yy[:, None] * _modes(n2)[None])
        for i, w in enumerate(W):
            out[i] += (e2 * w[a:a + step, None]).T @ Z
    return out.view(len(weights), n2, n1, n3).permute(0, 2, 1, 3)


def _shift(a, back=False):
    d = [n - n // 2 if back else n // 2 for n in a.shape[-2:]]
    return torch.roll(a, (-d[0], -d[1]), dims=(-2, -1))


def _exact_forward(x, dims, theta, gamma, rows, cols):
    x = x.to(F64)
    cg, sg = math.cos(gamma), math.sin(gamma)
    th = torch.tensor(np.asarray(theta, np.float64), device=DEV)
    vs, vc = _type2([sg * x[0] + cg * x[2], x[1]], dims, theta, gamma, rows, cols)
    P = torch.sin(th)[:, None, None] * vs + torch.cos(th)[:, None, None] * vc
    r, k = rows // 2, cols // 2  # fftshift, unnormalised inverse transform / N, ifftshift
    P = torch.roll(P, (-r, -k), dims=(-2, -1))
    return torch.roll(torch.fft.ifft2(P), (-(rows - r), -(cols - k)), dims=(-2, -1)).real


def _exact_adjoint(proj, dims, theta, gamma, rows, cols):
    cg, sg = math.cos(gamma), math.sin(gamma)
    th = torch.tensor(np.asarray(theta, np.float64), device=DEV)
    P = torch.fft.fft2(_shift(proj.to(C128)))
    P = _shift(P, back=True)
    ys, yc = _type1(P, dims, theta, gamma, rows, cols, [torch.sin(th).to(C128), torch.cos(th).to(C128)]).real
    return torch.stack([sg * ys, yc, cg * ys]) / float(rows * cols)


def _dirichlet(t, n):
    m = torch.round(t / n)
    f = t - n * m
    den = torch.sin(math.pi * f / n)
    near = f.abs() < 1e-9
    s = torch.where(near, torch.full_like(f, float(n)), torch.sin(math.pi * f) / torch.where(near, torch.ones_like(f), den))
    return s if n % 2 else s * (1 - 2 * (m.abs() % 2))


def _toeplitz(dims, thetas, gammas, rows, cols):
    """x -> sum over datasets of A^H A x: convolution with the closed-form kernel."""
    n1, n2, n3 = dims
    L1, L2, L3 = 2 * n1, 2 * n2, 2 * n3
    lag = [((torch.arange(l, device=DEV, dtype=F64) + n - 1) % l - (n - 1)) for l, n in ((L1, n1), (L2, n2), (L3, n3))]
    dz, dy, dx = lag[0][:, None, None], lag[1][None, :, None], lag[2][None, None, :]
    # slabs of lags, so that the temporaries stay small
    ss, cc, sc = (torch.zeros((L1, L2, L3), dtype=F64, device=DEV) for _ in range(3))
    T = [torch.zeros((L1, L2, L3), dtype=F64, device=DEV) for _ in range(6)]
    for th, g in zip(thetas, gammas):
        cg, sg = math.cos(g), math.sin(g)
        for v in (ss, cc, sc):
            v.zero_()
        Da = _dirichlet(dx * cg - dz * sg, cols)
        u = dx * sg + dz * cg
        for t in np.asarray(th, np.float64):
            P = Da * _dirichlet(math.cos(t) * u - dy * math.sin(t), rows)
            ss.add_(P, alpha=math.sin(t) ** 2)
            cc.add_(P, alpha=math.cos(t) ** 2)
            sc.add_(P, alpha=math.sin(t) * math.cos(t))
        for q, (a, b) in enumerate(((sg * sg, ss), (1, cc), (cg * cg, ss), (sg, sc), (sg * cg, ss), (cg, sc))):
            T[q].add_(b, alpha=a / (rows * cols))
    del ss, cc, sc
    K = [torch.fft.rfftn(v).real for v in T]
    idx = [[0, 3, 4], [3, 1, 5], [4, 5, 2]]

    def apply(x):
        X = [torch.fft.rfftn(x[i].to(F64), s=(L1, L2, L3)) for i in range(3)]
        return torch.stack([torch.fft.irfftn(sum(K[idx[i][j]] * X[j] for j in range(3)), s=(L1, L2, L3))[:n1, :n2, :n3]
                            for i in range(3)])
    return apply


def _too_many_lags(c, sets):
    n1, n2, n3 = _dims(c)
    return 8.0 * n1 * n2 * n3 * c["angles"] * sets > 3e10


def _exact_ramp(r):
    n2, n3 = r.shape[-2:]
    xf = torch.arange(n3 // 2 + 1, device=DEV, dtype=F64) / n3
    j = torch.arange(n2, device=DEV, dtype=F64)
    yf = torch.where(j <= n2 // 2, j, j - n2) / n2
    return torch.fft.irfft2(torch.fft.rfft2(r.to(F64)) * torch.sqrt(xf[None] ** 2 + yf[:, None] ** 2), s=(n2, n3))


def _exact_qggmrf(g, x, sigma, p):
    g, x = g.to(F64).clone(), x.to(F64)
    p = float(np.float32(p))
    sq, sqp = sigma ** 2, sigma ** (2 - p)
    wt = {0: 0.0, 1: 0.0523, 2: 0.037, 3: 0.0302}
    n1, n2, n3 = x.shape
    u = x[1:-1, 1:-1, 1:-1]
    for i in (-1, 0, 1):
        for j in (-1, 0, 1):
            for k in (-1, 0, 1):
                if i == j == k == 0:
                    continue
                d = x[1 + i:n1 - 1 + i, 1 + j:n2 - 1 + j, 1 + k:n3 - 1 + k] - u
                # the reference's table: 0.0532 at (0, 0, -1), 0.0523 at (0, 1, 0) and its like
                w = 0.0532 if (i, j, k) == (0, 0, -1) else wt[abs(i) + abs(j) + abs(k)]
                t1 = d.abs() ** (2 - p) / sqp
                v = d / ((0.001 + t1) * sq) * (2 - (2 - p) * t1 / (0.001 + t1))
                v = torch.where(d == 0, torch.full_like(v, 2 / (sq * 0.001)), v)
                g[1:-1, 1:-1, 1:-1] += float(np.float32(w)) * v
    return g


def _grad_u(u):
    g = torch.zeros((3,) + tuple(u.shape), dtype=F64, device=DEV)
    g[0, 1:-1, 1:-1, 1:-1] = (u[2:, 1:-1, 1:-1] - u[:-2, 1:-1, 1:-1]) / 2
    g[1, 1:-1, 1:-1, 1:-1] = (u[1:-1, 2:, 1:-1] - u[1:-1, :-2, 1:-1]) / 2
    g[2, 1:-1, 1:-1, 1:-1] = (u[1:-1, 1:-1, 2:] - u[1:-1, 1:-1, :-2]) / 2
    return g


def _divergence(d):
    o = torch.zeros(tuple(d.shape[1:]), dtype=F64, device=DEV)
    o[1:-1, 1:-1, 1:-1] = ((d[0][:-2, 1:-1, 1:-1] - d[0][2:, 1:-1, 1:-1]) + (d[1][1:-1, :-2, 1:-1] - d[1][1:-1, 2:, 1:-1])
                           + (d[2][1:-1, 1:-1, :-2] - d[2][1:-1, 1:-1, 2:])) / 2
    return o


def _cg(A, y, x, iters):
    x = x.clone()
    r = y - A(x)
    z = _exact_ramp(r)
    p, rs = z, float((z * r).sum())
    for _ in range(iters):
        Ap = A(p)
        pAp = float((p * Ap).sum())
        if abs(pAp) < 1e-10:
            break
        x = x + (rs / pAp) * p
        r = r - (rs / pAp) * Ap
        z = _exact_ramp(r)
        new = float((z * r).sum())
        p, rs = z + (new / rs) * p, new
    return x


def _split_bregman(A, yT, lam, mu, outer, inner):
    x = torch.zeros_like(yT)
    d = torch.zeros((3,) + tuple(yT.shape), dtype=F64, device=DEV)
    b = torch.zeros_like(d)
    Ap = lambda u: A(u) + mu * torch.stack([_divergence(_grad_u(u[i])) for i in range(3)])  # noqa: E731
    for _ in range(outer):
        x = _cg(Ap, yT + mu * torch.stack([_divergence(d[i] - b[i]) for i in range(3)]), x, inner)
        v = torch.stack([_grad_u(x[i]) for i in range(3)]) + b
        sk = torch.sqrt(1e-8 + (v ** 2).sum(dim=(0, 1)))
        d = torch.clamp(sk - lam / mu, min=0) * (v / sk)
        b = v - d
    return x


def _exact_mbir(c, data):
    dims = _vol(c["h"], c["t"])
    if c["method"] == 3:
        return None  # its line search takes decisions that rounding may turn
    f = PAD - np.float32(1) if c["method"] == 1 else PAD
    rows, cols = c["rows"] + _npad(c["rows"], f), c["cols"] + _npad(c["cols"], f)
    if _too_much(dims, len(data) * c["angles"] * rows * cols):
        return None
    yT = torch.zeros((3,) + dims, dtype=F64, device=DEV)
    for proj, th, gm in data:
        y = torch.zeros((c["angles"], rows, cols), dtype=F64, device=DEV)
        a, b = (rows - c["rows"]) // 2, (cols - c["cols"]) // 2
        y[:, a:a + c["rows"], b:b + c["cols"]] = proj.to(F64) / float(proj.max())
        yT += _exact_adjoint(y, dims, th, float(gm), rows, cols)
    A = _toeplitz(dims, [d[1] for d in data], [float(d[2]) for d in data], rows, cols)
    x = _cg(A, yT, torch.zeros_like(yT), c["iters"]) if c["method"] == 1 else \
        _split_bregman(A, yT, float(np.float32(0.1)), 10.0, c["iters"], 3)
    o = [(a - b) // 2 for a, b in zip(dims, (c["h"], c["t"], c["h"]))]
    return x[:, o[0]:o[0] + c["h"], o[1]:o[1] + c["t"], o[2]:o[2] + c["h"]].contiguous()


def exact(case, seed):
    c, kind = case, case["kind"]
    s = _inputs(c, seed)
    if kind == "ramp":
        return torch.stack([_exact_ramp(s["r"][i]) for i in range(3)])
    if kind == "qggmrf":
        return _exact_qggmrf(s["g"], s["x"], c["sigma"], c["p"])
    if kind == "mbir":
        return _exact_mbir(c, s["datasets"])
    dims, th = _dims(c), _angles(c, seed)
    gm = [float(np.float32(g)) for g in _gammas(c)]
    if kind in ("apply", "sysmat"):
        if _too_many_lags(c, len(gm)):
            return None
        return _toeplitz(dims, th, gm, c["rows"], c["cols"])(s["x"])
    if _too_much(dims, 2 * c["angles"] * c["rows"] * c["cols"]):
        return None
    geo = (dims, th[0], gm[0], c["rows"], c["cols"])
    if kind == "forward":
        return _exact_forward(s["x"], *geo)
    if kind == "adjoint":
        return _exact_adjoint(s["proj"], *geo)
    one = torch.ones(c["angles"], dtype=C128, device=DEV)
    return {"c": _type2([s["modes"]], *geo)[0], "modes": _type1(s["c"].to(C128), *geo, [one])[0].contiguous()}
