"""The work that a user of this package has it do, as a list of measurable cases.

A case is a dict of plain values. ``listed()`` gives the named cases, ``draw(rng)`` more of the same
ranges. Kinds:

- ``type1`` / ``type2``: one execute of a kept NUFFT plan (adjoint gridding / forward sampling) over
  all transforms;
- ``grad``: one step of trajectory optimisation: the optimiser has written new coordinates, the plan
  pair is re-pointed, the SENSE loss ``||S^H A^H (A S x - y)||^2`` is evaluated and differentiated
  with respect to the image and the coordinates;
- ``normal``: one fused Toeplitz SENSE apply ``sum_c conj(S_c) T(S_c x)``;
- ``cg``: a graph-captured conjugate-gradient reconstruction on that operator, one frame or several;
- ``kernel``: the Toeplitz kernel of a new trajectory.

Data are seeded and synthetic: a Gaussian image inside an ellipsoid, smooth coil maps with unit root
sum of squares, radial / cones-like / variable-density spiral trajectories in radians, turned by
an angle that the seed gives. The Toeplitz kernels of the ``normal`` and ``cg`` cases are the sampling density
of such a trajectory on the 2N grid.
"""
from __future__ import annotations

import math

import torch

import hastycucompute_b200 as hb
from hastycucompute_b200 import autograd as ag

DEVICE = "cuda"


# ---- the cases ------------------------------------------------------------------------------------

def _case(kind, dims, coils, points=0, width=0, traj="", frames=1, iters=0, name=None):
    c = {"kind": kind, "dims": "x".join(str(d) for d in dims), "coils": coils, "points": points, "width": width,
         "traj": traj, "frames": frames, "iters": iters}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one coil-combined 2-D slice sampled along spirals, the default tolerance: a call of a few launches
        _case("type2", (128, 128), 1, 16384, 6, "spiral", name="type2_2d_single"),
        # gridding of a small 3-D radial acquisition, all coils
        _case("type1", (64, 64, 64), 8, 131072, 4, "radial", name="type1_64_radial"),
        # forward sampling of one frame of a dynamic 3-D series: few spokes on a large grid
        _case("type2", (128, 128, 128), 16, 64000, 4, "radial", name="type2_128_frame"),
        # anisotropic volumes with odd counts of points and coils, an ordinary scan
        _case("type1", (120, 96, 150), 12, 700001, 6, "cones", name="type1_ragged"),
        _case("type2", (90, 110, 75), 5, 300007, 5, "radial", name="type2_ragged"),
        # a whole-brain acquisition: 6.1 million samples of 32 coils
        _case("type1", (160, 160, 160), 32, 6144000, 6, "cones", name="type1_160_cones"),
        _case("type2", (160, 160, 160), 32, 6144000, 6, "cones", name="type2_160_cones"),
        # one optimiser step of 2-D trajectory design
        _case("grad", (256, 256), 12, 65536, 4, "spiral", name="traj_grad_2d"),
        # a small iterative reconstruction, ten iterations
        _case("cg", (64, 64, 64), 8, traj="radial", iters=10, name="cg_64"),
        # one apply of the normal operator: an ordinary scanner matrix, and the whole-brain one
        _case("normal", (88, 104, 110), 6, traj="radial", name="normal_ragged"),
        _case("normal", (160, 160, 160), 32, traj="cones", name="normal_160"),
        # a new volume's trajectory arrives: its Toeplitz kernel
        _case("kernel", (128, 128, 128), 1, 2097152, 4, "radial", name="kernel_128"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# image edges N whose 2N has no prime factor above 13 (what the Toeplitz operators take)
_EDGES = [n for n in range(32, 161) if all(n % p for p in range(17, n + 1) if all(p % q for q in range(2, p)))]


def draw(rng):
    kind = rng.choice(["type1", "type2", "type1", "type2", "normal", "normal", "grad", "cg", "kernel"])
    if kind in ("type1", "type2"):
        if rng.random() < 0.25:
            dims = (_log(rng, 96, 320), _log(rng, 96, 320))
            return _case(kind, dims, _log(rng, 1, 32), _log(rng, 8000, 400000), rng.choice([4, 5, 6, 7]), "spiral")
        dims = tuple(_log(rng, 48, 160) for _ in range(3))
        return _case(kind, dims, _log(rng, 1, 32), _log(rng, 32000, 3000000), rng.choice([4, 5, 6, 7]),
                     rng.choice(["radial", "cones"]))
    if kind == "normal":
        if rng.random() < 0.25:
            dims = tuple(2 * rng.choice(_EDGES) for _ in range(2))
            return _case(kind, dims, _log(rng, 1, 32), traj="radial")
        return _case(kind, tuple(rng.choice(_EDGES) for _ in range(3)), _log(rng, 1, 32),
                     traj=rng.choice(["radial", "cones"]))
    if kind == "cg":
        dims = tuple(rng.choice([n for n in _EDGES if n <= 112]) for _ in range(3))
        return _case(kind, dims, _log(rng, 2, 12), traj=rng.choice(["radial", "cones"]), frames=rng.choice([1, 1, 2, 4]),
                     iters=rng.choice([5, 10, 15]))
    if kind == "grad":
        dims = (_log(rng, 96, 256), _log(rng, 96, 256))
        return _case(kind, dims, _log(rng, 2, 12), _log(rng, 8000, 65536), rng.choice([4, 5, 6]), "spiral")
    return _case(kind, tuple(rng.choice(_EDGES) for _ in range(3)), 1, _log(rng, 40000, 2000000), rng.choice([4, 6]),
                 rng.choice(["radial", "cones"]))


# ---- inputs ---------------------------------------------------------------------------------------

def _dims(case):
    return tuple(int(d) for d in case["dims"].split("x"))


def _gen(seed, salt=0):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 7919 + 104729 * salt + 1)
    return g


def _cnormal(shape, g):
    return torch.view_as_complex(torch.randn((*shape, 2), generator=g, device=DEVICE)) / math.sqrt(2.0)


def _axes(dims, scale=1.0):
    """Open grids of centred positions, one per axis, as fractions of the edge."""
    d = len(dims)
    out = []
    for i, n in enumerate(dims):
        a = (torch.arange(n, device=DEVICE, dtype=torch.float32) - n / 2 + 0.5) / n * scale
        out.append(a.reshape([n if j == i else 1 for j in range(d)]))
    return out


def _image(dims, g, lead=()):
    mask = sum((x / a) ** 2 for x, a in zip(_axes(dims), (0.84, 0.72, 0.6)[-len(dims):])) <= 0.25
    return (_cnormal((*lead, *dims), g) * mask).contiguous()


def _coils(coils, dims, g):
    """Gaussian magnitudes around points of a circle / sphere, a linear phase each, unit root sum of squares."""
    d = len(dims)
    pos = torch.randn((coils, d), generator=g, device=DEVICE)
    pos = 0.62 * pos / pos.norm(dim=1, keepdim=True)
    ph = (torch.rand((coils, d + 1), generator=g, device=DEVICE) - 0.5) * math.pi
    ax = _axes(dims)
    S = torch.empty((coils, *dims), dtype=torch.complex64, device=DEVICE)
    power = torch.zeros(dims, device=DEVICE)
    for c in range(coils):
        r2 = sum((x - pos[c, i]) ** 2 for i, x in enumerate(ax))
        mag = torch.exp(-r2 / (2 * 0.6 ** 2))
        S[c] = torch.polar(mag, sum(x * ph[c, i] for i, x in enumerate(ax)) + ph[c, d])
        power += mag * mag
    S /= power.sqrt()
    return S


def _rotation(d, g):
    q, _ = torch.linalg.qr(torch.randn((d, d), generator=g, device=DEVICE, dtype=torch.float64).cpu())
    return q.to(DEVICE)


def _trajectory(case, seed):
    """[dim, points] float32 in [-pi, pi)."""
    M, d, g = int(case["points"]), len(_dims(case)), _gen(seed, 3)
    f64 = dict(device=DEVICE, dtype=torch.float64)
    if d == 2:  # variable-density spirals
        ns = 2048
        ni = -(-M // ns)
        t = torch.arange(ns, **f64) / ns
        off = 2 * math.pi * torch.rand(1, generator=g, **f64)
        a = 2 * math.pi * 16 * t[None] + 2 * math.pi * torch.arange(ni, **f64)[:, None] / ni + off
        r = (math.pi * t ** 1.5)[None]
        k = torch.stack([r * torch.cos(a), r * torch.sin(a)])
    elif case["traj"] == "radial":  # golden-means spokes
        ns = 128
        ni = -(-M // ns)
        n = torch.arange(ni, **f64)
        z = torch.remainder(n * 0.4656, 1.0) * 2 - 1
        az = 2 * math.pi * torch.remainder(n * 0.6823, 1.0)
        st = torch.sqrt(1 - z * z)
        u = _rotation(3, g) @ torch.stack([z, st * torch.cos(az), st * torch.sin(az)])
        k = u[:, :, None] * ((torch.arange(ns, **f64) - ns / 2) * (2 * math.pi / ns))[None, None]
    else:  # cones: spirals around axes spread over the sphere, radius growing to pi
        ns = 256
        ni = -(-M // ns)
        n = torch.arange(ni, **f64)
        z = 1 - 2 * (n + 0.5) / ni
        az = math.pi * (3 - math.sqrt(5)) * n
        st = torch.sqrt(1 - z * z)
        axis = torch.stack([z, st * torch.cos(az), st * torch.sin(az)], 1) @ _rotation(3, g)
        ref = torch.where(axis[:, :1].abs() < 0.9, torch.tensor([[1.0, 0, 0]], **f64), torch.tensor([[0, 1.0, 0]], **f64))
        e1 = torch.linalg.cross(axis, ref)
        e1 = e1 / e1.norm(dim=1, keepdim=True)
        e2 = torch.linalg.cross(axis, e1)
        t = torch.arange(ns, **f64) / ns
        a = 2 * math.pi * 6 * t[None] + 2 * math.pi * torch.rand((ni, 1), generator=g, **f64)
        v = math.cos(0.35) * axis.T[:, :, None] + math.sin(0.35) * (torch.cos(a)[None] * e1.T[:, :, None]
                                                                  + torch.sin(a)[None] * e2.T[:, :, None])
        k = v * (math.pi * t)[None, None]
    k = k.reshape(d, -1)[:, :M]
    return k.clamp(-math.pi, math.pi * (1 - 1e-6)).to(torch.float32).contiguous()


def _density(case, dims, g):
    """Toeplitz kernel(s) [frames, 2N..]: the positive sampling density of a trajectory over the 2N grid, in FFT
    order, with the unevenness of a finite number of readouts, flattened by density compensation; the point
    spread function's centre lies at N - 1 of each axis, hence the ramp."""
    r, ramp = 0, 1
    for i, n in enumerate(dims):
        f = torch.fft.fftfreq(2 * n, device=DEVICE, dtype=torch.float64).reshape([2 * n if j == i else 1 for j in range(len(dims))])
        r = r + 4 * f * f
        ramp = ramp * torch.polar(torch.ones_like(f), -2 * math.pi * f * (n - 1)).to(torch.complex64)
    r = r.sqrt().to(torch.float32)
    base = 0.6 + (0.4 if case["traj"] == "radial" else 0.8) / (1 + 8 * r)
    F = int(case["frames"])
    K = torch.empty((F, *(2 * n for n in dims)), dtype=torch.complex64, device=DEVICE)
    for f in range(F):
        K[f] = ramp * (base * (1 + 0.2 * torch.rand(tuple(2 * n for n in dims), generator=g, device=DEVICE)))
    return K


def _inputs(case, seed):
    """Everything a case starts from, without the package's code."""
    kind, dims, C = case["kind"], _dims(case), int(case["coils"])
    d = {}
    if kind in ("type1", "type2", "grad", "kernel"):
        d["coords"] = _trajectory(case, seed)
    if kind == "type1":
        d["data"] = _cnormal((C, int(case["points"])), _gen(seed, 2))
    elif kind == "type2":
        d["data"] = _image(dims, _gen(seed, 0), (C,))
    elif kind == "kernel":
        k2 = sum(c.double() ** 2 for c in d["coords"])
        d["weights"] = (k2 / k2.mean()).to(torch.float32)
    elif kind == "grad":
        d["smaps"] = _coils(C, dims, _gen(seed, 1))
        d["x"] = _image(dims, _gen(seed, 0))
        d["y"] = _cnormal((C, int(case["points"])), _gen(seed, 2)) * 30
    else:
        d["smaps"] = _coils(C, dims, _gen(seed, 1))
        d["kernel"] = _density(case, dims, _gen(seed, 4))
        d["x"] = _image(dims, _gen(seed, 0), (int(case["frames"]),))
    return d


def prepare(case, seed):
    kind, dims, C = case["kind"], _dims(case), int(case["coils"])
    s = _inputs(case, seed)
    s["kind"], s["dims"], s["width"] = kind, dims, int(case["width"])
    if kind in ("type1", "type2"):
        plan = hb.NufftPlan(hb.NufftType.TYPE_1 if kind == "type1" else hb.NufftType.TYPE_2,
                            hb.NufftOpts(nmodes=dims, ntransf=C, kernel_width=s["width"]))
        plan.setpts(list(s["coords"]))
        s["plan"] = plan
        s["out"] = torch.empty((C, *dims) if kind == "type1" else (C, int(case["points"])), dtype=torch.complex64, device=DEVICE)
    elif kind == "grad":
        s["pair"] = ag.NufftPair(dims, C, kernel_width=s["width"])
        s["x"].requires_grad_(True)
        s["param"] = torch.zeros_like(s["coords"]).requires_grad_(True)
    elif kind == "normal":
        s["op"] = hb.NormalTT1Op(s.pop("kernel")[0], s["smaps"])
        s["x"] = s["x"][0]
        s["out"] = torch.empty_like(s["x"])
    elif kind == "cg":
        F = int(case["frames"])
        kernel = s.pop("kernel")
        if F == 1:
            s["x"] = s["x"][0]
            op = hb.NormalTT1Op(kernel[0], s["smaps"])
            s["solver"] = hb.CGSolver(lambda v, out: op.apply(v, out), dims, DEVICE, max_iter=int(case["iters"]), tol=0.0, graph=True)
        else:
            op = hb.BatchedNormalOp(kernel, s["smaps"])
            s["solver"] = hb.BatchedCGSolver(lambda v, out: op.apply(v, out), F, dims, DEVICE, max_iter=int(case["iters"]), tol=0.0,
                                             graph=True)
        s["x0"] = torch.zeros_like(s["x"])
    return s


def run(state):
    kind = state["kind"]
    if kind in ("type1", "type2"):
        return state["plan"].execute(state["data"], state["out"])
    if kind == "normal":
        return state["op"].apply(state["x"], state["out"])
    if kind == "cg":
        return state["solver"].solve(state["x0"], state["x"])
    if kind == "kernel":
        return hb.build_toeplitz_kernel(list(state["coords"]), state["dims"], state["weights"], kernel_width=state["width"])
    x, k, S, pair = state["x"], state["param"], state["smaps"], state["pair"]
    x.grad = k.grad = None
    with torch.no_grad():
        k.copy_(state["coords"])  # the optimiser's step
    r = ag.nufft_forward(S * x[None], k, pair) - state["y"]
    g = (torch.conj(S) * ag.nufft_adjoint(r, k, pair)).sum(0)
    loss = (g.abs() ** 2).sum()
    loss.backward()
    return {"loss": loss.detach(), "image": x.grad, "coords": k.grad}


def work(case):
    """Inputs read once and outputs written once; the multiply-adds of the w^d taps and of the FFTs over the fine
    (2x) grid, or of the 2N-point FFTs of the Toeplitz operator (pruned to the rows that are not zero)."""
    kind, dims, C = case["kind"], _dims(case), int(case["coils"])
    d, M, w, F, it = len(dims), int(case["points"]), int(case["width"]), int(case["frames"]), max(1, int(case["iters"]))
    n = math.prod(dims)
    nos = n * 2 ** d
    fft = 5.0 * nos * math.log2(nos)
    taps = 4.0 * w ** d * M
    if kind in ("type1", "type2"):
        return {"bytes": 8 * C * n + 8 * C * M + 4 * d * M, "flops": C * (taps + fft)}
    if kind == "kernel":
        return {"bytes": 4 * d * M + 4 * M + 8 * nos, "flops": 4.0 * w ** d * M + 5.0 * 2 ** d * nos * math.log2(nos) + fft}
    if kind == "grad":
        # forward, adjoint, their two backward transforms, and the coordinate gradient of both
        return {"bytes": 8 * C * n + 16 * n + 8 * C * M + 8 * d * M, "flops": C * (6 * taps + 4 * fft)}
    # apply: x in and out, coil maps, kernel
    one = F * (16 * n + 8 * nos) + 8 * C * n
    flops = F * C * 2 * 5.0 * n * sum((2 ** (d - i)) * math.log2(2 * dims[d - 1 - i]) for i in range(d))
    if kind == "normal":
        return {"bytes": one, "flops": flops}
    return {"bytes": one + 16 * F * n, "flops": (it + 1) * flops}


# ---- 64-bit results ---------------------------------------------------------------------------------

#: points x modes x transforms of a direct sum that still takes a few seconds
_DIRECT = 4e13


def _phases(x, n, sign, dtype=torch.complex128):
    k = torch.arange(n, device=DEVICE, dtype=torch.float64) - n // 2
    return torch.polar(torch.ones((), device=DEVICE, dtype=torch.float64), sign * x.double()[:, None] * k[None])


def _direct2(f, coords, sign=-1):
    """c[t, j] = sum_k f[t, k] exp(i sign k x_j)."""
    dims, T, M = tuple(f.shape[1:]), f.shape[0], coords.shape[1]
    out = []
    step = max(1, int(3e8 / (T * math.prod(dims[:-1]))))
    flat = f.reshape(-1, dims[-1]).T
    for j in range(0, M, step):
        x = coords[:, j:j + step]
        v = (_phases(x[-1], dims[-1], sign) @ flat).reshape(x.shape[1], T, *dims[:-1])
        for a in range(len(dims) - 2, -1, -1):
            e = _phases(x[a], dims[a], sign)
            v = torch.matmul(v.reshape(x.shape[1], -1, dims[a]), e[:, :, None])[..., 0]
            v = v.reshape(x.shape[1], T, *dims[:a])
        out.append(v.T)
    return torch.cat(out, 1)


def _direct1(c, coords, dims, sign=1):
    """f[t, k] = sum_j c[t, j] exp(i sign k x_j)."""
    T, M = c.shape
    step = max(1, int(3e8 / (T * math.prod(dims[:-1]))))
    acc = 0
    for j in range(0, M, step):
        x = coords[:, j:j + step]
        v = c[:, j:j + step].T  # [m, T]
        for a in range(len(dims) - 1):
            v = (v.reshape(x.shape[1], -1, 1) * _phases(x[a], dims[a], sign)[:, None, :]).reshape(x.shape[1], -1)
        acc = acc + v.T @ _phases(x[-1], dims[-1], sign)
    return acc.reshape(T, *dims)


def _apply(x, S, K):
    """sum_c conj(S_c) T(S_c x) by the zero-padded FFT, crop at [N-1, 2N-1) per axis."""
    d = x.dim()
    pad, at = tuple(K.shape), tuple(slice(n - 1, 2 * n - 1) for n in x.shape)
    out = torch.zeros_like(x)
    for c in range(S.shape[0]):
        s = S[c].to(torch.complex128)
        out += s.conj() * torch.fft.ifftn(torch.fft.fftn(s * x, s=pad, dim=tuple(range(d))) * K)[at]
    return out


def exact(case, seed):
    kind, dims, C, M = case["kind"], _dims(case), int(case["coils"]), int(case["points"])
    n, d = math.prod(dims), len(dims)
    c128 = torch.complex128
    if kind in ("type1", "type2") and M * n * C > _DIRECT:
        return None
    if kind == "kernel" and M * math.prod(2 * e - 1 for e in dims) > _DIRECT:
        return None
    s = _inputs(case, seed)
    if kind == "type1":
        return _direct1(s["data"].to(c128), s["coords"], dims)
    if kind == "type2":
        return _direct2(s["data"].to(c128), s["coords"])
    if kind == "kernel":
        psf = _direct1(s["weights"].to(c128)[None], s["coords"], tuple(2 * e - 1 for e in dims))[0]
        return torch.fft.fftn(psf, s=tuple(2 * e for e in dims)) / n
    if kind == "grad":
        S, y = s["smaps"].to(c128), s["y"].to(c128)
        x = s["x"].to(c128)
        k = s["coords"].double()
        # loss = ||g||^2, g = S^H A^H r, r = A S x - y; with p = A S g:
        # dL/dx* = 2 S^H A^H p, and the phases' derivatives give the coordinates'
        modes = [torch.arange(e, device=DEVICE, dtype=torch.float64) - e // 2 for e in dims]
        mul = [m.reshape([dims[i] if j == i else 1 for j in range(d)]) for i, m in enumerate(modes)]
        r = _direct2(S * x[None], k) - y
        g = (S.conj() * _direct1(r, k, dims)).sum(0)
        p = _direct2(S * g[None], k)
        gx = 2 * (S.conj() * _direct1(p, k, dims)).sum(0)
        gk = []
        for a in range(d):
            dr = _direct2(-1j * mul[a] * S * x[None], k)   # dr/dk_a at each point
            dp = _direct2(-1j * mul[a] * S * g[None], k)   # d(A S g)/dk_a with g held
            gk.append(2 * (p.conj() * dr + dp.conj() * r).real.sum(0))
        return {"loss": (g.abs() ** 2).sum(), "image": gx, "coords": torch.stack(gk)}
    K = s["kernel"].to(c128)
    S = s["smaps"]
    if kind == "normal":
        return _apply(s["x"][0].to(c128), S, K[0])
    out = []
    for f in range(int(case["frames"])):
        b = s["x"][f].to(c128)
        v, r = torch.zeros_like(b), b.clone()
        p, rz = r.clone(), (r.abs() ** 2).sum()
        for _ in range(int(case["iters"])):
            Ap = _apply(p, S, K[f])
            alpha = rz / (p.conj() * Ap).real.sum()
            v, r = v + alpha * p, r - alpha * Ap
            new = (r.abs() ** 2).sum()
            p, rz = r + (new / rz) * p, new
        out.append(v)
    return out[0] if len(out) == 1 else torch.stack(out)
