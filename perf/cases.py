"""Timed cases of the projectors and solvers: what programs that reconstruct with this library call.

A case names an operation (forward, adjoint, the gradient of a least-squares problem, a CGNE
solve), a projector, the volume, the detector and a circular trajectory. Volumes are random
ellipsoids, sinograms their analytic line integrals plus noise. ``exact`` restates the operators
in 64 bits with torch; its sample positions and geometry are 64-bit too, so it also shows the
drift of the float positions that the operators are defined with (a few 1e-6).
"""
import math

import numpy as np
import torch

import elsa_b200.pyelsa as elsa
from elsa_b200 import torch_ops

BLOB = {"radius": 2.0, "alpha": 10.83, "order": 2}
LUT = 100


def _case(name, op, projector, vol, views, det, s2c, c2d, arc=360.0, batch=1, iterations=0):
    c = {"op": op, "projector": projector, "dim": len(vol), "nx": vol[0], "ny": vol[1],
         "nz": vol[2] if len(vol) == 3 else 1, "views": views, "nu": det[0],
         "nv": det[1] if len(vol) == 3 else 1, "s2c": float(s2c), "c2d": float(c2d),
         "arc": float(arc), "batch": batch, "iterations": iterations}
    return dict({"name": name}, **c) if name else c


def listed():
    return [
        # a whole small solve: 20 iterations on one fan-beam slice, bound by launches and latency
        _case("fan128_cgne20", "cgne", "joseph", (128, 128), 180, (182,), 1000, 250,
              iterations=20),
        # one slice of ordinary size, each direction
        _case("fan512_forward", "forward", "joseph", (512, 512), 720, (730,), 5120, 1280),
        _case("fan512_adjoint", "adjoint", "joseph", (512, 512), 720, (730,), 5120, 1280),
        # the cone-beam scan of the benchmark, each direction: the largest calls
        _case("cone256_forward", "forward", "joseph", (256, 256, 256), 360, (384, 384), 2560, 640),
        _case("cone256_adjoint", "adjoint", "joseph", (256, 256, 256), 360, (384, 384), 2560, 640),
        # differentiable reconstruction: loss and gradient of a batch of eight volumes
        _case("cone128_batch8_gradient", "gradient", "joseph", (128, 128, 128), 180, (192, 192),
              1280, 320, batch=8),
        # exact-length ray tracing on a volume and a detector of odd sizes, a short arc
        _case("siddon_ragged_forward", "forward", "siddon", (171, 200, 149), 240, (250, 231), 1900,
              500, arc=220.0),
        _case("siddon_ragged_adjoint", "adjoint", "siddon", (171, 200, 149), 240, (250, 231), 1900,
              500, arc=220.0),
        # blob basis functions, the voxel-driven operator of the benchmark, each direction
        _case("blob128_forward", "forward", "blob", (128, 128, 128), 180, (192, 192), 1280, 320),
        _case("blob128_adjoint", "adjoint", "blob", (128, 128, 128), 180, (192, 192), 1280, 320),
        # differential phase contrast with B-splines: the gradient of one ragged volume
        _case("phase_ragged_gradient", "gradient", "phase_bspline", (101, 77, 90), 121, (143, 118),
              900, 260),
        # the ray-driven blob operator, a small volume: loss and gradient
        _case("rayblob64_gradient", "gradient", "ray_blob", (64, 64, 64), 60, (96, 96), 640, 160),
    ]


# per projector: the operations drawn, the edge ranges by dimension, most voxels times views in 3D
_DRAWN = [
    ("joseph", ("forward", "adjoint", "gradient", "cgne"), 3, (32, 256), 3.0e9),
    ("joseph", ("forward", "adjoint", "gradient", "cgne"), 2, (64, 512), 1.8e8),
    ("siddon", ("forward", "adjoint"), 3, (32, 200), 1.1e9),
    ("siddon", ("forward", "adjoint"), 2, (64, 512), 1.8e8),
    ("blob", ("forward", "adjoint", "gradient"), 3, (24, 128), 1.5e8),
    ("bspline", ("forward", "adjoint", "gradient"), 3, (24, 128), 1.5e8),
    ("phase_blob", ("forward", "adjoint"), 3, (24, 128), 1.5e8),
    ("phase_bspline", ("forward", "adjoint", "gradient"), 3, (24, 128), 1.5e8),
    ("blob", ("forward", "adjoint"), 2, (64, 512), 1.0e8),
    ("ray_blob", ("forward", "adjoint", "gradient"), 3, (24, 64), 1.6e7),
    ("ray_bspline", ("forward", "adjoint"), 3, (24, 64), 1.6e7),
]


def draw(rng):
    projector, ops, dim, (lo, hi), most = rng.choice(_DRAWN)
    op = rng.choice(ops)

    def size(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    edge = size(lo, hi)
    vol = [max(lo, min(hi, int(round(edge * rng.uniform(0.7, 1.15))))) for _ in range(dim)]
    views = size(30, 360 if dim == 3 else 720)
    det = [max(8, int(round(edge * rng.uniform(1.1, 1.5)))) for _ in range(dim - 1)]
    iterations = rng.randint(3, 20) if op == "cgne" else 0
    batch = rng.choice([1, 1, 2, 3, 4]) if op == "gradient" and dim == 3 else 1
    nvox = float(np.prod(vol))
    passes = 2 * batch if op == "gradient" else 2 * iterations + 1 if op == "cgne" else 1
    if op == "cgne" and dim == 3:
        passes *= 2
    views = max(3, min(views, int(most * (30 if dim == 2 else 1) / (nvox * passes))))
    s2c = edge * rng.uniform(4.0, 10.0)
    return _case(None, op, projector, vol, views, det, s2c, s2c * rng.uniform(0.2, 0.35),
                 arc=rng.choice([180.0, 200.0, 220.0, 360.0, 360.0]), batch=batch,
                 iterations=iterations)


# ---- geometry and inputs ------------------------------------------------------------------------


def _vol(case):
    return [case["nx"], case["ny"], case["nz"]][:case["dim"]]


def _det(case):
    return [case["nu"], case["nv"]][:case["dim"] - 1]


def _angles(case):
    n = case["views"]
    return [case["arc"] * math.pi / 180.0 * (i / (n - 1) if n > 1 else 0.0) for i in range(n)]


def _rotation(case, angle):
    """Rows: detector u, (v,) and the viewing direction, in voxel coordinates."""
    c, s = math.cos(angle), math.sin(angle)
    if case["dim"] == 2:
        return [[c, -s], [s, c]]
    return [[c, 0.0, s], [0.0, 1.0, 0.0], [-s, 0.0, c]]


def _source_and_rays(case, angle):
    """Source position [dim] and unit ray directions [nv * nu, dim] of one view."""
    dim = case["dim"]
    R = torch.tensor(_rotation(case, angle), dtype=torch.float64, device="cuda")
    centre = torch.tensor([0.5 * n for n in _vol(case)], dtype=torch.float64, device="cuda")
    sdd = case["s2c"] + case["c2d"]
    u = (torch.arange(case["nu"], dtype=torch.float64, device="cuda") + 0.5 - 0.5 * case["nu"]) / sdd
    if dim == 3:
        v = (torch.arange(case["nv"], dtype=torch.float64, device="cuda") + 0.5
             - 0.5 * case["nv"]) / sdd
        v, u = torch.meshgrid(v, u, indexing="ij")
        cam = torch.stack([u, v, torch.ones_like(u)], -1).reshape(-1, 3)
    else:
        cam = torch.stack([u, torch.ones_like(u)], -1)
    d = cam @ R
    return centre - case["s2c"] * R[dim - 1], d / d.norm(dim=1, keepdim=True)


def _ellipsoids(case, gen, count=20):
    """Centres, half axes (voxels) and amplitudes of random ellipsoids inside the volume."""
    dim = case["dim"]
    n = torch.tensor(_vol(case), dtype=torch.float64, device="cuda")
    r = torch.rand(count, 2 * dim + 1, dtype=torch.float64, device="cuda", generator=gen)
    half = n * (0.04 + 0.18 * r[:, :dim])
    centre = 0.5 * n + (r[:, dim:2 * dim] - 0.5) * (0.8 * n - 2 * half)
    half[0], centre[0] = 0.42 * n, 0.5 * n
    return centre, half, 0.1 + 0.9 * r[:, 2 * dim]


def _volume(case, ellipsoids):
    axes = [torch.arange(n, dtype=torch.float32, device="cuda") + 0.5 for n in _vol(case)]
    x = torch.zeros([len(a) for a in reversed(axes)], dtype=torch.float32, device="cuda")
    for centre, half, amp in zip(*(t.tolist() for t in ellipsoids)):
        q = 0.0
        for i, a in enumerate(axes):
            shape = [1] * len(axes)
            shape[len(axes) - 1 - i] = -1
            q = q + (((a - centre[i]) / half[i]) ** 2).reshape(shape)
        x += amp * (q <= 1.0)
    return x.reshape(-1)


def _sinogram(case, ellipsoids, gen):
    """Line integrals of the ellipsoids with 1 % noise (every pixel is non-zero, as in a scan)."""
    out = []
    for angle in _angles(case):
        o, d = _source_and_rays(case, angle)
        y = torch.zeros(d.shape[0], dtype=torch.float64, device="cuda")
        for centre, half, amp in zip(*ellipsoids):
            p, e = (o - centre) / half, d / half
            a, b, c = (e * e).sum(1), e @ p, (p * p).sum() - 1.0
            y += amp * 2.0 * (b * b - a * c).clamp(min=0.0).sqrt() / a
        out.append(y.float())
    y = torch.cat(out)
    noise = torch.randn(y.numel(), dtype=torch.float32, device="cuda", generator=gen)
    return y + noise * (0.01 * float(y.max()))


def _inputs(case, seed):
    """(volumes [batch, n] or None, sinograms [batch, m] or None) as the operation reads them."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    x, y = [], []
    for _ in range(case["batch"]):
        e = _ellipsoids(case, gen)
        if case["op"] in ("forward", "gradient"):
            x.append(_volume(case, e))
        if case["op"] != "forward":
            # the measurements of another object: the gradient is not small
            y.append(_sinogram(case, _ellipsoids(case, gen), gen))
    return torch.stack(x) if x else None, torch.stack(y) if y else None


def _operator(case):
    vol = elsa.VolumeDescriptor(_vol(case))
    sino = elsa.CircleTrajectoryGenerator.createTrajectory(
        case["views"], vol, case["arc"], case["s2c"], case["c2d"], detectorSize=_det(case))
    make = {"joseph": elsa.JosephsMethodCUDA, "siddon": elsa.SiddonsMethodCUDA,
            "blob": elsa.BlobVoxelProjectorCUDA, "bspline": elsa.BSplineVoxelProjectorCUDA,
            "phase_blob": elsa.PhaseContrastBlobVoxelProjectorCUDA,
            "phase_bspline": elsa.PhaseContrastBSplineVoxelProjectorCUDA,
            "ray_blob": elsa.BlobProjector, "ray_bspline": elsa.BSplineProjector}
    return make[case["projector"]](vol, sino), vol, sino


def prepare(case, seed):
    A, vol, sino = _operator(case)
    x, y = _inputs(case, seed)
    state = {"op": case["op"], "A": A}
    if case["op"] == "forward":
        state["x"] = elsa.DataContainer(x[0], vol)
    elif case["op"] == "adjoint":
        state["y"] = elsa.DataContainer(y[0], sino)
    elif case["op"] == "cgne":
        state["solver"] = elsa.CGNE(A, elsa.DataContainer(y[0], sino))
        state["iterations"] = case["iterations"]
    else:
        state["x"], state["y"] = x.requires_grad_(True), y
    return state


def run(state):
    if state["op"] == "forward":
        return state["A"].apply(state["x"]).tensor
    if state["op"] == "adjoint":
        return state["A"].applyAdjoint(state["y"]).tensor
    if state["op"] == "cgne":
        return state["solver"].solve(state["iterations"]).tensor
    r = torch_ops.project(state["x"], state["A"]) - state["y"]
    (g,) = torch.autograd.grad(0.5 * (r * r).sum(), state["x"])
    return {"residual": r.detach(), "gradient": g}


# ---- work and tolerances --------------------------------------------------------------------------


def work(case):
    nvox, nsino = float(np.prod(_vol(case))), float(np.prod(_det(case))) * case["views"]
    mag = (case["s2c"] + case["c2d"]) / case["s2c"]
    pairs = nvox * case["views"] * mag ** (case["dim"] - 1)  # rays that meet a voxel, over the views
    support = 2.0 if case["projector"].endswith("blob") else 1.5
    # per pair: Joseph interpolates on 0.9 planes from 2 or 4 taps, Siddon crosses 1.28 voxels,
    # a basis function covers (2 support)^(dim - 1) pixels with a distance and a table value each
    flops = {"joseph": 0.9 * (8 + 4 * case["dim"]), "siddon": 1.28 * 6}.get(
        case["projector"], (2 * support) ** (case["dim"] - 1) * 10) * pairs
    once = 4.0 * (nvox + nsino)
    if case["op"] == "gradient":  # volume and measurements read, residual and gradient written
        return {"bytes": 2 * case["batch"] * once, "flops": 2 * case["batch"] * flops}
    if case["op"] == "cgne":
        return {"bytes": once, "flops": (2 * case["iterations"] + 1) * flops}
    return {"bytes": once, "flops": flops}


def tolerance(case):
    if case["op"] == "cgne":  # the recurrence amplifies the rounding of ill-conditioned problems
        return {"rel": 2e-3}
    return {"rel": 1e-5}


# ---- the operators in 64 bits ----------------------------------------------------------------------


def _line_setup(case, o, d):
    """Per ray: driving axis (largest direction component, the first of equal ones), entry and
    exit parameters of the volume box."""
    n = torch.tensor(_vol(case), dtype=torch.float64, device="cuda")
    t1, t2 = -o / d, (n - o) / d
    near, far = torch.minimum(t1, t2), torch.maximum(t1, t2)
    near = torch.where(torch.isnan(near), torch.full_like(near, -math.inf), near)
    far = torch.where(torch.isnan(far), torch.full_like(far, math.inf), far)
    return d.abs().argmax(1), near.max(1).values, far.min(1).values


def _strides(case):
    s = [1, case["nx"], case["nx"] * case["ny"]][:case["dim"]]
    return torch.tensor(s, dtype=torch.int64, device="cuda")


def _groups(case, angle):
    """The rays of one view that meet the volume, by driving axis: (axis, ray numbers, o, d, t0,
    t1)."""
    o, d = _source_and_rays(case, angle)
    axis, t0, t1 = _line_setup(case, o, d)
    for g in range(case["dim"]):
        at = ((axis == g) & (t1 > t0)).nonzero().reshape(-1)
        if at.numel():
            yield g, at, o, d[at], t0[at], t1[at]


def _joseph(case, x, y):
    """One view at a time: y += A x (x given) or the adjoint's sums (y given)."""
    vol, stride = _vol(case), _strides(case).tolist()
    nrays = int(np.prod(_det(case)))
    out = torch.zeros(nrays * case["views"] if x is not None else int(np.prod(vol)),
                      dtype=torch.float64, device="cuda")
    for p, angle in enumerate(_angles(case)):
        for g, at, o, d, t0, t1 in _groups(case, angle):
            n = torch.tensor(vol, dtype=torch.float64, device="cuda")
            step = d / d[:, g:g + 1].abs()
            enter = torch.minimum((o + d * t0[:, None]).clamp(min=0.0), n)
            leave = torch.minimum((o + d * t1[:, None]).clamp(min=0.0), n)
            first = enter[:, g].floor()
            sign = d[:, g].sign()
            pos = enter + step * ((first + 0.5 - enter[:, g]) * sign)[:, None]
            count = (leave[:, g] - (first + 0.5)).abs().ceil()
            length = step.norm(dim=1)
            # all rays at once, plane by plane of the volume
            others = [i for i in range(case["dim"]) if i != g]
            acc = torch.zeros_like(length)
            w_in = None if y is None else y[p * nrays + at].double() * length
            for k in range(vol[g]):
                j = (k - first) * sign
                live = (j >= 0) & (j < count)
                if not bool(live.any()):
                    continue
                idx = torch.full_like(at, k * stride[g])
                taps = [(idx, live.double())]
                for i in others:
                    h = pos[:, i] + j * step[:, i] - 0.5
                    low = h.floor()
                    cw = h - low
                    low = low.long()
                    new = []
                    for e, w in ((0, 1.0 - cw), (1, cw)):
                        c = low + e
                        ok = (c >= 0) & (c < vol[i])
                        c = c.clamp(0, vol[i] - 1) * stride[i]
                        new += [(b + c, wt * w * ok) for b, wt in taps]
                    taps = new
                for b, wt in taps:
                    if x is not None:
                        acc += wt * x[b]
                    else:
                        out.index_add_(0, b, wt * w_in)
            if x is not None:
                out[p * nrays + at] = acc * length
    return out


def _siddon(case, x, y):
    vol, stride = _vol(case), _strides(case)
    nrays = int(np.prod(_det(case)))
    out = torch.zeros(nrays * case["views"] if x is not None else int(np.prod(vol)),
                      dtype=torch.float64, device="cuda")
    n = torch.tensor(vol, dtype=torch.float64, device="cuda")
    for p, angle in enumerate(_angles(case)):
        for _, at, o, d, t0, t1 in _groups(case, angle):
            enter = o + d * t0[:, None]
            cell = torch.minimum(torch.maximum((enter + 1e-9 * d).floor(), torch.zeros_like(n)),
                                 n - 1)
            t = t0.clone()
            acc = torch.zeros_like(t)
            w_in = None if y is None else y[p * nrays + at].double()
            delta = d.sign()
            for _ in range(int(sum(vol)) + 3):
                nxt = torch.where(d != 0, (cell + (d > 0) - o) / d, torch.full_like(d, math.inf))
                te = torch.minimum(nxt.min(1).values, t1)
                live = ((t < t1) & (cell >= 0).all(1) & (cell < n).all(1)).double()
                if not bool(live.any()):
                    break
                idx = (torch.minimum(cell.clamp(min=0), n - 1).long() * stride).sum(1)
                w = (te - t).clamp(min=0.0) * live
                if x is not None:
                    acc += w * x[idx]
                else:
                    out.index_add_(0, idx, w * w_in)
                cell = cell + delta * (nxt <= te[:, None])
                t = te
            if x is not None:
                out[p * nrays + at] = acc
    return out


def _bessel_half(m, z):
    """sqrt(pi / (2 z)) I_{m + 1/2}(z)."""
    s, c = math.sinh(z), math.cosh(z)
    return [s / z, (c - s / z) / z, ((3.0 / (z * z) + 1.0) * s - 3.0 / z * c) / z][m]


def _bessel_int(m, z):
    """I_m(z) by its power series."""
    term, k = (0.5 * z) ** m / math.factorial(m), 0
    total = term
    while term > 1e-18 * total:
        k += 1
        term *= 0.25 * z * z / (k * (k + m))
        total += term
    return total


def _bspline(x, m):
    return sum((-1) ** k * math.comb(m + 1, k) * max(0.0, x + 0.5 * (m + 1) - k) ** m
               for k in range(m + 2)) / math.factorial(m)


def _table(case):
    """(support, 100 samples) of the projected basis function, or of its derivative (divided by
    the distance in 3D) for phase contrast."""
    kind, dim = case["projector"], case["dim"]
    phase = kind.startswith("phase")
    if kind.endswith("blob"):
        a, alpha, m = BLOB["radius"], BLOB["alpha"], BLOB["order"]

        def f(s):
            w = 1.0 - (s / a) ** 2
            if w <= 1e-10:
                return 0.0
            z = alpha * math.sqrt(w)
            if not phase:
                return 2.0 * a / alpha * w * z * _bessel_half(2, z) / _bessel_int(2, alpha)
            v = -2.0 / (alpha * a) * z * z * _bessel_half(1, z) / _bessel_int(2, alpha)
            return v if dim == 3 else v * s
        support = a
    else:
        # the ray-driven operator takes the spline of one dimension for its projected table
        scale = 1.0
        for _ in range(dim - 2):
            scale *= _bspline(0.0, 2)

        def f(s):
            if not phase:
                return scale * _bspline(s, 2)
            v = (_bspline(s + 0.5, 1) - _bspline(s - 0.5, 1)) * scale
            return v if dim == 2 else v / max(s, 1e-10)
        support = 1.5
    return support, torch.tensor([f(support * i / (LUT - 1)) for i in range(LUT)],
                                 dtype=torch.float64, device="cuda")


def _lookup(table, support, dist):
    index = dist * ((LUT - 1) / support)
    low = index.floor().clamp(max=LUT - 1).long()
    t = index - low
    v = (1.0 - t) * table[low] + t * table[(low + 1).clamp(max=LUT - 1)]
    return v * (index <= LUT - 1)


def _voxel(case, x, y):
    """The footprint loop of the default mode: as many rows as the footprint has columns, each as
    long as the footprint has rows, starting where the previous one ended."""
    dim, vol = case["dim"], _vol(case)
    nu, nv = case["nu"], case["nv"]
    support, table = _table(case)
    phase = case["projector"].startswith("phase")
    npix = nu * nv
    out = torch.zeros(npix * case["views"] if x is not None else int(np.prod(vol)),
                      dtype=torch.float64, device="cuda")
    axes = [torch.arange(n, dtype=torch.float64, device="cuda") + 0.5 - 0.5 * n for n in vol]
    grid = torch.meshgrid(*reversed(axes), indexing="ij")
    centre = torch.stack([g.reshape(-1) for g in reversed(grid)], -1)
    sdd = case["s2c"] + case["c2d"]
    for p, angle in enumerate(_angles(case)):
        R = torch.tensor(_rotation(case, angle), dtype=torch.float64, device="cuda")
        cam = centre @ R.T
        cam[:, dim - 1] += case["s2c"]
        z = cam[:, dim - 1]
        s = sdd / cam.norm(dim=1)
        r = s * support
        c0 = sdd * cam[:, 0] / z + 0.5 * nu - 0.5
        lo0 = (c0 - r).ceil().clamp(min=0).long()
        ext0 = (c0 + r).floor().clamp(max=nu - 1).long() - lo0 + 1
        if dim == 3:
            c1 = sdd * cam[:, 1] / z + 0.5 * nv - 0.5
            lo1 = (c1 - r).ceil().clamp(min=0).long()
            ext1 = (c1 + r).floor().clamp(max=nv - 1).long() - lo1 + 1
        else:
            c1, lo1, ext1 = torch.zeros_like(c0), torch.zeros_like(lo0), torch.ones_like(ext0)
        rows, cols = (ext0, ext1) if dim == 3 else (ext1, ext0)
        any_ = (ext0 > 0) & (ext1 > 0)
        rows, cols = rows * any_, cols * any_
        view = out[p * npix:(p + 1) * npix] if x is not None else None
        for i in range(int(rows.max())):
            d1 = (c1 - (lo1 + i)) / s if dim == 3 else torch.zeros_like(c0)
            for j in range(int(cols.max())):
                u = lo0 + (i * (cols - ext0) + j if dim == 3 else j)
                lin = (lo1 + i) * nu + u
                d0 = (c0 - u) / s
                w = _lookup(table, support, (d0 * d0 + d1 * d1).sqrt())
                w = w * ((i < rows) & (j < cols) & (lin >= 0) & (lin < npix))
                if phase:
                    w = w * (d0 if dim == 3 else d0.sign())
                lin = lin.clamp(0, npix - 1)
                if x is not None:
                    view.index_add_(0, lin, w * x)
                else:
                    out += w * y[p * npix + lin].double()
    return out


def _ray_lut(case, x, y):
    """Per ray and slice along its driving axis: the voxels within the support's reach. The
    adjoint walks the box grown by that reach off the driving axis."""
    dim, vol, stride = case["dim"], _vol(case), _strides(case).tolist()
    support, table = _table(case)
    reach = 2
    nrays = int(np.prod(_det(case)))
    out = torch.zeros(nrays * case["views"] if x is not None else int(np.prod(vol)),
                      dtype=torch.float64, device="cuda")
    grow = 0 if x is not None else reach
    for p, angle in enumerate(_angles(case)):
        o, d = _source_and_rays(case, angle)
        axis = d.abs().argmax(1)
        for g in range(dim):
            at = (axis == g).nonzero().reshape(-1)
            if not at.numel():
                continue
            dg = d[at]
            acc = torch.zeros(at.numel(), dtype=torch.float64, device="cuda")
            w_in = None if y is None else y[p * nrays + at].double()
            others = [i for i in range(dim) if i != g]
            for k in range(vol[g]):
                pos = o + dg * ((k + 0.5 - o[g]) / dg[:, g])[:, None]
                inside = torch.ones_like(at, dtype=torch.bool)
                for i in others:
                    inside &= (pos[:, i] >= -grow) & (pos[:, i] <= vol[i] + grow)
                if not bool(inside.any()):
                    continue
                base = [pos[:, i].trunc().long() for i in range(dim)]
                ranges = [range(-reach, reach + 1) if i != g else (0,) for i in range(dim)]
                for e in np.ndindex(*[len(r) for r in ranges]):
                    ok, idx, diff = inside, 0, []
                    for i in range(dim):
                        c = base[i] + ranges[i][e[i]] if i != g else torch.full_like(at, k)
                        ok = ok & (c >= 0) & (c < vol[i])
                        idx = idx + c.clamp(0, vol[i] - 1) * stride[i]
                        diff.append(c + 0.5 - o[i])
                    diff = torch.stack(diff, -1)
                    perp = diff - (diff * dg).sum(1, keepdim=True) * dg
                    w = _lookup(table, support, perp.norm(dim=1)) * ok
                    if x is not None:
                        acc += w * x[idx]
                    else:
                        out.index_add_(0, idx, w * w_in)
            if x is not None:
                out[p * nrays + at] = acc
    return out


def _apply(case, x=None, y=None):
    kind = case["projector"]
    f = {"joseph": _joseph, "siddon": _siddon}.get(
        kind, _ray_lut if kind.startswith("ray") else _voxel)
    return f(case, None if x is None else x.double(), y)


def exact(case, seed):
    pairs = float(np.prod(_vol(case))) * case["views"]
    passes = {"gradient": 2 * case["batch"], "cgne": 2 * case["iterations"] + 1}.get(case["op"], 1)
    per = {"joseph": 1.0, "siddon": 8.0}.get(case["projector"], 25.0 if case["dim"] == 3 else 5.0)
    if pairs * passes * per > 2.5e10 or case["views"] * passes * max(_vol(case)) > 5e5:
        return None  # over about 20 seconds
    x, y = _inputs(case, seed)
    if case["op"] == "forward":
        return _apply(case, x=x[0])
    if case["op"] == "adjoint":
        return _apply(case, y=y[0])
    if case["op"] == "gradient":
        r = torch.stack([_apply(case, x=v) for v in x]) - y.double()
        return {"residual": r, "gradient": torch.stack([_apply(case, y=v) for v in r])}
    q = torch.zeros(x.shape[1] if x is not None else int(np.prod(_vol(case))),
                    dtype=torch.float64, device="cuda")
    r = _apply(case, y=y[0])
    s, gamma = r.clone(), r @ r
    for _ in range(case["iterations"]):
        z = _apply(case, y=_apply(case, x=s))
        alpha = gamma / (s @ z)
        q += alpha * s
        r -= alpha * z
        last, gamma = gamma, r @ r
        s = r + (gamma / last) * s
    return q
