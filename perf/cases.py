"""What is measured of this framework, and on which inputs.

Each case is one call (or one short sequence of calls) that a program using the
package makes: DFT and FFT gridding of a projection series, the
Fourier-constraint iteration from a gridded spectrum to a volume, batches of
such problems, the real-space projector, and the whole reconstructor class on
host arrays.  Inputs are synthetic: Gaussian atoms inside an ellipsoid, seen
from random Euler angles or a single-axis tilt series, with noise.  They are
made on the GPU by torch from the seed alone.

Arrays follow the package's MATLAB layout: a torch tensor of shape (dim 3,
dim 2, dim 1) is the column-major dim 1 x dim 2 x dim 3 array.

exact(case, seed) restates every path in 64 bits with torch alone.  The steps
the method itself defines in single precision (which grid points lie near a
plane, their in-plane coordinates and distances) are restated in single
precision, operation by operation, since they decide which points are filled.
"""
import math

import numpy as np
import torch

import genfire_gb300 as G

PRECISIONS = {"fp64": G.PREC_FP64, "mixed": G.PREC_MIXED, "fp16": G.PREC_FP16_SCALED}
ZYZ = ((0.0, 0.0, 1.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0))
ZYX = ((0.0, 0.0, 1.0), (0.0, 1.0, 0.0), (1.0, 0.0, 0.0))


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # the 64^3 tilt-series configuration (31 tilts, 5 degrees apart) gridded with the drop-in precision
        dict(name="grid_fp64_tilt64", kind="grid_dft", D1=64, D2=64, P=31, ratio=2.0, cutoff=0.125, precision="fp64",
             tilt=True),
        # the 256^3 configuration's gridding: 90 Euler triples, split-BF16 operands
        dict(name="grid_mixed_256", kind="grid_dft", D1=256, D2=256, P=90, ratio=2.0, cutoff=0.125,
             precision="mixed", tilt=False),
        # unequal, partly odd sizes at the class's oversampling of 3, a wider cutoff, scaled FP16 operands
        dict(name="grid_fp16_150x105", kind="grid_dft", D1=150, D2=105, P=40, ratio=3.0, cutoff=0.3,
             precision="fp16", tilt=False),
        # the class's default gridding method and cutoff at the 256^3 configuration's size
        dict(name="fftgrid_mixed_256", kind="grid_fft", D1=256, D2=256, P=90, ratio=2.0, cutoff=0.7,
             precision="mixed", tilt=False),
        # the smallest iteration: the 64^3 configuration with its own 200 iterations, bound by latency
        dict(name="recon_mixed_64", kind="recon", D1=64, D2=64, P=31, ratio=2.0, iters=200, mode=3, support=True,
             precision="mixed"),
        # lengths that are no power of two (300 x 225 x 300), unequal sizes, the class's default mode,
        # oversampling and iteration count, no support given
        dict(name="recon_mixed_100x75", kind="recon", D1=100, D2=75, P=40, ratio=3.0, iters=50, mode=1,
             support=False, precision="mixed"),
        # the 256^3 configuration's iteration (512^3 grid)
        dict(name="recon_mixed_256", kind="recon", D1=256, D2=256, P=90, ratio=2.0, iters=100, mode=3, support=True,
             precision="mixed"),
        # the drop-in precision at the 128^3 configuration's size
        dict(name="recon_fp64_128", kind="recon", D1=128, D2=128, P=60, ratio=2.0, iters=50, mode=3, support=True,
             precision="fp64"),
        # the largest configuration: a 512^3 object on a 1024^3 grid
        dict(name="recon_mixed_512", kind="recon", D1=512, D2=512, P=120, ratio=2.0, iters=10, mode=3, support=True,
             precision="mixed"),
        # several objects of the batched configuration's sizes iterated together
        dict(name="batch_mixed_8", kind="batch", sizes="48,64,64,96,96,128,160,192", P=40, ratio=2.0, iters=50,
             precision="mixed"),
        # simulated projections of a finished 256^3 volume (host arrays in and out)
        dict(name="project_mixed_256", kind="project", D1=256, D2=256, P=90, precision="mixed"),
        # the reconstructor class with its defaults (FFT gridding, oversampling 3, mode 1, FP64) on host arrays
        dict(name="class_fp64_64", kind="class", D1=64, D2=64, P=31, iters=50),
    ]


SMOOTH = sorted({2 ** a * 3 ** b * 5 ** c * 7 ** d for a in range(10) for b in range(6) for c in range(4)
                 for d in range(3) if 2 ** a * 3 ** b * 5 ** c * 7 ** d <= 1024})


def _size(rng, lo, hi):
    """A size in [lo, hi] spread over its logarithm whose transforms the library takes (factors 2, 3, 5, 7)."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((s for s in SMOOTH if lo <= s <= hi), key=lambda s: (abs(math.log(s / x)), s))


def draw(rng):
    kind = rng.choice(["grid_dft", "grid_dft", "grid_fft", "recon", "recon", "recon", "batch", "project", "class"])
    if kind == "grid_dft":
        precision = rng.choice(["fp64", "mixed", "fp16"])
        D1 = _size(rng, 24, 80 if precision == "fp64" else 240)
        D2 = D1 if rng.random() < 0.6 else _size(rng, max(24, D1 // 2), D1)
        return dict(kind=kind, D1=D1, D2=D2, P=rng.randint(8, 31 if precision == "fp64" else 80),
                    ratio=float(rng.choice([2, 2, 3])), cutoff=rng.choice([0.1, 0.125, 0.25]), precision=precision,
                    tilt=rng.random() < 0.3)
    if kind == "grid_fft":
        D = _size(rng, 24, 200)
        ratio = float(rng.choice([2, 3])) if D % 2 == 0 else 1.0  # odd sizes: 1 + (D - 1) ratio has to stay smooth
        return dict(kind=kind, D1=D, D2=D, P=rng.randint(8, 80), ratio=ratio, cutoff=rng.choice([0.3, 0.5, 0.7]),
                    precision=rng.choice(["fp64", "mixed"]), tilt=rng.random() < 0.3)
    if kind == "recon":
        precision = rng.choice(["fp64", "mixed", "mixed", "mixed"])
        D1 = _size(rng, 32, 128 if precision == "fp64" else 256)
        D2 = D1 if rng.random() < 0.6 else _size(rng, max(32, D1 // 2), D1)
        return dict(kind=kind, D1=D1, D2=D2, P=rng.randint(20, 60),
                    ratio=float(rng.choice([2, 2, 3] if D1 <= 120 else [2])), iters=rng.randint(20, 50),
                    mode=rng.choice([1, 2, 3]), support=rng.random() < 0.7, precision=precision)
    if kind == "batch":
        n = rng.randint(2, 8)
        return dict(kind=kind, sizes=",".join(str(rng.choice([48, 64, 96, 128, 160])) for _ in range(n)),
                    P=rng.randint(20, 60), ratio=2.0, iters=rng.randint(20, 50), precision="mixed")
    if kind == "project":
        D1 = _size(rng, 32, 243)
        return dict(kind=kind, D1=D1, D2=D1 if rng.random() < 0.5 else _size(rng, 32, D1), P=rng.randint(8, 80),
                    precision=rng.choice(["fp64", "mixed", "mixed"]) if D1 <= 128 else "mixed")
    return dict(kind=kind, D1=(D := rng.choice([24, 32, 36, 40, 48, 56, 60, 64])), D2=D, P=rng.randint(8, 40),
                iters=rng.randint(20, 50))


# --------------------------------------------------------------------------- inputs
_CTX = []


def _ctx():
    """The program's one library context."""
    if not _CTX:
        _CTX.append(G.Context(0))
    return _CTX[0]


def _rng(seed):
    return np.random.default_rng(int(seed) % (1 << 62)), torch.Generator("cuda").manual_seed(int(seed) % (1 << 62))


def _centred(n, dtype=torch.float32):
    return torch.arange(n, device="cuda", dtype=dtype) - n // 2


def _atoms(r, D1, D2):
    """Centres (atoms x 3: dims 1, 2, 3), amplitudes and width of Gaussian atoms in an ellipsoid inside the box."""
    n = 160
    d = r.normal(size=(n, 3))
    d *= (r.random((n, 1)) ** (1 / 3)) / np.linalg.norm(d, axis=1, keepdims=True)
    return d * np.array([0.38 * D1, 0.38 * D2, 0.28 * D1]), r.uniform(0.3, 1.0, n), max(1.0, D1 / 110.0)


def _volume(r, D1, D2):
    c, amp, sigma = _atoms(r, D1, D2)
    c = torch.tensor(c, device="cuda", dtype=torch.float32)
    e = [torch.exp(-(_centred(n)[None, :] - c[:, k, None]) ** 2 / (2 * sigma * sigma))
         for k, n in ((0, D1), (1, D2), (2, D1))]
    e[2] = e[2] * torch.tensor(amp, device="cuda", dtype=torch.float32)[:, None]
    return torch.einsum("az,ayx->zyx", e[2], e[1][:, :, None] * e[0][:, None, :])


def _angles(r, P, tilt):
    if tilt:
        return np.stack([np.zeros(P), np.linspace(-75, 75, P), np.zeros(P)], 1)
    return np.stack([r.uniform(0, 360, P), r.uniform(-72, 72, P), r.uniform(0, 360, P)], 1)


def _projections(r, g, D1, D2, P, R):
    """Line integrals of rotated Gaussian atoms with 2 % noise: a (P, D2, D1) double tensor."""
    c, amp, sigma = _atoms(r, D1, D2)
    out = torch.empty(P, D2, D1, device="cuda", dtype=torch.float64)
    a = torch.tensor(amp, device="cuda", dtype=torch.float64)
    for p in range(P):
        q = torch.tensor(c @ R[p], device="cuda", dtype=torch.float64)  # R' c
        ex = torch.exp(-(_centred(D1, torch.float64)[None, :] - q[:, 0, None]) ** 2 / (2 * sigma * sigma))
        ey = torch.exp(-(_centred(D2, torch.float64)[None, :] - q[:, 1, None]) ** 2 / (2 * sigma * sigma))
        out[p] = (ey * a[:, None]).T @ ex * (sigma * math.sqrt(2 * math.pi))
    out += 0.02 * out.std() * torch.randn(out.shape, device="cuda", dtype=torch.float64, generator=g)
    return out


def _support(D1, D2):
    x, y = _centred(D1), _centred(D2)
    return ((x[None, None, :] / (0.43 * D1)) ** 2 + (y[None, :, None] / (0.43 * D2)) ** 2
            + (x[:, None, None] / (0.31 * D1)) ** 2 <= 1).to(torch.uint8).contiguous()


def _padded(v, n1, n2):
    D1, D2 = v.shape[2], v.shape[1]
    o1, o2 = n1 // 2 - D1 // 2, n2 // 2 - D2 // 2
    out = torch.zeros(n1, n2, n1, device="cuda", dtype=v.dtype)
    out[o1:o1 + D1, o2:o2 + D2, o1:o1 + D1] = v
    return out


def _measured(r, g, D1, D2, n1, n2, P, cdtype):
    """A gridded spectrum: the noisy object's transform on the points near P planes, zero elsewhere, centred."""
    x = _padded(_volume(r, D1, D2), n1, n2)
    x += 0.02 * x.std() * torch.randn(x.shape, device="cuda", generator=g)
    near = torch.zeros(n1, n2, n1, device="cuda", dtype=torch.bool)
    k1, k2 = _centred(n1), _centred(n2)
    for p in range(P):
        th, ph = math.radians(r.uniform(0, 72)), r.uniform(0, 2 * math.pi)
        h = (math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th))
        near |= ((k1 * h[0])[None, None, :] + (k2 * h[1])[None, :, None] + (k1 * h[2])[:, None, None]).abs() < 0.125
    x = torch.fft.ifftshift(x)
    m = torch.fft.fftshift(torch.fft.fftn(x.to(torch.float64) if cdtype == torch.complex128 else x))
    return torch.where(near, m, torch.zeros((), device="cuda", dtype=m.dtype)).to(cdtype).contiguous()


def _params(case, D1, D2):
    p = G.default_params()
    p.Dim1, p.Dim2, p.NumProjs = D1, D2, case["P"]
    p.oversamplingRatio = case["ratio"]
    p.interpolationCutoffDistance = case.get("cutoff", 0.125)
    for name, v in zip(("vector1", "vector2", "vector3"), ZYX if case.get("tilt") else ZYZ):
        getattr(p, name)[:] = v
    p.precision = PRECISIONS[case["precision"]]
    p.griddingMethod = 1 if case["kind"] == "grid_fft" else 2
    if "iters" in case:
        p.numIterations = case["iters"]
        p.constraintEnforcementMode = case.get("mode", 3)
    return p


def _problem(case, D1, D2, seed):
    r, g = _rng(seed)
    p = _params(case, D1, D2)
    n1, n2 = G.grid_size(p)
    double = case["precision"] == "fp64"
    return dict(p=p, M=_measured(r, g, D1, D2, n1, n2, case["P"], torch.complex128 if double else torch.complex64),
                support=_support(D1, D2) if case.get("support", True) else None,
                rec=torch.empty(D1, D2, D1, device="cuda", dtype=torch.float64 if double else torch.float32),
                errK=torch.empty(case["iters"], device="cuda", dtype=torch.float64))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        state = dict(problems=[_problem(case, int(s), int(s), seed + 7919 * i)
                               for i, s in enumerate(case["sizes"].split(","))])
    elif kind == "recon":
        state = _problem(case, case["D1"], case["D2"], seed)
    else:
        r, g = _rng(seed)
        D1, D2, P = case["D1"], case["D2"], case["P"]
        angles = _angles(r, P, case.get("tilt", False))
        if kind == "project":
            v = _volume(r, D1, D2) + 0.01 * torch.rand(D1, D2, D1, device="cuda", generator=g)
            state = dict(vol=np.asfortranarray(v.cpu().numpy().T.astype("f8" if case["precision"] == "fp64" else "f4")),
                         angles=np.asfortranarray(angles))
        elif kind == "class":
            R = [_rot_zyz(*a) for a in angles]
            state = dict(projections=np.asfortranarray(_projections(r, g, D1, D2, P, R).cpu().numpy().T),
                         support=np.asfortranarray(_support(D1, D2).cpu().numpy().T != 0), angles=angles)
        else:
            p = _params(case, D1, D2)
            n1, n2 = G.grid_size(p)
            R = [_rot_zyz(*a) if kind == "grid_fft" else _rot(ZYX if case["tilt"] else ZYZ, a) for a in angles]
            double = case["precision"] == "fp64"
            state = dict(p=p, angles=np.asfortranarray(angles), projections=_projections(r, g, D1, D2, P, R),
                         M=torch.empty(n1, n2, n1, device="cuda",
                                       dtype=torch.complex128 if double else torch.complex64),
                         rec=torch.empty(D1, D2, D1, device="cuda", dtype=torch.float64 if double else torch.float32))
    state["case"] = case
    torch.cuda.synchronize()  # the library works on a stream of its own
    return state


# --------------------------------------------------------------------------- the calls
def _open(ctx, s):
    return ctx.recon(s["p"], s["M"].data_ptr(), support=None if s["support"] is None else s["support"].data_ptr(),
                     on_device=True)


def _close(r, s):
    r.result_device(s["rec"].data_ptr(), s["errK"].data_ptr())
    r.close()
    # the complex64 iteration's error record carries single precision
    return [s["rec"], s["errK"] if s["rec"].dtype == torch.float64 else s["errK"].float()]


def run(state):
    ctx, kind = _ctx(), state["case"]["kind"]
    if kind in ("grid_dft", "grid_fft"):
        call = ctx.grid_dft_device if kind == "grid_dft" else ctx.grid_fft_device
        n = call(state["p"], state["projections"].data_ptr(), state["angles"], state["M"].data_ptr(),
                 state["rec"].data_ptr())
        return [state["M"], state["rec"], n]
    if kind == "recon":
        r = _open(ctx, state)
        r.iterate(state["p"].numIterations)
        return _close(r, state)
    if kind == "batch":
        rs = [_open(ctx, s) for s in state["problems"]]
        b = G.ReconBatch(ctx, rs)
        b.iterate(state["case"]["iters"])
        b.close()
        return [_close(r, s) for r, s in zip(rs, state["problems"])]
    if kind == "project":
        return ctx.project(state["vol"], state["angles"], precision=PRECISIONS[state["case"]["precision"]])
    obj = G.GENFIRE_Reconstructor(InputProjections=state["projections"], InputAngles=state["angles"],
                                  Support=state["support"], numIterations=state["case"]["iters"])
    obj = obj.CheckPrepareData().runGridding().reconstruct()
    return [obj.measuredK, obj.recIFFT, obj.reconstruction, obj.errK]


# --------------------------------------------------------------------------- what a pass cannot do without
def _iteration_work(D1, D2, n1, n2, P, iters, double):
    S = 16 if double else 8
    N, half = n1 * n2 * n1, n1 // 2 + 1
    # in and out once; per iteration the object read and written and, since a volume's transform does not fit on
    # chip, one half spectrum of its box between two sweeps, each way; real transforms of the padded volume
    per = D1 * D2 * D1 * S + 4 * half * D2 * D1 * S
    return N * S + D1 * D2 * D1 * (S // 2 + 1) + iters * per, iters * 2 * 2.5 * N * math.log2(N)


def work(case):
    kind, P = case["kind"], case["P"]
    double = case.get("precision", "fp64") == "fp64"
    S = 16 if double else 8
    if kind == "batch":
        b = f = 0.0
        for s in case["sizes"].split(","):
            n = round(int(s) * case["ratio"])
            x, y = _iteration_work(int(s), int(s), n, n, P, case["iters"], double)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    D1, D2 = case["D1"], case["D2"]
    box = D1 * D2 * D1
    if kind == "project":
        return {"bytes": (box + D1 * D2 * P) * S / 2, "flops": 16.0 * box * P}
    if kind == "class":
        n = 3 * D2
        b, f = _iteration_work(D1, D2, n, n, P, case["iters"], True)
        return {"bytes": 8.0 * D1 * D2 * P + 16.0 * n ** 3 + b, "flops": f + P * 5.0 * n * n * math.log2(n * n)}
    n1, n2 = G.grid_size(_params(case, D1, D2))
    if kind == "recon":
        b, f = _iteration_work(D1, D2, n1, n2, P, case["iters"], double)
        return {"bytes": b, "flops": f}
    N = n1 * n2 * n1
    b = 8.0 * D1 * D2 * P + N * S + box * S / 2
    rec = 2.5 * N * math.log2(N)  # the inverse transform of the grid
    if kind == "grid_fft":
        return {"bytes": b, "flops": rec + P * 5.0 * n1 * n1 * math.log2(n1 * n1)}
    nk = P * 2 * case["cutoff"] * n1 * n2 / 2  # points within the cutoff of half a plane
    return {"bytes": b, "flops": rec + nk * (4.0 * D1 * D2 + 8.0 * D2)}


# --------------------------------------------------------------------------- the same in 64 bits
def _sincosd(x):
    r = math.remainder(x, 360.0)
    q = round(r / 90.0)
    t = (r - 90.0 * q) * (math.pi / 180.0)
    s, c = math.sin(t), math.cos(t)
    return [(s, c), (c, -s), (-s, -c), (-c, s)][q % 4]


def _rot_zyz(phi, theta, psi):
    (sf, cf), (st, ct), (sp, cp) = _sincosd(phi), _sincosd(theta), _sincosd(psi)
    return np.array([[cp * ct * cf - sp * sf, -sp * ct * cf - cp * sf, st * cf],
                     [cp * ct * sf + sp * cf, -sp * ct * sf + cp * cf, st * sf], [-cp * st, sp * st, ct]])


def _rot(vectors, angles):
    """The product of three axis rotations, element by element in double."""
    out = None
    for v, th in zip(vectors, angles):
        th = float(th) * math.pi / 180.0
        nv = math.sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2])
        w, s = math.cos(th / 2), -math.sin(th / 2)
        x, y, z = s * (v[0] / nv), s * (v[1] / nv), s * (v[2] / nv)
        q = [[1 - 2 * y * y - 2 * z * z, 2 * x * y + 2 * w * z, 2 * x * z - 2 * w * y],
             [2 * x * y - 2 * w * z, 1 - 2 * x * x - 2 * z * z, 2 * y * z + 2 * w * x],
             [2 * x * z + 2 * w * y, 2 * y * z - 2 * w * x, 1 - 2 * x * x - 2 * y * y]]
        out = q if out is None else [[out[i][0] * q[0][j] + out[i][1] * q[1][j] + out[i][2] * q[2][j]
                                      for j in range(3)] for i in range(3)]
    return np.array(out)


def _near_plane(R64, n1, n2, cutoff):
    """(index, distance, u, v) of the half grid's points near a plane, in the method's single precision."""
    f = np.float32
    R = R64.astype(f)
    nrm = R[:, 2]
    nn = f(np.sqrt(f(f(nrm[0] * nrm[0]) + f(nrm[1] * nrm[1])) + f(nrm[2] * nrm[2])))
    h = [float(f(x / nn)) for x in nrm]
    k1 = torch.arange(-(n1 // 2), 1, device="cuda", dtype=torch.float32)
    k2 = torch.arange(-(n2 // 2), n2 // 2 + 1, device="cuda", dtype=torch.float32)
    k3 = torch.arange(-(n1 // 2), n1 // 2 + 1, device="cuda", dtype=torch.float32)
    D = (((k1 * h[0])[None, None, :] + (k2 * h[1])[None, :, None]) + (k3 * h[2])[:, None, None]).abs()
    below = f(cutoff) if float(f(cutoff)) >= cutoff else np.nextafter(f(cutoff), f(np.inf))
    ind = torch.nonzero((D < float(below)).reshape(-1)).reshape(-1)
    D = D.reshape(-1)[ind]
    l1, l2 = k1.numel(), k2.numel()
    p = [k1[ind % l1], k2[(ind // l1) % l2], k3[ind // (l1 * l2)]]
    nr = [float(x) for x in nrm]
    nsq = float(f(f(f(nrm[0] * nrm[0]) + f(nrm[1] * nrm[1])) + f(nrm[2] * nrm[2])))
    s = (p[0] * nr[0] + p[1] * nr[1]) + p[2] * nr[2]
    t = (0.0 - s) / torch.full_like(s, nsq)
    b = [p[i] + t * nr[i] for i in range(3)]
    A, piv = R.copy(), []
    for k in range(3):
        j = k + int(np.argmax(np.abs(A[k:, k])))
        piv.append(j)
        A[[k, j]] = A[[j, k]]
        if A[k, k] != 0 and k < 2:
            A[k + 1:, k] = A[k + 1:, k] * f(f(1) / A[k, k])
        for j in range(k + 1, 3):
            for i in range(k + 1, 3):
                A[i, j] = f(A[i, j] - f(A[i, k] * A[k, j]))
    for k in range(3):
        b[k], b[piv[k]] = b[piv[k]], b[k]
    for k in range(3):
        for i in range(k + 1, 3):
            b[i] = b[i] - b[k] * float(A[i, k])
    for k in (2, 1, 0):
        b[k] = b[k] / torch.full_like(b[k], float(A[k, k]))
        for i in range(k):
            b[i] = b[i] - b[k] * float(A[i, k])
    ok = (b[0].abs() <= n1 / 2) & (b[1].abs() <= n2 / 2)
    return ind[ok], D[ok], b[0][ok], b[1][ok], (k3.numel(), l2, l1)


def _box_of(M, D1, D2):
    n1, n2 = M.shape[0], M.shape[1]
    o1, o2 = n1 // 2 - D1 // 2, n2 // 2 - D2 // 2
    x = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(M))).real
    return x[o1:o1 + D1, o2:o2 + D2, o1:o1 + D1].contiguous()


def _exact_dft(case, seed):
    s = prepare(case, seed)
    D1, D2 = case["D1"], case["D2"]
    n2, n1 = s["M"].shape[1], s["M"].shape[2]
    num = ws = hit = val = None
    counts = []
    a, b = _centred(D1, torch.float64), _centred(D2, torch.float64)
    for p, ang in enumerate(s["angles"]):
        ind, dist, u, v, shape = _near_plane(_rot(ZYX if case["tilt"] else ZYZ, ang), n1, n2, case["cutoff"])
        if num is None:
            n = shape[0] * shape[1] * shape[2]
            num = torch.zeros(n, device="cuda", dtype=torch.complex128)
            val = torch.zeros(n, device="cuda", dtype=torch.complex128)
            ws = torch.zeros(n, device="cuda", dtype=torch.float64)
            hit = torch.zeros(n, device="cuda", dtype=torch.bool)
        counts.append(ind.numel())
        F = torch.empty(ind.numel(), device="cuda", dtype=torch.complex128)
        P = s["projections"][p]  # (D2, D1)
        for j in range(0, ind.numel(), 1 << 18):
            t = (u[j:j + (1 << 18), None].double() * a) / n1
            t = -2 * math.pi * (t - t.round())
            w = (v[j:j + (1 << 18), None].double() * b) / n2
            w = -2 * math.pi * (w - w.round())
            q = torch.complex(torch.cos(t) @ P.T, torch.sin(t) @ P.T)
            F[j:j + (1 << 18)] = (q * torch.complex(torch.cos(w), torch.sin(w))).sum(1)
        exact = dist.double() < 1e-7
        wgt = torch.where(exact, torch.zeros((), device="cuda", dtype=torch.float64), 1.0 / dist.double().clamp_min(1e-30))
        num[ind] += F * wgt
        ws[ind] += wgt
        hit[ind[exact]] = True
        val[ind[exact]] = F[exact]
    fs = torch.where(hit, val, torch.where(ws > 0, num / ws.clamp_min(1e-300), torch.zeros_like(num))).reshape(shape)
    M = torch.zeros(n1, n2, n1, device="cuda", dtype=torch.complex128)
    c = n1 - n1 // 2 - 1
    M[:, :, :n1 // 2 + 1] = fs[:n1, :n2]
    M[:, :, n1 // 2 + 1:] = fs.flip(0, 1, 2)[:n1, :n2, 1:1 + c].conj()
    return [M, _box_of(M, D1, D2), np.array(counts, dtype=np.int64)]


def _fft_grid(projections, angles, m, cutoff):
    """FFT gridding of (P, D2, D1) projections onto an m^3 cube: (spectrum, number of gridded pairs)."""
    P, D2, D1 = projections.shape
    h = m // 2
    num = torch.zeros(m ** 3, device="cuda", dtype=torch.complex128)
    ws = torch.zeros(m ** 3, device="cuda", dtype=torch.float64)
    k = _centred(m)
    f = np.float32
    below = f(cutoff) if float(f(cutoff)) <= cutoff else np.nextafter(f(cutoff), f(-np.inf))
    s, pairs = int(math.floor(cutoff + 0.5)), 0
    for p in range(P):
        pad = torch.zeros(m, m, device="cuda", dtype=torch.float64)
        pad[h - D2 // 2:h - D2 // 2 + D2, h - D1 // 2:h - D1 // 2 + D1] = projections[p]
        F = torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(pad))).reshape(-1)
        R = _rot_zyz(*angles[p]).astype(f)
        c = [((k * float(R[i, 0]))[None, :] + (k * float(R[i, 1]))[:, None]).reshape(-1) for i in range(3)]
        near = [torch.sign(x) * torch.floor(x.abs() + 0.5) for x in c]
        for ys in range(-s, s + 1):
            for xs in range(-s, s + 1):
                for zs in range(-s, s + 1):
                    t = [near[0] + xs, near[1] + ys, near[2] + zs]
                    i = [x.long() + h for x in t]
                    d = [a - b for a, b in zip(c, t)]
                    d = torch.sqrt((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2])
                    ok = (d <= float(below))
                    for x in i:
                        ok &= (x >= 0) & (x < m)
                    w = (torch.ones((), device="cuda") / (d[ok] + 1e-5)).double()
                    at = i[0][ok] + m * (i[1][ok] + m * i[2][ok])
                    num.index_add_(0, at, F[ok] * w)
                    ws.index_add_(0, at, w)
                    pairs += at.numel()
    fs = torch.where(ws > 0, num / ws.clamp_min(1e-300), torch.zeros_like(num)).reshape(m, m, m)
    e = m + (m % 2 == 0)
    full = torch.zeros(e, e, e, device="cuda", dtype=torch.complex128)
    full[:m, :m, :m] = fs
    mate = full.flip(0, 1, 2)
    count = ((full != 0).double() + (mate != 0).double()).clamp_min(1)
    return ((full + mate.conj()) / count)[:m, :m, :m].contiguous(), pairs


def _iterate(M, support, D1, D2, iters, mode):
    """reconstruct's loop in double: (the best object, its error record)."""
    n1, n2 = M.shape[0], M.shape[1]
    E = torch.fft.ifftshift(M != 0)
    Ms = torch.fft.ifftshift(M.to(torch.complex128))
    S = torch.fft.ifftshift(_padded(torch.ones(D1, D2, D1, device="cuda", dtype=torch.float64) if support is None
                                    else support.to(torch.float64), n1, n2))
    m = {1: [0.95 + i * -0.1 for i in range(12)] + [-10.0] * 3 + [-0.15 + i * 0.1 for i in range(12)],
         2: [0.95 + i * -0.1 for i in range(12)] + [-10.0] * 2, 3: [-999.0] * 5}[mode]
    if mode != 3:
        # (divided by a tensor: torch multiplies by a scalar's reciprocal, which moves points across a threshold)
        k = [_centred(n, torch.float64) / torch.full((n,), float(n // 2), device="cuda", dtype=torch.float64)
             for n in (n1, n2)]
        # the first dimension's index takes the second dimension's vector and back; equal lengths 1 and 3
        q = torch.sqrt((k[1] * k[1])[None, :, None] + (k[0] * k[0])[None, None, :] + (k[0] * k[0])[:, None, None])
        ci = torch.fft.ifftshift(1 - q)
    at = [int(math.floor(1 + i * (iters - 1) / (len(m) - 1) + 0.5)) for i in range(len(m))]
    at[-1] = iters
    me = Ms[E].abs()
    denom = me.sum()
    x = torch.zeros(n1, n2, n1, device="cuda", dtype=torch.float64)
    best, best_err, cur, C = x, 1e30, 0, None
    err = torch.zeros(iters, dtype=torch.float64)
    for it in range(1, iters + 1):
        if cur < len(m) and it == at[cur]:
            last = max(i for i, y in enumerate(at) if y == it)
            C = E if m[last] < -2 else E & (ci > m[last])
            cur, best_err = last + 1, 1e30
        x = x.clamp_min(0) * S
        k = torch.fft.fftn(x)
        err[it - 1] = ((k[E].abs() - me).abs().sum() / denom).item()
        if err[it - 1] < best_err:
            best, best_err = x, float(err[it - 1])
        x = torch.fft.ifftn(torch.where(C, Ms, k)).real
    o1, o2 = n1 // 2 - D1 // 2, n2 // 2 - D2 // 2
    return torch.fft.fftshift(best)[o1:o1 + D1, o2:o2 + D2, o1:o1 + D1].contiguous(), err


def _exact_project(case, seed):
    s = prepare(case, seed)
    v = torch.tensor(s["vol"].T, device="cuda", dtype=torch.float64)  # (dim 3, dim 2, dim 1)
    n3, n2, n1 = v.shape
    V = v.reshape(-1)
    out = torch.empty(case["P"], n2, n1, device="cuda", dtype=torch.float64)
    X, Y, Z = _centred(n1, torch.float64), _centred(n2, torch.float64), _centred(n3, torch.float64)
    for p, ang in enumerate(s["angles"]):
        R = _rot_zyz(*ang)
        c = [((X * R[i, 0])[None, None, :] + (Y * R[i, 1])[None, :, None]) + (Z * R[i, 2])[:, None, None] + n // 2
             for i, n in enumerate((n1, n2, n3))]
        ok = torch.ones((), device="cuda", dtype=torch.bool)
        for x, n in zip(c, (n1, n2, n3)):
            ok = ok & (x >= 0) & (x <= n - 1)
        i = [x.floor().clamp(0, n - 2).long() for x, n in zip(c, (n1, n2, n3))]
        fr = [x - y for x, y in zip(c, i)]
        base = i[0] + n1 * (i[1] + n2 * i[2])
        acc = torch.zeros_like(fr[0])
        for dz in (0, 1):
            for dy in (0, 1):
                for dx in (0, 1):
                    w = (fr[0] if dx else 1 - fr[0]) * (fr[1] if dy else 1 - fr[1]) * (fr[2] if dz else 1 - fr[2])
                    acc += w * V[torch.where(ok, base + dx + n1 * (dy + n2 * dz), torch.zeros_like(base))]
        out[p] = torch.where(ok, acc, torch.zeros_like(acc)).sum(0)
    return out.permute(2, 1, 0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid_dft":
        return _exact_dft(case, seed)
    if kind == "grid_fft":
        s = prepare(case, seed)
        M, pairs = _fft_grid(s["projections"], s["angles"], s["M"].shape[0], case["cutoff"])
        return [M, _box_of(M, case["D1"], case["D2"]), pairs]
    if kind == "recon":
        s = prepare(case, seed)
        return list(_iterate(s["M"], s["support"], case["D1"], case["D2"], case["iters"], case["mode"]))
    if kind == "batch":
        s = prepare(case, seed)
        return [list(_iterate(q["M"], q["support"], q["p"].Dim1, q["p"].Dim2, case["iters"], 3)) for q in s["problems"]]
    if kind == "project":
        return _exact_project(case, seed)
    s = prepare(case, seed)
    D = case["D1"]
    pj = torch.tensor(s["projections"].T, device="cuda").contiguous()
    M, _ = _fft_grid(pj, s["angles"], 3 * D, 0.7)
    sup = torch.tensor(s["support"].T, device="cuda")
    rec, err = _iterate(M, sup, D, D, case["iters"], 1)
    return [M.permute(2, 1, 0).cpu().numpy(), _box_of(M, D, D).permute(2, 1, 0).cpu().numpy(),
            rec.permute(2, 1, 0).cpu().numpy(), err.numpy()]
