"""Performance cases of the framework's public entry points.

Each case is one call (or the few calls that belong together) that a reconstruction program makes on
device-resident data: the Toeplitz and SENSE normal operators, conjugate gradients, the NUFFT-based
SENSE operators, the construction of the Toeplitz diagonal and the locally-low-rank proximal step.
Sizes are those of the benchmark's workloads (64^3 x 8 coils; 128^3 x 16 coils, 20 frames x 5
encodings, 2000 spokes x 256 samples; the uneven mix of 96^3, 128^3 and 160 x 160 x 128) and generic
neighbours of them.

``prepare`` makes inputs, plans and operator data from a seed, ``run`` is one pass, ``exact`` the same
result in 64 bits with plain torch (direct non-uniform Fourier sums, FFTs, eigendecompositions).
"""
import math

import numpy as np
import torch

from hastycompute_b200 import synth
from hastycompute_b200.batched_sense import BatchedSenseNormal
from hastycompute_b200.llr import Normal3DBlocksSVT, admm_vectors
from hastycompute_b200.nufft import CUDANufft, NufftOptions, NufftPlan
from hastycompute_b200.toeplitz import ToeplitzPlan

DEV = "cuda"


def listed():
    return [
        # one image through the bare Toeplitz operator: the smallest call, three launches
        {"name": "toeplitz_64", "kind": "toeplitz", "n0": 64, "n1": 64, "n2": 64, "samples": 8192},
        # the single-frame SENSE normal operator, the inner call of an interactive reconstruction
        {"name": "normal_64_c8", "kind": "normal", "n0": 64, "n1": 64, "n2": 64, "coils": 8, "frames": 1, "encodings": 1,
         "samples": 8192, "lam": 1e-3},
        # the three image sizes of an uneven job mix; encodings of a frame share its diagonal
        {"name": "normal_96_c12", "kind": "normal", "n0": 96, "n1": 96, "n2": 96, "coils": 12, "frames": 1, "encodings": 5,
         "samples": 8192, "lam": 1e-3},
        {"name": "normal_128_c16", "kind": "normal", "n0": 128, "n1": 128, "n2": 128, "coils": 16, "frames": 2,
         "encodings": 5, "samples": 8192, "lam": 1e-3},
        {"name": "normal_160_c8", "kind": "normal", "n0": 160, "n1": 160, "n2": 128, "coils": 8, "frames": 1,
         "encodings": 5, "samples": 8192, "lam": 1e-3},
        # a short solve, as the x-update of an ADMM iteration makes it
        {"name": "cg_64_c8", "kind": "cg", "n0": 64, "n1": 64, "n2": 64, "coils": 8, "frames": 1, "encodings": 1,
         "samples": 8192, "lam": 0.02, "iters": 5},
        # right-hand side of the solve (type 1) and its forward model (type 2) for one frame of the 4D-flow scan
        {"name": "adjoint_128_c16", "kind": "adjoint", "n0": 128, "n1": 128, "n2": 128, "coils": 16, "spokes": 2000,
         "readout": 256, "tol": 1e-6},
        {"name": "forward_128_c16", "kind": "forward", "n0": 128, "n1": 128, "n2": 128, "coils": 16, "spokes": 2000,
         "readout": 256, "tol": 1e-6},
        # data-consistency gradient through the NUFFT pair with density weights, default tolerance
        {"name": "gradient_64_c8", "kind": "gradient", "n0": 64, "n1": 64, "n2": 64, "coils": 8, "spokes": 4096,
         "readout": 128, "tol": 1e-5},
        # a batch of 2-D slices there and back
        {"name": "slices_128", "kind": "slices", "n1": 128, "n2": 128, "transforms": 8, "spokes": 201, "readout": 256,
         "tol": 1e-5},
        # the Toeplitz diagonal of one frame, built once per frame and scan
        {"name": "diagonal_128", "kind": "diagonal", "n0": 128, "n1": 128, "n2": 128, "spokes": 2000, "readout": 256,
         "tol": 1e-6},
        # the proximal step of an ADMM iteration over the whole 4D-flow series
        {"name": "lowrank_128", "kind": "lowrank", "d0": 20, "d1": 5, "n0": 128, "n1": 128, "n2": 128, "b0": 8, "b1": 8,
         "b2": 8, "soft": True, "thresh": 60.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _toeplitz_shape(rng):
    """An image size that the Toeplitz plans take: (nz, ny) powers of two, 96^2 or 160^2."""
    which = rng.random()
    if which < 0.2:
        n0 = n1 = 96
    elif which < 0.4:
        n0 = n1 = 160
    else:
        n0, n1 = rng.choice([16, 32, 64, 128]), rng.choice([32, 64, 128])
        if rng.random() < 0.6:
            n0 = n1 = max(n0, n1)
    return n0, n1, rng.choice([32, 64, 96, 128, 160])


def draw(rng):
    kind = rng.choice(["toeplitz", "normal", "normal", "normal", "cg", "adjoint", "forward", "gradient", "slices", "diagonal",
                       "lowrank"])
    if kind in ("toeplitz", "normal", "cg"):
        n0, n1, n2 = _toeplitz_shape(rng)
        c = {"kind": kind, "n0": n0, "n1": n1, "n2": n2, "samples": _log_int(rng, 2000, 9000)}
        if kind == "toeplitz":
            return c
        budget = 160 * 128**3 // (2 if kind == "normal" else 16)  # image voxels x coils x systems
        slots = max(1, min(160, budget // (n0 * n1 * n2)))
        coils = _log_int(rng, 1, min(32, slots))
        systems = max(1, slots // coils)
        encodings = rng.randint(1, min(5, systems))
        frames = rng.randint(1, max(1, min(4, systems // encodings)))
        c.update(coils=coils, frames=frames, encodings=encodings, lam=1e-3 if kind == "normal" else 0.02)
        if kind == "cg":
            c["iters"] = rng.randint(2, 5)
        return c
    if kind == "lowrank":
        d0, d1 = rng.randint(4, 32), rng.randint(1, 5)
        side = min(128, int((100 * 128**3 / (d0 * d1)) ** (1 / 3) * 0.8))
        n = [rng.randint(32, max(33, side)) for _ in range(3)]
        b = rng.randint(4, 8)
        return {"kind": kind, "d0": d0, "d1": d1, "n0": n[0], "n1": n[1], "n2": n[2], "b0": b, "b1": b, "b2": rng.choice([b, 8]),
                "soft": rng.random() < 0.8, "thresh": 0.0}
    tol = rng.choice([1e-3, 1e-4, 1e-5, 1e-6])
    readout, spokes = rng.randint(65, 257), _log_int(rng, 101, 2000)
    if kind == "slices":
        return {"kind": kind, "n1": rng.choice([32, 64, 80, 96, 128, 160]), "n2": rng.choice([64, 96, 128, 160]),
                "transforms": rng.randint(1, 24), "spokes": _log_int(rng, 31, 800), "readout": readout, "tol": tol}
    if kind == "diagonal":
        n = rng.choice([32, 64, 128])
        return {"kind": kind, "n0": n, "n1": rng.choice([n, 64]), "n2": rng.choice([n, 64]), "spokes": spokes,
                "readout": readout, "tol": rng.choice([1e-5, 1e-6])}
    n = rng.choice([32, 48, 64, 80, 96, 128])
    c = {"kind": kind, "n0": rng.choice([n, n, 32]), "n1": n, "n2": rng.choice([n, n, 64]), "coils": _log_int(rng, 1, 16),
         "spokes": spokes, "readout": readout, "tol": tol}
    if kind == "gradient":
        c["coils"] = min(8, c["coils"])
    return c


# ---------------------------------------------------------------------------- inputs ----
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _cplx(shape, g):
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=g, device=DEV) * math.sqrt(0.5))


def _shape(c):
    return (c["n0"], c["n1"], c["n2"])


def _koosh(c, seed):
    return synth.kooshball(c["spokes"], c["readout"], frame=seed % 9973, nframes=20)


def _sparse_koosh(c, seed, frame):
    """The trajectory of a frame with few samples: 64 per spoke."""
    return synth.kooshball(c["samples"] // 64, 64, frame=seed % 9973 + 7 * frame, nframes=20)


def _radial2(c, seed):
    """Golden-angle radial 2-D trajectory, float32 [2, K]."""
    ang = (np.arange(c["spokes"]) + seed % 1009) * (math.pi * (math.sqrt(5.0) - 1) / 2)
    t = -math.pi + 2 * math.pi * np.arange(c["readout"]) / c["readout"]
    return np.stack([np.outer(np.sin(ang), t).ravel(), np.outer(np.cos(ang), t).ravel()]).astype(np.float32)


def _operator_inputs(c, seed):
    """Images, coil maps and (per frame) coordinates of the Toeplitz cases."""
    g = _gen(seed)
    shape = _shape(c)
    nsys = c["frames"] * c["encodings"]
    x = _cplx((nsys,) + shape, g)
    maps = synth.coil_maps_torch(c["coils"], shape, seed=seed, device=DEV)
    coords = [torch.from_numpy(_sparse_koosh(c, seed, f)).to(DEV) for f in range(c["frames"])]
    return x, maps, coords


def _kspace_inputs(c, seed):
    g = _gen(seed)
    coords = torch.from_numpy(_koosh(c, seed)).to(DEV)
    maps = synth.coil_maps_torch(c["coils"], _shape(c), seed=seed, device=DEV)
    return g, coords, maps


def _density(coords):
    """Radial density weights: |k|^2 with a floor at the centre."""
    r2 = (coords.double() ** 2).sum(0) / math.pi**2
    return (r2 + 1e-4).clamp(max=1.0).float()


def _lowrank_inputs(c, seed):
    """A series of smooth rank-3 frames with noise, and a dual variable."""
    g = _gen(seed)
    n = (c["d1"],) + _shape(c)
    basis = [_cplx(n, g) for _ in range(3)]
    coef = torch.randn(c["d0"], 3, generator=g, device=DEV)
    x = torch.empty((c["d0"],) + n, dtype=torch.complex64, device=DEV)
    u = torch.empty_like(x)
    for f in range(c["d0"]):
        x[f] = sum(float(coef[f, r]) * basis[r] for r in range(3)) + 0.3 * _cplx(n, g)
        u[f] = 0.1 * _cplx(n, g)
    return x, u


def _threshold(c):
    if not c["soft"]:
        return 3  # keep the three largest singular values
    rows = c["d1"] * c["b0"] * c["b1"] * c["b2"]
    return c["thresh"] or 0.5 * (math.sqrt(rows) + math.sqrt(c["d0"]))


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "toeplitz":
        plan = ToeplitzPlan(_shape(c))
        x = _cplx(_shape(c), _gen(seed))
        packed = plan.build_diagonal(torch.from_numpy(_sparse_koosh(c, seed, 0)).to(DEV))
        return {"case": c, "plan": plan, "x": x, "packed": packed,
                "storage": torch.empty(plan.grid, dtype=torch.complex64, device=DEV)}
    if k in ("normal", "cg"):
        plan = ToeplitzPlan(_shape(c))
        x, maps, coords = _operator_inputs(c, seed)
        packed = torch.stack([plan.build_diagonal(f) for f in coords])
        if k == "cg":  # an operator of unit mean
            packed *= 8.0 * float(np.prod(_shape(c))) / coords[0].shape[1]
        index = [f for f in range(c["frames"]) for _ in range(c["encodings"])]
        return {"case": c, "plan": plan, "x": x, "out": torch.empty_like(x), "maps": maps, "packed": packed, "index": index}
    if k in ("adjoint", "forward"):
        g, coords, maps = _kspace_inputs(c, seed)
        plan = NufftPlan(coords, _shape(c), tol=c["tol"])
        data = _cplx((c["coils"], coords.shape[1]), g) if k == "adjoint" else _cplx(_shape(c), g)
        return {"case": c, "plan": plan, "maps": maps, "data": data}
    if k == "gradient":
        g, coords, maps = _kspace_inputs(c, seed)
        x = _cplx((1, 1) + _shape(c), g)
        y = _cplx((1, c["coils"], coords.shape[1]), g)
        op = BatchedSenseNormal([coords], maps, kdata_vec=[y], weights_vec=[_density(coords)], tol=c["tol"])
        return {"case": c, "op": op, "x": x}
    if k == "slices":
        coords = torch.from_numpy(_radial2(c, seed)).to(DEV)
        modes = [c["transforms"], c["n1"], c["n2"]]
        return {"case": c, "f": _cplx(modes, _gen(seed)), "forward": CUDANufft(coords, modes, NufftOptions.type2(tol=c["tol"])),
                "adjoint": CUDANufft(coords, modes, NufftOptions.type1(tol=c["tol"]))}
    if k == "diagonal":
        return {"case": c, "plan": ToeplitzPlan(_shape(c)), "coords": torch.from_numpy(_koosh(c, seed)).to(DEV)}
    if k == "lowrank":
        x, u = _lowrank_inputs(c, seed)
        b = (c["b0"], c["b1"], c["b2"])
        svt = Normal3DBlocksSVT(tuple(x.shape), b, b, 1, _threshold(c), soft=c["soft"], seed=seed)
        return {"case": c, "x": x, "u": u, "z": torch.empty_like(x), "svt": svt}
    raise ValueError(k)


# ------------------------------------------------------------------------------ pass ----
def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "toeplitz":
        return s["plan"].apply(s["x"], s["packed"], s["storage"])
    if k == "normal":
        return s["plan"].sense_normal(s["x"], s["out"], s["maps"], s["packed"], diag_index=s["index"], lam=c["lam"])
    if k == "cg":
        x = torch.zeros_like(s["x"])
        s["plan"].cg(x, s["x"], s["maps"], s["packed"], iters=c["iters"], lam=c["lam"], diag_index=s["index"])
        return x
    if k == "adjoint":
        return s["plan"].sense_adjoint(s["data"], s["maps"])
    if k == "forward":
        return s["plan"].sense_forward(s["data"], s["maps"])
    if k == "gradient":
        return s["op"].apply(s["x"], manipulator="weighted_kdata")
    if k == "slices":
        y = torch.empty((c["transforms"], s["forward"].nfreq()), dtype=torch.complex64, device=DEV)
        s["forward"].apply(s["f"], y)
        f = torch.empty_like(s["f"])
        s["adjoint"].apply(y, f)
        return y, f
    if k == "diagonal":
        return s["plan"].build_diagonal(s["coords"], method="nufft", tol=c["tol"])
    admm_vectors(1, s["x"], s["z"], s["u"])  # z = x + u, then the proximal step in place
    return s["svt"].apply(s["z"])


# ------------------------------------------------------------------------------ work ----
def _fft_flops(m):
    return 5.0 * m * math.log2(m)


def work(case):
    c, k = case, case["kind"]
    if k in ("toeplitz", "normal", "cg"):
        n = float(np.prod(_shape(c)))
        if k == "toeplitz":
            return {"bytes": 8 * n + 8 * n + 32 * n, "flops": 2 * _fft_flops(8 * n)}
        nsys = c["frames"] * c["encodings"]
        one = nsys * 16 * n + c["coils"] * 8 * n + c["frames"] * 32 * n
        reps = 1 if k == "normal" else c["iters"] + 1
        return {"bytes": reps * one, "flops": reps * nsys * c["coils"] * 2 * _fft_flops(8 * n)}
    if k == "lowrank":
        n = float(c["d0"] * c["d1"] * np.prod(_shape(c)))
        return {"bytes": 3 * 8 * n, "flops": 12.0 * n * c["d0"]}
    w = math.ceil(math.log10(1 / c["tol"])) + 1
    samples = float(c["spokes"] * c["readout"])
    if k == "slices":
        n, t = float(c["n1"] * c["n2"]), c["transforms"]
        return {"bytes": t * 8 * (2 * n + 2 * samples) + 2 * 8 * samples, "flops": 2 * t * (_fft_flops(4 * n) + 4 * samples * w**2)}
    n = float(np.prod(_shape(c)))
    if k == "diagonal":
        return {"bytes": 12 * samples + 32 * n, "flops": _fft_flops(64 * n) + _fft_flops(8 * n) + 4 * samples * w**3}
    t = c["coils"]
    passes = 2 if k == "gradient" else 1
    data = 12 * samples + t * 8 * samples + (4 * samples if k == "gradient" else 0)
    return {"bytes": data + t * 8 * n + passes * 8 * n, "flops": passes * t * (_fft_flops(8 * n) + 4 * samples * w**3)}


# ----------------------------------------------------------------- 64-bit references ----
def _phasors(x, n, sign):
    """exp(sign i k x) for the centred modes k of an axis: [len(x), n] complex128."""
    k = torch.arange(n, device=DEV, dtype=torch.float64) - n // 2
    return torch.polar(torch.ones((), dtype=torch.float64, device=DEV), sign * x.double()[:, None] * k[None, :])


def _chunks(samples, row):
    """Sample ranges whose [chunk, row] complex128 temporaries stay near 1 GB."""
    step = max(64, int(2**26 // row))
    return [slice(a, min(samples, a + step)) for a in range(0, samples, step)]


def _type2(coords, f, sign=-1):
    """c[t, j] = sum_k f[t, k] exp(sign i k x_j), f [t, n0, n1, n2] complex128."""
    t, n0, n1, n2 = f.shape
    out = torch.empty((t, coords.shape[1]), dtype=torch.complex128, device=DEV)
    for sl in _chunks(coords.shape[1], n0 * n1):
        e = [_phasors(coords[a, sl], n, sign) for a, n in enumerate((n0, n1, n2))]
        for i in range(t):
            v = (e[2] @ f[i].reshape(n0 * n1, n2).T).reshape(-1, n0, n1)  # sum over x
            v = torch.matmul(v, e[1][:, :, None])[:, :, 0]
            out[i, sl] = (v * e[0]).sum(1)
    return out


def _type1(coords, y, shape, sign=+1):
    """f[t, k] = sum_j y[t, j] exp(sign i k x_j)."""
    n0, n1, n2 = shape
    out = torch.zeros((y.shape[0], n0 * n1, n2), dtype=torch.complex128, device=DEV)
    for sl in _chunks(coords.shape[1], n0 * n1):
        e = [_phasors(coords[a, sl], n, sign) for a, n in enumerate((n0, n1, n2))]
        zy = (e[0][:, :, None] * e[1][:, None, :]).reshape(-1, n0 * n1)
        for i in range(y.shape[0]):
            out[i] += zy.T @ (e[2] * y[i, sl, None])
    return out.reshape((-1,) + tuple(shape))


def _transfer(coords, shape):
    """FFT of the point-spread function on the doubled grid: complex128 [2 n0, 2 n1, 2 n2]."""
    grid = tuple(2 * n for n in shape)
    one = torch.ones((1, coords.shape[1]), dtype=torch.complex128, device=DEV)
    psf = _type1(coords, one, grid)[0] / float(np.prod(grid))
    return torch.fft.fftn(torch.fft.ifftshift(psf))


def _sense(x, maps, t):
    """sum_c conj(S_c) crop(ifft(T fft(pad(S_c x)))) in complex128."""
    n0, n1, n2 = x.shape
    out = torch.zeros_like(x)
    for s in maps:
        s = s.to(torch.complex128)
        out += s.conj() * torch.fft.ifftn(torch.fft.fftn(s * x, s=t.shape) * t)[:n0, :n1, :n2]
    return out


def _dot(a, b):
    return float(torch.sum(a.conj() * b).real)


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "toeplitz":
        t = _transfer(torch.from_numpy(_sparse_koosh(c, seed, 0)).to(DEV), _shape(c))
        x = _cplx(_shape(c), _gen(seed)).to(torch.complex128)
        return _sense(x, torch.ones((1, 1, 1, 1), device=DEV), t)
    if k in ("normal", "cg"):
        x, maps, coords = _operator_inputs(c, seed)
        out = torch.empty(x.shape, dtype=torch.complex128, device=DEV)
        for f, traj in enumerate(coords):
            t = _transfer(traj, _shape(c))
            if k == "cg":
                t *= 8.0 * float(np.prod(_shape(c))) / traj.shape[1]
            for i in range(f * c["encodings"], (f + 1) * c["encodings"]):
                v = x[i].to(torch.complex128)
                if k == "normal":
                    out[i] = _sense(v, maps, t) + c["lam"] * v
                    continue
                sol, r, p = torch.zeros_like(v), v.clone(), v.clone()
                rz = _dot(r, r)
                for _ in range(c["iters"]):
                    ap = _sense(p, maps, t) + c["lam"] * p
                    alpha = rz / _dot(p, ap)
                    sol += alpha * p
                    r -= alpha * ap
                    new = _dot(r, r)
                    p = r + (new / rz) * p
                    rz = new
                out[i] = sol
        return out
    if k in ("adjoint", "forward", "gradient"):
        g, coords, maps = _kspace_inputs(c, seed)
        s = maps.to(torch.complex128)
        if k == "adjoint":
            y = _cplx((c["coils"], coords.shape[1]), g).to(torch.complex128)
            return (s.conj() * _type1(coords, y, _shape(c))).sum(0)
        if k == "forward":
            return _type2(coords, s * _cplx(_shape(c), g).to(torch.complex128))
        x = _cplx((1, 1) + _shape(c), g)[0, 0].to(torch.complex128)
        y = _cplx((1, c["coils"], coords.shape[1]), g)[0].to(torch.complex128)
        d = (_type2(coords, s * x) - y) * _density(coords).double()
        return (s.conj() * _type1(coords, d, _shape(c))).sum(0)[None, None]
    if k == "slices":
        f = _cplx([c["transforms"], c["n1"], c["n2"]], _gen(seed)).to(torch.complex128)
        xy = torch.from_numpy(_radial2(c, seed)).to(DEV)
        coords = torch.cat([torch.zeros_like(xy[:1]), xy])
        y = _type2(coords, f[:, None])
        return y, _type1(coords, y, (1, c["n1"], c["n2"]))[:, 0]
    if k == "diagonal":
        return None  # the packed order of the diagonal is the library's own
    x, u = _lowrank_inputs(c, seed)
    z = x.add_(u)
    del u
    out = z.to(torch.complex128)
    b = (c["b0"], c["b1"], c["b2"])
    d0, d1 = c["d0"], c["d1"]
    # the grid of whole blocks; one that ends on the last index of an axis is left as it is
    m = [sum(1 for i in range(n // e) if i * e + e < n) for n, e in zip(_shape(c), b)]
    part = out[:, :, :m[0] * b[0], :m[1] * b[1], :m[2] * b[2]]
    if part.numel() == 0:
        return out
    for i0 in range(m[0]):
        row = part[:, :, i0 * b[0]:(i0 + 1) * b[0]].reshape(d0, d1, b[0], m[1], b[1], m[2], b[2])
        mat = row.permute(3, 5, 1, 2, 4, 6, 0).reshape(m[1] * m[2], -1, d0)
        lam, v = torch.linalg.eigh(mat.mH @ mat)
        sv = lam.clamp(min=0).sqrt()
        if c["soft"]:
            wt = torch.where(sv > _threshold(c), (sv - _threshold(c)) / sv.clamp(min=1e-300), 0.0)
        else:
            wt = torch.zeros_like(sv)
            wt[:, max(0, d0 - _threshold(c)):] = 1.0  # eigenvalues ascend
        mat = mat @ ((v * wt[:, None, :].to(v.dtype)) @ v.mH)
        row = mat.reshape(m[1], m[2], d1, b[0], b[1], b[2], d0).permute(6, 2, 3, 0, 4, 1, 5)
        part[:, :, i0 * b[0]:(i0 + 1) * b[0]] = row.reshape(d0, d1, b[0], m[1] * b[1], m[2] * b[2])
    return out
