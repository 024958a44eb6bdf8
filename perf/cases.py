"""Timed cases of the integral-equation path: what a program that uses this package has it do.

Kinds (each one pass through the public entry points):
  apply      one IE operator apply on device vectors, complex128 or complex64 (IEOperator.apply_device);
             nv = 2 applies two complex64 vectors of one operator together (apply_device_batch), as both
             polarisations of a plane wave do
  host       the reference-facing apply on host arrays (giem2g_apply_ie_operator), which a host program's own
             Krylov solver calls once per matrix-vector product
  solve      SolveEquation on host arrays, FP64
  batch      both polarisations of one or several frequencies as one lockstep batch; on device vectors as the
             frequency sweep runs it, or on host arrays as the input-file driver runs it
  setup      a frequency's set-up as the driver does it: the Green's tensor of the layered background, its
             spectrum, the conductivity, and the first apply of the new operator
  receivers  a frequency's receiver part: the receiver tensor, its spectrum, the conductivity, and the fields of
             one solution at the receivers

Grids are those of the package's configurations (32x32x8, 64x64x16, 128x128x32, 256x256x48) and ragged ones: the
lateral counts are powers of two (the operator's own limit) and need not be equal, the number of cells in z is
any.  The operators keep the default tile shapes, as the driver's do.  Operators of the apply and host kinds
take a tensor given by the caller (set_ie_kernel_spatial): the whole-space dyadic Green's function, whose
applies have a plain 64-bit statement (exact()); the other kinds, and the largest grid, compute the tensor of a
layered background.
"""
import math

import numpy as np
import torch

import giem2g_b200 as g2
from giem2g_b200.sources import plane_wave_integral
from giem2g_b200.synthetic import IEModel, THREE_LAYER_SIGMA, THREE_LAYER_THICK

MU0 = 4e-7 * math.pi

g2.set_logger(lambda line: None)  # the solver logs one line per outer iteration; a batch job drops them


def _apply(name, Nx, Ny, Nz, precision, nv=1, tensor="wholespace"):
    return {"name": name, "kind": "apply", "Nx": Nx, "Ny": Ny, "Nz": Nz, "precision": precision, "nv": nv,
            "tensor": tensor}


def listed():
    return [
        # the smallest grid in use: launches and call overhead count
        _apply("apply_c128_32x32x8", 32, 32, 8, 0),
        # the benchmark grid, the outer solver's apply
        _apply("apply_c128_128x128x32", 128, 128, 32, 0),
        # a ragged grid: unequal sides, 27 layers
        _apply("apply_c128_64x128x27", 64, 128, 27, 0),
        # the inner solver's apply: two right-hand sides per tensor read, complex64
        _apply("pair_c64_128x128x32", 128, 128, 32, 1, 2),
        _apply("pair_c64_128x64x41", 128, 64, 41, 1, 2),
        # the largest grid in use
        _apply("pair_c64_256x256x48", 256, 256, 48, 1, 2, "layered"),
        # one matrix-vector product of a host program's solver
        {"name": "host_c128_64x64x16", "kind": "host", "Nx": 64, "Ny": 64, "Nz": 16, "tensor": "wholespace"},
        # a small FP64 solve to the default tolerance: a chain of small kernels
        {"name": "solve_c128_32x32x8", "kind": "solve", "Nx": 32, "Ny": 32, "Nz": 8, "freq": 1.0, "tol": 1e-8},
        # the benchmark: both polarisations, mixed precision, device vectors
        {"name": "batch_mixed_128x128x32", "kind": "batch", "Nx": 128, "Ny": 128, "Nz": 32, "nf": 1, "freq": 0.1,
         "precision": 1, "tol": 1e-6, "host": False},
        # the driver's work on a ragged grid: two frequencies, both polarisations, host arrays
        {"name": "batch_mixed_64x64x20_2f", "kind": "batch", "Nx": 64, "Ny": 64, "Nz": 20, "nf": 2, "freq": 0.3,
         "precision": 1, "tol": 1e-6, "host": True},
        # what the driver does before each frequency's solves, and after them
        {"name": "setup_64x64x16", "kind": "setup", "Nx": 64, "Ny": 64, "Nz": 16, "freq": 0.1},
        {"name": "receivers_64x64x16", "kind": "receivers", "Nx": 64, "Ny": 64, "Nz": 16, "freq": 0.1, "Nr": 2},
    ]


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "apply", "host", "solve", "batch", "setup", "receivers"])
    limit = {"apply": 1 << 19, "host": 1 << 17, "solve": 1 << 14, "batch": 1 << 17, "setup": 1 << 16,
             "receivers": 1 << 16}[kind]
    while True:
        Nx, Ny = 2 ** rng.randint(4, 7), 2 ** rng.randint(4, 7)
        Nz = int(round(math.exp(rng.uniform(math.log(4), math.log(48)))))
        if 1 << 11 <= Nx * Ny * Nz <= limit:
            break
    case = {"kind": kind, "Nx": Nx, "Ny": Ny, "Nz": Nz}
    freq = round(10 ** rng.uniform(-2, 1), 4)
    if kind == "apply":
        precision = rng.randint(0, 1)
        case |= {"precision": precision, "nv": 1 + precision * rng.randint(0, 1), "tensor": "wholespace"}
    elif kind == "host":
        case |= {"tensor": "wholespace"}
    elif kind == "solve":
        case |= {"freq": freq, "tol": 1e-8}
    elif kind == "batch":
        case |= {"nf": 1 if Nx * Ny * Nz > 1 << 15 else rng.randint(1, 2), "freq": freq,
                 "precision": rng.randint(0, 1) if Nx * Ny * Nz <= 1 << 15 else 1, "tol": 1e-6,
                 "host": rng.random() < 0.5}
    elif kind == "setup":
        case |= {"freq": freq}
    else:
        case |= {"freq": freq, "Nr": rng.randint(1, 3)}
    return case


# ---- inputs ------------------------------------------------------------------------------------------------
def _spacing(case):
    """Cell sizes in metres: the same depth and width of the anomaly at every grid of its class."""
    return (50.0, 50.0, 25.0) if case["Nx"] * case["Ny"] > 64 * 64 else (100.0, 100.0, 50.0)


def _generator(seed, salt):
    return torch.Generator("cuda").manual_seed(1000003 * int(seed) + salt)


def _vector(case, seed, salt, dtype=torch.complex128):
    shape = (3, case["Nz"], case["Ny"], case["Nx"])
    return torch.randn(shape, dtype=torch.complex128, device="cuda", generator=_generator(seed, salt)).to(dtype)


def _sigma(case, seed):
    """Lognormal conductivity, correlated over four cells, mean log10 -2, deviation 0.7; [Nz, Ny, Nx]."""
    Nx, Ny, Nz = case["Nx"], case["Ny"], case["Nz"]
    f = torch.randn((Nz, Ny, Nx), dtype=torch.float64, device="cuda", generator=_generator(seed, 11))
    k = [torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) for n in (Nz, Ny, Nx)]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    f = torch.fft.ifftn(torch.fft.fftn(f) * torch.exp(-(2 * math.pi) ** 2 * k2 * 4.0)).real
    return 10.0 ** (-2.0 + 0.7 * (f - f.mean()) / f.std())


def _wholespace_tables(case):
    """The dyadic Green's function of a 0.01 S/m whole space between cells: {component: [Nx, Ny, Nz]} over the
    non-negative lags in x, y and z (xy odd in x and y, xz odd in x and z, yz odd in y and z)."""
    dx, dy, dz = _spacing(case)
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") * d
          for n, d in ((case["Nx"], dx), (case["Ny"], dy), (case["Nz"], dz))]
    x, y, z = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    r = torch.sqrt(x * x + y * y + z * z + (0.4 * min(dx, dy, dz)) ** 2)
    sb, iwm = 0.01, 1j * 2 * math.pi * 0.1 * MU0
    k = (iwm * sb) ** 0.5
    f = torch.exp(1j * k * r) / (4 * math.pi * r)
    d1 = f * (1j * k - 1 / r)
    d2 = f * ((1j * k - 1 / r) ** 2 + 1 / r ** 2)
    a, b = d1 / r, (d2 - d1 / r) / r ** 2
    vol = dx * dy * dz * dz
    return {"xx": (iwm * f + (a + b * x * x) / sb) * vol, "yy": (iwm * f + (a + b * y * y) / sb) * vol,
            "zz": (iwm * f + (a + b * z * z) / sb) * vol, "xy": b * x * y / sb * vol, "xz": b * x * z / sb * vol,
            "yz": b * y * z / sb * vol}


def _whole_space_operator(case, seed):
    Nx, Ny, Nz = case["Nx"], case["Ny"], case["Nz"]
    dx, dy, dz = _spacing(case)
    t = _wholespace_tables(case)
    col = [(i, j) for j in range(Nz) for i in range(j + 1)]  # packed upper: i + j (j + 1) / 2
    lag = torch.tensor([j - i for i, j in col], device="cuda")
    symm = torch.stack([t[c][:, :, lag] for c in ("xx", "xy", "yy", "zz")], dim=2).cpu().numpy()
    rc = torch.arange(Nz, device="cuda")
    step = (rc[None, :] - rc[:, None]).reshape(-1)  # row - column of a column-major block
    asym = torch.stack([t[c][:, :, step.abs()] * torch.sign(step) for c in ("xz", "yz")], dim=2).cpu().numpy()
    op = g2.IEOperator(Nx, Ny, Nz, dx, dy, np.arange(Nz + 1) * dz)
    op.set_background(np.array([1e-12, 0.01], complex), [], 2 * math.pi * 0.1)
    op.set_ie_kernel_spatial(symm, asym)
    op.calc_fft_of_ie_kernel()
    op.set_anomaly_conductivity(_sigma(case, seed).to(torch.complex128).cpu().numpy())
    return op


def _model(case, seed, freq):
    dx, dy, dz = _spacing(case)
    scale = 1.0 + 0.02 * (int(seed) % 17)  # another seed, another background
    return IEModel(case["Nx"], case["Ny"], case["Nz"], dx, dy, np.arange(case["Nz"] + 1) * dz,
                   THREE_LAYER_SIGMA * scale, THREE_LAYER_THICK.copy(), freq)


def _file_order(sigma):
    return np.ascontiguousarray(sigma.permute(1, 2, 0).cpu().numpy())  # [Ny, Nx, Nz], as the input files have it


def _layered_operator(case, seed, freq, sigma):
    m = _model(case, seed, freq)
    op = g2.IEOperator.from_model(m)
    op.calc_ie_kernel(m.csigma, m.thick, m.omega)
    op.calc_fft_of_ie_kernel()
    op.set_anomaly_sigma(sigma, freq)
    return m, op


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("apply", "host"):
        if case["tensor"] == "layered":
            _, s["op"] = _layered_operator(case, seed, 0.1, _file_order(_sigma(case, seed)))
        else:
            s["op"] = _whole_space_operator(case, seed)
    if kind == "apply":
        dt = torch.complex64 if case["precision"] else torch.complex128
        s["x"] = [_vector(case, seed, 21 + i, dt) for i in range(case["nv"])]
        s["y"] = [torch.empty_like(x) for x in s["x"]]
    elif kind == "host":
        s["x"] = _vector(case, seed, 21).cpu().numpy()
    elif kind == "solve":
        m, s["op"] = _layered_operator(case, seed, case["freq"], _file_order(_sigma(case, seed)))
        s["rhs"] = plane_wave_integral(m, 1)
    elif kind == "batch":
        sigma = _file_order(_sigma(case, seed))
        ops, rhs = [], []
        for i in range(case["nf"]):
            m, op = _layered_operator(case, seed, case["freq"] * 4.0 ** i, sigma)
            ops += [op, op]
            rhs += [plane_wave_integral(m, 1), plane_wave_integral(m, 0)]
        s["batch"] = g2.Batch(ops, precision=case["precision"])
        if case["host"]:
            s["rhs"] = rhs
        else:
            s["rhs"] = [torch.from_numpy(e).cuda() for e in rhs]
            s["sol"] = [torch.empty_like(e) for e in s["rhs"]]
    elif kind == "setup":
        s["model"] = _model(case, seed, case["freq"])
        s["op"] = g2.IEOperator.from_model(s["model"])
        s["sigma"] = _file_order(_sigma(case, seed))
        s["x"] = _vector(case, seed, 21)
        s["y"] = torch.empty_like(s["x"])
    else:
        s["model"] = _model(case, seed, case["freq"])
        depths = [0.0, 10.0, 2.5 * _spacing(case)[2]][: case["Nr"]]
        s["rc"] = g2.RCOperator.from_model(s["model"], depths)
        s["sigma"] = _file_order(_sigma(case, seed))
        s["x"] = torch.from_numpy(plane_wave_integral(s["model"], 1)).cuda() + 0.1 * _vector(case, seed, 21)
        s["y"] = [torch.empty((case["Ny"], case["Nx"], 3, case["Nr"]), dtype=torch.complex128, device="cuda")
                  for _ in range(2)]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "apply":
        if case["nv"] == 2:
            g2.apply_device_batch(s["op"], [x.data_ptr() for x in s["x"]], [y.data_ptr() for y in s["y"]],
                                  case["precision"])
        else:
            s["op"].apply_device(s["x"][0].data_ptr(), s["y"][0].data_ptr(), case["precision"])
        return s["y"]
    if kind == "host":
        return s["op"].apply_precond(s["x"])
    if kind == "solve":
        E, info = s["op"].solve_equation(s["rhs"], tol=case["tol"])
        return {"E": E, "iterations": info.iterations, "stat": info.stat}
    if kind == "batch":
        if case["host"]:
            E, infos = s["batch"].solve(s["rhs"], tol=case["tol"])
        else:
            E = s["sol"]
            infos = s["batch"].solve_device([e.data_ptr() for e in s["rhs"]], [e.data_ptr() for e in E],
                                            tol=case["tol"])
        return {"E": E, "iterations": [i.iterations for i in infos], "stat": [i.stat for i in infos]}
    m = s["model"]
    if kind == "setup":
        op = s["op"]
        op.calc_ie_kernel(m.csigma, m.thick, m.omega)
        op.calc_fft_of_ie_kernel()
        op.set_anomaly_sigma(s["sigma"], m.freq)
        op.apply_device(s["x"].data_ptr(), s["y"].data_ptr(), 0)
        return s["y"]
    rc = s["rc"]
    rc.calc_rc_kernel(m.csigma, m.thick, m.omega)
    rc.calc_fft_of_rc_kernel()
    rc.set_anomaly_sigma(s["sigma"], m.freq)
    rc.recalculate_device(s["x"].data_ptr(), s["y"][0].data_ptr(), s["y"][1].data_ptr())
    return s["y"]


# ---- what a pass cannot do without ---------------------------------------------------------------------------
def _apply_work(Nx, Ny, Nz, size, nv):
    """Tensor and per-cell coefficients read once, vectors read and written once; the padded 2-D transforms
    both ways and the 3Nz x 3Nz products at the 4 Nx Ny spectral points."""
    units, cells = Nx * Ny, Nx * Ny * Nz
    tensor = units * (2 * Nz * (Nz + 1) + 2 * Nz * Nz)
    fft = 2 * 3 * Nz * 4 * units * 5 * math.log2(4 * units)
    return size * (tensor + cells + 2 * nv * 3 * cells), nv * (4 * units * 9 * Nz * Nz * 8 + fft)


def work(case):
    Nx, Ny, Nz, kind = case["Nx"], case["Ny"], case["Nz"], case["kind"]
    units, cells = Nx * Ny, Nx * Ny * Nz
    if kind in ("apply", "host"):
        size = 8 if case.get("precision") else 16
        b, f = _apply_work(Nx, Ny, Nz, size, case.get("nv", 1))
    elif kind in ("solve", "batch"):
        # nested FGMRES: about 6 outer iterations for the small FP64 solves and 12 for the others, each with 11
        # inner applies and one outer apply, and the vectors of each Arnoldi step read once
        outer, mixed = (6, 0) if kind == "solve" else (12, case["precision"])
        si = 8 if mixed else 16
        pols = 2 if kind == "batch" else 1
        bi, fi = _apply_work(Nx, Ny, Nz, si, pols)
        bo, fo = _apply_work(Nx, Ny, Nz, 16, pols)
        basis = pols * 3 * cells * (si * 66 + 16 * 7)
        nf = case.get("nf", 1)
        b, f = nf * outer * (11 * bi + bo + basis), nf * outer * (11 * fi + fo)
    elif kind == "setup":
        tensor = 2 * Nz * (Nz + 1) + 2 * Nz * Nz
        b, f = _apply_work(Nx, Ny, Nz, 16, 1)
        b += units * tensor * (16 + 16 + 8)                        # spatial tensor, its spectra in both types
        f += 501 * 4 * units * (3 * Nz * (Nz + 1) + 2 * Nz * Nz)   # the sums over 501 wave numbers
        f += 5 * tensor * 4 * units * math.log2(4 * units) / 2     # the tensor's transform
    else:
        Nr = case["Nr"]
        tensor = 4 * units * 15 * Nr * Nz
        b = 16 * (2 * tensor + 3 * cells + 6 * units * Nr)
        f = 501 * 4 * 4 * units * 20 * Nr * Nz + 5 * tensor * math.log2(4 * units) + 4 * units * 8 * 17 * Nr * Nz
    return {"bytes": float(b), "flops": float(f)}


# ---- the same results in 64 bits, without this package's kernels ----------------------------------------------
def exact(case, seed):
    """The contracting-IE apply y = s (a x - (G * (g x)) / dz) with the whole-space tensor, as a 3-D linear
    convolution; None for the kinds that compute the layered background's tensor (its restatement in plain
    numpy takes minutes)."""
    if case["kind"] not in ("apply", "host") or case["tensor"] != "wholespace":
        return None
    Nx, Ny, Nz = case["Nx"], case["Ny"], case["Nz"]
    dz, sb = _spacing(case)[2], 0.01
    t = _wholespace_tables(case)
    n = (2 * Nz, 2 * Ny, 2 * Nx)

    def spectrum(c):
        k = torch.zeros(n, dtype=torch.complex128, device="cuda")
        v = t[c].permute(2, 1, 0)
        for mz in (1, -1):
            for my in (1, -1):
                for mx in (1, -1):
                    sign = 1.0
                    for axis, m in (("x", mx), ("y", my), ("z", mz)):
                        sign *= m if c in ("xy", "xz", "yz") and axis in c else 1
                    src = v[0 if mz > 0 else 1:, 0 if my > 0 else 1:, 0 if mx > 0 else 1:]
                    iz, iy, ix = ([i * m % size for i in range(0 if m > 0 else 1, cells)] for m, size, cells in
                                  ((mz, n[0], Nz), (my, n[1], Ny), (mx, n[2], Nx)))
                    k[torch.tensor(iz)[:, None, None], torch.tensor(iy)[None, :, None], torch.tensor(ix)] = sign * src
        return torch.fft.fftn(k)

    sa = _sigma(case, seed).to(torch.complex128)
    a = 2 * sb ** 0.5 / (sa + sb)
    g = (sa - sb) * a
    names = (("xx", "xy", "xz"), ("xy", "yy", "yz"), ("xz", "yz", "zz"))
    out = []
    dt = torch.complex64 if case.get("precision") else torch.complex128
    for i in range(case.get("nv", 1)):
        x = _vector(case, seed, 21 + i, dt).to(torch.complex128)
        u = [torch.fft.fftn(g * x[c], s=n) for c in range(3)]
        w = [sum(spectrum(names[c][d]) * u[d] for d in range(3)) for c in range(3)]
        w = torch.stack([torch.fft.ifftn(v)[:Nz, :Ny, :Nx] for v in w])
        out.append(sb ** 0.5 * (a * x - w / dz))
    return out if case["kind"] == "apply" else out[0].cpu().numpy()
