"""Performance cases of the simulation path: what a reconstruction program has this library do.

Every case goes through the public Python front-end (compas_b200), on device objects that such a program
keeps: the tissue parameters, the sequence, the trajectory, the coil maps and the measured or simulated
arrays. One pass is one call of the operation (one chain of calls for the "gradient" kind), its outputs are
the arrays it returns.

Kinds:
  fisp             FISP EPG simulation of the magnetization
  fisp_tangents    the same with the exact derivatives with respect to T1 and T2
  pssfp            pSSFP isochromat simulation
  signal           magnetization -> Cartesian or spiral k-space signal
  jacobian         J·v, Cartesian or spiral
  hermitian        Jᴴ·v, Cartesian or spiral
  gradient         tangents -> signal -> residual -> Jᴴ·r: the gradient of a parameter fit

Inputs are synthetic and follow the repository's workloads: tissue with T1 log-uniform in 0.1-4 s and T2 in
10-500 ms, off-resonance of 20 Hz, smooth flip-angle trains of 0-70 degrees, Gaussian slice profiles and
coil maps, complex normal echoes, directions and residuals.
"""
import math
import os
import sys

import numpy as np
import torch

# the package's front-end lives in a folder that is no Python identifier
sys.path.insert(0, os.path.join(os.getcwd(), "compas-toolkit_b200"))
import compas_b200 as cb  # noqa: E402

FOV = 22.4                                  # cm
FISP_TIMES = (8.7e-3, 4.35e-3, 25e-3)       # TR, TE, TI in s
PSSFP_TR, PSSFP_PULSE = 0.010, 0.001        # s
DT_CARTESIAN, DT_SPIRAL = 5e-6, 4e-6        # s between samples


def listed():
    return [
        # the reference's own small configuration: 64 x 64 voxels, one slice position, where launches and
        # the latency of the serial TR loop count
        {"name": "fisp_64", "kind": "fisp", "voxels": 4096, "trs": 400, "states": 8, "positions": 1, "complex_rf": False},
        # one MR-STAT slice, the headline workload
        {"name": "fisp_224", "kind": "fisp", "voxels": 50176, "trs": 1120, "states": 25, "positions": 35, "complex_rf": False},
        # RF-spoiled train (quadratic phases) on a masked brain: a ragged voxel count
        {"name": "fisp_rf_spoiled", "kind": "fisp", "voxels": 10007, "trs": 743, "states": 13, "positions": 9, "complex_rf": True},
        # derivatives for a fit of a 96 x 96 region with the MR-STAT sequence
        {"name": "tangents_96", "kind": "fisp_tangents", "voxels": 9216, "trs": 1120, "states": 25, "positions": 35, "complex_rf": False},
        # balanced sequence with a resolved slice-select pulse: one slice, and a small region
        {"name": "pssfp_224", "kind": "pssfp", "voxels": 50176, "trs": 320, "nz": 35, "rf_samples": 15},
        {"name": "pssfp_50", "kind": "pssfp", "voxels": 2500, "trs": 743, "nz": 35, "rf_samples": 15},
        # signal of the MR-STAT slice
        {"name": "signal_224", "kind": "signal", "trajectory": "cartesian", "voxels": 50176, "readouts": 1120, "samples": 224, "coils": 4},
        # the two Jacobian products of a Gauss-Newton step at MR-STAT scale
        {"name": "jacobian_224", "kind": "jacobian", "trajectory": "cartesian", "voxels": 50176, "readouts": 1120, "samples": 224, "coils": 8},
        {"name": "hermitian_224", "kind": "hermitian", "trajectory": "cartesian", "voxels": 50176, "readouts": 1120, "samples": 224, "coils": 8},
        # spiral readouts of a 128 x 128 slice, and the adjoint for a ragged region with few coils
        {"name": "spiral_signal_128", "kind": "signal", "trajectory": "spiral", "voxels": 16384, "readouts": 760, "samples": 1000, "coils": 8},
        {"name": "spiral_hermitian", "kind": "hermitian", "trajectory": "spiral", "voxels": 5003, "readouts": 401, "samples": 743, "coils": 3},
        # the gradient of a small fit, call by call
        {"name": "gradient_64", "kind": "gradient", "voxels": 4096, "trs": 400, "states": 8, "positions": 1, "samples": 64, "coils": 1},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fisp", "fisp", "fisp_tangents", "pssfp", "pssfp", "signal", "signal", "jacobian", "hermitian", "gradient"])
    while True:
        if kind in ("fisp", "fisp_tangents"):
            case = {"kind": kind, "voxels": log(1000, 64000), "trs": rng.randint(100, 1120), "states": rng.randint(2, 25),
                    "positions": rng.randint(1, 35), "complex_rf": rng.random() < 0.25}
            cost = case["voxels"] * case["trs"] * case["positions"] * max(8, case["states"])
            fits = cost <= 50176 * 1120 * 35 * 25 * (0.8 if kind == "fisp" else 0.12)
        elif kind == "pssfp":
            case = {"kind": kind, "voxels": log(1000, 100000), "trs": rng.randint(100, 1120), "nz": rng.randint(3, 35),
                    "rf_samples": rng.randint(5, 20)}
            fits = case["voxels"] * case["trs"] * case["nz"] * case["rf_samples"] <= 3 * 50176 * 320 * 35 * 15
        elif kind == "gradient":
            case = {"kind": kind, "voxels": log(500, 10000), "trs": rng.randint(100, 500), "states": rng.randint(5, 25),
                    "positions": rng.randint(1, 5), "samples": rng.randint(32, 128), "coils": rng.randint(1, 8)}
            fits = True
        else:
            spiral = rng.random() < 0.4
            case = {"kind": kind, "trajectory": "spiral" if spiral else "cartesian", "voxels": log(1000, 50176),
                    "readouts": rng.randint(50, 760) if spiral else rng.randint(100, 1120),
                    "samples": rng.randint(100, 1000) if spiral else rng.randint(32, 256), "coils": rng.randint(1, 16)}
            fits = case["voxels"] * case["readouts"] * case["samples"] * (8 + case["coils"]) <= 16 * 16384 * 760 * 1000 or not spiral
        if fits:
            return case


# ---------------------------------------------------------------------------------------------------
# inputs, on the host, from the seed alone
# ---------------------------------------------------------------------------------------------------

def _tissue(rng, nv):
    """float32 [9][nv]: T1, T2, B1, B0, rho_x, rho_y, x, y, z on the first nv points of a square grid."""
    t1 = np.exp(rng.uniform(np.log(0.1), np.log(4.0), nv))
    t2 = np.minimum(np.exp(rng.uniform(np.log(0.01), np.log(0.5), nv)), 0.8 * t1)
    mag, ph = rng.uniform(0.5, 1.0, nv), rng.uniform(0.0, 2 * np.pi, nv)
    side = math.ceil(math.sqrt(nv))
    lin = np.linspace(-FOV / 2, FOV / 2, side)
    y, x = np.divmod(np.arange(nv), side)
    return np.stack([t1, t2, rng.uniform(0.8, 1.2, nv), rng.normal(0.0, 20.0, nv), mag * np.cos(ph), mag * np.sin(ph),
                     lin[x], lin[y], np.zeros(nv)]).astype(np.float32)


def _coils(rng, nc, p):
    """Gaussian sensitivity maps around the field of view, with a seeded start angle."""
    a = 2 * np.pi * (np.arange(nc) / nc + rng.uniform())
    x, y = p[6].astype(np.float64), p[7].astype(np.float64)
    d2 = (x - FOV / 3 * np.cos(a)[:, None]) ** 2 + (y - FOV / 3 * np.sin(a)[:, None]) ** 2
    return (np.exp(-d2 / (2 * (FOV / 3) ** 2)) * np.exp(1j * a)[:, None]).astype(np.complex64)


def _fisp_sequence(rng, case):
    """(rf [nTR], slice profiles [P][nTR]): a smooth 0-70 degree train, with quadratic phases when it is
    RF-spoiled (117 degree increments)."""
    n, p = case["trs"], case["positions"]
    knots = rng.uniform(0.0, 70.0, 15)
    at = np.linspace(0, 14, n)
    i = np.minimum(at.astype(int), 13)
    f = 0.5 - 0.5 * np.cos(np.pi * (at - i))
    rf = (knots[i] * (1 - f) + knots[i + 1] * f).astype(np.complex128)
    if case.get("complex_rf"):
        k = np.arange(n)
        rf = rf * np.exp(1j * np.deg2rad(117.0) * ((k * (k + 1) // 2) % 360))
    pos = np.arange(p)
    prof = np.exp(-((pos - (p - 1) / 2) ** 2) / (2 * (max(p, 2) / 4.4) ** 2))
    return rf.astype(np.complex64), np.repeat(prof[:, None], n, axis=1).astype(np.complex64)


def _pssfp_sequence(rng, case):
    """A phase-cycled smooth train around 40 degrees with a Gaussian pulse normalised to 1 degree."""
    n, nrf = case["trs"], case["rf_samples"]
    i = np.arange(1, nrf + 1)
    g = np.exp(-((i - nrf / 2) ** 2) / nrf)
    rf = 40.0 * (1 + 0.25 * np.sin(2 * np.pi * (np.arange(n) * rng.uniform(1, 4) / n + rng.uniform())))
    rf[1::2] *= -1
    return {"rf": rf.astype(np.complex64), "gdtrf": ((np.pi / 180) * g / g.sum()).astype(np.complex64),
            "dt": (PSSFP_PULSE / nrf, 10.0, (PSSFP_TR - PSSFP_PULSE) / 2), "gz": (0.002 / nrf, 0.0, -0.01),
            "z": np.linspace(-1, 1, case["nz"]).astype(np.float32)}


def _trajectory(rng, case):
    """(k_start [R], Δk): lines of a Cartesian raster, or interleaves of a spiral with a step each."""
    r, s = case["readouts"], case["samples"]
    dk = 2 * np.pi / FOV
    if case["trajectory"] == "cartesian":
        lines = min(r, s)
        k0 = -s / 2 * dk + 1j * ((np.arange(r) + int(rng.integers(lines))) % lines - lines // 2) * dk
        return k0.astype(np.complex64), float(np.float32(dk))
    ang = 2 * np.pi * (np.arange(r) / r + rng.uniform())
    tangent = np.exp(1j * (ang + np.pi / 2)) * 0.7 + np.exp(1j * ang) * 0.3
    return (0.5 * dk * rng.uniform(0.5, 1.5) * np.exp(1j * ang)).astype(np.complex64), (dk * tangent / np.abs(tangent)).astype(np.complex64)


def _normal(gen, shape, scale):
    """Complex normal values, made on the GPU: complex64 tensor."""
    return torch.randn(tuple(shape) + (2,), generator=gen, device="cuda", dtype=torch.float32).mul_(scale / math.sqrt(2))


def _inputs(case, seed):
    """Everything the case's library objects are made of, as numpy arrays, numbers and, for the large
    random arrays, CUDA tensors of complex values as float pairs."""
    rng = np.random.default_rng([seed, 77])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, nv = case["kind"], case["voxels"]
    d = {"tissue": _tissue(rng, nv)}
    if kind in ("fisp", "fisp_tangents", "gradient"):
        d["rf"], d["slices"] = _fisp_sequence(rng, case)
    if kind == "pssfp":
        d["pssfp"] = _pssfp_sequence(rng, case)
    if kind == "gradient":
        case = dict(case, trajectory="cartesian", readouts=case["trs"])
    if "trajectory" in case:
        d["k_start"], d["dk"] = _trajectory(rng, case)
        d["coils"] = _coils(rng, case["coils"], d["tissue"])
        r, s, c = case["readouts"], case["samples"], case["coils"]
        if kind != "gradient":
            d["echos"] = _normal(gen, (r, nv), 0.1)
        if kind in ("jacobian", "hermitian"):
            d["dT1"], d["dT2"] = _normal(gen, (r, nv), 0.05), _normal(gen, (r, nv), 0.5)
        if kind == "jacobian":
            d["v"] = _normal(gen, (4, nv), 1.0)
        if kind == "hermitian":
            d["v"] = _normal(gen, (c, r, s), 1.0)
        if kind == "gradient":
            d["data"] = _normal(gen, (c, r, s), 5.0)
    return d


# ---------------------------------------------------------------------------------------------------
# library objects and one pass
# ---------------------------------------------------------------------------------------------------

def _array(ctx, a):
    if isinstance(a, torch.Tensor):
        a = a.cpu().numpy().view(np.complex64)[..., 0]
    return cb.CompasArray.from_numpy(ctx, a)


def prepare(case, seed):
    d = _inputs(case, seed)
    ctx = cb.Context(0)
    kind = case["kind"]
    s = {"kind": kind, "ctx": ctx, "params": cb.TissueParameters.from_soa(ctx, d["tissue"])}
    if "rf" in d:
        tr, te, ti = FISP_TIMES
        s["seq"] = cb.FispSequence(ctx, d["rf"], d["slices"], tr, te, case["states"], ti)
    if "pssfp" in d:
        q = d["pssfp"]
        s["seq"] = cb.pSSFPSequence(ctx, q["rf"], PSSFP_TR, q["gdtrf"], q["dt"], q["gz"], q["z"])
    if "k_start" in d:
        r = case.get("readouts", case.get("trs"))
        if case.get("trajectory") == "spiral":
            s["traj"] = cb.SpiralTrajectory(ctx, r, case["samples"], DT_SPIRAL, d["k_start"], d["dk"])
        else:
            s["traj"] = cb.CartesianTrajectory(ctx, r, case["samples"], DT_CARTESIAN, d["k_start"], d["dk"])
    for k in ("coils", "echos", "dT1", "dT2", "v", "data"):
        if k in d:
            s[k] = _array(ctx, d[k])
    ctx.synchronize()
    return s


def _view(a):
    """A result as a torch tensor of float pairs, without a copy."""
    return torch.as_tensor(a, device="cuda")


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind in ("fisp", "pssfp"):
        return _view(cb.simulate_magnetization(ctx, s["params"], s["seq"]))
    if kind == "fisp_tangents":
        return {k: _view(a) for k, a in cb.simulate_magnetization_tangents(ctx, s["params"], s["seq"]).items()}
    if kind == "signal":
        return _view(cb.magnetization_to_signal(ctx, s["echos"], s["params"], s["traj"], s["coils"]))
    if kind in ("jacobian", "hermitian"):
        product = cb.compute_jacobian if kind == "jacobian" else cb.compute_jacobian_hermitian
        return _view(product(ctx, s["echos"], {"T1": s["dT1"], "T2": s["dT2"]}, s["params"], s["traj"], s["coils"], s["v"]))
    m = cb.simulate_magnetization_tangents(ctx, s["params"], s["seq"])
    signal = cb.magnetization_to_signal(ctx, m["echos"], s["params"], s["traj"], s["coils"])
    objective, residual = cb.compute_residual(ctx, signal, s["data"])
    gradient = cb.compute_jacobian_hermitian(ctx, m["echos"], m, s["params"], s["traj"], s["coils"], residual)
    return {"signal": _view(signal), "objective": objective, "residual": _view(residual), "gradient": _view(gradient)}


# ---------------------------------------------------------------------------------------------------
# work and tolerances
# ---------------------------------------------------------------------------------------------------

def work(case):
    """Bytes: inputs once, outputs once. FLOPs: FISP 86 per state, position, voxel and TR (the 3 x 3 complex
    excitation and the relaxation), pSSFP the rotation of every RF sample, the products one complex
    multiply-add (8 flops) per voxel, coil, readout and sample, two in a Jacobian product."""
    kind, nv = case["kind"], case["voxels"]
    if kind in ("fisp", "fisp_tangents", "gradient"):
        echo = 8.0 * nv * case["trs"]
        sim = 86.0 * case["states"] * case["positions"] * nv * case["trs"]
        if kind == "fisp":
            return {"bytes": 36.0 * nv + echo, "flops": sim}
        if kind == "fisp_tangents":
            return {"bytes": 36.0 * nv + 3 * echo, "flops": 3 * sim}
        out = 8.0 * case["coils"] * case["trs"] * case["samples"]
        mac = 8.0 * nv * case["coils"] * case["trs"] * case["samples"]
        return {"bytes": (68.0 + 8 * case["coils"]) * nv + 3 * out, "flops": 3 * sim + 3 * mac}
    if kind == "pssfp":
        return {"bytes": 36.0 * nv + 8.0 * nv * case["trs"], "flops": case["nz"] * (54.0 * case["rf_samples"] + 24) * nv * case["trs"]}
    echo = 8.0 * nv * case["readouts"]
    space = 8.0 * case["coils"] * case["readouts"] * case["samples"]
    if kind == "signal":
        return {"bytes": echo + (36.0 + 8 * case["coils"]) * nv + space, "flops": space * nv}
    return {"bytes": 3 * echo + (68.0 + 8 * case["coils"]) * nv + space, "flops": 2 * space * nv}


def tolerance(case):
    """About four times the error measured against exact(): FP32 recurrences over up to 1120 TRs come out at
    7e-6 (EPG) and 3e-5 (pSSFP, whose pulse is a product of rotations per TR); the products, with operands split
    into two BF16 values and FP32 accumulation over the voxels, at 3e-5, the Hermitian ones, which sum over
    the samples, at 4e-6, and at 2e-5 behind a simulation, a signal and a residual."""
    kind = case["kind"]
    if kind in ("fisp", "fisp_tangents"):
        return {"rel": 3e-5}
    if kind == "hermitian":
        return {"rel": 2e-5}
    return {"rel": 8e-5 if kind == "gradient" else 1.2e-4}


# ---------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------

def _f64(a):
    return torch.as_tensor(np.asarray(a, np.float32).astype(np.float64), device="cuda")


def _c128(a):
    if isinstance(a, torch.Tensor):
        return torch.view_as_complex(a.double())
    return torch.as_tensor(np.asarray(a, np.complex64).astype(np.complex128), device="cuda")


def _pairs(a):
    return torch.view_as_real(a.contiguous())


def _f32(x):
    """A number as the library gets it: rounded to 32 bits."""
    return float(np.float32(x))


def _exact_fisp(case, d, tangents):
    """Extended phase graph in its textbook form, one position at a time: [nTR][nv] complex128, and the
    derivatives with respect to T1 and T2 by forward-mode differentiation of every step."""
    t1, t2, b1, b0 = _f64(d["tissue"][:4])
    tr, te, ti = (_f32(x) for x in FISP_TIMES)
    n, states, nv = case["trs"], case["states"], case["voxels"]
    rf = torch.as_tensor(d["rf"].astype(np.complex128))
    slices = torch.as_tensor(d["slices"].astype(np.complex128))
    nq = 3 if tangents else 1
    out = [torch.zeros((n, nv), dtype=torch.complex128, device="cuda") for _ in range(nq)]

    def relax(dt):
        e1, e2 = torch.exp(-dt / t1), torch.exp(-dt / t2)
        c = e2 * torch.exp(2j * math.pi * dt * b0)
        return e1, c, e1 * dt / t1 ** 2, c * dt / t2 ** 2

    e1_tr, c_tr, de1_tr, dc_tr = relax(tr)
    _, c_te, _, dc_te = relax(te)
    e1_ti, _, de1_ti, _ = relax(ti)
    # all nq quantities (value, d/dT1, d/dT2) ride in the first axis
    for p in range(case["positions"]):
        u, m, z = (torch.zeros((nq, states, nv), dtype=torch.complex128, device="cuda") for _ in range(3))  # F+, F-, Z
        z[0, 0] = 1 - 2 * e1_ti  # inversion and recovery over TI
        if tangents:
            z[1, 0] = -2 * de1_ti
        for k in range(n):
            a = complex(rf[k] * slices[p, k])
            half, phi = math.pi / 360 * abs(a) * b1, (a / abs(a) if abs(a) > 0 else 1.0 + 0j)
            si, co = torch.sin(half), torch.cos(half)
            # F+' = co² F+ + φ² si² F- - i φ sin(α) Z, F-' with the conjugate coefficients,
            # Z' = -i/2 conj(φ) sin(α) F+ + i/2 φ sin(α) F- + cos(α) Z
            c2, b = torch.complex(co * co, torch.zeros_like(co)), (phi * phi) * (si * si)
            w = (-1j * phi) * (2 * si * co)
            ca = torch.complex(co * co - si * si, torch.zeros_like(co))
            u2 = torch.addcmul(torch.addcmul(c2 * u, b, m), w, z)
            m2 = torch.addcmul(torch.addcmul(c2 * m, b.conj().resolve_conj(), u), w.conj().resolve_conj(), z)
            z = torch.addcmul(torch.addcmul(ca * z, -0.5 * w.conj().resolve_conj(), u), -0.5 * w, m)
            u, m = u2, m2
            out[0][k] += c_te * u[0, 0]
            if tangents:
                out[1][k] += c_te * u[1, 0]
                out[2][k] += c_te * u[2, 0] + dc_te * u[0, 0]
            if k == n - 1:
                break
            if tangents:
                d2u, d2m, d1z = dc_tr * u[0], dc_tr.conj() * m[0], de1_tr * z[0]
                d1z[0] -= de1_tr
            u.mul_(c_tr)
            m.mul_(c_tr.conj().resolve_conj())
            z.mul_(e1_tr)
            z[0, 0] += 1 - e1_tr
            if tangents:
                u[2] += d2u
                m[2] += d2m
                z[1] += d1z
            # the spoiler: F- one state down, F+ one state up, F+ of state 0 the conjugate of F-'s
            m = torch.cat([m[:, 1:], torch.zeros_like(m[:, :1])], 1)
            u = torch.cat([m[:, :1].conj(), u[:, :-1]], 1)
    return out


def _exact_pssfp(case, d):
    q = d["pssfp"]
    t1, t2, b1, b0 = _f64(d["tissue"][:4])
    dt_ex, dt_inv, dt_pr = (_f32(x) for x in q["dt"])
    gz_ex, _, gz_pr = (_f32(x) for x in q["gz"])
    z = _f64(q["z"])[:, None]
    g = q["gdtrf"].astype(np.complex128)
    rf = q["rf"].astype(np.complex128)

    def relax(dt, m):
        e1, e2 = torch.exp(-dt / t1), torch.exp(-dt / t2)
        return m[0] * e2, m[1] * e2, m[2] * e1 + (1 - e1)

    def precess(gz, dt, m):
        th = -gz * z - dt * 2 * math.pi * b0
        s, c = torch.sin(th), torch.cos(th)
        return c * m[0] - s * m[1], c * m[1] + s * m[0], m[2]

    az = -gz_ex * z - dt_ex * 2 * math.pi * b0

    def pulse(flip, m):
        for w in g:
            a = complex(flip * w)
            ax, ay = a.real * b1, -a.imag * b1
            th2 = ax * ax + ay * ay + az * az
            th = torch.sqrt(th2)
            s = torch.where(th > 1e-9, torch.sin(th) / th.clamp_min(1e-30), torch.ones_like(th))
            c = torch.cos(th)
            h = torch.where(th > 1e-9, (2 * torch.sin(th / 2) ** 2) / th2.clamp_min(1e-60), torch.full_like(th, 0.5)) * (ax * m[0] + ay * m[1] + az * m[2])
            m = (c * m[0] + s * (ay * m[2] - az * m[1]) + h * ax, c * m[1] + s * (az * m[0] - ax * m[2]) + h * ay,
                 c * m[2] + s * (ax * m[1] - ay * m[0]) + h * az)
            m = relax(dt_ex, m)
        return m

    nv = case["voxels"]
    zero = torch.zeros((case["nz"], nv), dtype=torch.float64, device="cuda")
    m = relax(dt_inv, (zero, zero, torch.cos(math.pi * b1) + zero))
    m = pulse(-rf[0] / 2, m)
    m = relax(dt_pr, precess(2 * gz_pr, dt_pr, m))
    out = torch.zeros((case["trs"], nv), dtype=torch.complex128, device="cuda")
    for k in range(case["trs"]):
        m = relax(dt_pr, precess(gz_pr, dt_pr, pulse(rf[k], m)))
        out[k] = torch.complex(m[0].sum(0), m[1].sum(0))
        m = relax(dt_pr, precess(gz_pr, dt_pr, m))
    return out


class _Model:
    """The k-space model of a readout in 64 bits: F[v][k], the factor of a voxel's magnetization in sample k
    (relaxation, off-resonance and gradients about the echo)."""

    def __init__(self, case, d):
        self.case = case
        self.t1, self.t2, _, self.b0, rx, ry, self.x, self.y, _ = _f64(d["tissue"])
        self.rho = torch.complex(rx, ry)
        self.spiral = case.get("trajectory") == "spiral"
        self.s = case["samples"]
        self.k0 = d["k_start"].astype(np.complex128)
        self.dk = d["dk"]
        self.dt = _f32(DT_SPIRAL if self.spiral else DT_CARTESIAN)
        self.k = torch.arange(self.s, dtype=torch.float64, device="cuda") - 0.5 * self.s
        self.cached = None

    def factor(self, r):
        """F of readout r about the echo: exp((k - S/2)(-Δt/T2 + iΘ)), times what the spiral's start adds."""
        if not self.spiral and self.cached is not None:
            return self.cached
        step = complex(self.dk[r]) if self.spiral else complex(self.dk)
        theta = step.real * self.x + step.imag * self.y + self.dt * 2 * math.pi * self.b0
        if self.spiral:
            # the rewind has relaxation and off-resonance of S/2 samples; the prephaser is the readout's start
            rate = torch.complex(-self.dt / self.t2, theta)
            kk = self.k + 0.5 * self.s
            lead = torch.complex(0.5 * self.s * self.dt / self.t2, self.k0[r].real * self.x - 0.5 * self.s * self.dt * 2 * math.pi * self.b0)
            return torch.exp(rate[:, None] * kk + lead[:, None])
        self.cached = torch.exp(torch.complex(-self.dt / self.t2, theta)[:, None] * self.k)
        return self.cached

    @property
    def slope(self):
        """dF/dT2 = (k - S/2)·slope·F"""
        return self.dt / self.t2 ** 2


def _exact_products(case, d):
    m = _Model(case, d)
    coils = _c128(d["coils"])
    nr, ns, nc = case.get("readouts", case.get("trs")), case["samples"], case["coils"]
    kind = case["kind"]
    if kind == "signal":
        out = torch.empty((nc, nr, ns), dtype=torch.complex128, device="cuda")
        if m.spiral:
            for r in range(nr):
                out[:, r] = (coils * (_c128(d["echos"][r]) * m.rho)) @ m.factor(r)
        else:
            f = m.factor(0)
            for c in range(nc):
                w = coils[c] * m.rho
                for r in range(0, nr, 128):
                    out[c, r : r + 128] = (_c128(d["echos"][r : r + 128]) * w) @ f
        return out
    v = _c128(d["v"])
    step = 1 if m.spiral else 128
    if kind == "jacobian":
        out = torch.empty((nc, nr, ns), dtype=torch.complex128, device="cuda")
        for r in range(0, nr, step):
            e, d1, d2 = (_c128(d[k][r : r + step]) for k in ("echos", "dT1", "dT2"))
            f = m.factor(r)
            a = v[0] * m.t1 * m.rho * d1 + v[1] * m.t2 * m.rho * d2 + (v[2] + 1j * v[3]) * e
            b = v[1] * m.t2 * m.rho * m.slope * e
            for c in range(nc):
                out[c, r : r + step] = (a * coils[c]) @ f + m.k * ((b * coils[c]) @ f)
        return out
    out = torch.zeros((4, case["voxels"]), dtype=torch.complex128, device="cuda")
    for r in range(0, nr, step):
        e, d1, d2 = (_c128(d[k][r : r + step]) for k in ("echos", "dT1", "dT2"))
        f = m.factor(r).conj().T  # [S][V]
        y = yk = 0
        for c in range(nc):
            u = v[c, r : r + step]
            y = y + coils[c].conj() * (u @ f)
            yk = yk + coils[c].conj() * ((u * m.k) @ f)
        out[0] += (m.t1 * m.rho).conj() * (y * d1.conj()).sum(0)
        out[1] += (m.t2 * m.rho).conj() * (y * d2.conj() + m.slope * yk * e.conj()).sum(0)
        out[2] += (y * e.conj()).sum(0)
    out[3] = -1j * out[2]
    return out


def exact(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    if kind == "fisp":
        return _pairs(_exact_fisp(case, d, False)[0])
    if kind == "fisp_tangents":
        return dict(zip(("echos", "T1", "T2"), (_pairs(a) for a in _exact_fisp(case, d, True))))
    if kind == "pssfp":
        return _pairs(_exact_pssfp(case, d))
    if kind in ("signal", "jacobian", "hermitian"):
        return _pairs(_exact_products(case, d))
    e, d1, d2 = _exact_fisp(case, d, True)
    at = dict(case, readouts=case["trs"])
    as_pairs = {k: _pairs(a) for k, a in (("echos", e), ("dT1", d1), ("dT2", d2))}
    signal = _exact_products(dict(at, kind="signal"), {**d, **as_pairs})
    residual = signal - _c128(d["data"])
    gradient = _exact_products(dict(at, kind="hermitian"), {**d, **as_pairs, "v": _pairs(residual)})
    return {"signal": _pairs(signal), "objective": float((residual.abs() ** 2).sum()), "residual": _pairs(residual), "gradient": _pairs(gradient)}
