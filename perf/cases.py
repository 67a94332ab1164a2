"""The workloads this framework is timed on: what a user has it do, through its Python API.

  calculate  one multislice call on host arrays (the drop-in's autoslic::calculate)
  tilt       a tilt series: orientations x thermal configurations x defoci, images on the device
  batch      many specimens of different sizes in one call (one CUDA graph)
  adjoint    images, misfit and its gradient for stacks of slice potentials on the device
  utr        the CTF-corrected 3D reconstruction from one image per orientation

`listed` gives the cases, `draw` more of the same ranges; `prepare` makes the inputs from a
seed, `run` is one pass, `work` its unavoidable bytes and operations, `exact` the same
results in 64 bits from torch and numpy alone.
"""
import math

import numpy as np
import torch

import utr_public_gb300 as msk

DEV = "cuda"
LIGHT = ((6, 0.50), (7, 0.17), (8, 0.30), (16, 0.03))  # C, N, O, S: the specimens' composition


# ------------------------------------------------------------------ the cases

def _calculate(name, nx, ny, atoms, fov, kev, dz):
    return {"name": name, "kind": "calculate", "nx": nx, "ny": ny, "atoms": atoms, "fov": fov,
            "kev": kev, "dz": dz}


def _tilt(name, nx, ny, atoms, fov, edge, kev, dz, angles, configs=1, thermal="none", defoci=2):
    return {"name": name, "kind": "tilt", "nx": nx, "ny": ny, "atoms": atoms, "fov": fov,
            "edge": edge, "kev": kev, "dz": dz, "angles": angles, "configs": configs,
            "thermal": thermal, "defoci": defoci}


def listed():
    return [
        # the smallest calls of the drop-in: MsctKirkland's per-orientation threads on a small
        # specimen, host arrays in and the host exit wave out -- latency and launches count
        _calculate("calculate_128", 128, 128, 300, 64.0, 200.0, 2.0),
        _calculate("calculate_256", 256, 256, 2000, 64.0, 200.0, 2.0),
        # one call at the tilt series' full size (an exit wave for one orientation)
        _calculate("calculate_1024", 1024, 1024, 20000, 160.0, 300.0, 1.0),
        # Debye-Waller thermal damping on a small grid, an odd number of orientations
        _tilt("tilt_dw_256", 256, 256, 2000, 64.0, 50.0, 200.0, 1.0, 45, thermal="dw"),
        # frozen phonons: every orientation averaged over displaced configurations
        _tilt("phonon_512", 512, 512, 2000, 64.0, 50.0, 200.0, 1.0, 5, configs=16,
              thermal="phonon", defoci=1),
        # a part of the headline tilt series on a grid that is not square
        _tilt("tilt_rect_512x1024", 512, 1024, 9001, 120.0, 90.0, 300.0, 1.0, 23),
        # the headline tilt series: a part of it, and all 180 orientations (the largest call)
        _tilt("tilt_1024_part", 1024, 1024, 20000, 160.0, 120.0, 300.0, 1.0, 16),
        _tilt("tilt_1024_full", 1024, 1024, 20000, 160.0, 120.0, 300.0, 1.0, 180),
        # a dense specimen (0.1 atoms/A^3, as in solid matter) on the finest common grid
        _tilt("tilt_dense_2048", 2048, 2048, 30011, 94.6, 66.9, 300.0, 1.0, 7),
        # specimens of uneven size, grid and orientation count in one graph
        {"name": "batch_uneven", "kind": "batch", "grids": "256,512,1024,256,512,1024,512",
         "atoms": "5016,12345,30007,8000,20011,6007,50021", "angles": "31,9,5,12,17,3,2",
         "kev": 300.0, "dz": 1.0},
        # the inversion's step: misfit and gradient, a checkpoint every 8 slices
        {"name": "adjoint_512", "kind": "adjoint", "nx": 512, "ny": 512, "slices": 64,
         "units": 16, "checkpoint": 8, "fov": 64.0, "kev": 200.0, "dz": 1.0},
        # the reconstruction of a tilt series' images into a volume
        {"name": "utr_512", "kind": "utr", "nx": 512, "ny": 512, "nz": 512, "images": 120,
         "xst": 0.3125},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fit(count, pixel_steps_each, most=2.0e10):
    """`count`, or as many as keep the call below the largest listed one."""
    return max(1, min(count, int(most / pixel_steps_each)))


def draw(rng):
    kind = rng.choice(["calculate", "calculate", "tilt", "tilt", "tilt", "batch", "adjoint", "utr"])
    if kind == "calculate":
        nx = 2 ** rng.randint(5, 10)
        ny = min(1024, max(32, nx * rng.choice([1, 1, 1, 2]) // rng.choice([1, 1, 2])))
        fov = round(rng.uniform(30.0, 160.0), 1)
        return {k: v for k, v in _calculate("", nx, ny, _log(rng, 60, 20000), fov,
                                            rng.choice([200.0, 300.0]),
                                            rng.choice([1.0, 1.5, 2.0])).items() if k != "name"}
    if kind == "tilt":
        nx = 2 ** rng.randint(6, 11)
        ny = min(2048, max(64, nx * rng.choice([1, 1, 1, 2]) // rng.choice([1, 1, 2])))
        fov = round(rng.uniform(40.0, 160.0), 1)
        edge = round(fov * rng.uniform(0.60, 0.75), 1)
        atoms = min(_log(rng, 500, 40000), int(0.1 * edge ** 3))
        thermal = rng.choice(["none", "none", "none", "dw", "phonon"])
        configs = rng.randint(2, 16) if thermal == "phonon" else 1
        # dense specimens cost more a pixel in the splat
        each = nx * ny * fov * configs * (1.0 + 8.0 * atoms / (0.1 * edge ** 3))
        c = _tilt("", nx, ny, atoms, fov, edge, rng.choice([200.0, 300.0]), 1.0,
                  _fit(_log(rng, 1, 180), each), configs, thermal, rng.randint(1, 3))
        return {k: v for k, v in c.items() if k != "name"}
    if kind == "batch":
        n = rng.randint(3, 9)
        grids = [2 ** rng.randint(7, 10) for _ in range(n)]
        atoms = [_log(rng, 2000, 50000) for _ in range(n)]
        angles = []
        for g, a in zip(grids, atoms):
            depth = math.sqrt(2.0) * (a / 0.1) ** (1.0 / 3.0)
            angles.append(_fit(_log(rng, 1, 60), 4.0 * g * g * depth, 2.0e10 / n))
        return {"kind": "batch", "grids": ",".join(map(str, grids)),
                "atoms": ",".join(map(str, atoms)), "angles": ",".join(map(str, angles)),
                "kev": 300.0, "dz": 1.0}
    if kind == "adjoint":
        nx = 2 ** rng.randint(6, 10)
        ny = min(1024, max(64, nx * rng.choice([1, 1, 2]) // rng.choice([1, 1, 2])))
        s = rng.randint(9, 90)
        units = _fit(_log(rng, 1, 64), 4.0 * nx * ny * s, 3.0e9)
        return {"kind": "adjoint", "nx": nx, "ny": ny, "slices": s, "units": units,
                "checkpoint": rng.choice([0, 5, 8]), "fov": round(rng.uniform(40.0, 100.0), 1),
                "kev": rng.choice([200.0, 300.0]), "dz": 1.0}
    nx = 2 ** rng.randint(6, 9)
    return {"kind": "utr", "nx": nx, "ny": nx, "nz": nx // rng.choice([1, 1, 2]),
            "images": rng.randint(31, 180), "xst": round(rng.uniform(0.2, 0.6), 3)}


# ------------------------------------------------------------------ inputs

_ctx = None


def _context():
    """The one context a program keeps."""
    global _ctx
    if _ctx is None:
        _ctx = msk.Context(0)
    return _ctx


def _atoms(count, fov, edge, seed):
    """Atoms uniform in a cube centred in the box."""
    rng = np.random.default_rng(seed)
    zs = np.array([z for z, _ in LIGHT], np.int32)
    ps = np.array([p for _, p in LIGHT])
    lo = 0.5 * (fov - edge)
    xyz = rng.uniform(lo, lo + edge, size=(3, count)).astype(np.float32)
    return (rng.choice(zs, size=count, p=ps / ps.sum()).astype(np.int32), xyz[0].copy(),
            xyz[1].copy(), xyz[2].copy(), np.ones(count, np.float32))


def _angles(count):
    """Rotations about y' in equal steps over half a turn."""
    return np.zeros(count), np.deg2rad(180.0 * np.arange(count) / count)


def _ints(text):
    return [int(t) for t in text.split(",")]


def _batch_geometry(case):
    """Per specimen: atoms, cube edge (0.1 atoms/A^3), field of view, grid, orientations."""
    out = []
    for n, a, k in zip(_ints(case["grids"]), _ints(case["atoms"]), _ints(case["angles"])):
        edge = (a / 0.1) ** (1.0 / 3.0)
        out.append((a, edge, float(np.float32(math.sqrt(2.0) * edge)), n, k))
    return out


_DEFOCI = (0.0, 500.0, 250.0)
_WOBBLE, _KELVIN = 0.08, 300.0


def _displacements(case, seed):
    rng = np.random.default_rng([seed, 7])
    return rng.normal(0.0, _WOBBLE, size=(case["configs"], 3, case["atoms"])).astype(np.float32)


def _stack_inputs(case, seed):
    """Slice potentials of scattered atoms (zero beyond 3 A of one) and shot-noisy images
    of a specimen 10% off them: what a step of the inversion has in hand."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    u, s, nx, ny, fov = (case[k] for k in ("units", "slices", "nx", "ny", "fov"))
    dx = (torch.fft.fftfreq(nx, device=DEV) * fov)[:, None]
    dy = (torch.fft.fftfreq(ny, device=DEV) * fov)[None, :]
    r2 = dx * dx + dy * dy
    peak = torch.where(r2 < 9.0, 250.0 * torch.exp(-r2 / 0.08) + 50.0 * torch.exp(-r2 / 0.7), 0.0)
    kernel = torch.fft.rfft2(peak)
    near = torch.fft.rfft2((r2 < 9.0).float())
    v = torch.empty((u, s, nx, ny), device=DEV)
    inner = ((dx.abs() < 0.4 * fov) & (dy.abs() < 0.4 * fov)).float()
    chance = 0.01 * fov * fov / (nx * ny)  # atoms per pixel of a 1 A slice
    for i in range(u):
        at = (torch.rand((s, nx, ny), generator=g, device=DEV) < chance).float() * inner
        f = torch.fft.rfft2(at)
        vi = torch.fft.irfft2(f * kernel, s=(nx, ny))
        v[i] = torch.where(torch.fft.irfft2(f * near, s=(nx, ny)) > 0.5, vi.clamp(min=0.0), 0.0)
    target = torch.empty((u, 1, nx, ny), device=DEV)
    for i in range(u):
        off = 1.0 + 0.1 * torch.randn((s, 1, 1), generator=g, device=DEV)
        image = _stack_images(case, v[i] * off, torch.complex64)
        target[i, 0] = image * (1.0 + 0.1 * torch.randn((nx, ny), generator=g, device=DEV))
    return v, target


def _utr_params(case):
    u = msk.Utr()
    u.modality, u.f1, u.f2 = 0, 1.0, 0.0
    u.nx, u.ny, u.xst = case["nx"], case["ny"], case["xst"]
    u.zlo, u.zhi = -0.5 * case["nz"] * case["xst"], 0.5 * case["nz"] * case["xst"]
    u.wl, u.aobj, u.ctf_mode, u.escc = 0.01968749, 40.0, 4, 1
    u.asigma, u.nsr, u.epsilon = 0.05, 0.03, 1e-4
    return u


def _utr_images(case, seed):
    """Flat-field corrected images: contrast about 1 at a few pixels' scale, and noise."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    n, ny, nx = case["images"], case["ny"], case["nx"]
    k2 = (torch.fft.fftfreq(ny, device=DEV)[:, None] ** 2 +
          torch.fft.rfftfreq(nx, device=DEV)[None, :] ** 2)
    smooth = torch.fft.irfft2(torch.fft.rfft2(torch.randn((n, ny, nx), generator=g, device=DEV)) *
                              torch.exp(-k2 * 300.0), s=(ny, nx))
    return 1.0 + 1.5 * smooth + 0.01 * torch.randn((n, ny, nx), generator=g, device=DEV)


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    if kind == "calculate":
        param = msk.make_param(case["fov"], case["fov"], case["nx"], case["ny"], case["kev"],
                               case["dz"])
        return {"kind": kind, "ctx": ctx, "param": param, "fov": case["fov"],
                "atoms": _atoms(case["atoms"], case["fov"], 0.78 * case["fov"], seed),
                "out": np.empty((case["nx"], case["ny"], 2), np.float32)}
    if kind == "tilt":
        s = msk.Series()
        s.nx, s.ny = case["nx"], case["ny"]
        s.ctblength = s.ctblengthz = case["fov"]
        s.v0, s.deltaz = case["kev"], case["dz"]
        state = {"kind": kind, "ctx": ctx, "series": s,
                 "atoms": _atoms(case["atoms"], case["fov"], case["edge"], seed),
                 "angles": _angles(case["angles"]), "defoci": np.array(_DEFOCI[:case["defoci"]]),
                 "configs": case["configs"], "displacements": None,
                 "images": torch.empty((case["angles"], case["defoci"], case["nx"], case["ny"]),
                                       device=DEV)}
        if case["thermal"] == "dw":
            state["wobble"] = np.full(case["atoms"], _WOBBLE, np.float32)
            s.lwobble, s.temperature, s.wobble = 1, _KELVIN, state["wobble"].ctypes.data
        if case["thermal"] == "phonon":
            state["displacements"] = _displacements(case, seed)
        return state
    if kind == "batch":
        s = msk.Series()
        s.v0, s.deltaz = case["kev"], case["dz"]
        specimens, images = [], []
        for i, (a, edge, fov, n, k) in enumerate(_batch_geometry(case)):
            spec = msk.specimen.Specimen(*_atoms(a, fov, edge, [seed, i]), np.zeros(a, np.float32),
                                         fov)
            specimens.append((spec, n, *_angles(k)))
            images.append(torch.empty((k, 2, n, n), device=DEV))
        return {"kind": kind, "ctx": ctx, "series": s, "specimens": specimens, "images": images,
                "defoci": np.array(_DEFOCI[:2])}
    if kind == "adjoint":
        v, target = _stack_inputs(case, seed)
        st = msk.Stack()
        st.nx, st.ny, st.ax, st.by = case["nx"], case["ny"], case["fov"], case["fov"]
        st.v0, st.deltaz = case["kev"], case["dz"]
        st.nslices, st.checkpoint = case["slices"], case["checkpoint"]
        return {"kind": kind, "ctx": ctx, "stack": st, "v": v, "target": target,
                "defoci": np.array([_stack_defocus(case)]), "grad": torch.empty_like(v)}
    ang = np.stack(_angles(case["images"]), axis=1) * (180.0 / np.pi)
    return {"kind": kind, "ctx": ctx, "utr": _utr_params(case), "angles": ang,
            "defocus": np.full(case["images"], 500.0), "images": _utr_images(case, seed),
            "volume": torch.empty((case["nz"], case["ny"], case["nx"]), device=DEV)}


def run(state):
    kind, ctx = state["kind"], state["ctx"]
    if kind == "calculate":
        return ctx.calculate(state["param"], *state["atoms"], state["fov"], state["fov"],
                             out=state["out"])
    if kind == "tilt":
        images, kept = ctx.tilt_series(state["series"], *state["atoms"], *state["angles"],
                                       state["defoci"], nconfig=state["configs"],
                                       displacements=state["displacements"],
                                       images=state["images"])
        return {"images": images, "kept": kept}
    if kind == "batch":
        images, kept = ctx.tilt_series_batch(state["series"], state["specimens"], state["defoci"],
                                             images=state["images"])
        return {"images": images, "kept": kept}
    if kind == "adjoint":
        loss, grad = ctx.adjoint(state["stack"], state["v"], state["defoci"], state["target"],
                                 grad=state["grad"])
        return {"loss": loss, "grad": grad}
    return ctx.utr_reconstruct(state["utr"], state["angles"], state["defocus"], state["images"],
                               volume=state["volume"])


# ------------------------------------------------------------------ bytes and operations

def _fft_flops(*n):
    total = math.prod(n)
    return 5.0 * total * math.log2(total)


def _multislice_flops(nx, ny, slices, units, atoms, fov):
    """Per slice: the transmission's 2D transform, its band limit back, the wave's two; per
    atom its pixels within 3 A at about 12 operations."""
    pixels = math.pi * 9.0 * nx * ny / (fov * fov)
    return units * (slices * 4.0 * _fft_flops(nx, ny) + atoms * 12.0 * pixels)


def work(case):
    kind = case["kind"]
    if kind == "calculate":
        n = case["nx"] * case["ny"]
        return {"bytes": 20.0 * case["atoms"] + 16.0 * n,
                "flops": _multislice_flops(case["nx"], case["ny"],
                                           math.ceil(case["fov"] / case["dz"]), 1, case["atoms"],
                                           case["fov"])}
    if kind == "tilt":
        n, units = case["nx"] * case["ny"], case["angles"] * case["configs"]
        disp = 12.0 * case["atoms"] * case["configs"] if case["thermal"] == "phonon" else 0.0
        flops = _multislice_flops(case["nx"], case["ny"], math.ceil(case["fov"] / case["dz"]),
                                  units, case["atoms"], case["fov"])
        flops += units * case["defoci"] * _fft_flops(case["nx"], case["ny"])
        return {"bytes": 20.0 * case["atoms"] + disp + 4.0 * n * case["angles"] * case["defoci"],
                "flops": flops}
    if kind == "batch":
        b = f = 0.0
        for a, _, fov, n, k in _batch_geometry(case):
            b += 20.0 * a + 8.0 * n * n * k
            f += _multislice_flops(n, n, math.ceil(fov / case["dz"]), k, a, fov)
            f += 2.0 * k * _fft_flops(n, n)
        return {"bytes": b, "flops": f}
    if kind == "adjoint":
        n, u, s = case["nx"] * case["ny"], case["units"], case["slices"]
        return {"bytes": u * n * (8.0 * s + 4.0),
                "flops": u * (9.0 * s + 3.0) * _fft_flops(case["nx"], case["ny"])}
    n, vol = case["nx"] * case["ny"], case["nx"] * case["ny"] * case["nz"]
    return {"bytes": 4.0 * (case["images"] * n + vol),
            "flops": case["images"] * (_fft_flops(case["nx"], case["ny"]) + 60.0 * n) +
            _fft_flops(case["nx"], case["ny"], case["nz"]) + 40.0 * vol}


# ------------------------------------------------------------------ the same in 64 bits

_PI = math.pi
# Kirkland's scattering-factor parameters: three Lorentzians (a, b), three Gaussians (c, d)
_FE = {
    6: (0.212080767, 0.208605417, 0.199811865, 0.208610186, 0.168254385, 5.57870773,
        0.14204836, 1.33311887, 0.363830672, 3.80800263, 0.000835012044, 0.040398262),
    7: (0.533015554, 0.290952515, 0.0529008883, 10.3547896, 0.0924159648, 10.3540028,
        0.261799101, 2.76252723, 0.000880262108, 0.0347681236, 0.110166555, 0.993421736),
    8: (0.339969204, 0.38157028, 0.307570172, 0.381571436, 0.130369072, 19.1919745,
        0.0883326058, 0.760635525, 0.1965867, 2.07401094, 0.000996220028, 0.0303266869),
    16: (1.01646916, 1.69181965, 0.441766748, 0.174180288, 0.121503863, 167.011091,
        0.82796667, 2.3034281, 0.0233022533, 0.15695415, 1.18302846, 5.85782891),
}
_I0S = (1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.0360768, 0.0045813)
_K0S = (-0.57721566, 0.42278420, 0.23069756, 0.03488590, 0.00262698, 0.00010750, 0.00000740)
_K0L = (1.25331414, -0.07832358, 0.02189568, -0.01062446, 0.00587872, -0.00251540, 0.00053208)


def _poly(c, x):
    s = np.zeros_like(x)
    for a in reversed(c):
        s = s * x + a
    return s


def _k0(x):
    """Abramowitz and Stegun 9.8.5 and 9.8.6, which Kirkland's potential is defined with."""
    small = np.minimum(x, 2.0)
    lo = -np.log(small / 2.0) * _poly(_I0S, (small / 3.75) ** 2) + _poly(_K0S, (small / 2.0) ** 2)
    hi = np.exp(-x) * _poly(_K0L, 2.0 / x) / np.sqrt(x)
    return np.where(x <= 2.0, lo, hi)


def _projected(z, r):
    p = _FE[z]
    x = 2.0 * 3.141592654 * r
    lorentz = sum(p[i] * _k0(x * math.sqrt(p[i + 1])) for i in (0, 2, 4))
    gauss = sum(p[i] * np.exp(-(3.141592654 * r) ** 2 / p[i + 1]) / p[i + 1] for i in (6, 8, 10))
    return 300.8242834 * lorentz + 150.4121417 * gauss


def _spline(z):
    """100 knots of r^2 and the cubic pieces of the Akima spline through the potential there."""
    r = 0.01 * np.exp(np.arange(100) * (math.log(500.0) / 99))
    x = r * r
    y = _projected(z, np.sqrt(x))
    m = np.diff(y) / np.diff(x)
    m = np.concatenate([[3 * m[0] - 2 * m[1], 2 * m[0] - m[1]], m, [2 * m[-1] - m[-2],
                                                                     3 * m[-1] - 2 * m[-2]]])
    w = np.abs(np.diff(m))
    left, right = w[2:], w[:-2]  # |m4 - m3| and |m2 - m1| about each knot
    total = left + right
    slope = np.where(total > 1e-25, (left * m[1:-2] + right * m[2:-1]) /
                     np.where(total > 1e-25, total, 1.0), 0.5 * (m[1:-2] + m[2:-1]))
    h, s = np.diff(x), m[2:-2]
    b, nb = slope[:-1], slope[1:]
    return x, np.stack([y[:-1], b, (3 * s - 2 * b - nb) / h, (b + nb - 2 * s) / (h * h)], axis=1)


def _wavelength(kev):
    return 12.3984244 / math.sqrt(kev * (2 * 510.99906 + kev))


def _sigma(kev):
    m = 510.99906
    return 2.0 * _PI * (m + kev) / (2.0 * m + kev) / (_wavelength(kev) * kev) / 1000.0


def _freq(n, a):
    i = np.arange(n)
    k = (np.where(i > n // 2, i - n, i).astype(np.float32) / np.float32(a)).astype(np.float32)
    return k, (k * k).astype(np.float32)


def _grid(nx, ny, a, kev, dz):
    """Band limit and propagator of a grid; the float frequencies decide what is in band."""
    (kx, kx2), (ky, ky2) = _freq(nx, a), _freq(ny, a)
    f = np.float32
    edge = min(f(nx) / (f(2.0) * f(a)), f(ny) / (f(2.0) * f(a)))
    k2max = f(f(2.0) / f(3.0) * edge) ** 2
    keep = (kx2[:, None] + ky2[None, :]).astype(f) < f(k2max)
    lam, scale = f(_wavelength(kev)), f(f(_PI) * f(dz))
    t = (scale * (kx2 * lam)).astype(np.float64)[:, None] + (scale * (ky2 * lam)).astype(np.float64)
    k2 = kx.astype(np.float64)[:, None] ** 2 + ky.astype(np.float64)[None, :] ** 2
    return (torch.from_numpy(keep).to(DEV), torch.from_numpy(np.where(keep, np.exp(-1j * t), 0)).to(DEV),
            torch.from_numpy(k2).to(DEV), float(lam))


def _slice_bounds(dz, depth):
    out, z, dz = [], float(np.float32(dz)), float(np.float32(dz))
    while z < float(np.float32(depth)) + dz:
        out.append(z)
        z += dz
    return np.array(out)


class _Splat:
    """Slice potentials of several units' atoms."""

    def __init__(self, units, nx, ny, fov, dz, depth):
        self.nx, self.ny, self.nu = nx, ny, len(units)
        self.bounds = _slice_bounds(dz, depth)
        zs = sorted(_FE)
        tabs = [_spline(z) for z in zs]
        self.knots = torch.from_numpy(tabs[0][0]).to(DEV)
        self.coef = torch.from_numpy(np.stack([t[1] for t in tabs])).to(DEV).reshape(-1, 4)
        self.sx, self.sy = (float(np.float32(fov) / np.float32(n)) for n in (nx, ny))
        self.rmin2 = 0.0625 * 0.5 * ((fov / nx) ** 2 + (fov / ny) ** 2)
        self.wx, self.wy = (int(n * 3.0 / fov) + 1 for n in (nx, ny))
        u = np.concatenate([np.full(len(a[0]), i) for i, a in enumerate(units)])
        num, x, y, z, occ = (np.concatenate([a[j] for a in units]) for j in range(5))
        at = np.searchsorted(self.bounds, z.astype(np.float64), side="right")
        order = np.argsort(at, kind="stable")
        self.first = np.searchsorted(at[order], np.arange(len(self.bounds) + 1))
        x, y, occ = (torch.from_numpy(q[order].astype(np.float64)).to(DEV) for q in (x, y, occ))
        self.u = torch.from_numpy(u[order]).to(DEV)
        self.elem = torch.from_numpy(np.searchsorted(zs, num[order])).to(DEV)
        self.x, self.y, self.occ = x, y, occ

    def potential(self, k):
        """The projected potentials [units, nx, ny] of slice k, or None where it has no atom."""
        a0, a1 = int(self.first[k]), int(self.first[k + 1])
        if a0 == a1:
            return None
        nx, ny = self.nx, self.ny
        v = torch.zeros(self.nu * nx * ny, dtype=torch.float64, device=DEV)
        ox = torch.arange(-self.wx, self.wx + 1, device=DEV)
        oy = torch.arange(-self.wy, self.wy + 1, device=DEV)
        step = max(1, (1 << 25) // (len(ox) * len(oy)))
        for b in range(a0, a1, step):
            c = slice(b, min(a1, b + step))
            x, y = self.x[c, None], self.y[c, None]
            ix, iy = (x / self.sx).long() + ox, (y / self.sy).long() + oy
            r2 = ((x - ix * self.sx) ** 2)[:, :, None] + ((y - iy * self.sy) ** 2)[:, None, :]
            inside = r2 <= 9.0
            r2 = r2.clamp(min=self.rmin2)
            i = (torch.searchsorted(self.knots, r2, right=True) - 1).clamp(0, 98)
            q = self.coef[i + 99 * self.elem[c, None, None]]
            d = r2 - self.knots[i]
            p = q[..., 0] + (q[..., 1] + (q[..., 2] + q[..., 3] * d) * d) * d
            p = torch.where(inside, p * self.occ[c, None, None], 0.0)
            to = (self.u[c, None, None] * nx + (ix % nx)[:, :, None]) * ny + (iy % ny)[:, None, :]
            v.index_add_(0, to.reshape(-1), p.reshape(-1))
        return v.reshape(self.nu, nx, ny)


def _exit_waves(units, nx, ny, fov, kev, dz, damping=None):
    """psi [units, nx, ny] behind the box, from a plane wave."""
    keep, prop, k2, _ = _grid(nx, ny, fov, kev, dz)
    s = _Splat(units, nx, ny, fov, dz, fov)
    psi = torch.ones((len(units), nx, ny), dtype=torch.complex128, device=DEV)
    for k in range(len(s.bounds)):
        v = s.potential(k)
        if v is not None:
            if damping is not None:
                v = torch.fft.ifft2(torch.fft.fft2(v) * torch.exp(damping * k2)).real
            t = torch.fft.fft2(torch.exp(1j * _sigma(kev) * v))
            psi = psi * torch.fft.ifft2(t * keep)
        psi = torch.fft.ifft2(torch.fft.fft2(psi) * prop)
    return psi


def _free_space(psi, k2, lam, distance):
    return torch.fft.ifft2(torch.fft.fft2(psi) * torch.exp(-1j * _PI * lam * distance * k2))


def _rotated(atoms, fov, depth, angle, shift=None):
    """Atoms about the y' axis through the centre in 32 bits, as the positions are defined,
    displaced, without those that leave the box."""
    num, x, y, z, occ = atoms
    f = np.float32
    c, s, m = f(math.cos(angle)), f(math.sin(angle)), f(fov / 2.0)
    x, z = (m + (x - m) * c) + (z - m) * s, (m + (-x + m) * s) + (z - m) * c
    if shift is not None:
        x, y, z = x + shift[0], y + shift[1], z + shift[2]
    fov, depth = f(fov), f(depth)
    ok = (x >= 0) & (x <= fov) & (y >= 0) & (y <= fov) & (z >= 0) & (z <= depth)
    return tuple(q[ok] for q in (num, x, y, z, occ))


def _series(atoms, nx, ny, fov, kev, dz, angles, defoci, shifts=(None,), damping=None):
    """Images [angles, defoci, nx, ny], averaged over the configurations."""
    _, _, k2, lam = _grid(nx, ny, fov, kev, dz)
    out = torch.zeros((len(angles), len(defoci), nx, ny), dtype=torch.float64, device=DEV)
    todo = [(i, s) for i in range(len(angles)) for s in shifts]
    some = max(1, (1 << 24) // (nx * ny))
    for b in range(0, len(todo), some):
        part = todo[b:b + some]
        psi = _exit_waves([_rotated(atoms, fov, fov, angles[i], s) for i, s in part], nx, ny, fov,
                          kev, dz, damping)
        for d, z in enumerate(defoci):
            image = _free_space(psi, k2, lam, z - 0.5 * fov).abs() ** 2
            for q, (i, _) in enumerate(part):
                out[i, d] += image[q] / len(shifts)
    return out


def _stack_defocus(case):
    return -0.5 * case["slices"] * case["dz"]


def _stack_images(case, v, dtype):
    """|psi|^2 in the detector plane of one stack of slice potentials."""
    keep, prop, k2, lam = _grid(case["nx"], case["ny"], case["fov"], case["kev"], case["dz"])
    prop = prop.to(dtype)
    psi = torch.ones_like(v[0]).to(dtype)
    for k in range(v.shape[0]):
        t = torch.fft.fft2(torch.exp(1j * _sigma(case["kev"]) * v[k]))
        psi = psi * torch.fft.ifft2(t * keep)
        psi = torch.fft.ifft2(torch.fft.fft2(psi) * prop)
    step = torch.exp(-1j * _PI * lam * _stack_defocus(case) * k2).to(dtype)
    psi = torch.fft.ifft2(torch.fft.fft2(psi) * step)
    return psi.real ** 2 + psi.imag ** 2


def _exact_utr(case, seed):
    p, images = _utr_params(case), _utr_images(case, seed).double()
    n, nx, ny, nz, xst = case["images"], case["nx"], case["ny"], case["nz"], case["xst"]
    f = np.float32
    v = torch.where(images > 0, images.clamp(min=1e-300).log(), 0.0)
    k2 = torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(v, dim=(1, 2))), dim=(1, 2))
    # gridding: every pixel onto its Ewald sphere, its coordinates and weights in 32 bits as the
    # method defines them, the sums in 64
    acc = torch.zeros((nz * ny * nx, 2), dtype=torch.float64, device=DEV)
    wsum = torch.zeros(nz * ny * nx, dtype=torch.float64, device=DEV)
    st = [1.0 / (xst * m) for m in (nx, ny, nz)]
    lo = [f(-s * (m // 2)) for s, m in zip(st, (nx, ny, nz))]
    st = [f(s) for s in st]
    at = [(l + s * np.arange(m).astype(f)).astype(np.float64) for l, s, m in zip(lo, st, (nx, ny))]
    dev = lambda q: torch.from_numpy(np.ascontiguousarray(q.astype(f))).to(DEV)  # noqa: E731
    ewald = dev(-0.5 * p.wl * at[0] ** 2)[None, :] + dev(-0.5 * p.wl * at[1] ** 2)[:, None]
    lost, ys = [float(l) for l in lo], dev(at[1])
    for a, angle in enumerate(np.deg2rad(np.rad2deg(_angles(n)[1]))):
        s, c = f(math.sin(angle)), f(math.cos(angle))
        x = dev(at[0] * float(c))[None, :] - ewald * float(s)
        z = dev(at[0] * float(s))[None, :] + ewald * float(c)
        y = (ys[:, None] - 0.0 * x)
        q = [(w - l) / float(t) for w, l, t in zip((x, y, z), lost, st)]
        i = [w.floor() for w in q]
        ok = ((i[0] >= 0) & (i[0] <= nx - 2) & (i[1] >= 0) & (i[1] <= ny - 2) & (i[2] >= 0) &
              (i[2] <= nz - 2))
        frac = [w - j for w, j in zip(q, i)]
        i = [j.long() for j in i]
        value = torch.view_as_real(k2[a])[ok]
        for ez in (0, 1):
            for ey in (0, 1):
                for ex in (0, 1):
                    part = [(w if e else 1.0 - w) for w, e in zip(frac, (ex, ey, ez))]
                    w = ((part[0] * part[1]) * part[2])[ok].double()
                    to = (((i[2] + ez) * ny + i[1] + ey) * nx + i[0] + ex)[ok]
                    wsum.index_add_(0, to, w)
                    acc.index_add_(0, to, value * w[:, None])
    # sampling normalisation with the signal-to-noise filter
    noise = p.nsr * math.sqrt(nx * ny)
    safe = wsum.clamp(min=1e-300)
    snr = acc.norm(dim=1) / (noise * safe.sqrt())
    scale = (0.5 + torch.atan(100.0 * (snr - 1.414213562373)) / _PI) / safe
    scale = torch.where(wsum > 0, scale, 0.0)
    vol = torch.view_as_complex(acc * scale[:, None]).reshape(nz, ny, nx)
    del acc, wsum, snr, scale, safe
    # the contrast transfer function's 3D correction inside the aperture
    sq = [torch.from_numpy(((np.arange(m) - m // 2) / (xst * m)) ** 2).to(DEV) for m in (nx, ny, nz)]
    r2 = sq[2][:, None, None] + sq[1][None, :, None] + sq[0][None, None, :]
    phase = _PI * p.wl * 500.0 * r2 - math.atan(p.asigma)
    s, c = torch.sin(phase), torch.cos(phase)
    fix = torch.complex(s / (s * s + p.epsilon), -c / (c * c + p.epsilon))
    vol = torch.where(r2 < (p.aobj * float(f(0.001)) / p.wl) ** 2, vol * fix, vol)
    del phase, s, c, fix, r2
    # the half spectrum's transform to real values: on the Nyquist plane the earlier of a pair of
    # points counts 3/4, the later 5/4
    k, j = torch.arange(nz, device=DEV)[:, None], torch.arange(ny, device=DEV)[None, :]
    mk, mj = (nz - k) % nz, (ny - j) % ny
    own = (mk == k) & (mj == j)
    half = torch.where(own, 1.0, torch.where((k < mk) | ((k == mk) & (j < mj)), 0.75, 1.25))
    vol[:, :, 0] *= half
    out = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(vol))).real
    del vol
    # the cylinder about y, its cupping compensation and the potential's scale
    rx, rz = (torch.arange(nx, device=DEV) - nx // 2) ** 2, (torch.arange(nz, device=DEV) - nz // 2) ** 2
    r2 = (rz[:, None, None] + rx[None, None, :]).double()
    mc2 = 9.1093837015e-31 * 299792458.0 ** 2
    chl2 = (299792458.0 * 6.62607004e-34) ** 2 / (p.wl ** 2 * 1e-20)
    volts = float((np.sqrt(np.longdouble(mc2) ** 2 + np.longdouble(chl2)) - np.longdouble(mc2)) /
                  np.longdouble(1.602176634e-19))
    norm = volts * p.wl / (2.0 * _PI * math.sqrt(1.0 + p.asigma ** 2) * xst)
    cup = 2.0 / ((nx // 2) ** 2 + (ny // 2) ** 2 + (nz // 2) ** 2)
    return torch.where(r2 > min(nx // 2, nz // 2) ** 2, 0.0, out * torch.exp(cup * r2) * norm)


def exact(case, seed):
    kind = case["kind"]
    if kind == "calculate":
        atoms = _atoms(case["atoms"], case["fov"], 0.78 * case["fov"], seed)
        psi = _exit_waves([atoms], case["nx"], case["ny"], case["fov"], case["kev"], case["dz"])
        return torch.view_as_real(psi[0])
    if kind == "tilt":
        if case["nx"] * case["ny"] * case["fov"] * case["angles"] * case["configs"] > 6.0e9:
            return None  # minutes in 64 bits
        atoms = _atoms(case["atoms"], case["fov"], case["edge"], seed)
        shifts, damping = (None,), None
        if case["thermal"] == "dw":
            damping = -0.25 * 2.0 * (2.0 * _PI) ** 2 * float(np.float32(_WOBBLE)) ** 2 * _KELVIN / 300.0
        if case["thermal"] == "phonon":
            shifts = tuple(_displacements(case, seed))
        return {"images": _series(atoms, case["nx"], case["ny"], case["fov"], case["kev"], case["dz"],
                                  _angles(case["angles"])[1], _DEFOCI[:case["defoci"]], shifts,
                                  damping), "kept": None}
    if kind == "batch":
        images = [_series(_atoms(a, fov, edge, [seed, i]), n, n, fov, case["kev"], case["dz"],
                          _angles(k)[1], _DEFOCI[:2])
                  for i, (a, edge, fov, n, k) in enumerate(_batch_geometry(case))]
        return {"images": images, "kept": None}
    if kind == "adjoint":
        v, target = _stack_inputs(case, seed)
        loss, grad = 0.0, torch.empty(v.shape, dtype=torch.float64, device=DEV)
        for i in range(v.shape[0]):
            w = v[i].double().requires_grad_()
            part = ((_stack_images(case, w, torch.complex128) - target[i, 0].double()) ** 2).sum()
            grad[i], = torch.autograd.grad(part, w)
            loss += float(part.detach())
        return {"loss": loss, "grad": grad}
    return _exact_utr(case, seed)
