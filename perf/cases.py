"""Performance cases of the 3D FFT backend: what its users run, over the range
of sizes, precisions and options they run it at.

A case is a dict of plain values; its "kind" says which entry points a pass
goes through:

  r2c        Engine.r2c then Engine.c2r: the forward and backward real
             transform of a solver step (decomp_2d_fft_3d, r2c and c2r);
  overwrite  the same on an engine created with OVERWRITE, whose c2r consumes
             its spectrum;
  c2c        Engine.c2c forward then backward;
  r2r        Dtt.r2r forward then backward: the DCT / DST solves of wall-bounded
             axes (decomp_2d_dtt_3d_r2r);
  transpose  the x -> y -> z -> y -> x chain of transpose_* calls;
  batch      Batch.run of many uneven grids, forward and backward (the
             multiple-grids use).

"prec" is 8 (double, the library's usual build) or 4 (single), "fmt" 1
(PHYSICAL_IN_X) or 3 (PHYSICAL_IN_Z).
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "2decomp-fft_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gbfft  # noqa: E402

DEVICE = "cuda"
FORWARD, BACKWARD = -1, 1
BATCH_LENGTHS = (32, 48, 64, 96, 128, 192, 256)
SMOOTH = sorted({2 ** a * 3 ** b * 5 ** c * 7 ** d for a in range(11) for b in range(6) for c in range(4)
                 for d in range(3) if 16 <= 2 ** a * 3 ** b * 5 ** c * 7 ** d <= 1024})


def _case(name, kind, nx=0, ny=0, nz=0, fmt=1, prec=8, **more):
    return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, fmt=fmt, prec=prec, **more)


def listed():
    return [
        # a small box (a test run, or one of many subdomains): launches and latency
        _case("r2c_64x64x64_f64", "r2c", 64, 64, 64),
        # the production double grids of mixed factors a simulation picks
        _case("r2c_384x400x243_f64", "r2c", 384, 400, 243),
        # a large double box that streams from HBM, the other pencil format
        _case("r2c_512x512x512_f64_z", "r2c", 512, 512, 512, fmt=3),
        # the benchmark's large single-precision box
        _case("r2c_1024x1024x512_f32", "r2c", 1024, 1024, 512, prec=4),
        # a mixed-factor box in single precision, the other pencil format
        _case("r2c_360x270x210_f32_z", "r2c", 360, 270, 210, fmt=3, prec=4),
        # an odd, ragged box (odd sides, factors 11 and 13) in single precision
        _case("r2c_225x143x105_f32", "r2c", 225, 143, 105, prec=4),
        # a double box of sizes without any special treatment, memory-saving OVERWRITE
        _case("overwrite_320x180x126_f64", "overwrite", 320, 180, 126),
        # complex fields in single precision (spectral solvers, post-processing)
        _case("c2c_256x256x256_f32", "c2c", 256, 256, 256, prec=4),
        # complex fields in double precision, a box of uneven sides
        _case("c2c_128x160x96_f64_z", "c2c", 128, 160, 96, fmt=3),
        # a wall-bounded Poisson solve: DCT-II along every axis of a 2^k + 1 grid
        _case("r2r_257x129x193_f64", "r2r", 257, 129, 193, kx=2, ky=2, kz=2),
        # the transposes of a solver's derivative sweeps on a double complex field
        _case("transpose_256x256x256_c128", "transpose", 256, 256, 256, complex=True),
        # many uneven single-precision grids in one call
        _case("batch_64_grids_f32", "batch", prec=4, grids=64, dims_seed=6),
    ]


def _length(rng, top):
    """A side of a grid: powers of two, 7-smooth lengths, odd lengths whose
    factors stay below 32, spread over the logarithm of the length."""
    want = 2.0 ** rng.uniform(4.0, math.log2(top))
    pick = rng.random()
    if pick < 0.3:
        return min(top, 2 ** max(4, round(math.log2(want))))
    if pick < 0.8:
        return min((s for s in SMOOTH if s <= top), key=lambda s: abs(math.log(s / want)))
    n = int(want) | 1
    while _largest_factor(n) > 31:
        n += 2
    return n


def _largest_factor(n):
    best, p = 1, 2
    while p * p <= n:
        while n % p == 0:
            best, n = max(best, p), n // p
        p += 1
    return max(best, n)


def _box(rng, top, least, most):
    while True:
        dims = [_length(rng, top) for _ in range(3)]
        if least <= dims[0] * dims[1] * dims[2] <= most:
            return dims


def draw(rng):
    kind = rng.choices(["r2c", "overwrite", "c2c", "r2r", "transpose", "batch"], [50, 10, 17, 13, 5, 5])[0]
    prec = 8 if rng.random() < 0.6 else 4
    fmt = rng.choice([1, 3])
    if kind == "batch":
        c = _case("", "batch", prec=4, grids=rng.randint(8, 64), dims_seed=rng.randint(0, 1 << 20))
    elif kind == "r2r":
        # windows leave out a point: sides of a smooth length plus one mostly
        while True:
            dims = [rng.choice([s for s in SMOOTH if s <= 384]) + (1 if rng.random() < 0.75 else 0) for _ in range(3)]
            # the FFT behind a window keeps factors below 32
            if all(_largest_factor(d - 1) <= 31 for d in dims) and 1 << 13 <= dims[0] * dims[1] * dims[2] <= 1 << 24:
                break
        # DCT-I, DCT-II / III and DST-I, DST-II / III as boundary conditions pair them
        kinds = [rng.choice([1, 2, 2, 2, 3, 4, 5, 6, 7, 8]) for _ in range(3)]
        c = _case("", "r2r", *dims, fmt=fmt, prec=prec, kx=kinds[0], ky=kinds[1], kz=kinds[2])
    elif kind == "transpose":
        c = _case("", "transpose", *_box(rng, 512, 1 << 13, 1 << 25), prec=prec, complex=rng.random() < 0.5)
    else:
        c = _case("", kind, *_box(rng, 1024, 1 << 13, 1 << 26), fmt=fmt, prec=prec)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
def _real(c):
    return torch.float64 if c["prec"] == 8 else torch.float32


def _cplx(c):
    return torch.complex128 if c["prec"] == 8 else torch.complex64


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _field(c, seed):
    """A real field: unit Gaussian noise plus a few low-wavenumber modes of
    amplitude 10, as a turbulent velocity component has."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    g = _generator(seed)
    x = torch.randn((nz, ny, nx), generator=g, dtype=_real(c), device=DEVICE)
    k = torch.randint(0, 4, (4, 3), generator=g, device=DEVICE).tolist()
    ph = torch.rand((4, 3), generator=g, device=DEVICE).tolist()
    for m in range(4):
        wave = [torch.cos(torch.arange(n, device=DEVICE, dtype=torch.float64) * (2 * math.pi * k[m][d] / n)
                          + 2 * math.pi * ph[m][d]).to(_real(c)) for d, n in enumerate((nx, ny, nz))]
        x += (10 * wave[2])[:, None, None] * wave[1][None, :, None] * wave[0][None, None, :]
    return x


def _complex_field(c, seed):
    return torch.randn((c["nz"], c["ny"], c["nx"]), generator=_generator(seed), dtype=_cplx(c), device=DEVICE)


def _grids(c):
    """The batch's grids: sides drawn from BATCH_LENGTHS, a format each."""
    rng = np.random.default_rng(c["dims_seed"])
    out = []
    for _ in range(c["grids"]):
        nx, ny, nz = (int(v) for v in rng.choice(BATCH_LENGTHS, size=3))
        out.append((nx, ny, nz, 1 if rng.random() < 0.5 else 3))
    return out


def _batch_fields(c, seed):
    """Every grid's field in one allocation: (flat values, [(offset, shape)])."""
    places, at = [], 0
    for nx, ny, nz, _ in _grids(c):
        places.append((at, (nz, ny, nx)))
        at += (nx * ny * nz + 63) // 64 * 64
    flat = torch.rand(at, generator=_generator(seed), dtype=torch.float32, device=DEVICE) * 2 - 1
    return flat, places


def _view(flat, place):
    at, shape = place
    return flat[at:at + shape[0] * shape[1] * shape[2]].view(shape)


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind in ("r2c", "overwrite"):
        s["engine"] = e = gbfft.Engine(c["fmt"], c["nx"], c["ny"], c["nz"], inplace=kind == "overwrite", prec=c["prec"])
        s["x"] = _field(c, seed)
        s["spec"], s["back"] = e.empty_spectral(), e.empty_physical()
    elif kind == "c2c":
        s["engine"] = gbfft.Engine(c["fmt"], c["nx"], c["ny"], c["nz"], prec=c["prec"])
        s["x"] = _complex_field(c, seed)
        s["spec"], s["back"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    elif kind == "r2r":
        s["dtt"] = gbfft.Dtt(c["fmt"], c["nx"], c["ny"], c["nz"], [c["kx"], c["ky"], c["kz"]], prec=c["prec"])
        s["x"] = _field(c, seed)
        for k in ("work", "spec", "back"):
            s[k] = torch.empty_like(s["x"])
    elif kind == "transpose":
        s["x"] = _complex_field(c, seed) if c["complex"] else _field(c, seed)
        for k in ("y", "z", "y2", "x2"):
            s[k] = torch.empty_like(s["x"])
    else:
        s["flat"], places = _batch_fields(c, seed)
        s["real"] = torch.empty_like(s["flat"])
        s["batch"], s["specs"], s["backs"] = gbfft.Batch(), [], []
        for (nx, ny, nz, fmt), place in zip(_grids(c), places):
            e = gbfft.Engine(fmt, nx, ny, nz, prec=4)
            real, spec = _view(s["real"], place), e.empty_spectral()
            s["batch"].add(e, real, spec)
            s["specs"].append(spec)
            s["backs"].append(real)
    return s


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind in ("r2c", "overwrite"):
        s["engine"].r2c(s["x"], s["spec"])
        s["engine"].c2r(s["spec"], s["back"])
        # an OVERWRITE engine's c2r leaves nothing of use in its spectrum
        return [s["back"]] if kind == "overwrite" else [s["spec"], s["back"]]
    if kind == "c2c":
        s["engine"].c2c(s["x"], s["spec"], FORWARD)
        s["engine"].c2c(s["spec"], s["back"], BACKWARD)
        return [s["spec"], s["back"]]
    if kind == "r2r":
        # r2r works in its input: the program keeps its field and spectrum
        s["work"].copy_(s["x"])
        s["dtt"].r2r(s["work"], s["spec"], FORWARD)
        s["work"].copy_(s["spec"])
        s["dtt"].r2r(s["work"], s["back"], BACKWARD)
        return [s["spec"], s["back"]]
    if kind == "transpose":
        chain = [s[k] for k in ("x", "y", "z", "y2", "x2")]
        for step, which in enumerate((gbfft.X_TO_Y, gbfft.Y_TO_Z, gbfft.Z_TO_Y, gbfft.Y_TO_X)):
            gbfft.transpose(which, chain[step], chain[step + 1], c["nx"], c["ny"], c["nz"], c["complex"], c["prec"])
        return chain[1:]
    # the batch's backward overwrites the fields: this step's fields first
    s["real"].copy_(s["flat"])
    s["batch"].run(3)
    # outputs: the first grids' spectra, then the fields of all grids
    return s["specs"][:48] + [s["real"]]


# ---------------------------------------------------------------------------
def _transform_work(nx, ny, nz, prec, cplx):
    """Input and output once each way, and 2.5 (5) N log2 N a direction."""
    n = nx * ny * nz
    if cplx:
        return {"bytes": 2 * 2 * n * 2 * prec, "flops": 2 * 5.0 * n * math.log2(n)}
    spec = n // nx * (nx // 2 + 1)
    return {"bytes": 2 * (n * prec + spec * 2 * prec), "flops": 2 * 2.5 * n * math.log2(n)}


def work(case):
    c, kind = case, case["kind"]
    n = c["nx"] * c["ny"] * c["nz"]
    if kind in ("r2c", "overwrite", "c2c"):
        return _transform_work(c["nx"], c["ny"], c["nz"], c["prec"], kind == "c2c")
    if kind == "r2r":
        return {"bytes": 2 * 2 * n * c["prec"], "flops": 2 * 2.5 * n * math.log2(n)}
    if kind == "transpose":
        return {"bytes": 4 * 2 * n * c["prec"] * (2 if c["complex"] else 1), "flops": 0}
    parts = [_transform_work(nx, ny, nz, 4, False) for nx, ny, nz, _ in _grids(c)]
    return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}


# ---------------------------------------------------------------------------
def _rfftn(x, fmt):
    x = x.double()
    return torch.fft.rfftn(x, dim=(0, 1, 2) if fmt == 1 else (1, 2, 0))


def _r2r_matrix(kind, n):
    """FFTW's unnormalised definition of kind 1..8 at n points, as the values
    rounded to 20 bits and the rest."""
    j, k = np.arange(n, dtype=np.int64)[None, :], np.arange(n, dtype=np.int64)[:, None]
    # angle = pi * num / den
    num, den = {1: (j * k, n - 1), 2: ((2 * j + 1) * k, 2 * n), 3: (j * (2 * k + 1), 2 * n),
                4: ((2 * j + 1) * (2 * k + 1), 4 * n), 5: ((j + 1) * (k + 1), n + 1),
                6: ((2 * j + 1) * (k + 1), 2 * n), 7: ((j + 1) * (2 * k + 1), 2 * n),
                8: ((2 * j + 1) * (2 * k + 1), 4 * n)}[kind]
    pi = np.longdouble("3.14159265358979323846264338327950288")
    a = pi * (num % (2 * den)).astype(np.longdouble) / np.longdouble(den)
    m = 2 * (np.cos(a) if kind <= 4 else np.sin(a))
    if kind in (1, 3):
        m[:, 0] /= 2
    if kind == 1:
        m[:, -1] /= 2
    if kind == 7:
        m[:, -1] /= 2
    hi = np.rint(m.astype(np.float64) * 2.0 ** 20) / 2.0 ** 20
    return torch.from_numpy(hi).to(DEVICE), torch.from_numpy((m - hi).astype(np.float64)).to(DEVICE)


def _r2r_axis(x, dim, kind, first, n):
    """Window [first, first + n) of axis `dim` transformed in float64: the
    leading parts of both factors hold 20 bits, so that their product sums
    are exact, and only the small rests round."""
    x = x.movedim(dim, 0)
    w = x[first:first + n].reshape(n, -1)
    scale = 2.0 ** (20 - math.frexp(float(w.abs().max()))[1])
    wh = torch.round(w * scale) / scale
    mh, ml = _r2r_matrix(kind, n)
    y = x.clone()
    y[first:first + n] = (mh @ wh + (mh @ (w - wh) + ml @ w)).reshape((n,) + tuple(x.shape[1:]))
    return y.movedim(0, dim)


def _r2r(x, c, isign):
    inverse = {1: 1, 2: 3, 3: 2, 4: 4, 5: 5, 6: 7, 7: 6, 8: 8}
    for dim, key, size in ((2, "kx", c["nx"]), (1, "ky", c["ny"]), (0, "kz", c["nz"])):
        k = c[key]
        first = 1 if k in (5, 7) else 0
        n = size - {1: 0, 5: 2}.get(k, 1)
        x = _r2r_axis(x, dim, k if isign == FORWARD else inverse[k], first, n)
    return x


def exact(case, seed):
    c, kind = case, case["kind"]
    n = c["nx"] * c["ny"] * c["nz"]
    if kind in ("r2c", "overwrite"):
        x = _field(c, seed)
        back = x.double() * n
        return [back] if kind == "overwrite" else [_rfftn(x, c["fmt"]), back]
    if kind == "c2c":
        x = _complex_field(c, seed).to(torch.complex128)
        return [torch.fft.fftn(x), x * n]
    if kind == "r2r":
        spec = _r2r(_field(c, seed).double(), c, FORWARD)
        return [spec, _r2r(spec, c, BACKWARD)]
    if kind == "transpose":
        return None  # copies: their outputs are the input, bit for bit
    flat, places = _batch_fields(c, seed)
    specs, back = [], flat.double()
    for (nx, ny, nz, fmt), place in zip(_grids(c), places):
        if len(specs) < 48:
            specs.append(_rfftn(_view(flat, place), fmt))
        _view(back, place).mul_(nx * ny * nz)
    return specs + [back]
