"""The work that is timed: gauge fixes, ensembles, configuration generation,
gluon propagators and configuration I/O, each through the library's public
entry points.

Inputs are beta 6.0 links: the committed 8^4 heatbath configuration repeated
over the lattice from a seeded origin, every link then multiplied by a small
seeded SU(3) matrix (so that no two copies are equal) and the whole lattice
gauge transformed by seeded random SU(3) matrices, as a fix meets them.
`smooth` mixes the identity into the links before that (a fine lattice, or
smeared links), and `turn` scales the gauge transformation's departure from
the identity: a configuration that has been fixed before, to less accuracy or
before it was smeared.

A fix to theta < 1e-14 of a thermalised lattice takes an iteration count that
depends on the summation order, so the larger fixes run a given number of
iterations (`iters`, with an accuracy out of reach), or to a theta that comes
early; the two smallest, the second of smooth links, run to their end.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from glu_b200 import _lib, cuts, nersc
from glu_b200.workload import base_config

DEV = "cuda"
C128 = torch.complex128


# --------------------------------------------------------------------------
# the cases

def _dims(case):
    return case["lx"], case["ly"], case["lz"], case["lt"]


def _d(lx, ly, lz, lt):
    return {"lx": lx, "ly": ly, "lz": lz, "lt": lt}


def listed():
    return [
        # the smallest fix in use, to its end: launches and latency
        {"name": "landau_8x8x8x8_whole", "kind": "landau", **_d(8, 8, 8, 8),
         "algo": "FACG", "precision": "FP64", "accuracy": 1e-12, "iters": 5000},
        # a small fine lattice, fixed to its end in mixed precision
        {"name": "landau_16x16x16x32_mixed_whole", "kind": "landau", **_d(16, 16, 16, 32),
         "algo": "FACG", "precision": "MIXED", "accuracy": 1e-12, "iters": 5000, "smooth": 1.0,
         "turn": 0.3},
        # extents with a factor 5, steepest descent
        {"name": "landau_20x20x20x40_fasd", "kind": "landau", **_d(20, 20, 20, 40),
         "algo": "FASD", "precision": "FP64", "accuracy": 1e-30, "iters": 12},
        # the usual production lattice, in both precisions
        {"name": "landau_32x32x32x64", "kind": "landau", **_d(32, 32, 32, 64),
         "algo": "FACG", "precision": "FP64", "accuracy": 1e-30, "iters": 12},
        {"name": "landau_32x32x32x64_mixed", "kind": "landau", **_d(32, 32, 32, 64),
         "algo": "FACG", "precision": "MIXED", "accuracy": 1e-30, "iters": 8},
        # the largest Landau lattice
        {"name": "landau_48x48x48x96_mixed", "kind": "landau", **_d(48, 48, 48, 96),
         "algo": "FACG", "precision": "MIXED", "accuracy": 1e-30, "iters": 5, "smooth": 0.5,
         "turn": 1.0},
        # an ensemble of two lattice sizes in one batch
        {"name": "ensemble_fasd_mixed", "kind": "batch", "n16": 6, "n24": 2,
         "algo": "FASD", "precision": "MIXED", "accuracy": 1e-30, "iters": 10},
        # Coulomb gauge of every time slice: the usual lattice, and the largest
        # spatial volume to its end in mixed precision
        {"name": "coulomb_32x32x32x64", "kind": "coulomb", **_d(32, 32, 32, 64),
         "algo": "FACG", "precision": "FP64", "accuracy": 0.1},
        {"name": "coulomb_64x64x64x16_mixed", "kind": "coulomb", **_d(64, 64, 64, 16),
         "algo": "FACG", "precision": "MIXED", "accuracy": 1e-12, "smooth": 2.0,
         "turn": 1.0},
        # one step of configuration generation: a heatbath and four
        # over-relaxation sweeps
        {"name": "heatbath_32x32x32x64", "kind": "heatbath", **_d(32, 32, 32, 64),
         "beta": 6.0, "steps": 1, "n_or": 4},
        # propagators of a fixed configuration with the shipped input file's cut
        {"name": "gluonprop_32x32x32x64", "kind": "cuts", **_d(32, 32, 32, 64),
         "mode": "GLUON_PROPS", "cut": "CYLINDER_CUT", "field": "LINEAR",
         "maxmom": 4, "width": 2.0},
        # a configuration read and written back (host buffers by nature)
        {"name": "nersc_16x16x16x32", "kind": "nersc", **_d(16, 16, 16, 32),
         "nreal": 12, "bytes": 8, "big": True},
    ]


_EXTENTS = [4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32, 36, 40,
            42, 45, 48]
_USUAL = [8, 16, 24, 32, 48]


def _draw_dims(rng, most, even=False, lo=1024):
    """Extents in use (cubic spatial volumes of the usual sizes, half the
    time) or any others the transforms take, with the volume spread over its
    logarithm."""
    target = math.exp(rng.uniform(math.log(lo), math.log(most)))
    ext = [e for e in _EXTENTS if not even or e % 2 == 0]
    usual = rng.random() < 0.5
    best = None
    for _ in range(200):
        if usual:
            s = rng.choice(_USUAL)
            d = (s, s, s, rng.choice([s, 2 * s, rng.choice(ext)]))
        else:
            s = rng.choice(ext)
            d = tuple(rng.choice([s, s, rng.choice(ext)]) for _ in range(3)) + (rng.choice(ext + [64, 96]),)
        v = d[0] * d[1] * d[2] * d[3]
        if d[0] * d[1] > 4096 or d[2] * d[3] > 4608 or v > most:
            continue
        off = abs(math.log(v / target))
        if best is None or off < best[0]:
            best = (off, d)
    return best[1] if best else (8, 8, 8, 8)


def draw(rng):
    kind = rng.choice(["landau", "landau", "landau", "batch", "coulomb", "coulomb", "heatbath",
                       "cuts", "cuts", "nersc"])
    if kind == "landau":
        d = _draw_dims(rng, 48 ** 3 * 96)
        v = d[0] * d[1] * d[2] * d[3]
        top = max(3, min(12, int(48 ** 3 * 96 * 8 / v)))
        return {"kind": kind, **_d(*d), "algo": rng.choice(["FACG", "FACG", "FASD"]),
                "precision": rng.choice(["FP64", "MIXED"]), "accuracy": 1e-30,
                "iters": rng.randint(3, 5 if v > 4e6 else top)}
    if kind == "batch":
        return {"kind": kind, "n16": rng.randint(1, 10), "n24": rng.randint(0, 3),
                "algo": rng.choice(["FACG", "FASD"]), "precision": rng.choice(["FP64", "MIXED"]),
                "accuracy": 1e-30, "iters": rng.randint(4, 12)}
    if kind == "coulomb":
        if rng.random() < 0.3:
            s = rng.choice([32, 48, 64])
            d = (s, s, s, rng.choice([4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16]))
        else:
            d = _draw_dims(rng, 32 ** 3 * 64)
        c = {"kind": kind, **_d(*d), "algo": rng.choice(["FACG", "FACG", "FASD"])}
        if rng.random() < 0.5:
            return {**c, "precision": "FP64", "accuracy": round(rng.uniform(0.1, 1.0), 3)}
        return {**c, "precision": "MIXED", "accuracy": 1e-12, "smooth": 2.0, "turn": 1.0}
    if kind == "heatbath":
        d = _draw_dims(rng, 32 ** 3 * 64, even=True)
        return {"kind": kind, **_d(*d), "beta": round(rng.uniform(5.7, 6.4), 2),
                "steps": rng.randint(1, 2), "n_or": rng.choice([0, 1, 4])}
    if kind == "cuts":
        d = _draw_dims(rng, 32 ** 3 * 64)
        return {"kind": kind, **_d(*d),
                "mode": rng.choice(["GLUON_PROPS", "GLUON_PROPS", "EXCEPTIONAL", "FIELDS"]),
                "cut": rng.choice(["CYLINDER_CUT", "SPHERICAL_CUT", "HYPERCUBIC_CUT"]),
                "field": rng.choice(["LINEAR", "LINEAR", "LOGARITHMIC"]),
                "maxmom": rng.choice([2, 4, 8, 20]), "width": rng.choice([1.0, 2.0])}
    d = _draw_dims(rng, 16 ** 3 * 32)
    return {"kind": kind, **_d(*d), "nreal": rng.choice([12, 18]), "bytes": rng.choice([4, 8]),
            "big": rng.choice([True, False])}


# --------------------------------------------------------------------------
# SU(3) algebra and lattices in torch

def _mm(a, b):
    return (a.unsqueeze(-1) * b.unsqueeze(-3)).sum(-2)


def _dag(a):
    return a.conj().transpose(-1, -2)


def _reunit(c0, c1):
    """Column Gram-Schmidt, third column the conjugate cross product."""
    c0 = c0 / torch.linalg.vector_norm(c0, dim=-1, keepdim=True)
    c1 = c1 - (c0.conj() * c1).sum(-1, keepdim=True) * c0
    c1 = c1 / torch.linalg.vector_norm(c1, dim=-1, keepdim=True)
    return torch.stack([c0, c1, torch.linalg.cross(c0, c1, dim=-1).conj()], dim=-1)


def _random_su3(n, gen, mean):
    z = torch.randn((2, n, 3), dtype=C128, generator=gen, device=DEV)
    return _reunit(mean[0] + z[0], mean[1] + z[1])


def _shift(f, mu, by):
    """f(x + by mu-hat) of f[Lt, Lz, Ly, Lx, ...]."""
    return torch.roll(f, -by, dims=3 - mu)


_base = {}


def _shape(case):
    return case.get("smooth", 0.0), case.get("turn", 0.0)


def _links(dims, seed, smooth=0.0, turn=0.0):
    """The seeded input links, complex128 (Lt, Lz, Ly, Lx, 4, 3, 3)."""
    if "b" not in _base:
        b, bd = base_config()
        _base["b"] = torch.from_numpy(b.reshape(*bd[::-1], 4, 3, 3)).to(DEV)
        _base["d"] = bd
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 13)
    o = torch.randint(0, 8, (4,), generator=gen, device=DEV).tolist()
    ix = [(torch.arange(dims[a], device=DEV) + o[a]) % _base["d"][a] for a in range(4)]
    V = math.prod(dims)
    lat = tuple(dims[::-1])
    U = torch.empty(lat + (4, 3, 3), dtype=C128, device=DEV)
    one = torch.eye(3, dtype=C128, device=DEV)
    g = _random_su3(V, gen, one / turn if turn else 0 * one).reshape(lat + (3, 3))
    for mu in range(4):
        b = _base["b"][..., mu, :, :]
        u = b[ix[3]][:, ix[2]][:, :, ix[1]][:, :, :, ix[0]]
        if smooth:
            u = _reunit(u[..., 0] + smooth * one[0], u[..., 1] + smooth * one[1])
        noise = _random_su3(V, gen, 20.0 * one).reshape(lat + (3, 3))
        U[..., mu, :, :] = _mm(_mm(g, _mm(noise, u)), _dag(_shift(g, mu, 1)))
    return U


# --------------------------------------------------------------------------
# the passes

def _params(case):
    p = _lib.GfixParams()
    p.gf_alpha = 0.08
    p.accuracy = case["accuracy"]
    p.max_iters = case.get("iters", 5000)
    p.algo = {"FACG": 0, "FASD": 1}[case["algo"]]
    p.precision = {"FP64": 0, "MIXED": 1}[case["precision"]]
    p.switch_theta = 1e-9
    return p


def _flat(U):
    return torch.view_as_real(U).reshape(-1)


def _cd(dims):
    return (C.c_size_t * 4)(*dims)


class _Batch:
    """A batch handle over device links, freed with the state."""

    def __init__(self, p, bufs, dims):
        self.lib = _lib.load()
        self.h = self.lib.gfix_batch_create(C.byref(p))
        for b, d in zip(bufs, dims):
            if self.lib.gfix_batch_add_device(self.h, b.data_ptr(), _cd(d)) < 0:
                _lib.check(-1)

    def __del__(self):
        if self.h:
            self.lib.gfix_batch_destroy(self.h)
            self.h = None


def _batch_dims(case):
    return [(16, 16, 16, 32)] * case["n16"] + [(24, 24, 24, 48)] * case["n24"]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "nersc":
        dims = _dims(case)
        U = _links(dims, seed).reshape(-1, 4, 3, 3).cpu().numpy()
        r = U.reshape(-1, 4, 9)[..., : case["nreal"] // 2].view(np.float64)
        t = np.dtype({8: "f8", 4: "f4"}[case["bytes"]]).newbyteorder(">" if case["big"] else "<")
        s["payload"] = np.ascontiguousarray(r.astype(t)).tobytes()
        return s
    if kind == "batch":
        ds = _batch_dims(case)
        s["in"] = [_flat(_links(d, seed * 64 + i)) for i, d in enumerate(ds)]
        s["work"] = [x.clone() for x in s["in"]]
        s["batch"] = _Batch(_params(case), s["work"], ds)
        return s
    U = _links(_dims(case), seed, *_shape(case))
    if kind == "cuts":
        s["links"] = U
        s["info"] = cuts.CutInfo(case["mode"], case["cut"], case["field"], case["maxmom"], 60,
                                 case["width"])
        return s
    s["in"] = _flat(U)
    s["work"] = torch.empty_like(s["in"])
    s["seed"] = int(seed)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    lib = _lib.load()
    if kind == "landau":
        s["work"].copy_(s["in"])
        r = _lib.GfixResult()
        _lib.check(lib.gfix_landau_device(s["work"].data_ptr(), _cd(_dims(case)),
                                          C.byref(_params(case)), C.byref(r)))
        out = {"links": s["work"]}
        if _bounded(case):  # (the last theta of a whole fix is rounding)
            out["theta"] = float(r.theta)
        return out
    if kind == "batch":
        for w, i in zip(s["work"], s["in"]):
            w.copy_(i)
        _lib.check(lib.gfix_batch_run(s["batch"].h))
        return {"links": s["work"]}
    if kind == "coulomb":
        s["work"].copy_(s["in"])
        r = _lib.GfixResult()
        T = case["lt"]
        th = np.zeros(T)
        it = np.zeros(T, dtype=np.uintp)
        _lib.check(lib.gfix_coulomb_device(
            s["work"].data_ptr(), _cd(_dims(case)), C.byref(_params(case)), C.byref(r),
            th.ctypes.data_as(C.POINTER(C.c_double)), it.ctypes.data_as(C.POINTER(C.c_size_t))))
        if case["precision"] == "MIXED":  # (the last thetas are rounding)
            return {"links": s["work"]}
        return {"links": s["work"], "theta": th, "iters": it.astype(np.int64)}
    if kind == "heatbath":
        s["work"].copy_(s["in"])
        plaq = np.zeros(case["steps"])
        if lib.gfix_heatbath_device(s["work"].data_ptr(), _cd(_dims(case)), case["beta"],
                                    case["steps"], case["n_or"], s["seed"], 0,
                                    plaq.ctypes.data_as(C.POINTER(C.c_double))) != 0:
            raise RuntimeError(lib.gfix_update_error().decode())
        return {"links": s["work"], "plaquette": plaq}
    if kind == "cuts":
        r = cuts.measure_device(s["links"], _dims(case), s["info"])
        return {k: v for k, v in r.items()}
    links, ck = nersc.decode(s["payload"], _dims(case), case["nreal"], case["bytes"], case["big"])
    pay, ck2 = nersc.encode(links, _dims(case), case["nreal"], case["bytes"], case["big"])
    return {"links": links, "payload": np.frombuffer(pay, dtype=np.uint8),
            "checksums": np.array([ck, ck2], dtype=np.int64)}


def _bounded(case):
    return case["accuracy"] < 1e-20


# --------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    """Bytes: the links in and out of the call once (1152 per site), and per
    iteration, whose two global sums force it over the lattice again, in the
    types of the phase: the links (96 bytes each in FP64, two columns) read
    for the line search, read and written by the update, and the fields
    through the derivative, the three FFT passes, the line search and the
    update (768 per site in FP64)."""
    kind = case["kind"]
    if kind == "batch":
        n = [_landau_work(case, math.prod(d), case["iters"]) for d in _batch_dims(case)]
        return {"bytes": sum(x[0] for x in n), "flops": sum(x[1] for x in n)}
    V = math.prod(_dims(case))
    if kind == "landau":
        # (whole fixes: 93 iterations, or 14 in each phase of the smooth one)
        whole = 14 if case["precision"] == "MIXED" else 93
        b, f = _landau_work(case, V, case["iters"] if _bounded(case) else whole)
        return {"bytes": b, "flops": f}
    if kind == "coulomb":
        # 15 (FP32) and 4 steps to the end of a smooth configuration, 30 to an
        # early theta of a rough one: per step the three spatial links and g
        # read for the derivative and for the probes, g read and written, the
        # fields as above
        per = 2 * (288 + 144) + 288 + 768
        n32, n64 = (15, 4) if case["precision"] == "MIXED" else (0, 30)
        return {"bytes": V * (1152 + n32 * per / 2 + n64 * per), "flops": V * (n32 + n64) * 5000.0}
    if kind == "heatbath":
        # links in and out, and per sweep and (direction, colour) the links
        # updated read and written, the others read (two columns)
        sweeps = case["steps"] * (1 + case["n_or"])
        return {"bytes": V * (1152.0 + sweeps * 8 * 432 / 1.0),
                "flops": V * 4.0 * sweeps * 3500}
    if kind == "cuts":
        # the links read once (what is kept of their transforms is small)
        return {"bytes": 576.0 * V, "flops": 4.0 * V * (60 + 4 * 5 * 2 * math.log2(V))}
    nb = V * 4 * case["nreal"] * case["bytes"]
    return {"bytes": 2.0 * nb + 2 * 576 * V, "flops": 0.0}


def _landau_work(case, V, iters):
    links, fields = 3 * 384.0, 768.0
    it64 = links + fields
    phases = ([(links + fields) / 2, links + fields / 2] if case["precision"] == "MIXED"
              else [it64])
    return V * (1152 + iters * sum(phases)), V * iters * len(phases) * 6000.0


def tolerance(case):
    """Four times what runs with sums in another order, and the 64-bit
    restatement below, differ by."""
    kind = case["kind"]
    mixed = case.get("precision") == "MIXED"
    if kind == "landau" and not _bounded(case):
        # theta < 1e-12 leaves the links this free
        return {"rel": 2e-6, "max": 1e-3} if mixed else {"rel": 5e-9, "max": 1e-7}
    if kind in ("landau", "batch"):
        return {"rel": 1e-5, "max": 1e-3} if mixed else {"rel": 1e-9, "max": 1e-7}
    if kind == "coulomb":
        return {"rel": 1e-6, "max": 1e-4} if mixed else {"rel": 1e-8, "max": 1e-6}
    if kind == "heatbath":
        return {"rel": 1e-11, "max": 1e-8}
    if kind == "cuts":
        return {"rel": 1e-11, "max": 1e-8}
    return {"rel": 1e-12, "max": 1e-11}


# --------------------------------------------------------------------------
# the same in 64 bits, restated in torch

def _re_tr(a):
    return a[..., 0, 0].real + a[..., 1, 1].real + a[..., 2, 2].real


def _pack(D):
    """The su(3) packing of a sum of link differences D (4 fields), and the
    sum of squares that is theta's numerator per site."""
    i0, i1, i2 = D[..., 0, 0].imag, D[..., 1, 1].imag, D[..., 2, 2].imag
    r0, r3 = 2 * i0 - i1 - i2, 2 * i1 - i0 - i2
    off = [D[..., a, b] - D[..., b, a].conj() for a, b in ((0, 1), (0, 2), (1, 2))]
    f = torch.stack([torch.complex(-r3 / 3, r0 / 3)] + [0.5 * o for o in off])
    th = 4.0 / 9.0 * (r0 * r0 + r3 * (r3 + r0))
    for o in off:
        th = th + o.real ** 2 + o.imag ** 2
    return f, th


def _gauge(f, al):
    """reunit(1 + alpha A) of the packed fields; al broadcasts over sites."""
    zero = torch.zeros_like(f[0].real)
    one = zero + 1.0
    a1, a2, a3 = al * f[1], al * f[2], al * f[3]
    c0 = torch.stack([torch.complex(one, al * f[0].imag), -a1.conj(), -a2.conj()], dim=-1)
    c1 = torch.stack([a1, torch.complex(one, -al * f[0].real), -a3.conj()], dim=-1)
    return _reunit(c0, c1)


def _accelerate(f, dims, nd):
    """FFT, times maxp / p^2, FFT back, over the last nd of the axes of
    f[4, Lt, Lz, Ly, Lx]."""
    k = torch.zeros((1, 1, 1, 1), dtype=torch.float64, device=DEV)
    for mu in range(nd):
        n = torch.arange(dims[mu], dtype=torch.float64, device=DEV)
        sh = [1, 1, 1, 1]
        sh[3 - mu] = dims[mu]
        k = k + torch.cos(2 * math.pi * n / dims[mu]).reshape(sh)
    p2 = torch.where((nd - k) < 1e-14, torch.ones_like(k), 2 * (nd - k))
    maxp = 4.0 * nd / math.prod(dims[:nd])
    ax = tuple(range(-nd, 0))
    out = torch.empty_like(f)
    for c in range(4):
        out[c] = torch.fft.ifftn(torch.fft.fftn(f[c], dim=ax) * (maxp / p2), dim=ax,
                                 norm="forward")
    return out


def _sums(f, old):
    """The conjugate-gradient sums per time slice: insum, sumconj."""
    t = f - old
    s = f.real ** 2 + f.imag ** 2
    c = f.real * t.real + f.imag * t.imag
    s0, c0 = f[0].real * f[0].imag, f[0].real * t[0].imag + f[0].imag * t[0].real
    ax = (-3, -2, -1)
    ins = 2 * (s.sum(ax).sum(0) + s0.sum(ax))
    con = 2 * c.sum(ax).sum(0) + c0.sum(ax)
    return ins, con


def _minimum(al, f):
    """The parabola's minimum of GLU's approx_minimum."""
    A = f[0] / ((al[0] - al[1]) * (al[0] - al[2]))
    B = f[1] / ((al[1] - al[0]) * (al[1] - al[2]))
    D = f[2] / ((al[2] - al[0]) * (al[2] - al[1]))
    den = 2 * (A + B + D)
    if den == 0:
        return 0.08
    s = (al[0] * (B + D) + al[1] * (A + D) + al[2] * (A + B)) / den
    if s > al[2]:
        return al[2]
    return 0.08 if math.isnan(s) or math.isinf(s) or s < al[0] else s


class _Landau:
    def __init__(self, U, dims):
        self.U, self.dims, self.V = U, dims, math.prod(dims)

    def derivative(self):
        f, th = None, None
        D = torch.zeros(self.U.shape[:4] + (3, 3), dtype=C128, device=DEV)
        for mu in range(4):
            u = self.U[..., mu, :, :]
            D += _shift(u, mu, -1) - u
        f, th = _pack(D)
        return f, float(th.sum()) / (3.0 * self.V)

    def probe(self, f):
        d = [0.0, 0.0]
        for k, al in enumerate((0.15, 0.30)):
            g = _gauge(f, al)
            for mu in range(4):
                u = self.U[..., mu, :, :]
                w = _mm(g, u)
                gy = _shift(g, mu, 1)
                d[k] += float(((w.real * gy.real + w.imag * gy.imag).sum((-1, -2))
                               - _re_tr(u)).sum())
        return _minimum((0.0, 0.15, 0.30), (0.0, -d[0], -d[1]))

    def update(self, f, al):
        g = _gauge(f, al)
        for mu in range(4):
            self.U[..., mu, :, :] = _mm(_mm(g, self.U[..., mu, :, :]), _dag(_shift(g, mu, 1)))

    def solve(self, algo, acc, iters):
        if 2 * self.derivative()[1] < acc:
            return 0.0
        old = sn = None
        inold = 0.0
        if algo == "FACG":
            f = _accelerate(self.derivative()[0], self.dims, 4)
            self.update(f, self.probe(f))
            old = sn = f
            inold = float(2 * ((f.real ** 2 + f.imag ** 2).sum()
                               + (f[0].real * f[0].imag).sum()))
        for it in range(iters):
            f, tr = self.derivative()
            f = _accelerate(f, self.dims, 4)
            if algo == "FACG":
                a, b = (float(x.sum()) for x in _sums(f, old))
                beta = max(b / inold, 0.0) if tr >= 5e-11 else a / inold
                inold = a
                sn = f + beta * sn
                old = f
                self.update(sn, self.probe(sn) if tr > 5e-11 else 0.08)
            else:
                self.update(f, self.probe(f))
            if not tr > acc:
                break
        return tr


class _Coulomb:
    def __init__(self, U, dims):
        self.U, self.dims = U, dims
        self.lcu = dims[0] * dims[1] * dims[2]
        self.g = torch.eye(3, dtype=C128, device=DEV).expand(U.shape[:4] + (3, 3)).contiguous()
        self.T = dims[3]

    def rotated(self, mu):
        return _mm(_mm(self.g, self.U[..., mu, :, :]), _dag(_shift(self.g, mu, 1)))

    def solve(self, acc, iters, algo):
        T = self.T
        theta, count = np.zeros(T), np.zeros(T, dtype=np.int64)
        live = np.ones(T, dtype=bool)
        sd = True
        inold = np.ones(T)
        old = torch.zeros((4,) + self.U.shape[:4], dtype=C128, device=DEV)
        sn = old
        per = lambda v: torch.tensor(v, dtype=torch.float64, device=DEV).reshape(T, 1, 1, 1)  # noqa: E731
        while live.any():
            W = [self.rotated(mu) for mu in range(3)]
            D = sum(_shift(w, mu, -1) - w for mu, w in enumerate(W))
            f = _accelerate(_pack(D)[0], self.dims, 3)
            ins, con = (x.cpu().numpy() for x in _sums(f, old))
            tr = ins / (3.0 * self.lcu)
            beta = np.zeros(T) if sd else np.where(tr < 5e-11, ins / inold,
                                                   np.maximum(con / inold, 0.0))
            inold = ins
            sn = f if sd else f + per(beta) * sn
            old = f
            d = []
            for al in (0.17, 0.34):
                A = _gauge(sn, al)
                t = 0.0
                for mu, w in enumerate(W):
                    x, y = _mm(A, w), _shift(A, mu, 1)
                    t = t + ((x.real * y.real + x.imag * y.imag).sum((-1, -2))
                             - _re_tr(w)).sum((1, 2, 3))
                d.append(t.cpu().numpy())
            al = np.array([_minimum((0.0, 0.17, 0.34), (0.0, -d[0][t], -d[1][t]))
                           if sd or tr[t] > 5e-11 else 0.08 for t in range(T)])
            G = _mm(_gauge(sn, per(al)), self.g)
            m = torch.tensor(live, device=DEV)
            self.g = torch.where(m.reshape(T, 1, 1, 1, 1, 1), G, self.g)
            theta = np.where(live, tr, theta)
            if not sd or algo == "FASD":
                count += live
                live &= (tr > acc) & (count < iters)
            sd = algo == "FASD"
        return theta, count

    def reunit(self):
        self.g = _reunit(self.g[..., 0], self.g[..., 1])

    def links(self):
        for mu in range(4):
            self.U[..., mu, :, :] = self.rotated(mu)
        return self.U


def _philox(c, k0, k1):
    """Philox4x32-10 of counters c[4] (int64 tensors) under key (k0, k1)."""
    M = 0xFFFFFFFF

    def mul(a, b):  # 32 x 32 -> (hi, lo)
        p0, p1 = a * (b & 0xFFFF), a * (b >> 16)
        lo = (p0 + ((p1 & 0xFFFF) << 16))
        return (p1 >> 16) + (lo >> 32), lo & M

    c = list(c)
    for _ in range(10):
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c


class _Draws:
    def __init__(self, h, tag, it, seed):
        self.h, self.tag, self.it = h, tag, it
        self.k = (seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF)
        self.w = torch.zeros_like(h)

    def pair(self, sel):
        w = self.w[sel]
        z = torch.zeros_like(w)
        c = _philox([self.h[sel], z + self.tag, z + self.it, w], *self.k)
        self.w[sel] = w + 1
        # the upper 53 of 64 bits, put together without overflow
        mk = lambda a, b: ((a << 21 | b >> 11).double() + 0.5) * 2.0 ** -53  # noqa: E731
        return mk(c[0], c[1]), mk(c[2], c[3])


def _heatbath_sweep(U, dims, hb, invbeta, seed, it):
    co = torch.meshgrid(*[torch.arange(d, device=DEV) for d in dims[::-1]], indexing="ij")
    par = sum(co) % 2
    half = (torch.arange(par.numel(), device=DEV).reshape(par.shape)) // 2
    for mu in range(4):
        for p in range(2):
            st = torch.zeros(U.shape[:4] + (3, 3), dtype=C128, device=DEV)
            m = U[..., mu, :, :]
            for nu in range(4):
                if nu == mu:
                    continue
                n = U[..., nu, :, :]
                top = _mm(_mm(n, _shift(m, nu, 1)), _dag(_shift(n, mu, 1)))
                bot = _mm(_mm(_dag(n), m), _shift(n, mu, 1))
                st += top + _shift(bot, nu, -1)
            sel = par == p
            S, M, h = st[sel], m[sel], half[sel]
            rng = _Draws(h, 2 * mu + p, it, seed)
            every = torch.ones_like(h, dtype=torch.bool)
            for a, b in ((0, 1), (1, 2), (2, 0)):
                X = _mm(M, _dag(S))
                m0 = X[:, a, a] + X[:, b, b].conj()
                m1 = X[:, a, b] - X[:, b, a].conj()
                z = 1.0 / torch.sqrt(m0.abs() ** 2 + m1.abs() ** 2)
                s0, s1 = m0 * z, m1 * z
                if hb:
                    d = torch.zeros_like(z)
                    act = every.clone()
                    for _ in range(43):
                        x4, x3 = rng.pair(act)
                        x3 = torch.cos(2 * math.pi * x3)
                        l1, l2 = rng.pair(act)
                        dn = -(torch.log(l1) + torch.log(l2) * x3 * x3) * (invbeta * z[act])
                        d[act] = dn
                        again = act.clone()
                        again[act] = (1.0 - 0.5 * dn) < x4 * x4
                        act = again
                        if not bool(act.any()):
                            break
                    a0 = 1.0 - d
                    ar2 = (1.0 - a0 * a0).abs()
                    u, v = rng.pair(every)
                    a3 = torch.sqrt(ar2) * (2 * u - 1)
                    rho = torch.sqrt((ar2 - a3 * a3).abs())
                    a1, a2 = rho * torch.cos(2 * math.pi * v), rho * torch.sin(2 * math.pi * v)
                    # the draw times the conjugate of the staple's element
                    q0, q1 = torch.complex(a0, a3), torch.complex(a2, a1)
                    s0, s1 = q0 * s0.conj() + q1 * s1.conj(), q1 * s0 - q0 * s1
                else:
                    q0, q1 = s0.conj(), -s1
                    s0, s1 = q0 * q0 - q1 * q1.conj(), q0 * q1 + q1 * q0.conj()
                N = M.clone()
                N[:, a] = s0[:, None] * M[:, a] + s1[:, None] * M[:, b]
                N[:, b] = s0.conj()[:, None] * M[:, b] - s1.conj()[:, None] * M[:, a]
                M = N
            if hb:
                M = _reunit(M[..., 0], M[..., 1])
            m[sel] = M


def _plaquette(U):
    t = 0.0
    for mu in range(1, 4):
        for nu in range(mu):
            a, b = U[..., mu, :, :], U[..., nu, :, :]
            x, y = _mm(a, _shift(b, mu, 1)), _mm(b, _shift(a, nu, 1))
            t += float((x.real * y.real + x.imag * y.imag).sum())
    return t / (18.0 * math.prod(U.shape[:4]))


def _momenta(dims, case):
    """The kept momenta, t slowest, and their 2 sin(p / 2)."""
    small = min(dims)
    ax = [torch.arange(-(d // 2), d - d // 2, dtype=torch.float64) for d in dims]
    n = torch.stack([x.reshape(-1) for x in torch.meshgrid(*ax[::-1], indexing="ij")][::-1], -1)
    L = torch.tensor(dims, dtype=torch.float64)
    r = n * (small / L)
    p = 2 * torch.sin(math.pi * n / L)
    if case["cut"] == "HYPERCUBIC_CUT":
        ok = (r.abs() <= math.sqrt(case["maxmom"])).all(-1)
    else:
        ok = (r * r).sum(-1) <= case["maxmom"]
        if case["cut"] == "CYLINDER_CUT":
            near = torch.zeros_like(ok)
            for d in range(16):
                x = torch.tensor([1.0 if d >> mu & 1 else -1.0 for mu in range(4)],
                                 dtype=torch.float64)
                t = p - 0.25 * (p @ x)[:, None] * x
                near |= torch.sqrt((t * t).sum(-1)) <= 2 * math.pi * case["width"] / small
            ok &= near
    return n[ok].to(torch.int64), p[ok]


def _exact_cuts(case, seed):
    dims = _dims(case)
    n, p = _momenta(dims, case)
    U = _links(dims, seed)
    G = torch.empty((len(n), 4, 3, 3), dtype=C128)
    at = tuple((n % torch.tensor(dims)).T.flip(0).to(DEV))
    for mu in range(4):
        u = U[..., mu, :, :]
        A = (u - _dag(u)) / 2j
        tr = (A[..., 0, 0] + A[..., 1, 1] + A[..., 2, 2]) / 3
        A = A - tr[..., None, None] * torch.eye(3, dtype=C128, device=DEV)
        half = 0.5 * p[:, mu]
        ph = torch.complex(torch.sqrt(1 - half * half), half)
        for a in range(3):
            for b in range(3):
                F = torch.fft.ifftn(A[..., a, b], dim=(0, 1, 2, 3), norm="forward")
                G[:, mu, a, b] = F[at].cpu() * ph
    V = math.prod(dims)
    out = {"mom": n.numpy().astype(np.int32)}
    err = (G * p[..., None, None]).sum((1, 2, 3)).abs() / 9
    out["pspace_err"] = float(err.mean())
    psq = (p * p).sum(-1)
    psq = torch.where(psq < 3e-14, torch.ones_like(psq), psq)
    zero = len(n) // 2
    g2 = torch.full_like(psq, 2.0 / (8 * 3 * V))
    g2[zero] = 2.0 / (8 * 4 * V)
    if case["mode"] == "FIELDS":
        out["fields"] = G.numpy()
    elif case["mode"] == "GLUON_PROPS":
        re = torch.einsum("imab,inab->imn", G, G.conj()).real
        c = p[:, :, None] * p[:, None, :] / psq[:, None, None] * re
        lo = c.sum((1, 2))
        T = (torch.einsum("imm->i", re) - lo) * g2
        lo = lo * (2.0 / (8 * V))
        back = torch.arange(len(n))
        back = torch.where(back > zero, len(n) - 1 - back, back)
        out["transverse"], out["longitudinal"] = T[back].numpy(), lo[back].numpy()
    else:
        Gc = G.flip(0)
        tr = lambda a, b: torch.einsum("iab,iba->i", a, b)  # noqa: E731
        out["g2"] = (sum(tr(G[:, m], Gc[:, m]).real for m in range(4)) * g2).numpy()
        w = p[..., None, None]
        AA = sum(G[:, m] @ Gc[:, m] for m in range(4))
        Ar, AP = (w * G[zero]).sum(1), (w * G).sum(1)
        AM = (w * Gc).sum(1) / -psq[:, None, None]
        g3 = (tr(AA, Ar).real + tr(Ar @ AP, AM).real) / psq
        out["g3"] = (g3 * (4.0 / (2.0 * 3 * 8 * 3 * V))).numpy()
    return out


def _exact_landau(case, dims, seed):
    L = _Landau(_links(dims, seed, *_shape(case)), dims)
    th = None
    for _ in range(2 if case["precision"] == "MIXED" and _bounded(case) else 1):
        th = L.solve(case["algo"], case["accuracy"], case["iters"])
    return L.U, th


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"links": [_flat(_exact_landau(case, d, seed * 64 + i)[0])
                          for i, d in enumerate(_batch_dims(case))]}
    dims = _dims(case)
    if kind == "landau":
        U, th = _exact_landau(case, dims, seed)
        return {"links": _flat(U), "theta": th} if _bounded(case) else {"links": _flat(U)}
    if kind == "coulomb":
        S = _Coulomb(_links(dims, seed, *_shape(case)), dims)
        n = 0
        if case["precision"] == "MIXED":
            S.solve(1e-9, 5000, case["algo"])
            S.reunit()
        th, it = S.solve(case["accuracy"], 5000, case["algo"])
        S.reunit()
        if case["precision"] == "MIXED":
            return {"links": _flat(S.links())}
        return {"links": _flat(S.links()), "theta": th, "iters": it}
    if kind == "heatbath":
        U = _links(dims, seed)
        plaq = np.zeros(case["steps"])
        for i in range(case["steps"]):
            _heatbath_sweep(U, dims, True, 3.0 / case["beta"], int(seed), i)
            for _ in range(case["n_or"]):
                _heatbath_sweep(U, dims, False, 0.0, 0, 0)
            plaq[i] = _plaquette(U)
        return {"links": _flat(U), "plaquette": plaq}
    if kind == "cuts":
        if case["field"] != "LINEAR":
            return None  # a matrix logarithm of every link: minutes in torch
        return _exact_cuts(case, seed)
    pay = prepare(case, seed)["payload"]
    t = np.dtype({8: "f8", 4: "f4"}[case["bytes"]]).newbyteorder(">" if case["big"] else "<")
    r = np.frombuffer(pay, dtype=t)
    u = np.zeros((r.size // case["nreal"], 3, 3), dtype=np.complex128)
    rows = r.astype(np.float64).view(np.complex128).reshape(-1, case["nreal"] // 6, 3)
    u[:, : rows.shape[1]] = rows
    if case["nreal"] == 12:
        u[:, 2] = np.conj(np.cross(u[:, 0], u[:, 1]))
    words = r.astype(r.dtype.newbyteorder("=")).view(np.uint32)
    ck = int(words.sum(dtype=np.uint64) & np.uint64(0xFFFFFFFF))
    return {"links": u.reshape(-1, 4, 3, 3), "payload": np.frombuffer(pay, dtype=np.uint8),
            "checksums": np.array([ck, ck], dtype=np.int64)}
