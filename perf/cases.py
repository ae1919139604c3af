"""Cases of use of the framework, timed through its public entry points.

A case is one pass of a user's program: a noise field turned into a potential
or a power spectrum with Grid_FFT, the source terms of the second and third
order built with a convolver, a whole initial condition of ICGenerator, or a
recorded Batch of them.  Every pass ends where such a program has its results:
device tensors over the library's buffers, or host arrays where the entry point
returns those.

`exact` gives the same results in 64 bits from plain torch: the noise generator
(Philox4x32-10 and Box-Muller), the unitary transforms, the 3/2-padded products
and the LPT recursion are written out there from their definitions.
"""
import math

import numpy as np
import torch

import monofonic_gb300 as mf
from monofonic_gb300 import _lib, ic, serve

SIZES = (16, 32, 64, 96, 128, 192, 256, 384, 512)  # the grid sizes the library accepts

# cosmology::calculator's scalars of the default Cosmology at the two starting redshifts used here
SCALARS = {
    24: {"Dplus": 0.05116311398069919, "vfac": 278.0459699590209},
    49: {"Dplus": 0.025690268235906342, "vfac": 392.8002345716269},
}
PNORM, N_S, H0, OMEGA_M, OMEGA_B, TCMB = 12095.967112802226, 0.9667, 67.74, 0.3099, 0.0488, 2.7255

SHIFTS = {  # sub-lattices of the particle loads, in cells
    "sc": [(0, 0, 0)],
    "bcc": [(0, 0, 0), (0.5, 0.5, 0.5)],
    "fcc": [(0, 0, 0), (0, 0.5, 0.5), (0.5, 0, 0.5), (0.5, 0.5, 0)],
    "rsc": [(0, 0, 0), (0, 0, 0.5), (0, 0.5, 0), (0, 0.5, 0.5), (0.5, 0, 0), (0.5, 0, 0.5), (0.5, 0.5, 0),
            (0.5, 0.5, 0.5)],
}
PAIRS = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))


def listed():
    return [
        # the smallest call: noise and its potential on a 64^3 grid, where launches and latency count
        {"name": "field_n64_f32", "kind": "field", "n": 64, "prec": "f32", "box": 128.0},
        # a large field on a grid that is not a power of two
        {"name": "field_n384_f32", "kind": "field", "n": 384, "prec": "f32", "box": 768.0},
        # the check a user makes of a noise field: P(k) of the default-precision grid
        {"name": "spectrum_n256_f64", "kind": "spectrum", "n": 256, "prec": "f64", "box": 500.0},
        # the 2LPT source of a small grid, term by term, as code written against the convolver builds it
        {"name": "source2_n128_f32", "kind": "source2", "n": 128, "prec": "f32", "box": 256.0, "conv": "orszag"},
        # the same in double precision (the default) on a grid with a factor of three
        {"name": "source2_n192_f64", "kind": "source2", "n": 192, "prec": "f64", "box": 384.0, "conv": "orszag"},
        # the aliased convolver
        {"name": "source2_n256_f32_naive", "kind": "source2", "n": 256, "prec": "f32", "box": 500.0, "conv": "naive"},
        # triple products of the third order, each two chained padded convolutions
        {"name": "triple_n256_f32", "kind": "triple", "n": 256, "prec": "f32", "box": 500.0, "conv": "orszag"},
        # the plain 2LPT run: noise from the host, displacement and velocity fields back to the host
        {"name": "ic_n64_2lpt_fields_host", "kind": "ic", "n": 64, "prec": "f64", "box": 100.0, "z": 49, "order": 2,
         "lattice": "sc", "plt": False, "host": True},
        # 3LPT on a simple cubic lattice, 256^3 particles, in both precisions
        {"name": "ic_n256_3lpt_f64", "kind": "ic", "n": 256, "prec": "f64", "box": 500.0, "z": 24, "order": 3,
         "lattice": "sc", "plt": False, "host": False},
        {"name": "ic_n256_3lpt_f32", "kind": "ic", "n": 256, "prec": "f32", "box": 500.0, "z": 24, "order": 3,
         "lattice": "sc", "plt": False, "host": False},
        # the largest: 3LPT with PLT corrections on a BCC lattice, 2 x 512^3 particles
        {"name": "ic_n512_bcc_plt_f32", "kind": "ic", "n": 512, "prec": "f32", "box": 1000.0, "z": 24, "order": 3,
         "lattice": "bcc", "plt": True, "host": False},
        # many realizations of uneven sizes as one recorded batch
        {"name": "batch_10_f32", "kind": "batch", "sizes": "64 64 64 64 96 96 96 128 128 192", "orders": "2 3 2 3 2 3 2 3 2 3",
         "streams": 8},
    ]


def draw(rng):
    """One more case of the same ranges: every kind, grid size, precision, order and lattice, boxes of 1 to 4 per cell."""
    kind = rng.choice(["field", "field", "spectrum", "source2", "triple", "ic", "ic", "ic", "batch"])
    prec = rng.choice(["f32", "f32", "f64"])
    if kind == "batch":
        n = rng.randint(3, 12)
        return {"kind": kind, "sizes": " ".join(str(rng.choice([64, 96, 128, 192])) for _ in range(n)),
                "orders": " ".join(str(rng.choice([2, 3])) for _ in range(n)), "streams": rng.choice([4, 8])}
    top = {"field": 512, "spectrum": 384, "source2": 256, "triple": 256, "ic": 384}[kind]
    if prec == "f64" and kind == "ic":
        top = 192
    n = rng.choice([s for s in SIZES if s <= top])
    c = {"kind": kind, "n": n, "prec": prec, "box": round(n * rng.uniform(1.0, 4.0), 2)}
    if kind == "spectrum":
        c["prec"] = "f64"
    if kind in ("source2", "triple"):
        # (the aliased convolver takes grids that are a power of two)
        c["conv"] = rng.choice(["orszag", "orszag", "orszag", "naive"]) if n & (n - 1) == 0 else "orszag"
    if kind == "ic":
        lattice = rng.choice(["sc", "sc", "bcc", "bcc", "fcc", "rsc"])
        if n > 256 and lattice == "rsc":
            lattice = "fcc"
        c |= {"z": rng.choice([24, 49]), "order": rng.choice([1, 2, 3, 3]), "lattice": lattice,
              "plt": rng.random() < 0.3, "host": False}
    return c


# --------------------------------------------------------------------------
# what a program has in hand, and one pass
# --------------------------------------------------------------------------
_ctx = None


def _context():
    """the program's one device context"""
    global _ctx
    if _ctx is None:
        torch.zeros(1, device="cuda")
        _ctx = mf.Context(0)
    return _ctx


class _Buffer:
    """library memory as an array; its owner lives as long as a tensor over it"""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": typestr,
                                         "version": 3, "strides": None}


def _tensor(owner, ptr, shape, typestr):
    return torch.as_tensor(_Buffer(owner, ptr, shape, typestr), device="cuda")


def _real_view(g):
    n = g.n
    return _tensor(g, g.device_ptr(), (n, n, n + 2), "<f8" if g.dtype == np.float64 else "<f4")[:, :, :n]


def _k_view(g):
    n = g.n
    return _tensor(g, g.device_ptr(), (n, n, n // 2 + 1), "<c16" if g.dtype == np.float64 else "<c8")


def _noise_seed(seed, i=0):
    return (int(seed) * 1000003 + 7919 * i + 12345) % (1 << 62)


def _noise_field(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.randn((n, n, n), generator=g, dtype=torch.float64, device="cuda")


def _scalars(z):
    return ic.cosmology_scalars(ic.Cosmology(), float(z))


def _ic_config(c):
    f64 = c["prec"] == "f64"
    return ic.ICConfig(ngrid=c["n"], boxlen=c["box"], zstart=float(c["z"]), lpt_order=c["order"], lattice=c["lattice"],
                       precision=c["prec"], plt=c["plt"], lunit=c["box"], vunit=c["box"],
                       out_kind="fields" if c["host"] else "particles", pos64=f64, id64=True)


def prepare(case, seed):
    kind = case["kind"]
    ctx = _context()
    if kind in ("field", "spectrum"):
        g = mf.Grid_FFT(ctx, case["n"], case["box"], case["prec"])
        s = {"kind": kind, "grid": g, "seed": _noise_seed(seed)}
        s["view"] = _real_view(g) if kind == "field" else _k_view(g)
        return s
    if kind in ("source2", "triple"):
        n, box, prec = case["n"], case["box"], case["prec"]
        phi = mf.Grid_FFT(ctx, n, box, prec)
        phi.fill_white_noise(_noise_seed(seed))
        phi.apply_InverseLaplacian()
        out = mf.Grid_FFT(ctx, n, box, prec, "k")
        conv = (mf.OrszagConvolver if case["conv"] == "orszag" else mf.NaiveConvolver)(ctx, n, box, prec)
        ctx.synchronize()
        return {"kind": kind, "phi": phi, "out": out, "conv": conv, "view": _k_view(out)}
    if kind == "ic":
        gen = ic.ICGenerator(ctx, _ic_config(case), _scalars(case["z"]))
        noise = _noise_field(case["n"], seed)
        if case["host"]:
            noise = noise.cpu().numpy()
        else:
            torch.cuda.synchronize()
        return {"kind": kind, "gen": gen, "noise": noise, "host": case["host"]}
    sizes = [int(x) for x in case["sizes"].split()]
    orders = [int(x) for x in case["orders"].split()]
    reqs = [serve.Request(ngrid=n, boxlen=2.0 * n, zstart=24.0, lpt_order=o, lattice="sc", precision="f32",
                          seed=_noise_seed(seed, i), pos64=False, id64=True)
            for i, (n, o) in enumerate(zip(sizes, orders))]
    return {"kind": kind, "batch": serve.Batch(reqs, nstreams=case["streams"]), "sizes": sizes}


def _particles(owner, pos, vel, ids, n, f64):
    t = "<f8" if f64 else "<f4"
    return {"pos": _tensor(owner, pos, (n, 3), t), "vel": _tensor(owner, vel, (n, 3), t), "ids": _tensor(owner, ids, (n,), "<i8")}


def run(state):
    kind = state["kind"]
    if kind == "field":
        g = state["grid"]
        g.fill_white_noise(state["seed"])
        g.FourierTransformForward()
        g.apply_InverseLaplacian()
        g.FourierTransformBackward()
        return {"potential": state["view"]}
    if kind == "spectrum":
        g = state["grid"]
        g.fill_white_noise(state["seed"])
        k, P, eP, count = g.Compute_PowerSpectrum()
        return {"k": k, "P": P, "eP": eP, "count": count, "modes": state["view"]}
    if kind == "source2":
        cv, p, o = state["conv"], state["phi"], state["out"]
        cv.convolve_SumOfHessians(p, (0, 0), p, (1, 1), (2, 2), mf.op.assign_to(o))
        cv.convolve_Hessians(p, (1, 1), p, (2, 2), mf.op.add_to(o))
        cv.convolve_Hessians(p, (0, 1), p, (0, 1), mf.op.subtract_from(o))
        cv.convolve_Hessians(p, (0, 2), p, (0, 2), mf.op.subtract_from(o))
        cv.convolve_Hessians(p, (1, 2), p, (1, 2), mf.op.subtract_from(o))
        return {"source": state["view"]}
    if kind == "triple":
        cv, p, o = state["conv"], state["phi"], state["out"]
        cv.convolve_Hessians(p, (0, 0), p, (1, 1), p, (2, 2), mf.op.assign_to(o))
        cv.convolve_Hessians(p, (0, 1), p, (0, 2), p, (1, 2), mf.op.multiply_add_to(o, 2.0))
        return {"sum": state["view"]}
    if kind == "ic":
        gen = state["gen"]
        if state["host"]:
            gen.set_noise(state["noise"])
            pos, vel, _ = gen.run()
            return {"pos": pos, "vel": vel}
        gen.set_noise_device(state["noise"].data_ptr())
        pos, vel, ids = gen.run(to_host=False)
        return _particles(gen, pos, vel, ids, gen.npart, gen.cfg.pos64)
    b = state["batch"]
    b.run()
    out = []
    for i, n in enumerate(state["sizes"]):
        p = _lib.mf_particles()
        b._check(mf.lib().mf_batch_particles(b.ptr, i, p), "mf_batch_particles")
        out.append(_particles(b, p.pos, p.vel, p.ids, n ** 3, False))
    return out


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _fft_flops(n):
    return 2.5 * n ** 3 * math.log2(float(n) ** 3)


def _ic_work(n, order, lattice, size, id_bytes=8, noise_bytes=8):
    """bytes: the noise in, the particles (or two fields) out; flops: the noise's
    transform, each distinct padded operand and product once, three
    components of positions and velocities on each sub-lattice"""
    m, sub = 3 * n // 2, len(SHIFTS[lattice])
    padded = {1: 0, 2: 7, 3: 27}[order]
    return {"bytes": n ** 3 * noise_bytes + sub * n ** 3 * (6 * size + id_bytes),
            "flops": (1 + 6 * sub) * _fft_flops(n) + padded * _fft_flops(m)}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [_ic_work(int(n), int(o), "sc", 4, noise_bytes=0)
             for n, o in zip(case["sizes"].split(), case["orders"].split())]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    n, size = case["n"], 8 if case["prec"] == "f64" else 4
    if kind == "ic":
        return _ic_work(n, case["order"], case["lattice"], size, id_bytes=0 if case["host"] else 8)
    grid = n * n * (n + 2) * size
    if kind == "field":
        return {"bytes": n ** 3 * size, "flops": 2 * _fft_flops(n)}
    if kind == "spectrum":
        return {"bytes": grid, "flops": _fft_flops(n)}
    m = 3 * n // 2 if case["conv"] == "orszag" else n
    # source2: six Hessians and one sum of products; triple: six Hessians, two pairs there and back, one sum
    # (the aliased convolver's triple product needs no pair transform)
    t = 7 if kind == "source2" else (11 if case["conv"] == "orszag" else 7)
    return {"bytes": 2 * grid, "flops": t * _fft_flops(m)}


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------
def _white_noise(n, seed):
    """N(0,1) draws: cells 2p, 2p+1 from Philox4x32-10 (Salmon et al. 2011) at counter p, Box-Muller"""
    p = torch.arange(n ** 3 // 2, dtype=torch.int64, device="cuda")
    lo = 0xFFFFFFFF
    c = [p & lo, p >> 32, torch.zeros_like(p), torch.zeros_like(p)]
    k0, k1 = seed & lo, (seed >> 32) & lo
    for _ in range(10):
        a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # 64-bit products, wrapped; the halves are masked
        c = [((b >> 32) & lo) ^ c[1] ^ k0, b & lo, ((a >> 32) & lo) ^ c[3] ^ k1, a & lo]
        k0, k1 = (k0 + 0x9E3779B9) & lo, (k1 + 0xBB67AE85) & lo
    b1 = (c[1] << 21) | (c[0] >> 11)
    b2 = (c[3] << 21) | (c[2] >> 11)
    r = torch.sqrt(-2.0 * torch.log((b1.double() + 0.5) * 2.0 ** -53))
    t = (b2.double() + 0.5) * 2.0 ** -53 * (2 * math.pi)
    return torch.stack([r * torch.cos(t), r * torch.sin(t)], -1).reshape(n, n, n)


class _Exact:
    """Unitary transforms, gradients and products on an n^3 grid, with Grid_FFT's conventions"""

    def __init__(self, n, box, orszag=True):
        self.n, self.box, self.orszag = n, box, orszag
        self.m = 3 * n // 2 if orszag else n
        i = torch.arange(n, device="cuda")
        f = (i - torch.where(i > n // 2, n, 0)).double() * (2 * math.pi / box)
        g = torch.where(i == n // 2, torch.zeros_like(f), f)  # the gradient is zero at the Nyquist index
        kz = n // 2 + 1
        self.k = (f[:, None, None], f[None, :, None], f[None, None, :kz])
        self.g = (g[:, None, None], g[None, :, None], g[None, None, :kz])
        self.k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2

    def r2c(self, x):
        return torch.fft.rfftn(x) / math.sqrt(self.n ** 3)

    @staticmethod
    def _back(X, m):
        """complex over x and y, then the half-complex z lines whose end terms count by their real parts"""
        Y = torch.fft.ifftn(X, dim=(0, 1), norm="forward")
        Y[:, :, 0].imag.zero_()
        Y[:, :, m // 2].imag.zero_()
        return torch.fft.irfft(Y, n=m, dim=2, norm="forward")

    def c2r(self, X):
        return self._back(X, self.n) / math.sqrt(self.n ** 3)

    def inverse_laplacian(self, X):
        Y = -X / self.k2
        Y[0, 0, 0] = 0
        return Y

    def hessian(self, X, a, b):
        return -(self.g[a] * self.g[b]) * X

    def padded(self, X):
        """the operand in (padded) real space"""
        n, m, h = self.n, self.m, self.n // 2
        if not self.orszag:
            return self._back(X, n) / math.sqrt(n ** 3)
        P = torch.zeros((m, m, m // 2 + 1), dtype=torch.complex128, device="cuda")
        lo, hi = slice(0, h + 1), slice(m - h + 1, m)
        a, b = slice(0, h + 1), slice(h + 1, n)
        for d, s in ((lo, a), (hi, b)):
            for e, t in ((lo, a), (hi, b)):
                P[d, e, : h + 1] = X[s, t]
        return self._back(P, m) * (1.5 ** 1.5 / math.sqrt(m ** 3))

    def product(self, x):
        """a real-space product back in the n-cube, Nyquist planes zeroed for the dealiased form"""
        n, m, h = self.n, self.m, self.n // 2
        P = torch.fft.rfftn(x)
        if not self.orszag:
            return P / math.sqrt(n ** 3)
        X = torch.empty((n, n, h + 1), dtype=torch.complex128, device="cuda")
        lo, hi = slice(0, h + 1), slice(m - h + 1, m)
        a, b = slice(0, h + 1), slice(h + 1, n)
        for d, s in ((lo, a), (hi, b)):
            for e, t in ((lo, a), (hi, b)):
                X[s, t] = P[d, e, : h + 1]
        X *= math.sqrt(n ** 3) / m ** 3
        X[h], X[:, h], X[:, :, h] = 0, 0, 0
        return X

    def hessians(self, X):
        H = {p: self.padded(self.hessian(X, *p)) for p in PAIRS}
        return lambda a, b: H[(min(a, b), max(a, b))]

    def phi2_source(self, H):
        return (H(0, 0) * (H(1, 1) + H(2, 2)) + H(1, 1) * H(2, 2) - H(0, 1) ** 2 - H(0, 2) ** 2 - H(1, 2) ** 2)


def _transfer(k):
    """Eisenstein & Hu (1998), the full fit with baryons, k in h/Mpc"""
    h = H0 * 0.01
    om = OMEGA_M * h * h
    fb = OMEGA_B / OMEGA_M
    ob = om * fb
    th = TCMB / 2.7
    z_eq = 2.50e4 * om / th ** 4
    k_eq = 0.0746 * om / th ** 2
    b1 = 0.313 * om ** -0.419 * (1 + 0.607 * om ** 0.674)
    b2 = 0.238 * om ** 0.223
    z_d = 1291 * om ** 0.251 / (1 + 0.659 * om ** 0.828) * (1 + b1 * ob ** b2)
    R_d = 31.5 * ob / th ** 4 * 1000 / (1 + z_d)
    R_eq = 31.5 * ob / th ** 4 * 1000 / z_eq
    s = 2 / 3 / k_eq * math.sqrt(6 / R_eq) * math.log((math.sqrt(1 + R_d) + math.sqrt(R_d + R_eq)) / (1 + math.sqrt(R_eq)))
    k_silk = 1.6 * ob ** 0.52 * om ** 0.73 * (1 + (10.4 * om) ** -0.95)
    a1 = (46.9 * om) ** 0.670 * (1 + (32.1 * om) ** -0.532)
    a2 = (12.0 * om) ** 0.424 * (1 + (45.0 * om) ** -0.582)
    alpha_c = a1 ** -fb * a2 ** -(fb ** 3)
    beta_c = 1 / (1 + 0.944 / (1 + (458 * om) ** -0.708) * ((1 - fb) ** ((0.395 * om) ** -0.0266) - 1))
    y = z_eq / (1 + z_d)
    G = y * (-6 * math.sqrt(1 + y) + (2 + 3 * y) * math.log((math.sqrt(1 + y) + 1) / (math.sqrt(1 + y) - 1)))
    alpha_b = 2.07 * k_eq * s * (1 + R_d) ** -0.75 * G
    beta_node = 8.41 * om ** 0.435
    beta_b = 0.5 + fb + (3 - 2 * fb) * math.sqrt((17.2 * om) ** 2 + 1)
    kk = k * h
    q = kk / 13.41 / k_eq
    x = kk * s
    lb, ln = torch.log(2.718282 + 1.8 * beta_c * q), torch.log(2.718282 + 1.8 * q)
    tail = 386 / (1 + 69.9 * q ** 1.08)
    C0, C1 = 14.2 + tail, 14.2 / alpha_c + tail
    f = 1 / (1 + (x / 5.4) ** 4)
    Tc = f * lb / (lb + C0 * q * q) + (1 - f) * lb / (lb + C1 * q * q)
    xt = kk * s * (1 + (beta_node / x) ** 3) ** (-1 / 3)
    Tb = torch.sin(xt) / xt * (ln / (ln + C0 * q * q) / (1 + (x / 5.2) ** 2)
                               + alpha_b / (1 + (beta_b / x) ** 3) * torch.exp(-((kk / k_silk) ** 1.4)))
    return fb * Tb + (1 - fb) * Tc


def _exact_ic(n, box, z, order, lattice, noise, fields):
    """displacements and velocities (or particles) of the LPT run from an n^3 noise field, box units"""
    E = _Exact(n, box)
    D, vf = SCALARS[z]["Dplus"], SCALARS[z]["vfac"]
    k = torch.sqrt(E.k2)
    k[0, 0, 0] = 1.0
    amp = k ** (0.5 * N_S) * _transfer(k) * math.sqrt(PNORM)
    wn = E.r2c(noise) / (box / n / 2 / math.pi) ** 1.5
    phi = -wn * amp / (k * k)
    phi[0, 0, 0] = 0
    P2 = P3 = None
    A = None
    if order > 1:
        H = E.hessians(phi)
        P2 = E.inverse_laplacian(E.product(E.phi2_source(H)))
    if order > 2:
        G = E.hessians(P2)
        T = lambda x: E.padded(E.product(x))  # noqa: E731  the first stage of a triple product
        src = T(H(0, 0) * H(1, 1)) * H(2, 2) + 2 * T(H(0, 1) * H(0, 2)) * H(1, 2)
        src -= T(H(1, 2) ** 2) * H(0, 0) + T(H(0, 2) ** 2) * H(1, 1) + T(H(0, 1) ** 2) * H(2, 2)
        src -= 5 / 7 * (H(0, 0) * (G(1, 1) + G(2, 2)) + H(1, 1) * (G(2, 2) + G(0, 0)) + H(2, 2) * (G(0, 0) + G(1, 1)))
        src += 10 / 7 * (H(0, 1) * G(0, 1) + H(0, 2) * G(0, 2) + H(1, 2) * G(1, 2))
        P3 = E.inverse_laplacian(E.product(src))
        A = []
        for d in range(3):
            p, q = (d + 1) % 3, (d + 2) % 3
            s = G(d, p) * H(d, q) - G(d, q) * H(d, p) + H(p, q) * (G(p, p) - G(q, q)) - G(p, q) * (H(p, p) - H(q, q))
            A.append(E.inverse_laplacian(E.product(s)))
    out = []
    for vel in (False, True):
        w = [-D, -3 / 7 * D ** 2, 1 / 3 * D ** 3, 1 / 7 * D ** 3]
        if vel:
            w = [vf * w[0], 2 * vf * w[1], 3 * vf * w[2], 3 * vf * w[3]]
        tot = w[0] * phi
        if order > 1:
            tot = tot + w[1] * P2
        if order > 2:
            tot = tot + w[2] * P3
        comp = []
        for d in range(3):
            X = 1j * E.g[d] * tot
            if A:
                p, q = (d + 1) % 3, (d + 2) % 3
                X = X + w[3] * 1j * (E.g[p] * A[q] - E.g[q] * A[p])
            X[0, 0, 0] = 0
            r, last, sub = E.c2r(X), (0, 0, 0), []
            for sh in SHIFTS[lattice]:
                if sh != last:  # the field is read through relative shifts, one after the other
                    step = [a - b for a, b in zip(sh, last)]
                    ph = sum(s * kk for s, kk in zip(step, E.k)) * (box / n)
                    r = E.c2r(E.r2c(r) * torch.exp(1j * ph))
                    last = sh
                v = r  # in units of the box: lunit / L = 1
                if not vel and not fields:
                    idx = torch.arange(n, device="cuda", dtype=torch.float64).reshape([-1 if e == d else 1 for e in range(3)])
                    v = r + (idx + sh[d]) / n * box
                sub.append(v.reshape(-1))
            comp.append(torch.cat(sub))
        out.append(torch.stack(comp).reshape(3, n, n, n) if fields else torch.stack(comp, -1))
    return {"pos": out[0], "vel": out[1], "ids": None} if not fields else {"pos": out[0], "vel": out[1]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sizes, orders = [int(x) for x in case["sizes"].split()], [int(x) for x in case["orders"].split()]
        return [_exact_ic(n, 2.0 * n, 24, o, "sc", _white_noise(n, _noise_seed(seed, i)), False)
                for i, (n, o) in enumerate(zip(sizes, orders))]
    n, box = case["n"], case["box"]
    if kind == "ic":
        if case["plt"]:
            return None  # the eigenmodes of the lattice's dynamical matrix take too long here
        r = _exact_ic(n, box, case["z"], case["order"], case["lattice"], _noise_field(n, seed), case["host"])
        return {k: v.cpu().numpy() for k, v in r.items()} if case["host"] else r
    E = _Exact(n, box, case.get("conv") != "naive")
    wn = E.r2c(_white_noise(n, _noise_seed(seed)))
    if kind == "field":
        return {"potential": E.c2r(E.inverse_laplacian(wn))}
    if kind == "spectrum":
        # |k| rounded as the library rounds it: modes of integer norm lie on bin edges
        kf = 2 * math.pi / box
        b = (torch.sqrt(E.k2) / torch.full_like(E.k2, kf)).to(torch.int64)  # divided, not times a reciprocal
        nb = int(kf * (n // 2) / kf)
        ok = (torch.sqrt(E.k2) >= kf) & (torch.sqrt(E.k2) < kf * (n // 2))
        w = torch.full_like(E.k2, 2.0)
        w[:, :, 0] = 1.0
        p = wn.real ** 2 + wn.imag ** 2
        hist = lambda x: torch.bincount(b[ok], weights=(w * x)[ok], minlength=nb)[:nb].cpu().numpy()  # noqa: E731
        cnt, sp, sp2, sk = hist(torch.ones_like(p)), hist(p), hist(p * p), hist(torch.sqrt(E.k2))
        f = box ** 3 / (2 * math.pi) ** 3 / n ** 3
        with np.errstate(all="ignore"):
            has = cnt > 0
            P = np.where(has, sp / cnt * f, sp)
            eP = np.where(has, np.sqrt(sp2 / cnt - P * P) / np.sqrt(cnt) * f, sp2)
            kk = np.where(has, sk / cnt, sk)
        return {"k": kk, "P": P, "eP": eP, "count": None, "modes": wn}
    phi = E.inverse_laplacian(wn)
    H = E.hessians(phi)
    if kind == "source2":
        return {"source": E.product(E.phi2_source(H))}
    T = (lambda x: E.padded(E.product(x))) if E.orszag else (lambda x: x)
    return {"sum": E.product(T(H(0, 0) * H(1, 1)) * H(2, 2)) + 2.0 * E.product(T(H(0, 1) * H(0, 2)) * H(1, 2))}
