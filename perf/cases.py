"""The workloads this framework is timed on, each through the calls that a
program makes: the nonsubsampled and the decimated surfacelet transform, their
gradients, the denoiser and bfloat16 coefficients, over the volume sizes they
are used at.

`listed()` names the cases, `draw(rng)` gives one more of the same ranges,
`prepare` and `run` execute a case, `work` counts the bytes and operations a
pass cannot do without, and `exact` restates the transforms in 64-bit torch.
"""

import importlib.util
import math
import os
import sys
from fractions import Fraction

import torch


def _package():
    """The package (its folder name is not an identifier)."""
    name = "surfacelets_b200"
    if name in sys.modules:
        return sys.modules[name]
    folder = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "surfacelets.jl_b200")
    spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"),
                                                  submodule_search_locations=[folder])
    mod = importlib.util.module_from_spec(spec)
    sys.modules[name] = mod
    spec.loader.exec_module(mod)
    return mod


# A case: `bank` "ns" or "dec", `do` what the pass runs, the volume n1 x n2 x
# n3, the directional levels coarse to fine as digits, `type` of the volume,
# and for the decimated transform its pyramid ratio.


def _case(name, bank, do, dims, levels, kind="float32", ratio=0):
    c = {"bank": bank, "do": do, "n1": dims[0], "n2": dims[1], "n3": dims[2], "levels": levels, "type": kind,
         "ratio": ratio}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest volumes in use (a patch, a unit test, the benchmark suite's 32^3): launches and latency
        _case("ns_analyze_32", "ns", "analyze", (32, 32, 32), "12"),
        # a patch or a small scan analyzed and put back together
        _case("ns_roundtrip_64", "ns", "roundtrip", (64, 64, 64), "223"),
        # the usual volume with the usual parameters, each direction by itself
        _case("ns_analyze_128", "ns", "analyze", (128, 128, 128), "223"),
        _case("ns_synthesize_128", "ns", "synthesize", (128, 128, 128), "223"),
        # a scan whose axes are round numbers and no powers of two
        _case("ns_roundtrip_120x100x90", "ns", "roundtrip", (120, 100, 90), "122"),
        # a scan as it comes, odd and prime lengths (the grid of a 2 mm brain template)
        _case("ns_roundtrip_91x109x91", "ns", "roundtrip", (91, 109, 91), "12"),
        # reconstruction from complex data: the transform, its adjoint and both gradients
        _case("ns_grad_complex_96", "ns", "grad", (96, 96, 96), "12", "complex64"),
        # coefficients kept in 16 bits, axes of different lengths
        _case("ns_bf16_160x128x96", "ns", "bf16", (160, 128, 96), "122"),
        # the largest volume: denoised without its coefficients ever being held
        _case("ns_denoise_256", "ns", "denoise", (256, 256, 256), "2233"),
        # the decimated transform at its usual size, both directions
        _case("dec_roundtrip_128", "dec", "roundtrip", (128, 128, 128), "223", ratio=2),
        # the decimated transform inside an optimiser, with the pyramid ratio it has by default
        _case("dec_grad_96", "dec", "grad", (96, 96, 96), "12", ratio=1.5),
        # a large decimated volume with unequal axes, default pyramid
        _case("dec_roundtrip_192x144x96", "dec", "roundtrip", (192, 144, 96), "122", ratio=1.5),
    ]


_ROUND = (24, 32, 36, 40, 48, 54, 60, 64, 72, 80, 90, 96, 100, 108, 112, 120, 128, 140, 144, 150, 160, 176, 180, 192,
          200, 216, 224, 240, 256)


def draw(rng):
    sfl = _package()
    while True:
        if rng.random() < 0.3:
            ratio = rng.choice([1.5, 1.5, 2])
            axes = (48, 72, 96, 120, 144, 168, 192, 240) if ratio == 1.5 else (32, 48, 64, 80, 96, 112, 128, 160, 192)
            c = _case(None, "dec", rng.choice(["roundtrip", "grad"]), [rng.choice(axes) for _ in range(3)],
                      rng.choice(["1", "2", "11", "12", "22", "112", "122", "223"]), ratio=ratio)
            if rng.random() < 0.2:
                c["type"] = "complex64"
        else:
            do = rng.choice(["analyze", "synthesize", "roundtrip", "roundtrip", "grad", "bf16", "denoise"])
            lo, hi = 24, 256
            kind = rng.random()
            if kind < 0.2:       # a cube of a usual length
                dims = [rng.choice((32, 64, 96, 128, 160))] * 3
            elif kind < 0.75:    # round lengths, spread over their logarithm
                dims = []
                for _ in range(3):
                    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
                    dims.append(min(_ROUND, key=lambda r: abs(math.log(r / want))))
            else:                # any lengths, odd ones among them
                dims = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3)]
            c = _case(None, "ns", do, dims, rng.choice(["1", "12", "13", "22", "112", "122", "223"]))
            if do not in ("bf16", "denoise") and rng.random() < 0.25:
                c["type"] = "complex64"
        dims = (c["n1"], c["n2"], c["n3"])
        try:   # sizes that the transform refuses (an empty scale, an axis that does not divide) are drawn again
            sizes = sfl.subband_sizes(_transform(c), dims)
        except sfl.ArgumentError:
            continue
        coefs = sum(math.prod(s) for s in sizes) * (2 if c["type"] == "complex64" else 1)
        # at most the coefficients of 128^3 with levels 2, 2, 3 (its cost is below the largest listed case's)
        if coefs <= 128 ** 3 * 49:
            return c


def _transform(c):
    sfl = _package()
    levels = [int(d) for d in c["levels"]]
    if c["bank"] == "ns":
        return sfl.NSSurfacelet(direction_levels=levels)
    return sfl.Surfacelet(direction_levels=levels, pyramid_ratio=c["ratio"])


def _colmajor(t):
    """The same shape and values, axis 1 fastest."""
    rev = tuple(reversed(range(t.dim())))
    return t.permute(*rev).contiguous().permute(*rev)


def _phantom(dims, gen, complex_):
    """Twelve ellipsoids and noise; complex volumes carry a smooth phase."""
    g = [torch.linspace(-1, 1, n, device="cuda").reshape([-1 if a == d else 1 for a in range(3)])
         for d, n in enumerate(dims)]
    x = torch.zeros(dims, device="cuda")
    p = torch.rand((12, 7), generator=gen, device="cuda").tolist()
    for q in p:
        r = sum(((g[d] - (1.2 * q[d] - 0.6)) / (0.1 + 0.5 * q[3 + d])) ** 2 for d in range(3))
        x += (0.2 + 0.8 * q[6]) * (r < 1)
    x += 0.05 * torch.randn(dims, generator=gen, device="cuda")
    if complex_:
        x = x * torch.exp(1j * (p[0][0] * g[0] + p[1][0] * g[1] + p[2][0] * g[2]))
    return _colmajor(x.to(torch.complex64 if complex_ else torch.float32))


def _inputs(c, seed):
    """The arrays a pass reads, from the seed alone."""
    dims = (c["n1"], c["n2"], c["n3"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    cplx = c["type"] == "complex64"
    dt = torch.complex64 if cplx else torch.float32
    s = {}
    if c["do"] != "synthesize":
        s["x"] = _phantom(dims, gen, cplx)
    if c["do"] in ("synthesize", "grad"):
        sfl = _package()
        sizes = sfl.subband_sizes(_transform(c), dims)
        shape = dims + (len(sizes),) if c["bank"] == "ns" else (sum(math.prod(z) for z in sizes),)
        rev = tuple(reversed(range(len(shape))))
        make = lambda: torch.randn(shape[::-1], generator=gen, device="cuda", dtype=dt).permute(*rev)   # noqa: E731
        s["c"] = make()
        if c["do"] == "grad":
            s["gc"] = make()
            s["gx"] = _colmajor(torch.randn(dims, generator=gen, device="cuda", dtype=dt))
    return s


_TAU = 0.05


def prepare(case, seed):
    sfl = _package()
    s = _inputs(case, seed)
    s["do"] = case["do"]
    s["ws"] = sfl.make_workspace(_transform(case), case["type"], (case["n1"], case["n2"], case["n3"]))
    return s


def run(s):
    sfl = _package()
    ws, do = s["ws"], s["do"]
    if do == "analyze":
        return sfl.analyze(ws, s["x"])
    if do == "synthesize":
        return sfl.synthesize(ws, s["c"])
    if do == "roundtrip":
        c = sfl.analyze(ws, s["x"])
        return c, sfl.synthesize(ws, c)
    if do == "bf16":
        c, scales = sfl.analyze_bf16(ws, s["x"])
        return c, scales, sfl.synthesize_bf16(ws, c, scales)
    if do == "denoise":
        return sfl.denoise(ws, s["x"], _TAU)
    x = s["x"].detach().requires_grad_()
    a = sfl.analyze_ad(ws, x)
    a.backward(s["gc"])
    c = s["c"].detach().requires_grad_()
    y = sfl.synthesize_ad(ws, c)
    y.backward(s["gx"])
    return a.detach(), x.grad, y.detach(), c.grad


def _coefficients(case):
    """Number of values of the coefficients and of subbands."""
    sizes = _package().subband_sizes(_transform(case), (case["n1"], case["n2"], case["n3"]))
    return sum(math.prod(s) for s in sizes), len(sizes)


def work(case):
    n = case["n1"] * case["n2"] * case["n3"]
    m, subbands = _coefficients(case)
    ch = 2 if case["type"] == "complex64" else 1
    directions = {"analyze": 1, "synthesize": 1, "roundtrip": 2, "bf16": 2, "denoise": 2, "grad": 4}[case["do"]]
    values = {"analyze": n + m, "synthesize": n + m, "roundtrip": 2 * (n + m), "bf16": 2 * n + m, "denoise": 2 * n,
              "grad": 4 * (n + m)}[case["do"]]
    # one real FFT of the volume and one of every subband's points, each direction
    flops = ch * directions * 2.5 * (n + m) * math.log2(n)
    return {"bytes": 4 * ch * values, "flops": flops}


# ── the transforms in 64 bits ────────────────────────────────────────────────

_D = {"dtype": torch.float64, "device": "cuda"}


def _rcos(n, w, t):
    """Square root of the raised-cosine lowpass on an n-point DFT axis, and its edge."""
    P = math.ceil(Fraction(n, 2) * (w + t))
    Q = math.floor(Fraction(n, 2) * (w - t))
    k = torch.arange(n, **_D)
    f = torch.where(k <= n // 2, k, n - k)
    u = ((P - f) / (P - Q)).clamp(0, 1)
    return torch.where(f <= P, torch.sqrt((1 - torch.cos(math.pi * u)) / 2), torch.zeros_like(f)), P


def _split(x):
    """The half-band step of order 1: ((1+x)/2)^2 (1 + 2 (1-x)/2)."""
    return ((1 + x) / 2) ** 2 * (1 + (1 - x))


class _NS64:
    def __init__(self, dims, levels, order=12):
        self.dims, self.levels, self.J = dims, levels, len(levels)
        n, self.h = dims, (dims[0] // 2 + 1, dims[1], dims[2])
        b = []
        for d in range(3):
            s = torch.sin(math.pi * torch.arange(self.h[d], **_D) / n[d]) ** 2
            b.append(torch.stack([math.comb(order, j) * s ** j * (1 - s) ** (order - j) for j in range(order + 1)]))
        j = torch.arange(order + 1, **_D)
        s3 = torch.sign(j[:, None, None] - torch.maximum(j[None, :, None], j[None, None, :]))
        s2 = torch.sign(j[:, None] - j[None, :])
        m1 = _split(torch.einsum("abc,ax,by,cz->xyz", s3, *b))
        m2 = _split(torch.einsum("ab,ay,bz->yz", s2, b[1], b[2]))[None]
        self.hg = [torch.sqrt(w.clamp(min=0)) for w in (m1, (1 - m1) * m2, (1 - m1) * (1 - m2))]
        acc, self.band = [torch.ones(k, **_D) for k in self.h], []
        for lv in range(1, self.J + 1):
            l = [_rcos(n[d], Fraction(1, 2 ** lv), Fraction(1, 3 * 2 ** lv))[0][:self.h[d]] for d in range(3)]
            self.band.append(self._outer(acc) * torch.sqrt((1 - self._outer(l) ** 2).clamp(min=0)))
            acc = [p * q for p, q in zip(acc, l)]
        self.low = self._outer(acc)

    @staticmethod
    def _outer(v):
        return v[0][:, None, None] * v[1][None, :, None] * v[2][None, None, :]

    def _wedges(self, ref, tr, level):
        """Square-rooted wedge planes of axes (ref, tr), laid out on the half grid."""
        if level == 0:
            return [torch.ones((1, 1, 1), **_D)]
        w = []
        for d in (ref, tr):
            k = torch.arange(self.h[d], **_D)
            w.append(torch.where(2 * k > self.dims[d], k - self.dims[d], k) * (2 * math.pi / self.dims[d]))
        own = [(2 * torch.arange(self.h[d], device="cuda")) % self.dims[d] == 0 for d in (ref, tr)]
        R, T = w[0][:, None].expand(-1, len(w[1])), w[1][None].expand(len(w[0]), -1)
        s = torch.where(own[0][:, None], T.abs() / R.abs(), torch.where(own[1][None], T / R.abs(), T / R))
        s = torch.where(R == 0, torch.zeros_like(s), s)
        nw = 1 << level
        step = [torch.ones_like(s)] + [_split(((s + 1 - 2 * i / nw) * (nw / 2)).clamp(-1, 1)) for i in range(1, nw)] + \
               [torch.zeros_like(s)]
        shape = [1, 1, 1]
        shape[ref], shape[tr] = len(w[0]), len(w[1])
        planes = [torch.sqrt((step[i] - step[i + 1]).clamp(min=0)) for i in range(nw)]
        return [(p if ref < tr else p.T).reshape(shape) for p in planes]

    def masks(self):
        """(0-based subband, its mask), the lowpass last."""
        s = 1
        for j, level in enumerate(self.levels):
            for i in range(3):
                a, b = [d for d in range(3) if d != i]
                G = self.band[self.J - 1 - j] * self.hg[i]
                for wa in self._wedges(i, a, (level + 1) // 2):
                    for wb in self._wedges(i, b, level // 2):
                        yield s, G * wa * wb
                        s += 1
        yield 0, self.low

    def fft(self, x):
        return torch.fft.rfftn(x, dim=(1, 2, 0))

    def ifft(self, X):
        return torch.fft.irfftn(X, s=(self.dims[1], self.dims[2], self.dims[0]), dim=(1, 2, 0))

    def analyze(self, x):
        X = self.fft(x)
        count = 1 + sum(3 << v for v in self.levels)
        c = torch.empty((count,) + tuple(reversed(self.dims)), **_D).permute(3, 2, 1, 0)
        for s, M in self.masks():
            c[..., s] = self.ifft(X * M)
        return c

    def synthesize(self, c):
        return self.ifft(sum(self.fft(c[..., s].double()) * M for s, M in self.masks()))

    def denoise(self, x, tau):
        X, A = self.fft(x), 0
        for s, M in self.masks():
            c = self.ifft(X * M)
            if s:
                c = torch.sign(c) * (c.abs() - tau).clamp(min=0)
            A = A + self.fft(c) * M
        return self.ifft(A)


class _Dec64:
    LADDER = (-0.6299909650161403, -0.19294788893803155, -0.09719811683520764, -0.05257765509290852,
              -0.027224347419537415, -0.014421093056370137)

    def __init__(self, dims, levels, ratio):
        first, later = {1.5: ((Fraction(1, 2), Fraction(1, 7), Fraction(3, 2)), (Fraction(3, 8), Fraction(1, 9), 2)),
                        2: ((Fraction(1, 3), Fraction(1, 7), 2),) * 2}[ratio]
        self.dims, self.lv, n = dims, [], tuple(dims)
        for j in range(len(levels)):
            w, t, D = first if j == 0 else later
            low = tuple(int(k / D) for k in n)
            at, to, prof = [], [], []
            for d in range(3):
                f, P = _rcos(n[d], w, t)
                at.append(torch.cat([torch.arange(P + 1), torch.arange(n[d] - P, n[d])]).cuda())
                to.append(torch.cat([torch.arange(P + 1), torch.arange(low[d] - P, low[d])]).cuda())
                prof.append(f[at[d]])
            level = levels[len(levels) - 1 - j]
            self.lv.append({"n": n, "low": low, "D": float(D) ** 1.5, "at": at, "to": to, "L": _NS64._outer(prof),
                            "V": self._hourglass(n), "stages": [self._stages(n, K, level) for K in range(3)],
                            "parts": [self._parts(K, level) for K in range(3)]})
            n = low

    @staticmethod
    def _parts(K, level):
        a, b = [d for d in range(3) if d != K]
        p = [1, 1, 1]
        p[a], p[b] = 1 << ((level + 1) // 2), 1 << (level // 2)
        return p

    @staticmethod
    def _hourglass(n, size=15, beta=2.5, power=4):
        def bessel(x):
            x, y, z, k = x / 2, 1.0, 1.0, 1
            while True:
                z *= x / k
                k += 1
                y += z * z
                if z * z <= 1e-10 * y:
                    return y
        half = size // 2
        u = torch.arange(-half, half + 1, **_D)
        win = torch.tensor([bessel(beta * math.sqrt(1 - (i / half) ** 2)) for i in range(-half, half + 1)], **_D)
        win = win / bessel(beta) * torch.sinc(u / 2)

        def plane(nK, nm):
            a = 2 * math.pi * torch.arange(nK, **_D)[:, None] / nK + math.pi
            b = 2 * math.pi * torch.arange(nm, **_D)[None] / nm
            even, odd = (u % 2 == 0), (u % 2 != 0)
            f = lambda w, s: (win[s, None, None] * torch.cos(u[s, None, None] * w)).sum(0)   # noqa: E731
            p, q = (a + b) / 2, (a - b) / 2
            return (f(p, even) * f(q, even) + f(p, odd) * f(q, odd)) ** power
        hg = []
        for K in range(3):
            acc = torch.ones(n, **_D)
            for m in range(3):
                if m != K:
                    P = plane(n[K], n[m])
                    shape = [n[d] if d in (K, m) else 1 for d in range(3)]
                    acc = acc * (P if K < m else P.T).reshape(shape)
            hg.append(acc)
        total = sum(hg)
        return [torch.sqrt(3 * hg[K] / total).narrow(K, 0, n[K] // 2 + 1) for K in range(3)]

    def _stages(self, n, K, level):
        """(axis, half block, analysis channels, synthesis channels) in analysis order."""
        b = lambda w: 2 * sum(t * torch.sin((2 * i + 1) * w) for i, t in enumerate(self.LADDER))   # noqa: E731
        out = []
        for m in range(3):
            parts = self._parts(K, level)[m]
            for le in range(1, parts.bit_length()):
                W = n[m] >> (le - 1)
                c = torch.arange(n[m], device="cuda")
                wK = 2 * math.pi * torch.arange(n[K] // 2 + 1, **_D)[:, None] / n[K]
                wm = 2 * math.pi * (c % W).double()[None] / W + ((1 << (le - 1)) - 1 - 2 * (c // W))[None] * wK
                B, r = -b(wK) * b(wm), 1 / math.sqrt(2.0)
                turn = torch.polar(torch.ones_like(wm), wm)
                f = (0.5 * r * (1 + B) + 0j, 0.5 * r * turn * (2 - B - B * B),
                     r * (2 + B - B * B) + 0j, r * turn.conj() * (1 - B))
                shape = [n[K] // 2 + 1 if d == K else n[m] if d == m else 1 for d in range(3)]
                f = [(v if K < m else v.T).reshape(shape) for v in f]
                out.append((m, n[m] >> le, f[:2], f[2:]))
        return out

    @staticmethod
    def _halves(S, m, b):
        v = S.unflatten(m, (-1, 2, b))
        return v.select(m + 1, 0), v.select(m + 1, 1)

    def _stage(self, S, m, b, f, back):
        A, B = self._halves(S, m, b)
        (f0a, f0b), (f1a, f1b) = (self._halves(g, m, b) for g in f)
        p, q = (f0a * A + f1a * B, f0b * A + f1b * B) if back else (f0a * A + f0b * B, f1a * A + f1b * B)
        return torch.stack([p, q], m + 1).flatten(m, m + 2)

    def _blocks(self, n, K, parts):
        """Slices of the half spectrum's blocks, the first axis fastest."""
        size = [n[d] // 2 + 1 if d == K else n[d] // parts[d] for d in range(3)]
        for i2 in range(parts[2]):
            for i1 in range(parts[1]):
                for i0 in range(parts[0]):
                    yield tuple(slice(i * z, (i + 1) * z) for i, z in zip((i0, i1, i2), size))

    @staticmethod
    def _flat(t):
        return t.permute(2, 1, 0).reshape(-1)

    def analyze(self, x):
        X, bands = torch.fft.fftn(x), []
        for v in self.lv:
            ix = tuple(a.reshape([-1 if e == d else 1 for e in range(3)]) for d, a in enumerate(v["at"]))
            il = tuple(a.reshape([-1 if e == d else 1 for e in range(3)]) for d, a in enumerate(v["to"]))
            box = X[ix]
            low = torch.zeros(v["low"], dtype=torch.complex128, device="cuda").index_put(il, v["L"] / v["D"] * box)
            X = X.index_put(ix, box * torch.sqrt(1 - v["L"] ** 2))
            out = []
            for K in range(3):
                n, (a, b) = v["n"], [d for d in range(3) if d != K]
                S = X.narrow(K, 0, n[K] // 2 + 1) * v["V"][K]
                for m, h, f, _ in v["stages"][K]:
                    S = self._stage(S, m, h, f, False)
                for sl in self._blocks(n, K, v["parts"][K]):
                    blk = S[sl]
                    out.append(self._flat(torch.fft.irfftn(blk, s=(blk.shape[a], blk.shape[b], n[K]), dim=(a, b, K))))
            bands = out + bands
            X = low
        return torch.cat([self._flat(torch.fft.ifftn(X).real)] + bands)

    def synthesize(self, c):
        at = math.prod(self.lv[-1]["low"])
        C = torch.fft.fftn(c[:at].reshape(self.lv[-1]["low"][::-1]).permute(2, 1, 0) + 0j)
        for v in reversed(self.lv):
            n, X = v["n"], 0
            for K in range(3):
                a, b = [d for d in range(3) if d != K]
                parts, h = v["parts"][K], n[K] // 2 + 1
                size = [n[d] // parts[d] for d in range(3)]
                S = torch.zeros([h if d == K else n[d] for d in range(3)], dtype=torch.complex128, device="cuda")
                for sl in self._blocks(n, K, parts):
                    k = math.prod(size)
                    S[sl] = torch.fft.rfftn(c[at:at + k].reshape(size[::-1]).permute(2, 1, 0), dim=(a, b, K))
                    at += k
                for m, w, _, f in reversed(v["stages"][K]):
                    S = self._stage(S, m, w, f, True)
                S = S * v["V"][K] / 3
                # the other half is the conjugate mirror
                src = torch.arange(n[K] - h, 0, -1, device="cuda")
                mir = S.index_select(K, src).conj()
                for d in (a, b):
                    mir = mir.index_select(d, (-torch.arange(n[d], device="cuda")) % n[d])
                X = X + torch.cat([S, mir], K)
            ix = tuple(q.reshape([-1 if e == d else 1 for e in range(3)]) for d, q in enumerate(v["at"]))
            il = tuple(q.reshape([-1 if e == d else 1 for e in range(3)]) for d, q in enumerate(v["to"]))
            C = X.index_put(ix, torch.sqrt(1 - v["L"] ** 2) * X[ix] + v["L"] * v["D"] * C[il])
        return torch.fft.ifftn(C).real


def _by_channel(f, t):
    """Complex data are two real channels."""
    return torch.complex(f(t.real.double()), f(t.imag.double())) if t.is_complex() else f(t.double())


def _transpose(f, like, g):
    """The transpose of the linear map f at g."""
    z = torch.zeros(like, **_D, requires_grad=True)
    with torch.enable_grad():
        return torch.autograd.grad(f(z), z, g)[0]


def exact(case, seed):
    dims = (case["n1"], case["n2"], case["n3"])
    levels, do, s = [int(d) for d in case["levels"]], case["do"], _inputs(case, seed)
    T = _NS64(dims, levels) if case["bank"] == "ns" else _Dec64(dims, levels, case["ratio"])
    if do == "synthesize":
        return _by_channel(T.synthesize, s["c"])
    if do == "denoise":
        return T.denoise(s["x"].double(), _TAU)
    c = _by_channel(T.analyze, s["x"])
    if do == "analyze":
        return c
    if do == "roundtrip":
        return c, s["x"].to(torch.complex128 if s["x"].is_complex() else torch.float64)
    if do == "bf16":
        # subbands over the smallest power of two at or above their peak
        scale = 2.0 ** (torch.frexp(c.abs().amax((0, 1, 2)))[1]).double()
        return c / scale, scale, s["x"].double()
    if case["bank"] == "ns":     # tight: each direction is the other's transpose
        gx, gc = _by_channel(T.synthesize, s["gc"]), _by_channel(T.analyze, s["gx"])
    else:
        gx = _by_channel(lambda g: _transpose(T.analyze, dims, g), s["gc"])
        gc = _by_channel(lambda g: _transpose(T.synthesize, s["c"].shape, g), s["gx"])
    return c, gx, _by_channel(T.synthesize, s["c"]), gc
