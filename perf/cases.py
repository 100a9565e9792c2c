"""The work that users of this framework give it, as cases that can be timed and checked.

Every case goes through the public entry points (``SHT``, ``Batch``).  A case is a dict:

  kind       t2alm | alm2t | qu2eb | eb2qu   one call of that ``SHT`` method on device tensors
             roundtrip                       t2alm, convert_alm_healpy, alm2t on device tensors
             host                            t2alm from page-locked NumPy maps to NumPy alm
             batch                           one replay of a ``Batch`` of mixed jobs
  precision  "fp64" (the default of ``SHT``) or "split" (tensor-core digit products)
  nside, lmax, nmaps (Q/U or E/B pairs count once), niter, method   as ``SHT`` takes them

Ranges that the listed cases stand for (``draw`` spreads over them): nside 16..2048 (powers of
two), lmax nside..3 nside - 1, 1..200 maps, both precisions, both directions, spin 0 and 2,
0..3 iterations; FP64 to nside 1024.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fastsht_gb300 import SHT
from fastsht_gb300.batch import Batch
from fastsht_gb300.sht import pinned_empty

DEV = "cuda"


def _case(name, kind, precision, nside, lmax, nmaps, niter=0, method="old"):
    return {"name": name, "kind": kind, "precision": precision, "nside": nside, "lmax": lmax,
            "nmaps": nmaps, "niter": niter, "method": method}


def listed():
    return [
        # one small map, as an interactive user or a small serving request has it: latency
        _case("t2alm 32 one map", "t2alm", "fp64", 32, 95, 1),
        # the plain round trip of 100 white-noise maps (nside 64, lmax 191) with healpy-order alm
        _case("roundtrip 64", "roundtrip", "fp64", 64, 191, 100),
        # the reference's demonstration: nside 128, lmax 383, 100 maps, three iterations
        _case("t2alm 128 niter 3", "t2alm", "fp64", 128, 383, 100, niter=3),
        # polarisation sets of simulation pipelines (nside 256, lmax 767), both directions; the
        # inverse with an odd number of maps
        _case("qu2eb 256", "qu2eb", "fp64", 256, 767, 128),
        _case("eb2qu 256 odd", "eb2qu", "fp64", 256, 767, 67),
        # high-resolution maps in the default precision
        _case("t2alm 1024", "t2alm", "fp64", 1024, 2047, 64),
        # a large batch of high-resolution maps in the split form: the throughput case
        _case("split t2alm 1024", "t2alm", "split", 1024, 2047, 160),
        # split form with one refinement step, maps of a ragged count
        _case("split t2alm 512 niter 1", "t2alm", "split", 512, 1023, 75, niter=1,
              method="new"),
        # split synthesis at lmax = 3 nside - 1
        _case("split alm2t 512", "alm2t", "split", 512, 1535, 96),
        # split polarisation analysis, lmax = 2 nside as serving requests have it
        _case("split qu2eb 512", "qu2eb", "split", 512, 1024, 48),
        # maps and alm in page-locked host memory, the way the reference's arrays are held
        _case("host split 1024", "host", "split", 1024, 2047, 24),
        # a mix of small jobs of several sizes as one graph launch
        _case("batch mix", "batch", "fp64", 128, 300, 24),
    ]


def _odd(rng, lo, hi):
    """An integer, uniform over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    top = _legendre(_case("", "t2alm", "fp64", 1024, 2047, 64))
    while True:
        kind = rng.choice(["t2alm", "t2alm", "alm2t", "qu2eb", "eb2qu", "roundtrip", "host",
                           "batch"])
        precision = rng.choice(["fp64", "fp64", "split"])
        nside = 2 ** rng.randint(4, 11)
        lmax = rng.randint(nside, 3 * nside - 1)
        c = {"kind": kind, "precision": precision, "nside": nside, "lmax": lmax,
             "nmaps": _odd(rng, 1, 200), "niter": 0, "method": "old"}
        if kind == "batch":
            c["precision"] = "fp64"
            c["nside"] = min(nside, 256)
            c["lmax"] = rng.randint(c["nside"], 3 * c["nside"] - 1)
            c["nmaps"] = min(c["nmaps"], 48)
        if kind in ("t2alm", "qu2eb") and rng.random() < 0.3:
            c["niter"] = rng.randint(1, 3)
            if kind == "t2alm":
                c["method"] = rng.choice(["old", "new"])
        # contractions work on tiles of maps: a few maps cost as much as a tile of 64
        tiled = dict(c, nmaps=-(-c["nmaps"] // 64) * 64)
        if c["precision"] == "fp64" and (c["nside"] > 1024 or _legendre(tiled) > 0.9 * top):
            continue
        if c["precision"] == "split" and _legendre(tiled) > 8 * top:
            continue
        fields = 2 if kind in ("qu2eb", "eb2qu") else 1
        per_map = 12 * c["nside"] ** 2 * 8 + (c["lmax"] + 1) ** 2 * 8
        bufs = 4 if c["niter"] else 2
        per_map += bufs * (c["lmax"] + 1) * 2 * c["nside"] * 32
        if fields * c["nmaps"] * per_map > 35e9:
            continue
        return c


# ------------------------------------------------------------------ work
def _fields(case):
    return 2 if case["kind"] in ("qu2eb", "eb2qu") else 1


def _legendre(case):
    """Flops of the north/south-folded Legendre sums."""
    ns, L = case["nside"], case["lmax"] + 1
    one = 4.0 * ns * L * (L + 1) * case["nmaps"] * (4 if _fields(case) == 2 else 1)
    return one * (2 if case["kind"] == "roundtrip" else 1 + 2 * case.get("niter", 0))


def _fft_flops(nside):
    """5 n log2 n per ring of real data, two rings per complex transform."""
    f = 0.0
    for i in range(4 * nside - 1):
        n = _ring_len(nside, i)
        f += 2.5 * n * math.log2(n)
    return f


def _batch_jobs(case):
    ns, lm, k = case["nside"], case["lmax"], case["nmaps"]
    jobs = [("t2alm", ns, lm, k), ("qu2eb", ns, lm, max(1, k // 3)), ("alm2t", ns, lm, k)]
    if ns >= 32:
        jobs += [("t2alm", ns // 2, lm // 2, k + 5), ("eb2qu", ns // 2, lm // 2, max(1, k // 2)),
                 ("qu2eb", ns // 2, lm // 2, k)]
    return jobs


def work(case):
    if case["kind"] == "batch":
        parts = [work(_case("", kd, "fp64", ns, lm, k)) for kd, ns, lm, k in _batch_jobs(case)]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    ns, L, k = case["nside"], case["lmax"] + 1, case["nmaps"]
    maps, alm = 8.0 * 12 * ns * ns * k, 8.0 * L * L * k
    flops = _legendre(case) + _fields(case) * k * _fft_flops(ns)
    if case["kind"] == "roundtrip":
        # maps in; alm, healpy alm and maps out (the transforms read the alm once more)
        nbytes = 2 * maps + 2 * alm + 16.0 * (L * (L + 1) // 2) * k
        flops += k * _fft_flops(ns)
    else:
        nbytes = _fields(case) * (maps + alm)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ inputs
def _ring_start(ns, i):
    if i < ns:
        return 2 * i * (i + 1)
    if i < 3 * ns - 1:
        return 2 * ns + 4 * ns * i - 2 * ns * ns
    r = 4 * ns - i
    return 12 * ns * ns - 2 * (r - 1) * r


def _ring_len(ns, i):
    return 4 * min(i + 1, ns, 4 * ns - 1 - i)


def _ring_shift(ns, i):
    """phi of the first pixel of a ring in units of pi / n."""
    if i < ns or i >= 3 * ns - 1:
        return 1
    return 1 if (i + 1 - ns) % 2 == 0 else 0


def _ring_z_sin(ns, i):
    """cos and sin of a ring's colatitude."""
    j = min(i + 1, 4 * ns - 1 - i)
    if j < ns:
        t = j * j / (3.0 * ns * ns)
        z, s = 1.0 - t, math.sqrt(t * (2.0 - t))
    else:
        z = (2 * ns - j) * 2.0 / (3.0 * ns)
        s = math.sqrt((1.0 - z) * (1.0 + z))
    return (z if i + 1 <= 2 * ns else -z), s


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _sky(nside, nmaps, seed):
    """(nmaps, npix): smooth large-scale structure (plane waves through the sphere, amplitude
    falling with the wave number) under white pixel noise."""
    g = _gen(seed)
    nr = 4 * nside - 1
    ln = torch.tensor([_ring_len(nside, i) for i in range(nr)], device=DEV)
    st = torch.tensor([_ring_start(nside, i) for i in range(nr)], device=DEV)
    sh = torch.tensor([_ring_shift(nside, i) for i in range(nr)], device=DEV)
    zs = torch.tensor([_ring_z_sin(nside, i) for i in range(nr)], dtype=torch.float64, device=DEV)
    ring = torch.repeat_interleave(torch.arange(nr, device=DEV), ln)
    j = torch.arange(12 * nside * nside, device=DEV) - st[ring]
    phi = (2.0 * j + sh[ring]) * math.pi / ln[ring]
    z, s = zs[ring, 0], zs[ring, 1]
    x, y = s * torch.cos(phi), s * torch.sin(phi)
    nw = 12
    basis = torch.empty((nw, 12 * nside * nside), dtype=torch.float64, device=DEV)
    for w in range(nw):
        k = 1.5 * (0.5 * nside) ** (w / nw)
        d = torch.randn(3, generator=g, device=DEV, dtype=torch.float64)
        d = (d / d.norm() * k).tolist()
        basis[w] = torch.cos((d[0] * x + d[1] * y + d[2] * z).float()).double() / k
    coef = torch.randn((nmaps, nw), generator=g, device=DEV, dtype=torch.float64)
    out = torch.randn((nmaps, 12 * nside * nside), generator=g, device=DEV, dtype=torch.float64)
    out.mul_(0.3)
    for a in range(0, nmaps, 32):
        out[a:a + 32] += coef[a:a + 32] @ basis
    return out


def _white(nside, nmaps, seed):
    return torch.randn((nmaps, 12 * nside * nside), generator=_gen(seed), device=DEV,
                       dtype=torch.float64)


def _gauss_alm(lmax, nmaps, seed, lmin=0, amp=1.0):
    """(L, L, nmaps) square-real alm: Gaussian with C_l = amp / (l (l+1)); slot [m][l] holds
    Re a_lm, slot [L - m][l - m] Im a_lm."""
    L = lmax + 1
    c = torch.arange(L, device=DEV).view(L, 1)
    r = torch.arange(L, device=DEV).view(1, L)
    l = torch.where(r >= c, r, r + L - c).double()
    var = amp / (l * (l + 1)).clamp(min=1.0)
    var = torch.where((c == 0) & (r >= c), var, var / 2)
    var = torch.where(l < lmin, torch.zeros_like(var), var)
    out = torch.randn((L, L, nmaps), generator=_gen(seed), device=DEV, dtype=torch.float64)
    return out.mul_(var.sqrt().unsqueeze(-1))


def _inputs(case, seed):
    """Input tensors in the library's layout: maps (nmaps, npix) or alm (L, L, nmaps)."""
    ns, lm, k = case["nside"], case["lmax"], case["nmaps"]
    kind, seed = case["kind"], 7919 * int(seed)
    if kind == "roundtrip":
        return [_white(ns, k, seed + 1)]
    if kind in ("t2alm", "host"):
        return [_sky(ns, k, seed + 1)]
    if kind == "qu2eb":
        return [_sky(ns, k, seed + 1), _sky(ns, k, seed + 2)]
    if kind == "alm2t":
        return [_gauss_alm(lm, k, seed + 1)]
    return [_gauss_alm(lm, k, seed + 1, 2), _gauss_alm(lm, k, seed + 2, 2, 0.1)]


def prepare(case, seed):
    ns, lm, k = case["nside"], case["lmax"], case["nmaps"]
    if case["kind"] == "batch":
        b = Batch(nslots=4, workspace_budget=8 << 30)
        for n, (kd, jns, jlm, jk) in enumerate(_batch_jobs(case)):
            ins = _inputs(_case("", kd, "fp64", jns, jlm, jk), 100 * int(seed) + n)
            b.add(kd, jns, jlm, jk, inputs=ins)
        b.build()
        return {"kind": "batch", "batch": b}
    sht = SHT(ns, lm, k, niter=case["niter"], pol=_fields(case) == 2,
              precision=case["precision"])
    ins = _inputs(case, seed)
    if case["kind"] == "host":
        maps = pinned_empty((12 * ns * ns, k))
        torch.from_numpy(maps.T).copy_(ins[0])
        return {"kind": "host", "sht": sht, "maps": maps,
                "alm": pinned_empty((k, lm + 1, lm + 1))}
    if case["kind"] in ("alm2t", "eb2qu"):
        ins = [x.permute(2, 1, 0) for x in ins]     # (nmaps, L, L) in Fortran strides
    else:
        ins = [x.T for x in ins]                    # (npix, nmaps) in Fortran strides
    return {"kind": case["kind"], "sht": sht, "ins": ins, "method": case["method"]}


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].run()
        return [j.outputs for j in state["batch"].jobs]
    sht = state["sht"]
    if kind == "host":
        sht.t2alm(state["maps"], state["alm"])
        return state["alm"]
    ins = state["ins"]
    if kind == "roundtrip":
        alm = sht.t2alm(ins[0])
        return {"alm": alm, "healpy": sht.convert_alm_healpy(alm), "maps": sht.alm2t(alm)}
    if kind == "t2alm":
        return sht.t2alm(ins[0], method=state["method"])
    if kind == "alm2t":
        return sht.alm2t(ins[0])
    if kind == "qu2eb":
        return sht.qu2eb(ins[0], ins[1])
    return sht.eb2qu(ins[0], ins[1])


# ------------------------------------------------------------------ 64-bit values
# The transform written out in torch: per-ring FFTs, the associated Legendre functions from the
# three-term recursion (values carried as v 2^(600 e), so that no seed underflows), dense sums.
class _Exact:
    def __init__(self, nside, lmax):
        self.ns, self.lmax, self.R = nside, lmax, 2 * nside
        zs = torch.tensor([_ring_z_sin(nside, i) for i in range(self.R)], dtype=torch.float64,
                          device=DEV)
        self.x, self.s = zs[:, 0].contiguous(), zs[:, 1].contiguous()
        # block of orders: the table of a block stays near 2 GB
        per = (lmax + 1) * self.R * 8
        self.block = max(1, min(lmax + 1, int(2.2e9 // per), 128))

    def rings(self):
        for i in range(4 * self.ns - 1):
            n = _ring_len(self.ns, i)
            south = i + 1 > 2 * self.ns
            yield i, _ring_start(self.ns, i), n, _ring_shift(self.ns, i), south

    def _phase(self, n, shift, sign):
        m = torch.arange(self.lmax + 1, device=DEV, dtype=torch.float64)
        a = torch.remainder(m * shift, 2.0 * n) * (math.pi / n)
        return torch.complex(torch.cos(a), sign * torch.sin(a))

    def fourier(self, maps):
        """maps (K, npix) -> F_N, F_S, each complex (L, R, K); F_S of the equator is zero."""
        K, L = maps.shape[0], self.lmax + 1
        out = [torch.zeros((L, self.R, K), dtype=torch.complex128, device=DEV) for _ in range(2)]
        m = torch.arange(L, device=DEV)
        for i, st, n, sh, south in self.rings():
            F = torch.fft.fft(maps[:, st:st + n], dim=1)
            F = F[:, m % n] * self._phase(n, sh, -1.0)
            out[1 if south else 0][:, 4 * self.ns - 2 - i if south else i] = F.T
        return out

    def pixels(self, GN, GS):
        """G_N, G_S (L, R, K) -> maps (K, npix)."""
        K, L = GN.shape[2], self.lmax + 1
        maps = torch.empty((K, 12 * self.ns * self.ns), dtype=torch.float64, device=DEV)
        m = torch.arange(L, device=DEV)
        w = torch.full((L, 1), 2.0, dtype=torch.float64, device=DEV)
        w[0] = 1.0
        for i, st, n, sh, south in self.rings():
            G = (GS if south else GN)[:, 4 * self.ns - 2 - i if south else i]
            c = G * (self._phase(n, sh, 1.0).unsqueeze(1) * w)
            bins = torch.zeros((n, K), dtype=torch.complex128, device=DEV)
            torch.view_as_real(bins).index_add_(0, m % n, torch.view_as_real(c.contiguous()))
            maps[:, st:st + n] = (torch.fft.ifft(bins, dim=0).real * n).T
        return maps

    def legendre(self, m0, m1):
        """lambda_lm on the north rings for m0 <= m < m1: (m, L, R), zero for l < m."""
        L, R, nb = self.lmax + 1, self.R, m1 - m0
        lam = torch.zeros((nb, L, R), dtype=torch.float64, device=DEV)
        mm = np.arange(m0, m1, dtype=np.float64)
        # seeds: log2 |lambda_mm| = 0.5 log2(prod (2k+1)/(2k) / 4 pi) + m log2 sin
        k = np.arange(1, m1, dtype=np.longdouble)
        lg = np.concatenate([[0.0], np.cumsum(np.log2((2 * k + 1) / (2 * k)))])[m0:m1]
        s = self.s.cpu().numpy().astype(np.longdouble)
        seed = 0.5 * (lg[:, None] - np.log2(4 * np.pi)) + mm[:, None] * np.log2(s)[None, :]
        e = np.minimum(0, np.ceil((seed - 300) / 600))
        v = np.exp2(seed - 600 * e).astype(np.float64) * np.where(mm[:, None] % 2, -1.0, 1.0)
        seed = torch.from_numpy(np.ascontiguousarray(v)).to(DEV)
        e = torch.from_numpy(e.astype(np.float64)).to(DEV)
        ll = np.arange(L, dtype=np.float64)[:, None]
        with np.errstate(divide="ignore", invalid="ignore"):
            a = np.sqrt((4 * ll * ll - 1) / (ll * ll - mm * mm))
            b = np.sqrt(((ll - 1) ** 2 - mm * mm) / (4 * (ll - 1) ** 2 - 1)) * a
        a = torch.from_numpy(np.where(ll > mm, a, 0.0)).to(DEV).unsqueeze(-1)
        b = torch.from_numpy(np.where(ll > mm, b, 0.0)).to(DEV).unsqueeze(-1)
        cur = torch.zeros((nb, R), dtype=torch.float64, device=DEV)
        prev = torch.zeros_like(cur)
        for l in range(m0, L):
            nx = torch.addcmul(cur * (a[l] * self.x), prev, b[l], value=-1.0)
            if l < m1:
                nx[l - m0] = seed[l - m0]
            prev, cur = cur, nx
            if l % 8 == 0:
                up = (cur.abs() > 2.0 ** 300) & (e < 0)
                cur = torch.where(up, cur * 2.0 ** -600, cur)
                prev = torch.where(up, prev * 2.0 ** -600, prev)
                e = e + up
            torch.where(e >= 0, cur, torch.zeros_like(cur), out=lam[:, l])
        return lam

    def spin2(self, lam, m0, m1):
        """The two spin-2 functions from lambda: (m, L, R) each, zero for l < 2."""
        L = self.lmax + 1
        m = torch.arange(m0, m1, device=DEV, dtype=torch.float64).view(-1, 1, 1)
        l = torch.arange(L, device=DEV, dtype=torch.float64).view(1, -1, 1)
        s2 = (self.s * self.s).view(1, 1, -1)
        x = self.x.view(1, 1, -1)
        nl = torch.where(l >= 2, ((l + 2) * (l + 1) * l * (l - 1)).clamp(min=1.0).rsqrt(), 0.0)
        lf = torch.where(l > m, 2 * ((2 * l + 1) / (2 * l - 1) * (l * l - m * m)).clamp(min=0).sqrt(),
                         0.0)
        one, two = torch.zeros_like(lam), torch.zeros_like(lam)
        for b in range(m1 - m0):                      # one order at a time: small temporaries
            prev = torch.zeros_like(lam[b])
            prev[1:] = lam[b, :-1]
            mb, cur = m[b], lam[b]
            f, n = lf[b], nl[0]
            one[b] = (prev * f * (x[0] / s2[0]) -
                      cur * (2 * (l[0] - mb * mb) / s2[0] + l[0] * (l[0] - 1))) * n
            two[b] = (prev * f - cur * (2 * (l[0] - 1)) * x[0]) * (mb / s2[0]) * n
        return one, two

    def _put(self, alm, m0, A):
        """A complex (m, L, K) -> square-real alm (L, L, K)."""
        L = self.lmax + 1
        for b in range(A.shape[0]):
            m = m0 + b
            alm[m, m:] = A[b, m:].real
            if m:
                alm[L - m, :L - m] = A[b, m:].imag

    def _get(self, alm, m0, m1):
        L = self.lmax + 1
        A = torch.zeros((m1 - m0, L, alm.shape[2], 2), dtype=torch.float64, device=DEV)
        for b in range(m1 - m0):
            m = m0 + b
            A[b, m:, :, 0] = alm[m, m:]
            if m:
                A[b, m:, :, 1] = alm[L - m, :L - m]
        return A.flatten(2)                           # (m, L, 2K), re and im interleaved

    def _blocks(self):
        for m0 in range(0, self.lmax + 1, self.block):
            yield m0, min(self.lmax + 1, m0 + self.block)

    def _fold(self, F, m0, m1):
        """(sum, difference) of north and south with even l - m first: even-l and odd-l sides."""
        S = torch.view_as_real(F[0][m0:m1] + F[1][m0:m1]).flatten(2)
        D = torch.view_as_real(F[0][m0:m1] - F[1][m0:m1]).flatten(2)
        odd = torch.arange(m0, m1, device=DEV).remainder(2).bool().view(-1, 1, 1)
        return torch.where(odd, D, S), torch.where(odd, S, D)

    def _rows(self, lam, even, odd):
        out = torch.empty((lam.shape[0], lam.shape[1], even.shape[2]), dtype=torch.float64,
                          device=DEV)
        out[:, 0::2] = torch.bmm(lam[:, 0::2], even)
        if lam.shape[1] > 1:
            out[:, 1::2] = torch.bmm(lam[:, 1::2], odd)
        return torch.view_as_complex(out.unflatten(2, (-1, 2)))

    def analyse(self, fields):
        """Maps (K, npix) of T, or of Q and U -> alm (L, L, K) of T, or of E and B."""
        L, K = self.lmax + 1, fields[0].shape[0]
        pa = 4 * math.pi / (12.0 * self.ns * self.ns)
        F = [self.fourier(f) for f in fields]
        alm = [torch.zeros((L, L, K), dtype=torch.float64, device=DEV) for _ in fields]
        for m0, m1 in self._blocks():
            lam = self.legendre(m0, m1)
            if len(fields) == 1:
                self._put(alm[0], m0, self._rows(lam, *self._fold(F[0], m0, m1)) * pa)
                continue
            one, two = self.spin2(lam, m0, m1)
            del lam
            Q, U = self._fold(F[0], m0, m1), self._fold(F[1], m0, m1)
            E = self._rows(one, *Q) + 1j * self._rows(two, U[1], U[0])
            B = self._rows(one, *U) - 1j * self._rows(two, Q[1], Q[0])
            self._put(alm[0], m0, E * -pa)
            self._put(alm[1], m0, B * -pa)
        return alm

    def _sums(self, lam, A, m0, m1, flip):
        """sum_l lam A on the north and (with the parity sign) the south rings."""
        ev = torch.bmm(lam[:, 0::2].transpose(1, 2), A[:, 0::2])
        od = torch.bmm(lam[:, 1::2].transpose(1, 2), A[:, 1::2])
        odd = torch.arange(m0, m1, device=DEV).remainder(2).bool().view(-1, 1, 1)
        ev, od = torch.where(odd, od, ev), torch.where(odd, ev, od)
        c = [torch.view_as_complex(t.unflatten(2, (-1, 2)).contiguous())
             for t in (ev + od, od - ev if flip else ev - od)]
        return c

    def synthesise(self, alm):
        """alm (L, L, K) of T, or of E and B -> maps (K, npix) of T, or of Q and U."""
        L, K = self.lmax + 1, alm[0].shape[2]
        G = [[torch.zeros((L, self.R, K), dtype=torch.complex128, device=DEV) for _ in range(2)]
             for _ in alm]
        for m0, m1 in self._blocks():
            lam = self.legendre(m0, m1)
            if len(alm) == 1:
                A = self._get(alm[0], m0, m1)
                G[0][0][m0:m1], G[0][1][m0:m1] = self._sums(lam, A, m0, m1, False)
                continue
            one, two = self.spin2(lam, m0, m1)
            del lam
            E, B = self._get(alm[0], m0, m1), self._get(alm[1], m0, m1)
            e1, b1 = (self._sums(one, a, m0, m1, False) for a in (E, B))
            e2, b2 = (self._sums(two, a, m0, m1, True) for a in (E, B))
            for h in range(2):
                G[0][h][m0:m1] = -(e1[h] + 1j * b2[h])
                G[1][h][m0:m1] = 1j * e2[h] - b1[h]
        return [self.pixels(*g) for g in G]


def _exact_seconds(case):
    """About how long exact() takes: the dense sums, the recursion's steps, the ring loops."""
    ns, L = case["nside"], case["lmax"] + 1
    per = L * 2 * ns * 8
    blocks = -(-L // max(1, min(L, int(2.2e9 // per), 128)))
    turns = 2 if case["kind"] == "roundtrip" else 1 + 2 * case["niter"]
    spin = 3.0 if _fields(case) == 2 else 1.0
    one = blocks * L * 40e-6 + L * L * ns * spin * 4e-10 + 4 * ns * _fields(case) * 5e-4
    return turns * one + 2.2 * _legendre(case) / 0.6e12 + 2e-3 * ns


def _exact_one(case, seed):
    if _exact_seconds(case) > 18:
        return None
    kind, ns, lm = case["kind"], case["nside"], case["lmax"]
    T = _Exact(ns, lm)
    ins = _inputs(case, seed)
    if kind in ("alm2t", "eb2qu"):
        maps = [x.T for x in T.synthesise(ins)]
        return maps[0] if kind == "alm2t" else tuple(maps)
    alm = T.analyse(ins)
    if kind == "roundtrip":
        back = T.synthesise(alm)
        L = lm + 1
        hp = torch.empty((L * (L + 1) // 2, case["nmaps"]), dtype=torch.complex128, device=DEV)
        at = 0
        for m in range(L):
            im = alm[0][L - m, :L - m] if m else torch.zeros_like(alm[0][0])
            hp[at:at + L - m] = torch.complex(alm[0][m, m:], im)
            at += L - m
        return {"alm": alm[0].permute(2, 1, 0), "healpy": hp, "maps": back[0].T}
    for _ in range(case["niter"]):
        # Jacobi step: the analysis of what the maps have beyond the synthesis
        back = T.synthesise(alm)
        alm = [a + d for a, d in zip(alm, T.analyse([x - y for x, y in zip(ins, back)]))]
    alm = [a.permute(2, 1, 0) for a in alm]
    return tuple(alm) if kind == "qu2eb" else alm[0]


def exact(case, seed):
    if case["method"] == "new" and case["niter"]:
        return None       # the one-sided iteration has no plain map-space form
    if case["kind"] == "batch":
        out = []
        for n, (kd, ns, lm, k) in enumerate(_batch_jobs(case)):
            c = _case("", kd, "fp64", ns, lm, k)
            r = _exact_one(c, 100 * int(seed) + n)
            r = [r] if torch.is_tensor(r) else list(r)
            # the batch's buffers are in the library's layout
            out.append([x.permute(2, 1, 0) if x.dim() == 3 else x.T for x in r])
        return out
    r = _exact_one(case, seed)
    if case["kind"] == "host" and r is not None:
        return r.cpu().numpy()
    return r
