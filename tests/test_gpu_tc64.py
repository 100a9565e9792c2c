"""FP64 plans on the tensor cores (digit-product contraction, matrix-form ring transforms) against
the general path: the same calls on plans whose workspace limit leaves no room for digit tiles run
the FMA contraction and the ring FFTs.  Tolerance: the parity bar of the FP64 method, 1e-11 of the
largest value of a map; both sides meet it against the oracle.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TOL = 1e-11


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fastsht_gb300 import build
    build.build()


def _plans(kind, ns, lmax, nsim, niter=0):
    """The plan, and one that the limit keeps on the general path (in chunks below a tile)."""
    from fastsht_gb300 import SHT
    pol = kind in ("qu2eb", "eb2qu")
    nbuf = (2 if pol else 1) * (2 if niter else 1)
    limit = nbuf * min(nsim, 60) * 2 * ns * (lmax + 1) * 32
    general = SHT(ns, lmax, nsim, niter=niter, pol=pol, workspace_limit=limit)
    assert general.plan_info()["maps_per_chunk"] == min(nsim, 60)
    return SHT(ns, lmax, nsim, niter=niter, pol=pol), general


def _inputs(kind, ns, lmax, nsim, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = 2 if kind in ("qu2eb", "eb2qu") else 1
    if kind in ("t2alm", "qu2eb"):
        return [torch.randn((nsim, 12 * ns * ns), dtype=torch.float64, device="cuda",
                            generator=g).T for _ in range(n)]
    return [torch.randn((lmax + 1, lmax + 1, nsim), dtype=torch.float64, device="cuda",
                        generator=g).permute(2, 1, 0) for _ in range(n)]


def _run(sht, kind, ins):
    out = getattr(sht, kind)(*[x.clone() for x in ins])
    return [o.clone() for o in (out if isinstance(out, (tuple, list)) else (out,))]


def _per_map(kind, x, nsim):
    # maps (npix, nsim), alm (nsim, l, m)
    return (x.T if kind in ("alm2t", "eb2qu") else x).reshape(nsim, -1)


# edges: one map; 128-row l tiles of a parity (lmax 255, 256, 257); 128-ring blocks; 64-map tiles
# (63, 64, 65, 129 maps); the maps per tile from which the ring transforms change form, with the
# rest of a tile on either side; belt in matrix form (nside <= 256) and not (512)
SIZES = [(32, 95, 1), (32, 127, 63), (32, 63, 64), (32, 95, 65), (32, 70, 129),
         (64, 191, 19), (64, 191, 20), (64, 255, 38), (64, 256, 37), (128, 257, 102),
         (128, 300, 14), (128, 300, 15), (128, 383, 79), (256, 511, 31), (256, 300, 30),
         (512, 530, 23), (512, 530, 67)]


@pytest.mark.parametrize("kind", ["t2alm", "alm2t", "qu2eb", "eb2qu"])
@pytest.mark.parametrize("ns,lmax,nsim", SIZES)
def test_equals_general_path(kind, ns, lmax, nsim):
    tc, general = _plans(kind, ns, lmax, nsim)
    ins = _inputs(kind, ns, lmax, nsim, ns + lmax + nsim)
    for a, b in zip(_run(tc, kind, ins), _run(general, kind, ins)):
        a, b = _per_map(kind, a, nsim), _per_map(kind, b, nsim)
        assert torch.isfinite(a).all()
        assert ((a - b).abs().amax(1) <= TOL * b.abs().amax(1)).all()


@pytest.mark.parametrize("kind", ["t2alm", "qu2eb"])
@pytest.mark.parametrize("ns,lmax,nsim", [(32, 95, 5), (64, 130, 70)])
def test_iterations_equal_general_path(kind, ns, lmax, nsim):
    tc, general = _plans(kind, ns, lmax, nsim, niter=2)
    ins = _inputs(kind, ns, lmax, nsim, 5)
    for a, b in zip(_run(tc, kind, ins), _run(general, kind, ins)):
        a, b = _per_map(kind, a, nsim), _per_map(kind, b, nsim)
        assert ((a - b).abs().amax(1) <= TOL * b.abs().amax(1)).all()


@pytest.mark.parametrize("kind", ["t2alm", "alm2t", "qu2eb", "eb2qu"])
@pytest.mark.parametrize("ns,lmax,nsim", [(32, 95, 9), (64, 200, 66)])
def test_columns_outside_the_digit_range(kind, ns, lmax, nsim):
    """Maps of 2^+-1000 and a NaN take the FMA kernels in their tile; zeros and the others of the
    tile come out as ever."""
    tc, general = _plans(kind, ns, lmax, nsim)
    ins = [x.clone() for x in _inputs(kind, ns, lmax, nsim, 7)]
    for x in ins:
        v = x.T if kind in ("t2alm", "qu2eb") else x           # map first
        v[1] *= 2.0 ** 1000
        v[3] *= 2.0 ** -1000
        v[4] = 0.0
        if kind in ("t2alm", "qu2eb"):
            v[6, 17] = float("nan")
    for a, b in zip(_run(tc, kind, ins), _run(general, kind, ins)):
        a, b = _per_map(kind, a, nsim), _per_map(kind, b, nsim)
        assert torch.equal(torch.isnan(a), torch.isnan(b))
        ok = ~torch.isnan(b).any(1)
        assert ok.sum() == nsim - (kind in ("t2alm", "qu2eb"))
        assert (a[4] == 0).all()
        assert ((a - b)[ok].abs().amax(1) <= TOL * b[ok].abs().amax(1)).all()


def test_ragged_maps_do_not_depend_on_their_tile():
    """A map's result has the same bits wherever its tile's other columns come from."""
    from fastsht_gb300 import SHT
    ns, lmax = 64, 150
    ins = _inputs("t2alm", ns, lmax, 128, 3)[0]
    a = SHT(ns, lmax, 128).t2alm(ins)
    b = SHT(ns, lmax, 64).t2alm(ins[:, 64:].T.contiguous().T)
    assert torch.equal(a[64:], b)
