"""FP64 plans on the tensor cores with operands that fill their fixed-point scales, against the
general path (plans whose workspace limit leaves no room for digit tiles).  Tolerance: the parity
bar of the FP64 method, 1e-11 of the largest value of a map.
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


def _top_of_scale(lmax, spin):
    """a_lm for which every fixed-point column entry a Dm 2^EA(l) is 0.999 of one power of two:
    Dm the mantissa of D_l = prod a_k (spin 2: of N_l), 2^EA the power of two above bound / Dm."""
    l = np.arange(lmax + 1)[:, None].astype(float)
    m = np.arange(lmax + 1)[None].astype(float)
    with np.errstate(all="ignore"):
        if spin == 0:
            a2 = np.where(l > m, (4 * l * l - 1) / (l * l - m * m), 1.0)
            log_d = 0.5 * np.cumsum(np.log2(a2), 0)
        else:
            log_d = np.where(l >= 2, -0.5 * np.log2((l + 2) * (l + 1) * l * (l - 1)), 0.0) + 0 * m
    dm = np.exp2(log_d - np.floor(log_d))
    bound = np.sqrt((2 * l + 1) / (4 * np.pi)) * (1 + 2.0 ** -30)
    ea = np.floor(np.log2(bound / dm)) + 1
    return np.where(l >= m, 0.999 / dm / np.exp2(ea), 0.0)


def _one_sign(lmax, spin):
    """alm (4, l, m), square-real packing: a_l0 = 1, a_l0 = 1.1, the top of scale for m = 0, and
    for every order, real and imaginary."""
    top = _top_of_scale(lmax, spin)
    a = np.zeros((4, lmax + 1, lmax + 1))
    a[0, :, 0], a[1, :, 0], a[2, :, 0] = 1.0, 1.1, top[:, 0]
    a[3] = top
    for m in range(1, lmax + 1):                 # Im a_lm: column lmax + 1 - m, row l - m
        a[3, :lmax + 1 - m, lmax + 1 - m] = top[m:, m]
    return a


def _device(a):
    """alm (nsim, l, m) as the device tensor of the same shape and Fortran strides."""
    return torch.tensor(np.ascontiguousarray(a.transpose(2, 1, 0)), device="cuda").permute(2, 1, 0)


# 128 / 63 and 512 / 255 (a_l0 = 1) and 64 / 63 (1.1) reach 1.05 to 1.09 of a 0.4 (lmax/2 + 1) bound
# a parity, the others up to 1.63; 1024 / 3071 and 2048 / 4200: columns with spare bits
@pytest.mark.parametrize("ns,lmax", [(32, 64), (64, 63), (64, 64), (128, 63), (128, 153), (128, 254),
                                     (512, 255), (512, 1018), (1024, 1228), (1024, 3071),
                                     (2048, 4200)])
@pytest.mark.parametrize("kind", ["alm2t", "eb2qu"])
def test_synthesis_of_one_sign_columns(kind, ns, lmax):
    from fastsht_gb300 import SHT
    pol = kind == "eb2qu"
    if pol and ns > 512:
        pytest.skip("spin 2 shares the units; the smaller sizes reach them")
    alm = _one_sign(lmax, 2 if pol else 0)
    ins = [_device(alm)] * (2 if pol else 1)
    out = []
    for limit in (None, (2 if pol else 1) * 4 * 2 * ns * (lmax + 1) * 32):
        kw = {} if limit is None else {"workspace_limit": limit}
        sht = SHT(ns, lmax, 4, pol=pol, **kw)
        res = getattr(sht, kind)(*ins)
        out.append([x.T.clone() for x in (res if pol else (res,))])
        sht.close()
    for got, want in zip(*out):
        assert ((got - want).abs().amax(1) <= TOL * want.abs().amax(1)).all()


@pytest.mark.parametrize("ns,lmax", [(64, 64), (128, 153)])
def test_iterations_on_zonal_maps(ns, lmax):
    """Iterations synthesise what the analysis found: maps of a_l0 at the top of their scale."""
    from fastsht_gb300 import SHT
    alm = _device(_one_sign(lmax, 0)[1:3])
    general = SHT(ns, lmax, 2, workspace_limit=2 * 2 * ns * (lmax + 1) * 32)
    maps = general.alm2t(alm).clone()
    out = []
    for kw in ({}, {"workspace_limit": 2 * 2 * 2 * ns * (lmax + 1) * 32}):
        sht = SHT(ns, lmax, 2, niter=1, **kw)
        out.append(sht.t2alm(maps).reshape(2, -1).clone())
        sht.close()
    assert ((out[0] - out[1]).abs().amax(1) <= TOL * out[1].abs().amax(1)).all()


@pytest.mark.parametrize("ns,lmax", [(1024, 1100), (2048, 1300)])
def test_largest_inverse_ring_transforms(ns, lmax):
    """alm2t with the cap rings in matrix form (24 maps) against the same maps by FFT (12): bins of
    one sign at the top of their scale, and random ones."""
    from fastsht_gb300 import SHT
    g = torch.Generator(device="cuda").manual_seed(ns)
    alm = torch.randn((lmax + 1, lmax + 1, 24), dtype=torch.float64, device="cuda", generator=g)
    alm[..., ::2].abs_()
    out = []
    for k in (24, 12):
        sht = SHT(ns, lmax, k, workspace_limit=64 << 30)
        out.append(sht.alm2t(alm[..., :k].contiguous().permute(2, 1, 0)).T[:12].clone())
        sht.close()
    got, want = out
    assert ((got - want).abs().amax(1) <= TOL * want.abs().amax(1)).all()
