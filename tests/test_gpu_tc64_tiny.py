"""Ring transforms in matrix form on values below FP64's normal range, against the FFT route."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fastsht_gb300 import build
    build.build()


@pytest.mark.parametrize("kind", ["t2alm", "alm2t"])
def test_subnormal_maps(kind):
    """64 maps in matrix form against 8 by FFT: white values of 2^-1000 (normal) and 2^-1040.  The
    sums round in units of 2^-1074, a few thousand times a result at most."""
    from fastsht_gb300 import SHT
    ns, lmax = 64, 127
    g = torch.Generator(device="cuda").manual_seed(1)
    shape = (64, 12 * ns * ns) if kind == "t2alm" else (64, lmax + 1, lmax + 1)
    x = torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
    x[::2] *= 2.0 ** -1000
    x[1::2] *= 2.0 ** -1000
    x[1::2] *= 2.0 ** -40
    out = []
    for k in (64, 8):
        sht = SHT(ns, lmax, k)
        if kind == "t2alm":
            out.append(sht.t2alm(x[:k].contiguous().T)[:8].reshape(8, -1).clone())
        else:
            y = x[:k].permute(2, 1, 0).contiguous().permute(2, 1, 0)
            out.append(sht.alm2t(y).T[:8].clone())
        sht.close()
    got, want = out
    top = want.abs().amax(1)
    assert (top > 0).all()
    assert ((got - want).abs().amax(1) <= 1e-11 * top + 2.0 ** -1062).all()
