"""FP64 plans of small lmax: which form the ring transforms take, results and times against the
general path (a limit without room for digit tiles: ring FFTs and FMA kernels)."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fastsht_gb300 import build
    build.build()


def _input(kind, ns, lmax, nsim):
    g = torch.Generator(device="cuda").manual_seed(ns + lmax + nsim)
    if kind == "t2alm":
        return torch.randn((nsim, 12 * ns * ns), dtype=torch.float64, device="cuda", generator=g).T
    return torch.randn((lmax + 1, lmax + 1, nsim), dtype=torch.float64, device="cuda",
                       generator=g).permute(2, 1, 0)


def _plans(ns, lmax, nsim):
    from fastsht_gb300 import SHT
    return SHT(ns, lmax, nsim), SHT(ns, lmax, nsim,
                                    workspace_limit=nsim * 2 * ns * (lmax + 1) * 32)


# short waves of rings (few orders a plan), on both sides of the rule; one tile, two, a rest
@pytest.mark.parametrize("kind", ["t2alm", "alm2t"])
@pytest.mark.parametrize("ns,lmax,nsim", [(32, 0, 64), (32, 1, 70), (32, 16, 48), (32, 64, 128),
                                          (32, 95, 192), (64, 3, 64), (64, 16, 40), (64, 63, 129),
                                          (128, 2, 65), (128, 32, 96), (128, 128, 100),
                                          (256, 10, 40), (256, 32, 96), (512, 15, 24),
                                          (32, 0, 1), (64, 31, 16), (64, 32, 16), (64, 31, 17),
                                          (256, 15, 1), (256, 16, 1)])
def test_small_lmax_equals_general_path(kind, ns, lmax, nsim):
    x = _input(kind, ns, lmax, nsim)
    out = []
    for sht in _plans(ns, lmax, nsim):
        r = getattr(sht, kind)(x.clone())
        out.append((r.T if kind == "alm2t" else r).reshape(nsim, -1).clone())
        sht.close()
    assert ((out[0] - out[1]).abs().amax(1) <= 1e-11 * out[1].abs().amax(1)).all()


@pytest.mark.parametrize("kind", ["t2alm", "alm2t"])
@pytest.mark.parametrize("ns,lmax,nsim", [(32, 3, 64), (64, 20, 40), (128, 2, 64), (256, 10, 40)])
def test_small_lmax_is_not_slower(kind, ns, lmax, nsim):
    """The matrix form of the ring transforms took up to twenty times the FFT's time here; twice
    the general path's is left for noise."""
    x = _input(kind, ns, lmax, nsim)
    ms = []
    for sht in _plans(ns, lmax, nsim):
        f = getattr(sht, kind)
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            f(x)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        ms.append(min(times))
        sht.close()
    assert ms[0] <= 2.0 * ms[1]


def test_more_maps_than_a_grid_dimension():
    """262,208 maps of nside 32 in one call: the ring slices' grids stay within their limits."""
    from fastsht_gb300 import SHT
    ns, lmax, nsim = 32, 1, 262208
    maps = torch.full((nsim, 12 * ns * ns), 2.0, dtype=torch.float64, device="cuda")
    x = _input("t2alm", ns, lmax, 64)
    maps[-64:] = x.T
    sht = SHT(ns, lmax, nsim)
    alm = sht.t2alm(maps.T)
    want = SHT(ns, lmax, 64).t2alm(x)
    assert ((alm[-64:] - want).abs().max() <= 1e-13 * want.abs().max())
    assert ((alm[:-64, 0, 0] - 2.0 * (4 * torch.pi) ** 0.5).abs().max() <= 1e-12)
