"""The split synthesis' size rules against the FP64 form, at the form's 1e-7 bar: few maps (rings on
the TMEM lanes up to 32 maps, columns above), slicing in clusters (512 / 1040) and sums in two parts
(lmax > 2047)."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fastsht_gb300 import build
    build.build()


@pytest.mark.parametrize("ns,lmax,nsim", [(16, 40, 1), (64, 160, 7), (64, 160, 31), (64, 160, 32),
                                          (64, 160, 33), (64, 191, 65), (512, 1040, 2),
                                          (1024, 2100, 3)])
def test_split_synthesis_sizes_match_fp64(ns, lmax, nsim):
    from fastsht_gb300 import SHT
    g = torch.Generator(device="cuda").manual_seed(ns + nsim)
    alm = torch.randn((lmax + 1, lmax + 1, nsim), dtype=torch.float64, device="cuda", generator=g)
    out = []
    for precision in ("fp64", "split"):
        sht = SHT(ns, lmax, nsim, precision=precision)
        out.append(sht.alm2t(alm.permute(2, 1, 0)).T.clone())
        sht.close()
    want, got = out
    assert ((got - want).abs().amax(1) <= 1e-7 * want.abs().amax(1)).all()
