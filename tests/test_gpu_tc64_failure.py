"""Expired device waits of FP64 calls, which return before the device is done: the plan's next call
reports them, and so does a call whose result goes to a host array.  (The wait is the library's
self-test: a bounded one that nothing satisfies.)"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fastsht_gb300 import build
    build.build()


def test_expired_wait_is_reported_by_the_next_call():
    from fastsht_gb300 import SHT, _lib
    lib = _lib.load()
    ns, lmax = 32, 64
    sht = SHT(ns, lmax, 2, pol=True)
    maps = torch.randn((2, 12 * ns * ns), dtype=torch.float64, device="cuda").T
    want = sht.t2alm(maps).clone()
    for call in (lambda: sht.t2alm(maps), lambda: sht.alm2t(want), lambda: sht.qu2eb(maps, maps),
                 lambda: sht.eb2qu(want, want)):
        assert lib.fsht_selftest_wait_timeout(sht._plan) == _lib.FSHT_OK
        torch.cuda.synchronize()
        with pytest.raises(_lib.FshtError) as ei:
            call()
        assert ei.value.code == _lib.FSHT_ETIMEOUT and "earlier" in str(ei.value)
        call()                                                     # cleared
    assert torch.equal(sht.t2alm(maps), want)
    assert lib.fsht_plan_sync(sht._plan) == _lib.FSHT_OK


def test_expired_wait_is_reported_with_a_host_result():
    from fastsht_gb300 import SHT, _lib
    lib = _lib.load()
    ns, lmax = 32, 64
    sht = SHT(ns, lmax, 1)
    alm = np.zeros((1, lmax + 1, lmax + 1), order="F")
    alm[0, 0, 0] = 1.0
    assert lib.fsht_selftest_wait_timeout(sht._plan) == _lib.FSHT_OK   # still running at the call
    with pytest.raises(_lib.FshtError) as ei:
        sht.alm2t(alm)
    assert ei.value.code == _lib.FSHT_ETIMEOUT
    assert np.abs(sht.alm2t(alm) - 1 / np.sqrt(4 * np.pi)).max() < 1e-12


def test_more_plans_than_shared_error_words():
    """1,030 plans at once, each with a word of its own; the last one's expiry is its own."""
    from fastsht_gb300 import SHT, _lib
    lib = _lib.load()
    plans = [SHT(4, 4, 1) for _ in range(1030)]
    assert lib.fsht_selftest_wait_timeout(plans[-1]._plan) == _lib.FSHT_OK
    torch.cuda.synchronize()
    assert [lib.fsht_plan_check(p._plan) for p in plans] == [_lib.FSHT_OK] * 1029 + [_lib.FSHT_ETIMEOUT]
    for p in plans:
        p.close()
    assert lib.fsht_plan_check(SHT(4, 4, 1)._plan) == _lib.FSHT_OK
