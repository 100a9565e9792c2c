"""What an FP64 plan does where its digit tiles find no room: the limit or the device leaves the FMA
form, which needs the phase matrices only."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fastsht_gb300 import build
    build.build()


@pytest.mark.parametrize("share", [0.1, 0.14, 0.18, 0.22, 0.26, 0.3, 0.34, 0.38, 0.42, 0.46, 0.5])
def test_plan_whose_tiles_do_not_fit_the_device(share):
    """Phase matrices of `share` of the free memory and no limit of the plan's own: the tiles take
    a few times as much, so they fit, fit alone but not beside the matrices, or do not fit."""
    from fastsht_gb300 import SHT
    ns, lmax = 256, 767
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    nsim = int(share * free / (2 * ns * (lmax + 1) * 32))
    sht = SHT(ns, lmax, nsim, workspace_limit=1 << 50)
    assert sht.plan_info()["maps_per_chunk"] == nsim
    sht.close()
    # the thread's next calls are not disturbed by the allocations that failed
    maps = torch.ones((12 * 16 * 16, 1), dtype=torch.float64, device="cuda")
    alm = SHT(16, 20, 1).t2alm(maps)
    assert abs(float(alm[0, 0, 0]) - (4 * torch.pi) ** 0.5) < 1e-12


@pytest.mark.parametrize("precision,pol,limit", [("fp64", False, 0), ("fp64", True, 0),
                                                 ("fp64", True, 2 << 30), ("split", True, 0)])
def test_plan_info_counts_what_the_plan_holds(precision, pol, limit):
    """device_bytes against the device's own count: digit tiles, tables, and a limit that leaves
    the FMA form.  (64 MiB for the blocks that the device rounds up to, and its streams.)"""
    from fastsht_gb300 import SHT
    ns, lmax = 256, 767

    def plan():
        return SHT(ns, lmax, 64, pol=pol, precision=precision, workspace_limit=limit)
    plan().close()                              # kernels that load on first use
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    sht = plan()
    torch.cuda.synchronize()
    held = free - torch.cuda.mem_get_info()[0]
    assert abs(held - sht.plan_info()["device_bytes"]) <= 64 << 20
    sht.close()


def test_stages_take_the_maps_of_a_chunk_without_tiles():
    """A limit that holds 640 maps' phase matrices, and 64 maps with their digit tiles: the
    stages, which need no tiles, run on all 640."""
    import ctypes as C
    from fastsht_gb300 import _lib
    ns, lmax, nsim = 64, 191, 640
    plan = C.c_void_p()
    _lib.call("fsht_plan_create", ns, lmax, nsim, 0, _lib.FSHT_PREC_FP64,
              nsim * 2 * ns * (lmax + 1) * 32, None, C.byref(plan))
    try:
        k = C.c_int()
        _lib.call("fsht_plan_info", plan, None, C.byref(k))
        assert 64 <= k.value < nsim and k.value % 64 == 0
        maps = torch.ones((nsim, 12 * ns * ns), dtype=torch.float64, device="cuda")
        W = torch.zeros((lmax + 1, 2 * ns, nsim, 2, 2), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        _lib.call("fsht_run_stage", plan, 0, C.c_void_p(maps.data_ptr()), C.c_void_p(W.data_ptr()),
                  nsim)
        _lib.call("fsht_plan_sync", plan)
        # m = 0, every ring but the equator: S = F_N + F_S = 2 n, D = 0
        assert (W[0, :-1, :, 0, 0] > 7).all() and W[0, :-1, :, 1].abs().max() < 1e-10
        with pytest.raises(ValueError):
            _lib.call("fsht_run_stage", plan, 0, C.c_void_p(maps.data_ptr()),
                      C.c_void_p(W.data_ptr()), nsim + 1)
    finally:
        _lib.load().fsht_plan_destroy(plan)
