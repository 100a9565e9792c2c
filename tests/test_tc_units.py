"""The integer units of the FP64 digit products (fastsht_gb300/csrc/tc_units.h) hold the largest
sums the kernels can form: sum over the operands |row| |column| with both at most one, times 2^12,
in units of 2^-bits, within 2^63.

Synthesis, every lmax from 1 to 4 nside: the running sum over l of one order and ring, rows in the
kernel's own scale (the power of two above bound / Dm for the mantissa Dm of D_l, spin 2: of N_l),
columns of one sign at the top of their scale.  Ring transforms: all accepted nside.
"""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastsht_gb300" / "csrc"
SHIM = """
#include "tc_units.h"
static int put(FshtTcUnits u, int* head) { *head = u.head; return u.bits; }
extern "C" int synthesis(int lmax, int* head) { return put(fsht_tc_units_synthesis(lmax), head); }
extern "C" int analysis(int ns, int lmax, int* head) {
  return put(fsht_tc_units_analysis(ns, lmax), head);
}
extern "C" int dft(int nk, int extra, int* head) { return put(fsht_tc_units_dft(nk, extra), head); }
"""


@pytest.fixture(scope="module")
def units(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("units")
    (d / "u.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CSRC),
                    str(d / "u.cpp"), "-o", str(d / "u.so")], check=True)
    lib = C.CDLL(str(d / "u.so"))

    def call(name, *args):
        head = C.c_int()
        bits = getattr(lib, name)(*args, C.byref(head))
        assert 40 <= bits <= 46 and 0 <= head.value <= 3      # what the drains take
        return bits - head.value
    return call


def _row_sums(ns, mmax):
    """Per l: the largest running sum over l' <= l of |row| over orders m <= mmax and rings, spin 0
    and 2; and the largest row."""
    lmax, nn = 4 * ns, 2 * ns
    i = np.arange(nn) + 1
    z = np.where(i < ns, 1 - i * i / (3.0 * ns * ns), (2 * ns - i) * 2 / (3.0 * ns))
    s = np.sqrt((1 - z) * (1 + z))
    m = np.arange(mmax + 1)[:, None].astype(float)
    k = np.arange(1, mmax + 1)
    lg = np.concatenate([[0], np.cumsum(np.log2((2 * k + 1) / (2 * k)))])[:, None]
    lg = 0.5 * (lg - np.log2(4 * np.pi)) + m * np.log2(s)[None]
    e = np.minimum(0, np.ceil((lg - 300) / 600))
    seed = np.exp2(lg - 600 * e)
    cur, prev = np.zeros((2, mmax + 1, nn))
    log_d = np.zeros((mmax + 1, 1))           # log2 D_l = sum log2 a_k
    run = np.zeros((2, mmax + 1, nn))
    sums, top = np.zeros((lmax + 1, 2)), 0.0
    for l in range(lmax + 1):
        with np.errstate(all="ignore"):
            a2 = np.where(l > m, (4.0 * l * l - 1) / (l * l - m * m), 1.0)
            a = np.where(l > m, np.sqrt(a2), 0.0)
            b = np.nan_to_num(np.where(
                l > m, np.sqrt(((l - 1) ** 2 - m * m) / (4.0 * (l - 1) ** 2 - 1)) * a, 0))
        log_d += 0.5 * np.log2(a2)
        nx = a * z * cur - b * prev
        if l <= mmax:
            nx[l] = seed[l]
        prev, cur = cur, nx
        up = (np.abs(cur) > 2.0 ** 300) & (e < 0)
        cur, prev = np.where(up, cur * 2.0 ** -600, cur), np.where(up, prev * 2.0 ** -600, prev)
        e = e + up
        w = (m <= l) & (e >= 0)
        lam, lp = np.where(w, cur, 0), np.where(w, prev, 0)
        bound = np.sqrt((2 * l + 1) / (4 * np.pi)) * (1 + 2.0 ** -30)
        dm = np.exp2(log_d - np.floor(log_d))                       # mantissa in [1, 2)
        row = np.abs(lam) / dm / np.exp2(np.floor(np.log2(bound / dm)) + 1)
        run[0] += row
        top = max(top, row.max())
        if l >= 2:
            nl = 1 / np.sqrt((l + 2.0) * (l + 1.0) * l * (l - 1.0))
            lf = 2 * np.sqrt(np.maximum((2 * l + 1.0) / (2 * l - 1.0) * (l * l - m * m), 0))
            l1 = (lp * lf * z / s ** 2 - lam * (2 * (l - m * m) / s ** 2 + l * (l - 1.0))) * nl
            l2 = (lp * lf - lam * 2 * z * (l - 1.0)) * m / s ** 2 * nl
            dm = nl / np.exp2(np.floor(np.log2(nl)))
            row = ((np.abs(l1) + np.abs(l2)) / dm / np.exp2(np.floor(np.log2(bound / dm)) + 1))
            run[1] += row
            top = max(top, row.max())
        sums[l] = run.max((1, 2))
    return sums, top


@pytest.mark.parametrize("ns,mmax", [(32, 128), (64, 256), (128, 40), (512, 2), (1024, 2)])
def test_synthesis_sums_fit(units, ns, mmax):
    sums, top = _row_sums(ns, mmax)
    assert top < 1.0
    for lmax in range(1, 4 * ns + 1):
        bits = units("synthesis", lmax)
        assert sums[lmax].max() * 2.0 ** (12 + bits) < 2.0 ** 63, (ns, lmax)
        assert lmax + 1 <= 2.0 ** (63 - 12 - bits)             # every row and column at its top


@pytest.mark.parametrize("ns", [32, 256, 2048])
def test_analysis_sums_fit(units, ns):
    # (sum over rings of |lambda| < 0.85 nside: test_tc_bounds.py)
    for lmax in (1, ns, 2 * ns, 3 * ns - 1):
        eag = int(np.floor(np.log2(np.sqrt((2 * lmax + 1) / (4 * np.pi)) * (1 + 2.0 ** -30)))) + 1
        assert 0.85 * ns * 2.0 ** (12 + units("analysis", ns, lmax) - eag) < 2.0 ** 63


@pytest.mark.parametrize("ns", [32, 64, 128, 256, 512, 1024, 2048])
def test_ring_transform_sums_fit(units, ns):
    # forward (folds of two rings), inverse (four mirrored samples); the matrices hold cos 2^61
    nk = ns + 1 if ns <= 256 else ns - 1
    for extra in (1, 2):
        assert nk * 0.5 * 2.0 ** extra * 2.0 ** (12 + units("dft", nk, extra)) <= 2.0 ** 63
