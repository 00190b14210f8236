"""Quotients that share a reciprocal round as the division does, for every
numerator and divisor (csrc/quotient.cuh compiled for the host; both its
multiply-add and the device's round once, and 1/b is the IEEE quotient on
both)."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "mfix-cfd-dem_b200" / "csrc"
SRC = """
#include "quotient.cuh"
template <int N> static long run(long n, const double* a, const double* b, double* q) {
  long shared = 0;
  for (long k = 0; k < n; ++k) shared += demb::quotients<N>(a + N * k, b[k], 1.0 / b[k], q + N * k);
  return shared;
}
extern "C" long quotients3(long n, const double* a, const double* b, double* q) { return run<3>(n, a, b, q); }
extern "C" long quotients5(long n, const double* a, const double* b, double* q) { return run<5>(n, a, b, q); }
extern "C" void contacts(long n, const double* dist, const double* dmag, const double* r, double* nrm, double* arm) {
  for (long k = 0; k < n; ++k)
    demb::contact_quotients(dist + 3 * k, dmag[k], r[2 * k], r[2 * k + 1], nrm + 3 * k, arm[2 * k], arm[2 * k + 1]);
}
extern "C" void in_place(long n, double* a, const double* b) {
  for (long k = 0; k < n; ++k) demb::div3(a + 3 * k, b[k], a + 3 * k);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotient")
    (d / "q.cc").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-march=native", "-ffp-contract=off", "-Wno-unknown-pragmas", "-shared",
                    "-fPIC", "-I", str(CSRC), str(d / "q.cc"), "-o", str(d / "q.so")], check=True)
    lib = C.CDLL(str(d / "q.so"))
    lib.quotients3.restype = lib.quotients5.restype = C.c_long
    return lib


def _p(x):
    return x.ctypes.data_as(C.POINTER(C.c_double))


def _check(lib, width, a, b):
    """a[n, width] / b[n] bit for bit; the number of rows that shared 1/b."""
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    q = np.empty_like(a)
    shared = getattr(lib, f"quotients{width}")(C.c_long(len(b)), _p(a), _p(b), _p(q))
    with np.errstate(all="ignore"):
        want = a / b[:, None]
    same = (q.view(np.int64) == want.view(np.int64)) | (np.isnan(q) & np.isnan(want))
    bad = np.argwhere(~same)
    assert not len(bad), (len(bad), a[bad[0][0]].tolist(), b[bad[0][0]])
    if width == 3:
        c = a.copy()
        lib.in_place(C.c_long(len(b)), _p(c), _p(b))
        assert ((c.view(np.int64) == want.view(np.int64)) | (np.isnan(c) & np.isnan(want))).all()
    return shared


def _mantissas(rng, shape):
    """Random ones, and ones within a few units of 1 and of 2."""
    m = 1.0 + rng.random(shape)
    near = rng.integers(0, 4, shape) * 2.0 ** -52
    kind = rng.integers(0, 4, shape)
    m = np.where(kind == 0, 1.0 + near, np.where(kind == 1, 2.0 - 2.0 ** -52 - near, m))
    return m * rng.choice([-1.0, 1.0], shape)


@pytest.mark.parametrize("width", [3, 5])
def test_ordinary_quotients(lib, width):
    """Magnitudes of the contact arithmetic: all share."""
    rng = np.random.default_rng(7)
    n = 400_000
    a = _mantissas(rng, (n, width)) * 2.0 ** rng.integers(-120, 120, (n, width))
    a[rng.random((n, width)) < 0.1] = 0.0
    a[rng.random((n, width)) < 0.05] = -0.0
    b = np.abs(_mantissas(rng, n)) * 2.0 ** rng.integers(-60, 60, n)
    assert _check(lib, width, a, b) == n


@pytest.mark.parametrize("width", [3, 5])
@pytest.mark.parametrize("ea", [(-1074, -900), (-1000, -480), (-510, -490), (380, 420), (560, 640), (900, 1023)])
@pytest.mark.parametrize("eb", [(-1074, -1000), (-410, -390), (-5, 5), (390, 410), (900, 1023)])
def test_range_edges(lib, width, ea, eb):
    """Exponents around each bound of the range, down to subnormal numerators
    and up to quotients that overflow; one ordinary numerator beside them."""
    rng = np.random.default_rng(abs(ea[0]) * 7 + abs(eb[0]))
    n = 20_000
    with np.errstate(all="ignore"):
        a = np.ldexp(_mantissas(rng, (n, width)), rng.integers(*ea, (n, width)))
        a[:, 0] = np.ldexp(_mantissas(rng, n), rng.integers(-20, 20, n))
        b = np.ldexp(np.abs(_mantissas(rng, n)), rng.integers(*eb, n))
    _check(lib, width, a, b)


@pytest.mark.parametrize("width", [3, 5])
def test_special_values(lib, width):
    v = np.array([0.0, -0.0, 5e-324, -5e-324, 2.0 ** -1022, 2.0 ** -500, 2.0 ** -500 * (1 - 2.0 ** -53), 1.0, -3.0,
                  2.0 ** 600, 1.7976931348623157e308, np.inf, -np.inf, np.nan])
    w = np.concatenate([v, -v, [2.0 ** -400, 2.0 ** 400, 2.0 ** 400 * (1 - 2.0 ** -53)]])
    rng = np.random.default_rng(3)
    _check(lib, width, rng.choice(v, (40_000, width)), rng.choice(w, 40_000))


@pytest.mark.parametrize("scale", [0, -160, -199, -201, -440, 199, 399, 401, 500])
def test_contact_quotients(lib, scale):
    """Normals and lever arms of overlapping spheres, equal radii and aligned
    or nearly aligned centres among them, at lengths around 2^scale."""
    rng = np.random.default_rng(500 + scale)
    n = 60_000
    r = np.ldexp(1.0 + rng.random((n, 2)), scale + rng.integers(-1, 2, (n, 2)))
    r[: n // 3, 1] = r[: n // 3, 0]
    r[n // 3: n // 2, 1] = np.nextafter(r[n // 3: n // 2, 0], 0.0)
    u = rng.normal(size=(n, 3))
    u[rng.random((n, 3)) < 0.2] = 0.0
    few = rng.random((n, 3)) < 0.1
    u = np.where(few, np.ldexp(u, rng.integers(-900, 0, (n, 3))), u)
    u[np.abs(u).max(1) < 0.1] = [1.0, 0.0, -0.0]
    u /= np.abs(u).max(1)[:, None] * np.sqrt(3.0)
    dist = u * (0.95 * r.sum(1))[:, None]
    dmag = np.sqrt((dist * dist).sum(1))
    ok = (dmag > 0.0) & (dmag <= r.sum(1))
    dist, dmag, r = (np.ascontiguousarray(x[ok]) for x in (dist, dmag, r))
    nrm, arm = np.empty_like(dist), np.empty_like(r)
    lib.contacts(C.c_long(len(dmag)), _p(dist), _p(dmag), _p(r), _p(nrm), _p(arm))
    with np.errstate(all="ignore"):
        rl2, ri2 = r[:, 0] * r[:, 0], r[:, 1] * r[:, 1]
        wn = dist / dmag[:, None]
        wa = np.stack([(dmag * dmag + rl2 - ri2) / (2.0 * dmag), (rl2 - ri2) / (2.0 * dmag)], 1)
    for got, want in ((nrm, wn), (arm, wa)):
        same = (got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want))
        assert same.all(), int((~same).sum())
    assert len(dmag) > n // 2 or abs(scale) > 400
