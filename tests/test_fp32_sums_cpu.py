"""The three-float sums and quotients of the FP32 PCG against FP64's.

Both forms of a dot are formed on the host: a thread's products into a
two-float sum and an FP64 tree over the threads, and three floats all the way,
from the header that the kernels use, over as many threads as the kernels run.
Exact values are rationals.  The limits are FP64's own: on no data may the
three-float form's error, over many dots, exceed the FP64 tree's.
"""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "specfem3d_geotech_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SRC = r"""
#include <vector>
#include "sg_sum3.cuh"
using namespace sg;
// thread i takes products i, i + nt, ... as the kernels do; the forms of a thread's sum:
enum { ONE_BY_ONE, FEW, MANY, FOURS, HALVES };
static Sum3 thread_sum(const float* a, const float* b, int n, int nt, int i, int form) {
  const int cnt = i < n ? (n - 1 - i) / nt + 1 : 0;
  CompSum c, half;
  CompSum3 m;
  for (int k = 0; k < cnt; ++k) {
    const float x = a[i + (size_t)k * nt], y = b[i + (size_t)k * nt];
    if (form == MANY) {
      m.add(x, y);
    } else if (form == FOURS) {
      CompSum g;
      g.set(x, y);
      for (int q = 1; q < 4 && k + 1 < cnt; ++q) { ++k; g.add(a[i + (size_t)k * nt], b[i + (size_t)k * nt]); }
      c.add(g);
    } else if (form == FEW && k == 0) {
      c.set(x, y);
    } else {
      c.add(x, y);
    }
    if (form == HALVES && k + 1 == 2 * ((cnt + 3) / 4)) { half = c; c = CompSum(); }
  }
  Sum3 s = form == MANY ? m.sum() : c.sum();
  if (form == HALVES) s.add(half.sum());
  return s;
}
// lanes by halves, the block's warps and then the blocks one after the other
template <typename S, typename ADD>
static S tree(std::vector<S>& x, int block, S zero, ADD add) {
  S all = zero;
  for (size_t b0 = 0; b0 < x.size(); b0 += block) {
    S bl = zero;
    for (size_t w = b0; w < b0 + block && w < x.size(); w += 32) {
      for (int o = 16; o >= 1; o >>= 1)
        for (int i = 0; i < o; ++i)
          if (w + i + o < x.size()) add(x[w + i], x[w + i + o]);
      add(bl, x[w]);
    }
    add(all, bl);
  }
  return all;
}
extern "C" double dot64(const float* a, const float* b, int n, int nt) {
  std::vector<double> x;
  for (int i = 0; i < nt; ++i) {
    const Sum3 s = thread_sum(a, b, n, nt, i, ONE_BY_ONE);
    x.push_back((double)s.h + (double)s.l);
  }
  return tree(x, 256, 0.0, [](double& s, double y) { s += y; });
}
extern "C" void dot3(const float* a, const float* b, int n, int nt, int block, int form, float* out) {
  std::vector<Sum3> x;
  for (int i = 0; i < nt; ++i) x.push_back(thread_sum(a, b, n, nt, i, form));
  const Sum3 s = tree(x, block, zero3(), [](Sum3& s, const Sum3& y) { s.add(y); });
  out[0] = s.h; out[1] = s.l; out[2] = s.m;
}
extern "C" float quotient(const float* a, const float* b) {
  return div3(norm3(Sum3{a[0], a[1], a[2]}), norm3(Sum3{b[0], b[1], b[2]}));
}
extern "C" void parts(double x, float* out) {
  const Sum3 s = split3(x);
  out[0] = s.h; out[1] = s.l; out[2] = s.m;
}
extern "C" double joined(const float* a) { return Sum3{a[0], a[1], a[2]}.value(); }
extern "C" int le(const float* a, const float* b) { return at_most(norm3(Sum3{a[0], a[1], a[2]}), norm3(Sum3{b[0], b[1], b[2]})); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sums")
    (d / "s.cpp").write_text(SRC)
    so = str(d / "s.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-I",
                    CUDA + "/include", str(d / "s.cpp"), "-o", so], check=True, timeout=300)
    L = ctypes.CDLL(so)
    L.dot64.restype = L.joined.restype = ctypes.c_double
    L.quotient.restype = ctypes.c_float
    vp, i = ctypes.c_void_p, ctypes.c_int
    L.parts.argtypes = [ctypes.c_double, vp]
    L.dot64.argtypes = [vp, vp, i, i]
    L.dot3.argtypes = [vp, vp, i, i, i, i, vp]
    L.quotient.argtypes = L.le.argtypes = [vp, vp]
    L.joined.argtypes = [vp]
    return L


def f3(fn, *args):
    out = np.zeros(3, np.float32)
    fn(*(a.ctypes.data if isinstance(a, np.ndarray) else a for a in args), out.ctypes.data)
    return out


def exact(t):
    return sum((Fraction(float(v)) for v in t), Fraction(0))


def vectors(kind, n, rng):
    r = (rng.standard_normal(n) * np.exp(3.0 * rng.standard_normal(n))).astype(np.float32)
    if kind == "rr":
        return r, r
    if kind == "rz":                    # z = D r with a diagonal of wide range
        return r, (r * np.exp(2.0 * rng.standard_normal(n)).astype(np.float32))
    # p.Kp: terms of both signs whose sum is a hundredth of their size
    q = rng.standard_normal(n).astype(np.float32)
    return r, ((q + 0.01 * r / np.float32(np.abs(r).mean())).astype(np.float32))


ONE_BY_ONE, FEW, MANY, FOURS, HALVES = range(5)


def forms(kr, n):
    """Threads per column of the FP64-tree kernels and of today's for n rows and
    kr columns, with the block size and how a thread adds its products."""
    q = max(1, kr // 4)                           # threads of a row: four columns each
    few = -(-n * q // 4 // 256) * 256 // q        # at least four rows a thread, up to 608 blocks
    update, gather = min(155648 // q, few), min({4: 145920, 8: 72960, 16: 29184}[kr], few)
    nt = 72960 // q
    yield "persistent", [min(155648 // q, -(-n // 256) * 256)], (nt, 480, FEW if n <= 4 * nt else MANY)
    yield "update", [max(256, update)], (77824 // q, 512, FOURS)
    yield "gather", [max(256, gather)], ({4: 116736, 8: 58368, 16: 29184}[kr], 384, HALVES)


@pytest.mark.parametrize("kr, n, dots", [(4, 200, 60), (4, 9000, 60), (16, 9000, 60), (8, 120000, 30), (16, 120000, 30),
                                         (8, 500000, 10), (4, 1600000, 5), (8, 1600000, 5)])
def test_dots_are_no_further_off_than_with_fp64_trees(lib, kr, n, dots):
    """Rows of 8 elements to 62,000 (1.6 million rows).  Either error is a random
    one whose size is set by few of the products: the median over the dots."""
    rng = np.random.default_rng(n)
    errs = {}
    for i in range(dots):
        for kind in ("rr", "rz", "pkp"):
            a, b = vectors(kind, n, rng)
            # products of 24-bit numbers are exact in FP64: add them as integers, exponent by exponent
            p = a.astype(np.float64) * b.astype(np.float64)
            mant, expo = np.frexp(p)
            ex = sum(Fraction(sum(np.ldexp(mant[expo == v], 53).astype(np.int64).tolist()))
                     * Fraction(2) ** (int(v) - 53) for v in np.unique(expo))
            for name, before, now in forms(kr, n):
                if name == ("update" if kind == "pkp" else "gather"):
                    continue                      # that kernel forms no such dot
                e64, e3 = errs.setdefault(name, ([], []))
                e64 += [float(abs((Fraction(lib.dot64(a.ctypes.data, b.ctypes.data, n, nt)) - ex) / ex)) for nt in before]
                e3.append(float(abs((exact(f3(lib.dot3, a, b, n, *now)) - ex) / ex)))
    for name, (e64, e3) in errs.items():
        print(kr, n, name, "FP64 tree %.1e, three floats %.1e" % (np.median(e64), np.median(e3)))
        assert np.median(e3) <= np.median(e64), name


def rounded(x):
    """x (a rational) to FP32, to nearest even."""
    f = np.float32(float(x))
    near = [f, np.nextafter(f, np.float32(-np.inf)), np.nextafter(f, np.float32(np.inf))]
    return min(near, key=lambda v: (abs(Fraction(float(v)) - x), int(v.view(np.uint32)) & 1))


def test_quotients_are_rounded_once(lib):
    """Any three-float numbers, and quotients 2^-46 of themselves beside the
    middle of two FP32 numbers: an FP64 quotient of sums that are FP64 sums
    decides those no better."""
    rng = np.random.default_rng(5)
    for i in range(20000):
        b = f3(lib.parts, float(np.ldexp(1 + rng.random(), rng.integers(-20, 40))))
        b[2] += np.float32(rng.standard_normal() * 2.0 ** -50) * b[0]
        if i % 2:
            a = f3(lib.parts, float(np.ldexp(1 + rng.random(), rng.integers(-20, 40))))
        else:
            q = np.float32(1 + rng.random())
            mid = (Fraction(float(q)) + Fraction(float(np.nextafter(q, np.float32(4))))) / 2
            x = exact(b) * mid * (1 + rng.choice([-1, 1]) * Fraction(1, 1 << 46))
            h = np.float32(float(x))
            m = np.float32(float(x - Fraction(float(h))))
            a = np.array([h, m, np.float32(float(x - Fraction(float(h)) - Fraction(float(m))))], np.float32)
        assert lib.quotient(a.ctypes.data, b.ctypes.data) == rounded(exact(a) / exact(b))


def test_parts_compare_and_join(lib):
    rng = np.random.default_rng(6)
    for _ in range(5000):
        x = float(np.ldexp(1 + rng.random(), rng.integers(-40, 60)))
        t = f3(lib.parts, x)
        assert exact(t) == Fraction(x) and lib.joined(t.ctypes.data) == x
        for y in (x, np.nextafter(x, 0.0), np.nextafter(x, np.inf), 0.5 * x, 2.0 * x):
            u = f3(lib.parts, float(y))
            assert lib.le(t.ctypes.data, u.ctypes.data) == (x <= y)
    inf, nan, zero = (np.array([v, 0, 0], np.float32) for v in (np.inf, np.nan, 0.0))
    one = np.array([1, 0, 0], np.float32)
    div = lambda x, y: lib.quotient(x.ctypes.data, y.ctypes.data)  # noqa: E731
    assert div(one, zero) == np.inf and np.isnan(div(zero, zero)) and div(zero, one) == 0
    assert np.isnan(div(nan, one)) and np.isnan(div(one, nan)) and div(inf, one) == np.inf
    assert not lib.le(nan.ctypes.data, one.ctypes.data) and not lib.le(one.ctypes.data, nan.ctypes.data)
