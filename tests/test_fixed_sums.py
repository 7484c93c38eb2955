"""The fixed-point stencil sums (csrc/swg_fixed.cuh) on the CPU, where the
header's functions compile as plain C++: words and weights are exact, and a
sum of N products is within its stated distance of the exact one, over mixed
magnitudes, signs and cancelling terms; what cannot be represented is
flagged."""
import ctypes
import math
import os
import random
import struct
import subprocess
from fractions import Fraction

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "omega_playground_gb300",
                    "csrc")
SRC = r"""
#include "swg_fixed.cuh"
using namespace swg;
template <int N>
static double sum(const double *w, const double *x, unsigned *flag) {
  Wt W[N];
  fx_t X[N];
  long long s = 0;
  unsigned f = 0;
  for (int j = 0; j < N; ++j) {
    W[j] = fx_weight(w[j], f);
    X[j] = fx_word(x[j]);
    s += W[j].hi;
  }
  double r = fx_sum(W, X, fx_start(s), f);
  *flag = f;
  return r;
}
template <int N>
static double raw(const double *w, const double *x, unsigned *slow) {
  Wt W[N];
  double X[N];
  unsigned f = 0;
  for (int j = 0; j < N; ++j) {
    W[j] = fx_raw_weight(w[j], f);
    X[j] = x[j];
  }
  bool s = f != 0;
  double r = fx_raw_sum(W, X, s);
  *slow = s;
  return r;
}
extern "C" {
double raw3(const double *w, const double *x, unsigned *f) { return raw<3>(w, x, f); }
double raw6(const double *w, const double *x, unsigned *f) { return raw<6>(w, x, f); }
unsigned long long word(double x) { return fx_word(x); }
void weight(double w, long long *W, int *e, unsigned *flag) {
  *flag = 0;
  Wt t = fx_weight(w, *flag);
  *W = ((long long)t.hi << 28) + t.lo;
  *e = t.e;
}
double sum7(const double *w, const double *x, unsigned *f) { return sum<7>(w, x, f); }
double sum8(const double *w, const double *x, unsigned *f) { return sum<8>(w, x, f); }
double sum14(const double *w, const double *x, unsigned *f) { return sum<14>(w, x, f); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fx")
    src, so = d / "fx.cpp", d / "fx.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC,
                    "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.word.restype = ctypes.c_uint64
    lib.word.argtypes = [ctypes.c_double]
    lib.weight.argtypes = [ctypes.c_double, ctypes.POINTER(ctypes.c_int64),
                           ctypes.POINTER(ctypes.c_int),
                           ctypes.POINTER(ctypes.c_uint)]
    for f in [getattr(lib, f"sum{n}") for n in (7, 8, 14)] + [lib.raw3,
                                                              lib.raw6]:
        f.restype = ctypes.c_double
        f.argtypes = [ctypes.POINTER(ctypes.c_double),
                      ctypes.POINTER(ctypes.c_double),
                      ctypes.POINTER(ctypes.c_uint)]
    return lib


def _sum(lib, w, x):
    n = len(w)
    f = ctypes.c_uint()
    r = getattr(lib, f"sum{n}")((ctypes.c_double * n)(*w),
                                (ctypes.c_double * n)(*x), ctypes.byref(f))
    return r, f.value


EDGES = [1.0, -1.0, 1.5, -2.0, 2.0 - 2.0**-52, -(2.0 - 2.0**-52),
         2.0**-314, -(2.0**-314), 2.0**66, (2.0 - 2.0**-52) * 2.0**66]


def test_words_and_weights_are_exact(lib):
    rng = random.Random(1)
    xs = EDGES + [rng.choice((-1, 1)) * (1 + rng.random()) * 2.0**rng.randint(-314, 66)
                  for _ in range(3000)]
    for x in xs:
        w = lib.word(x)
        q = w & 0xff
        X = struct.unpack("<q", struct.pack("<Q", w & ~0xff))[0]
        assert 1 <= q <= 127 and 2**60 <= abs(X) < 2**63
        assert Fraction(X) * Fraction(2)**(3 * q - 377) == Fraction(x)
        W, e, f = ctypes.c_int64(), ctypes.c_int(), ctypes.c_uint()
        lib.weight(x, W, e, f)
        assert f.value == 0 and 2**55 <= abs(W.value) < 2**56
        assert Fraction(W.value) * Fraction(2)**e.value == Fraction(x)
    assert lib.word(0.0) == 0 and lib.word(-0.0) == 0


def test_what_cannot_be_represented_is_flagged(lib):
    one = [1.0] * 7
    for bad in (math.inf, -math.inf, math.nan, 2.0**67, 2.0**-315, 5e-324,
                -1.7e308):
        assert lib.word(bad) & 0x80
        for j in range(7):
            x = list(one)
            x[j] = bad
            assert _sum(lib, one, x)[1] & 0x80
    for bad in (math.inf, math.nan, 2.0**402, 2.0**-401, 5e-324):
        w = list(one)
        w[3] = bad
        assert _sum(lib, w, one)[1] & 0x80
    assert _sum(lib, [0.0] * 7, one) == (0.0, 0)
    assert _sum(lib, one, [0.0] * 7) == (0.0, 0)
    assert _sum(lib, [0.0, 1.0] + [0.0] * 5, [3.0] * 7) == (3.0, 0)


def test_a_sum_of_zero_products_is_zero(lib):
    rng = random.Random(9)
    for _ in range(500):
        w = [rng.uniform(-1, 1) for _ in range(7)]
        assert _sum(lib, w, [0.0] * 7) == (0.0, 0)
        x = [rng.uniform(-1, 1) for _ in range(7)]
        for j in range(7):  # every product has one zero factor
            (w if rng.random() < 0.5 else x)[j] = 0.0
        assert _sum(lib, w, x) == (0.0, 0)


@pytest.mark.parametrize("n", [7, 8, 14])
@pytest.mark.parametrize("spread_w,spread_x", [(0, 0), (3, 3), (30, 30),
                                               (60, 5), (5, 60), (300, 150)])
def test_sum_error(lib, n, spread_w, spread_x):
    """|sum - exact| <= n (2^-56 + 2^-59) M + 2^-56 M + 2^-53 |sum|, with M the
    largest |w_j x_j|: the dropped partial products and shifts, and the two
    roundings (fixed point, then to double)."""
    rng = random.Random(1000 * n + 7 * spread_w + spread_x)

    def val(s):
        return rng.choice((-1, 1)) * (1 + rng.random()) * 2.0**rng.randint(-s, 0)

    for trial in range(1500):
        w = [val(spread_w) for _ in range(n)]
        x = [val(spread_x) for _ in range(n)]
        kind = trial % 5
        if kind == 1:    # a difference: the last weight cancels the others
            w[-1] = -math.fsum(w[:-1])
            x = [1.0 + 1e-6 * v for v in x]
        elif kind == 2:  # zeros among the values and the weights
            x[rng.randrange(n)] = 0.0
            w[rng.randrange(n)] = 0.0
        elif kind == 3:  # extreme mantissas
            x = [math.copysign((2 - 2.0**-52) * 2.0**rng.randint(-2, 2), v)
                 for v in x]
            w = [math.copysign(2 - 2.0**-52, v) for v in w]
        elif kind == 4:  # the largest weight meets the smallest value
            w.sort(key=abs)
            x.sort(key=abs, reverse=True)
        r, flag = _sum(lib, w, x)
        assert flag == 0
        prods = [Fraction(a) * Fraction(b) for a, b in zip(w, x)]
        exact, M = sum(prods), max(abs(p) for p in prods)
        tol = (n * (Fraction(1, 2**56) + Fraction(1, 2**59))
               + Fraction(1, 2**56)) * M + Fraction(1, 2**53) * abs(exact)
        assert abs(Fraction(r) - exact) <= tol * Fraction(1001, 1000)


@pytest.mark.parametrize("n", [7, 8, 14])
@pytest.mark.parametrize("spread", [20, 40, 60, 100, 300])
@pytest.mark.parametrize("zeros", [1, 3])
def test_zeros_under_the_largest_weights(lib, n, spread, zeros):
    """Values as small as the words hold, with weights 2^-spread and smaller,
    beside zeros under the largest weights: the bound of test_sum_error, M
    being the largest product that is not zero."""
    rng = random.Random(31 * n + spread + zeros)
    for trial in range(600):
        w = [rng.choice((-1, 1)) * (1 + rng.random()) * 2.0**rng.randint(-2, 60)
             if j < zeros else
             rng.choice((-1, 1)) * (1 + rng.random())
             * 2.0**-(spread + rng.randint(0, 9)) for j in range(n)]
        x = [0.0 if j < zeros else rng.choice((-1, 1)) * (1 + rng.random())
             * 2.0**rng.randint(-314, -300 + trial % 200) for j in range(n)]
        if trial % 3 == 0:
            x[-1] = 0.0
        if trial % 3 == 1:
            w[-1] = 0.0
        order = rng.sample(range(n), n)
        w, x = [w[j] for j in order], [x[j] for j in order]
        r, flag = _sum(lib, w, x)
        assert flag == 0
        prods = [Fraction(a) * Fraction(b) for a, b in zip(w, x)]
        exact, M = sum(prods), max(abs(p) for p in prods)
        tol = (n * (Fraction(1, 2**56) + Fraction(1, 2**59))
               + Fraction(1, 2**56)) * M + Fraction(1, 2**53) * abs(exact)
        assert abs(Fraction(r) - exact) <= tol * Fraction(1001, 1000)


LEFT_SRC = r"""
#include "swg_fixed.cuh"
using namespace swg;
extern "C" double sum12(const double *w, const double *x, unsigned *flag) {
  Wt W[12];
  fx_t X[12];
  long long s = 0;
  unsigned f = 0;
  for (int j = 0; j < 12; ++j) {
    W[j] = fx_weight<FX_TOP>(w[j], f);
    X[j] = fx_word(x[j]);
    s += W[j].hi;
  }
  double r = fx_sum<12, FX_LEAVE>(W, X, fx_start(s), FX_TOP, f);
  *flag = f;
  return r;
}
"""


PV_SRC = r"""
#include "swg_fixed.cuh"
using namespace swg;
extern "C" unsigned long long word(double x) { return fx_word<FX_PV_MINQ>(x); }
extern "C" int spread() { return FX_PV_SPREAD; }
extern "C" double sum8(const double *w, const double *x, unsigned *flag) {
  Wt W[8];
  fx_t X[8];
  long long s = 0;
  unsigned f = 0;
  for (int j = 0; j < 8; ++j) {
    W[j] = fx_weight(w[j], f);
    X[j] = fx_word<FX_PV_MINQ>(x[j]);
    s += W[j].hi;
  }
  double r = fx_sum<8, FX_NONE>(W, X, fx_start(s), FX_TOP, f);
  *flag = f;
  return r;
}
"""


def test_pv_sums_need_no_look_at_zeros(tmp_path):
    """The PV sums' words: with weights within their spread of each other the
    bound holds for every mixture of zeros and values down to the smallest
    word; smaller values are flagged."""
    src, so = tmp_path / "pv.cpp", tmp_path / "pv.so"
    src.write_text(PV_SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC,
                    "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.sum8.restype = ctypes.c_double
    lib.sum8.argtypes = [ctypes.POINTER(ctypes.c_double),
                         ctypes.POINTER(ctypes.c_double),
                         ctypes.POINTER(ctypes.c_uint)]
    lib.word.restype = ctypes.c_uint64
    lib.word.argtypes = [ctypes.c_double]
    least = 2.0**-293
    for x in (least, -least, 1.5 * least, 2.0**66, 0.0):
        assert not lib.word(x) & 0x80
    for x in (math.nextafter(least, 0.0), -least / 2, 2.0**-314, 5e-324, 2.0**67,
              math.inf, math.nan):
        assert lib.word(x) & 0x80
    spread = lib.spread()
    rng = random.Random(8)
    for trial in range(6000):
        w = [rng.choice((-1, 1)) * (1 + rng.random())
             * 2.0**(rng.randint(0, spread) if rng.random() < 0.7
                     else rng.choice((0, spread))) for _ in range(8)]
        x = [rng.choice((-1, 1)) * (1 + rng.random())
             * 2.0**-rng.randint(293 - trial % 2 * 9, 293) for _ in range(8)]
        for _ in range(rng.randint(0, 7)):
            x[rng.randrange(8)] = 0.0
        if trial % 3 == 0:
            w[rng.randrange(8)] = 0.0
        r, flag = _sum(lib, w, x)
        assert flag == 0
        prods = [Fraction(a) * Fraction(b) for a, b in zip(w, x)]
        exact, M = sum(prods), max(abs(p) for p in prods)
        tol = (8 * (Fraction(1, 2**56) + Fraction(1, 2**59))
               + Fraction(1, 2**56)) * M + Fraction(1, 2**53) * abs(exact)
        assert abs(Fraction(r) - exact) <= tol * Fraction(1001, 1000)


def test_sums_that_leave_small_products_to_fp64(tmp_path):
    """The tracer passes' form: within the bound, or left to FP64, which no
    sum with a product of 2^-278 and more is, nor one of zero
    weights or values alone."""
    src, so = tmp_path / "left.cpp", tmp_path / "left.so"
    src.write_text(LEFT_SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC,
                    "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.sum12.restype = ctypes.c_double
    lib.sum12.argtypes = [ctypes.POINTER(ctypes.c_double),
                          ctypes.POINTER(ctypes.c_double),
                          ctypes.POINTER(ctypes.c_uint)]
    rng = random.Random(5)
    left = 0
    for trial in range(6000):
        lo, wlo = (-284, -200) if trial % 2 else (-30, -40)
        w = [rng.choice((-1, 1)) * (1 + rng.random()) * 2.0**rng.randint(wlo, 34)
             for _ in range(12)]
        x = [rng.choice((-1, 1)) * (1 + rng.random()) * 2.0**rng.randint(lo - 30, lo)
             for _ in range(12)]
        for _ in range(rng.randint(0, 8)):
            (w if rng.random() < 0.5 else x)[rng.randrange(12)] = 0.0
        r, flag = _sum(lib, w, x)
        prods = [Fraction(a) * Fraction(b) for a, b in zip(w, x)]
        exact, M = sum(prods), max(abs(p) for p in prods)
        if flag:
            left += 1
            assert flag == 0x80
            assert M < Fraction(1, 2**278)
            continue
        tol = (12 * (Fraction(1, 2**56) + Fraction(1, 2**59))
               + Fraction(1, 2**56)) * M + Fraction(1, 2**53) * abs(exact)
        assert abs(Fraction(r) - exact) <= tol * Fraction(1001, 1000)
    assert left > 100
    assert _sum(lib, [2.0**36] + [1.0] * 11, [1.0] * 12)[1] == 0x80
    assert _sum(lib, [3.0] * 12, [0.0] * 12) == (0.0, 0)
    assert _sum(lib, [0.0] * 12, [3.0, 1e-90] * 6) == (0.0, 0)
    assert _sum(lib, [0.0] * 11 + [2.0], [1e-90] * 11 + [3.0]) == (6.0, 0)


def _raw(lib, w, x):
    n = len(w)
    f = ctypes.c_uint()
    r = (lib.raw3 if n == 3 else lib.raw6)(
        (ctypes.c_double * n)(*w), (ctypes.c_double * n)(*x), ctypes.byref(f))
    return r, f.value


@pytest.mark.parametrize("n", [3, 6])
@pytest.mark.parametrize("spread_w,spread_x", [(0, 0), (3, 3), (30, 30),
                                               (60, 5), (5, 60), (100, 400)])
def test_raw_sum_error(lib, n, spread_w, spread_x):
    """As the sums of words, with one more 2^-60 of each negative term (its
    complement for its negation) and with values that keep 2^60 <= |X|."""
    rng = random.Random(77 * n + 7 * spread_w + spread_x)

    def val(s):
        return rng.choice((-1, 1)) * (1 + rng.random()) * 2.0**rng.randint(-s, 0)

    for trial in range(2000):
        w = [val(spread_w) for _ in range(n)]
        x = [val(spread_x) for _ in range(n)]
        kind = trial % 4
        if kind == 1:
            w[-1] = -math.fsum(w[:-1])
            x = [1.0 + 1e-6 * v for v in x]
        elif kind == 2:
            x[rng.randrange(n)] = rng.choice((0.0, -0.0))
            w[rng.randrange(n)] = 0.0
        elif kind == 3:
            x = [math.copysign((2 - 2.0**-52) * 2.0**rng.randint(-2, 2), v)
                 for v in x]
            w = [math.copysign(2 - 2.0**-52, v) for v in w]
        prods = [Fraction(a) * Fraction(b) for a, b in zip(w, x)]
        exact, M = sum(prods), max(abs(p) for p in prods)
        r, slow = _raw(lib, w, x)
        if M == 0 or abs(w[-1]) < 2.0**-120:
            continue
        assert not slow
        tol = (n * (Fraction(1, 2**56) + Fraction(1, 2**59)
                    + Fraction(1, 2**59))
               + Fraction(1, 2**56)) * M + Fraction(1, 2**53) * abs(exact)
        assert abs(Fraction(r) - exact) <= tol * Fraction(1001, 1000)


def test_raw_sum_leaves_the_rest_to_fp64(lib):
    one = [1.0] * 6
    for bad in (math.inf, -math.inf, math.nan, 1e300):
        for j in range(6):
            x = list(one)
            x[j] = bad
            assert _raw(lib, one, x)[1]
    for x in ([0.0] * 6, [-0.0] * 6, [5e-324] * 6, [1e-290] * 6):
        assert _raw(lib, one, x)[1]
    assert _raw(lib, [2.0**121] + [1.0] * 5, one)[1]
    assert _raw(lib, [2.0**-121] + [1.0] * 5, one)[1]
    assert _raw(lib, [0.0, 0.0, 2.0], [math.pi, 1.0, 3.0]) == (6.0, 0)
    assert _raw(lib, [1.0] * 3, [0.0, -0.0, 3.0]) == (3.0, 0)
