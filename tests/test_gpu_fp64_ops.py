"""The branch-free division and square root of the plain FP64 form
(flux_fp64.cuh), called directly: bit for bit IEEE (numpy's, and CUDA's own
operations for the random operands) at the operands nearest to a rounding
boundary, at both ends of every range they are said to hold on, and with
zero numerators."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import fp64_operands as X

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
RECIP, ROOT, QUOTIENT = 0, 1, 2
# the stated ranges, as exponents: recip_rn and sqrt_rn take operands in
# [2^-500, 2^500]; quotient_by a zero or a numerator in [2^-850, 2^700] over a
# divisor in [2^-320, 2^320], with the quotient in [2^-950, 2^950]
RANGE = 500


@pytest.fixture(scope="module")
def ops(tmp_path_factory):
    so = tmp_path_factory.mktemp("fp64") / "fp64_ops.so"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(HERE, "..", "amr-demo_b200", "csrc"),
                    "-o", str(so), os.path.join(HERE, "fp64_ops.cu")], check=True)
    L = C.CDLL(str(so))
    f64p = C.POINTER(C.c_double)
    L.fp64_ops.argtypes = [C.c_int, f64p, f64p, f64p, C.c_longlong]
    L.fp64_marked.argtypes = [f64p, C.POINTER(C.c_int), C.c_int]
    L.fp64_random.argtypes = [C.c_int, C.c_ulonglong, C.c_longlong] + [C.c_int] * 4 + [C.POINTER(C.c_ulonglong)]
    return L


def check(ops, op, a, b):
    a, b = (np.ascontiguousarray(v, np.float64) for v in np.broadcast_arrays(a, b))
    got = np.zeros(a.size)
    p = [v.ctypes.data_as(C.POINTER(C.c_double)) for v in (a, b, got)]
    assert ops.fp64_ops(op, *p, a.size) == 0
    want = 1.0 / b if op == RECIP else np.sqrt(b) if op == ROOT else a / b
    bad = np.nonzero(got != want)[0]
    assert bad.size == 0, (bad.size, [(a[k], b[k], got[k], want[k]) for k in bad[:3]])


def scaled(m, exponents):
    return (m[None, :] * (2.0 ** np.asarray(exponents, float))[:, None]).ravel()


def test_reciprocals_at_binade_ends(ops):
    m = X.binade_ends(4096)
    b = scaled(m, [-RANGE, -RANGE + 1, -134, -1, 0, 1, 170, RANGE - 2, RANGE - 1])
    check(ops, RECIP, 1.0, np.concatenate([b, -b, [2.0 ** RANGE, -(2.0 ** RANGE)]]))


def test_roots_nearest_to_a_tie(ops):
    m = np.concatenate([X.near_tie_roots(4000), X.binade_ends(4096), 2.0 * X.binade_ends(4096)])
    check(ops, ROOT, 0.0, np.concatenate([scaled(m, [-RANGE, -300, -2, 0, 2, 300, RANGE - 2]), [2.0 ** RANGE]]))


def test_quotients_nearest_to_a_tie(ops):
    a, b = X.near_tie_quotients(np.random.default_rng(0), 20000)
    # (numerator, divisor) exponents at the corners of the range
    for ea, eb in ((0, 0), (699, 319), (699, -249), (-850, 99), (-850, -320), (-630, 319), (-700, -200), (512, -301)):
        for s in (1.0, -1.0):
            check(ops, QUOTIENT, s * a * 2.0 ** ea, b * 2.0 ** eb)


def test_quotients_by_binade_ends(ops):
    rng = np.random.default_rng(1)
    b = X.binade_ends(2048)
    a = np.concatenate([X.binade_ends(2048), rng.uniform(1.0, 2.0, 4096), b * rng.choice(b, b.size)])
    for k in range(64):
        check(ops, QUOTIENT, a, rng.choice(b, a.size))


def test_zero_numerators(ops):
    b = scaled(X.binade_ends(64), [-320, 0, 319])
    check(ops, QUOTIENT, 0.0, np.concatenate([b, -b]))
    check(ops, QUOTIENT, -0.0, b)  # compares equal to a zero of either sign


@pytest.mark.parametrize("op,a,b", [
    (RECIP, (0, 0), (-RANGE, RANGE - 1)),
    (ROOT, (0, 0), (-RANGE, RANGE - 1)),
    (QUOTIENT, (-850, 628), (-320, 99)),
    (QUOTIENT, (-629, 699), (-249, 319)),
    (QUOTIENT, (-60, 60), (-60, 60)),
])
def test_random_operands(ops, op, a, b):
    """2^30 operands each."""
    bad = C.c_ulonglong(1)
    assert ops.fp64_random(op, 0x1234, 1 << 30, *a, *b, C.byref(bad)) == 0
    assert bad.value == 0


@pytest.mark.parametrize("rho,speed", [(1.0, 1.0), (1e-24, 1e6), (1e-31, 1e9), (1.2, 340.0), (1.2e-3, 3.4e4),
                                       (1e30, 1.0), (1.0, 1e-12)])
def test_states_in_any_units_are_not_marked(ops, rho, speed):
    """Densities and speeds of CGS, SI and scaled units, with one velocity
    zero, tiny (ahead of a shock) or as large as the other."""
    q = np.array([[rho, rho * speed * m, rho * speed * k, rho * speed ** 2 * 2.5]
                  for m in (1.0, -0.3) for k in (0.0, -0.0, 1.0, 1e-30)])
    marked = np.ones(len(q), np.int32)
    assert ops.fp64_marked(q.ctypes.data_as(C.POINTER(C.c_double)), marked.ctypes.data_as(C.POINTER(C.c_int)),
                           len(q)) == 0
    assert not marked.any()


def test_states_out_of_range_are_marked(ops):
    t = 2.0 ** -52
    bad = [[0.0, 0, 0, 1], [-1.0, 0, 0, 1], [np.nan, 0, 0, 1], [np.inf, 0, 0, 1], [1.0, 0, 0, 0], [1.0, 0, 0, -1.0],
           [1.0, 0, 0, np.nan], [2.0 ** 110, 0, 0, 2.0 ** 110], [2.0 ** -110 * (1 - t), 0, 0, 2.0 ** -110],
           [1.0, 0, 0, 2.0 ** 80], [1.0, 0, 0, 2.0 ** -80 * (1 - t)], [1.0, 2.0 ** 100, 0, 1], [1.0, 0, -2.0 ** 100, 1],
           [1.0, 2.0 ** -160 * (1 - t), 0, 1], [1.0, 0, 2.0 ** -161, 1], [1.0, np.nan, 0, 1], [1.0, 0, np.inf, 1],
           [2.0 ** 109, 5e-324, 0, 2.0 ** 109]]
    good = [[2.0 ** 110 * (1 - t), 0, 0, 2.0 ** 110], [2.0 ** -110, 0, 0, 2.0 ** -110], [1.0, 0, 0, 2.0 ** 80 * (1 - t)],
            [1.0, 0, 0, 2.0 ** -80], [1.0, 2.0 ** 99, -2.0 ** -160, 1]]
    q = np.array(bad + good, float)
    marked = np.full(len(q), -1, np.int32)
    assert ops.fp64_marked(q.ctypes.data_as(C.POINTER(C.c_double)), marked.ctypes.data_as(C.POINTER(C.c_int)),
                           len(q)) == 0
    assert marked.tolist() == [1] * len(bad) + [0] * len(good)
