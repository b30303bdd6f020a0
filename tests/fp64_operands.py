"""Operands whose reciprocal, quotient or root lies next to a rounding
boundary, for test_gpu_fp64_ops.py."""
import numpy as np

ULP = 2.0 ** -52


def binade_ends(count):
    """Mantissas in [1, 2): the `count` at each end, all ones among them.
    Their reciprocals are the ones nearest to a rounding boundary:
    1 / (2 - j 2^-52) = (1 + j 2^-53 + j^2 2^-106 + ...) / 2."""
    j = np.arange(count)
    return np.concatenate([1.0 + j * ULP, 2.0 - (j + 1) * ULP])


def near_tie_quotients(rng, count):
    """(a, b) in [1, 2) with a / b within 2^-103 of the middle between two
    doubles: A 2^54 = B (2 Q + 1) + c for 53-bit integers A and B and a small
    odd c, solved for 2 Q + 1 modulo 2^54 (B odd); A 2^53 likewise for
    quotients in [1, 2)."""
    out = []
    while len(out) < count:
        B = int(rng.integers(2 ** 52, 2 ** 53)) | 1
        for bits in (53, 54):
            inv = pow(B, -1, 2 ** bits)
            for c in (1, -1, 3, -3, 5, -5):
                M = (-c * inv) % 2 ** bits
                A = (B * M + c) >> bits
                if not (A << bits == B * M + c and 2 ** 53 < M < 2 ** 54):
                    continue  # 2 Q + 1 has 54 bits: Q is a mantissa
                if 2 ** 52 <= A < 2 ** 53:
                    out.append((A * 2.0 ** -52, B * 2.0 ** -52))
    a, b = np.array(out[:count]).T
    return a, b


def near_tie_roots(most):
    """x in [1, 4) whose root is nearest to the middle between two doubles:
    x = k^2 + k + c for a 53-bit k and |c| <= most, a multiple of 2^52 or
    2^53 so that x fits 53 bits. The two solutions k modulo 2^52 (2^53) of
    each even c are found bit by bit (2 k + 1 is odd)."""
    out = []
    for bits in (52, 53):
        for c in range(-most, most + 1, 2):
            for k in (0, 1):
                for t in range(1, bits + 1):
                    if (k * k + k + c) % 2 ** t:
                        k ^= 1 << (t - 1)
                k %= 2 ** bits
                if bits == 52:
                    k += 2 ** 52
                v = k * k + k + c
                assert v % 2 ** bits == 0
                X = v >> bits
                if k < 2 ** 52 or X >= 2 ** 53:
                    continue
                out.append(float(X) * 2.0 ** (bits - 104))
    return np.array(out)
