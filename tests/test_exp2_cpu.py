"""The exponential that the prompt attention evaluates in the multiply-add unit (attention_tcgen05.cu: exp2_fma), step by step in
32-bit on the host with the constants that stand in the source: its error over the whole range against 64 bits."""
import os
import re

import numpy as np

import nanoinfer_b200

F = np.float32


def _constants():
    """(degree 0 .. 5, the number whose low bits are whole numbers) as the source has them."""
    with open(os.path.join(os.path.dirname(nanoinfer_b200.__file__), "csrc", "attention_tcgen05.cu")) as f:
        body = f.read().split("void exp2_fma(")[1].split("\n}\n")[0]
    pairs = re.findall(r"two\((-?[0-9.e+-]+)f, (-?[0-9.e+-]+)f\)", body)
    assert all(a == b for a, b in pairs)
    values = [F(a) for a, _ in pairs]
    assert len(values) == 9 and values[0] == -values[1] and values[2] == -1       # magic, -magic, -1, then degrees 5 .. 0
    return values[:2:-1], values[0]


def _fma(a, b, c):
    # 24-bit factors: the product is exact in 64 bits; the sum is rounded there (2^-53) and then to 32
    return (a.astype(np.float64) * b + c).astype(F)


def test_exp2_by_multiply_adds():
    c, magic = _constants()
    halves = np.arange(-126, 8.5, 0.5)                      # where the nearest whole number changes, and the ends of the range
    x = np.concatenate([np.linspace(-126, 8, 4_000_001), np.linspace(-1, 1, 2_000_001), halves, np.nextafter(halves, -200).clip(-126),
                        np.nextafter(F(halves), F(9)).clip(-126, 8)]).astype(F)
    n = x + magic
    f = _fma(n - magic, F(-1), x)
    assert np.abs(f).max() <= 0.5
    p = np.full_like(x, c[5])
    for k in (4, 3, 2, 1, 0):
        p = _fma(p, f, c[k])
    got = (p.view(np.int32) + (n.view(np.int32) << 23)).view(F).astype(np.float64)
    want = np.exp2(x.astype(np.float64))
    assert (np.abs(got - want) / want).max() <= 2.2e-7       # 2.1e-7 as measured; ex2.approx.ftz allows itself 2^-22 = 2.4e-7
