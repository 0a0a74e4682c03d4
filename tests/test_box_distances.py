"""The 8-wide traversal's box-plane distances, emulated in FP32 step by step: how far a near plane can come out beyond the
plane itself, which would cut off what the box holds.

A plane's distance is (2^15 + q) * s + a, with s the quantum over the direction, a the node's origin distance p minus
2^15 s, widened outward by 2^-21 |a|.  p, a and the sum carry five roundings of 2^-24 each.  From 2^17 quanta on |a| is at
least three quarters of |p| and the widening, eight times 2^-24 |a|, covers them all.  Nearer, where p and 2^15 s may cancel,
the five come to at most 5 * 2^17 / 2^24 quanta; the builders put every child plane at least half a quantum outside its box,
so no hit is lost.
"""
import re
from pathlib import Path

import numpy as np

F = np.float32
TRAVERSE = Path(__file__).resolve().parents[1] / "selas_gb300" / "csrc" / "traverse.cuh"
OUT = 1.0 / float(re.search(r"kOut = 1\.0f / (\d+)", TRAVERSE.read_text()).group(1))


def _fma(a, b, c):
    # the product of two floats is exact in double; the sum is rounded to double, then to float
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def _excess(rng, n, near_node):
    """Near plane's distance beyond the plane, in quanta (negative: outside)."""
    scale = np.ldexp(F(1.0), rng.integers(-12, 8, n)).astype(F)
    d = rng.uniform(0.05, 1.0, n).astype(F) * rng.choice([-1.0, 1.0], n).astype(F)
    origin = rng.uniform(-500, 500, n).astype(F)
    q = rng.integers(0, 256, n)
    # the ray's origin: near_node quanta before the node, against the direction
    o = (origin.astype(np.float64) - np.sign(d) * near_node * scale * rng.uniform(0.9, 1.1, n)).astype(F)
    ix = (F(1.0) / d).astype(F)
    s = (scale * ix).astype(F)
    p = ((origin - o).astype(F) * ix).astype(F)
    a = _fma(np.full(n, -32768.0, F), s, p)
    a = _fma(np.full(n, -OUT, F), np.abs(a), a)
    got = _fma((32768 + q).astype(F), s, a).astype(np.longdouble)
    plane = (origin.astype(np.longdouble) + q * scale.astype(np.longdouble) - o.astype(np.longdouble)) / d.astype(np.longdouble)
    return np.asarray((got - plane) / np.abs(scale.astype(np.longdouble) / d.astype(np.longdouble)), np.float64)


def test_near_planes_stay_within_the_builders_slack():
    rng = np.random.default_rng(17)
    for k in range(0, 30):
        worst = _excess(rng, 200_000, 2.0 ** k).max()
        assert worst <= (5.0 * 2.0 ** (17 - 24) if k < 18 else 0.0), (k, worst)
