"""The error bound of the tensor cores' filter of feature-space neighbours (csrc/feature_filter.cu): what splitting numbers into
two bf16 leaves out, measured, and the constant that has to cover it together with the roundings.  Host arithmetic."""
import os
import re

import numpy as np

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "torkit3d_b200", "csrc", "feature_filter.cu")


def _bf16(x):
    """Nearest bf16, ties to even."""
    b = x.astype(np.float32).view(np.uint32)
    return ((b + 0x7fff + ((b >> 16) & 1)) & np.uint32(0xffff0000)).view(np.float32)


def _left_out():
    """Largest |a b - (ah bh + ah bl + al bh)| / |a b| found: random pairs, and pairs around the worst upper halves."""
    g = np.random.default_rng(0)
    worst = np.float32(1 + 2 ** -8) + np.arange(-64, 65, dtype=np.float32) * np.float32(2 ** -23)
    pairs = [(np.repeat(worst, worst.size), np.tile(worst, worst.size)),
             (g.uniform(1, 2, 1 << 20).astype(np.float32), g.uniform(1, 2, 1 << 20).astype(np.float32))]
    top = 0.0
    for a, b in pairs:
        ah, bh = _bf16(a), _bf16(b)
        al, bl = _bf16(a - ah), _bf16(b - bh)
        d = np.float64
        err = np.abs(a.astype(d) * b - (ah.astype(d) * bh + ah.astype(d) * bl + al.astype(d) * bh)) / (a.astype(d) * b)
        top = max(top, err.max())
    return top


def test_the_constant_covers_the_halves_and_the_roundings():
    with open(SOURCE) as f:
        per_channel, fixed = map(float, re.search(r"return \(float\)C \* ([0-9.e-]+)f \+ ([0-9.e-]+)f;", f.read()).groups())
    left_out = _left_out()
    assert 2 ** -16 < left_out <= 2 ** -15
    u = 2.0 ** -24  # of X^2; v has 2 |a||b| <= X^2 / 2
    for C in range(1, 129):
        halves = 2 ** -15 / 2
        product = 3 * (C + -(-C // 16)) * u
        roundings = (2 * (C + 2) + 2 + 4) * u
        assert halves + product + roundings <= per_channel * C + fixed
