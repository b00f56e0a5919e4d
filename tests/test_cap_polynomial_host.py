"""The short polynomial of capped prompt scores (csrc/prefill_umma.cu), from its source, against tanh in 64 bits."""
import os
import re

import numpy as np

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nano-vllm-ascend_b200", "csrc", "prefill_umma.cu")


def _constants():
    with open(SOURCE) as f:
        text = f.read()
    c = [float(x) for x in re.search(r"kCapShort\[4\] = \{([^}]*)\}", text).group(1).split(",")]
    return c, float(re.search(r"kCapShortTo = ([0-9.]+)f", text).group(1))


def test_it_cuts_off_less_than_fp32_shows():
    """2e-10 of a score: a hundredth of its rounding, and less than the long polynomial's 1.2e-8 at the end of its range."""
    c, top = _constants()
    y = np.linspace(1e-3, top, 100001)
    off = np.polynomial.polynomial.polyval(y * y, c) * y / np.tanh(y) - 1
    assert np.abs(off).max() < 2e-10


def test_in_fp32_it_is_as_near_as_the_long_polynomial():
    """Both as the kernel computes them, rounding for rounding, over scores up to the short one's end and caps of common scales."""
    c, top = _constants()
    F = np.float32
    fma = lambda a, b, x: (a.astype(np.float64) * np.float64(b) + np.float64(x)).astype(F)  # noqa: E731
    rng = np.random.default_rng(1)
    for cap, scale in ((30.0, 0.125), (50.0, 128 ** -0.5), (4.0, 0.125), (0.7, 0.3)):
        scale = F(scale)
        pre = F(scale / F(cap))
        x = (rng.uniform(0, top, 400000) / float(pre)).astype(F)
        want = cap * np.tanh(x.astype(np.float64) * float(scale) / cap)
        b = [scale]
        for _ in range(3):
            b.append(b[-1] * (pre * pre))
        a = [F(ci) * bi for ci, bi in zip(c, b)]
        x2 = x * x
        short = x * fma(x2, fma(x2, fma(x2, a[3], a[2]).astype(F), a[1]), a[0])
        y = x * pre
        y2 = y * y
        t = np.full_like(x, F(-1382 / 155925))
        for k in (62 / 2835, -17 / 315, 2 / 15, -1 / 3, 1.0):
            t = fma(y2, t, F(k))
        long = t * (x * F(F(cap) * pre))
        off = [np.sqrt(((r.astype(np.float64) / want - 1) ** 2).mean()) for r in (short, long)]
        assert off[0] <= 1.01 * off[1], (cap, off)
