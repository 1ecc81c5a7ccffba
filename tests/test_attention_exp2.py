"""The exponential that ns_attention_prompt.cu computes as a polynomial, operation for operation in numpy with the constants that stand in the source, against 2^x."""
import os
import re

import numpy as np

from nn_b200 import build

f = np.float32


def _fma(a, b, c):
    return (a.astype(np.float64) * np.float64(b) + c).astype(f)


def _exp2(x):
    text = open(os.path.join(build.CSRC, "ns_attention_prompt.cu")).read()
    body = re.search(r"void pa_exp2_pair\(.*?\n\}", text, re.S).group(0)
    first, *rest = [f(c) for c in re.findall(r"pa_pair\((\S+?)f, \1f\)", body[body.index("uint64_t y ="):])]
    assert len(rest) == 5
    x = np.maximum(x, f(-127))
    shift = f(12582912.0)
    t = x + shift
    n = t - shift
    r = _fma(n, -1, x)
    y = np.full_like(x, first)
    for k in rest:
        y = _fma(y, r, k)
    return (y.view(np.int32) + (t.view(np.int32) << 23)).view(f)


def test_polynomial():
    x = np.concatenate([np.linspace(-126, 8, 2_000_001), np.linspace(-1, 1, 200_001)]).astype(f)
    want = np.exp2(x.astype(np.float64))
    assert np.abs(_exp2(x) / want - 1).max() < 2.0 ** -22.5
    assert np.array_equal(_exp2(np.array([-127, -200, -np.inf, 0], f)), [0, 0, 0, 1])
