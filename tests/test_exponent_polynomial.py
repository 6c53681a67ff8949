"""The polynomial that takes 2^t of a part of the scores at head_dim 64 (ex2_poly in csrc/fwd_sm100.cu), restated in f32 steps
with the constants that the source holds, against f64."""
import os
import re

import numpy as np

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flat-attention_b200", "csrc", "fwd_sm100.cu")


def coefficients():
    """Highest degree first, as the source evaluates them."""
    text = open(SOURCE).read()
    body = text[text.index("void ex2_poly("):]
    body = body[:body.index("\n}\n")]
    out = []
    for a, b in re.findall(r'pack2\(((?:0x)?[0-9.a-fp+-]+?)f?, ((?:0x)?[0-9.a-fp+-]+?)f?\)', body):
        assert a == b
        out.append(float.fromhex(a) if a.startswith("0x") else float(a))
    assert out[0] == -1.0 and len(out) == 7  # the factor of the reduction, then degree 5 to 0
    assert "kRound = 12582912.f + 127.f" in body
    return np.array(out[1:], np.float32)



def ex2_poly(t):
    """A fused step is formed in f64, where the product of two f32 is exact, and rounded to f32."""
    round_ = np.float32(12582912.0 + 127.0)
    t = np.maximum(t, np.float32(-127.0))  # keeps NaN
    n = t + round_
    f = (t.astype(np.float64) - (n - round_)).astype(np.float32)
    c = coefficients()
    r = np.full_like(t, c[0])
    for k in c[1:]:
        r = (r.astype(np.float64) * f + np.float64(k)).astype(np.float32)
    scale = (n.view(np.uint32) << np.uint32(23)).view(np.float32)
    return r * scale


def test_relative_error_over_the_range_of_scores():
    t = np.linspace(-126.0, 8.0, 4_000_001).astype(np.float32)
    error = np.abs(ex2_poly(t).astype(np.float64) / np.exp2(t.astype(np.float64)) - 1.0)
    assert error.max() <= 2.4e-7, error.max()  # 2^-22, the bound of ex2.approx
    whole = np.arange(-126, 9, dtype=np.float32)
    assert np.array_equal(ex2_poly(whole), np.exp2(whole))


def test_error_of_the_polynomial_itself():
    f = np.linspace(-0.5, 0.5, 1_000_001)
    error = np.abs(np.polyval(coefficients().astype(np.float64), f) / np.exp2(f) - 1.0).max()
    assert 1.5e-7 < error < 1.65e-7, error


def test_far_below_is_exactly_zero_and_nan_stays():
    assert np.all(ex2_poly(np.array([-127.0, -128.0, -1e4, -3e38, -np.inf], np.float32)) == 0.0)
    t = np.linspace(-127.0, -126.0, 1001).astype(np.float32)  # below the normal range: off by less than its smallest number
    assert np.abs(ex2_poly(t).astype(np.float64) - np.exp2(t.astype(np.float64))).max() < 2.0 ** -126
    with np.errstate(invalid="ignore"):
        assert np.isnan(ex2_poly(np.array([np.nan], np.float32))).all()
