"""The heavy tier's phase (csrc/k2_fast.cu, heavy_tile), emulated operation by operation with exact rounding,
against the exact phase frac(v G + psi): the table index and remainder lie within 2^-48 turn of it for
any 64.64 v and 32.128 G, the limbs' extremes and the table cells' edges included; and the rotation of
the 256-entry table by the remainder is within 1e-14 of the exact cosine and sine (truncation 4.7e-15,
roundings of unit order 2e-16)."""
import random
from fractions import Fraction as Fr

import pytest

from test_tier_phase_models import M32, bits, exact_phase, fma, from_bits, limbs, turn_distance

MAGIC35 = 51539607552.0            # 1.5 2^35


def model(vi, vf, G, ps):
    """(q, d): table index and remainder in units of 2^-49 turn."""
    a1, a0, d1, d0, gi, b1, b0, c1, c0 = limbs(vi, vf, G)
    pair = lambda x, y: fma(float(y), 2.0**-64, x * 2.0**-32)  # noqa: E731
    B0, C1, B1, GI = pair(b0, c1), pair(c1, c0), pair(b1, b0), pair(gi, b1)
    psi_hi, psi_lo = ((ps >> 32) + (1 << 23)) & M32, (ps & M32) * 2.0**-32
    L = (a1 * b0 + a0 * b1 + d1 * gi + psi_hi) & M32
    p1 = fma(float(a0), B0, fma(float(a1), C1, psi_lo))
    p2 = fma(float(d0), GI, fma(float(d1), B1, MAGIC35))
    w = (L * 131072 + bits(float(Fr(p1) + Fr(p2)))) & ((1 << 64) - 1)
    wh = w >> 32
    d = from_bits((((wh & 0x1FF) | 0x43300000) << 32) | (w & M32)) - 4504699138998272.0
    return (wh >> 9) & 255, d


def points():
    rng = random.Random(31)
    ones = (1 << 64) - 1
    for vi, vf, G in ((ones, ones, (1 << 160) - 1), (0, 0, 0), (1, 0, 1 << 120), (ones, ones, ((1 << 32) - 1) << 128)):
        for ps in (0, ones, 1 << 63, (1 << 55) - 1, 1 << 55, (1 << 56) - 1):
            yield vi, vf, G, ps
    for i in range(1500):
        vi = rng.getrandbits(64) if i % 2 else 3_500_000_000_000_000_000 + rng.getrandbits(56)
        yield vi, rng.getrandbits(64), (rng.getrandbits(32 if i % 3 else 19) << 128) | rng.getrandbits(128), rng.getrandbits(64)


def test_index_and_remainder_within_2_pow_minus_48():
    worst = 0
    for vi, vf, G, ps in points():
        q, d = model(vi, vf, G, ps)
        assert 0 <= q < 256 and abs(d) <= 2.0**40
        worst = max(worst, turn_distance(Fr(q, 256) + Fr(d) / 2**49, exact_phase(vi, vf, G, ps)))
    assert worst <= Fr(1, 1 << 48), float(worst)


@pytest.mark.parametrize("edge", [0.0, 1.0, -2.0**40, 2.0**40, 2.0**40 - 1])
def test_rotation_within_1e_14(edge):
    import mpmath as mp
    mp.mp.prec = 120
    rng = random.Random(32)
    a = 6.283185307179586 * 2.0**-49
    for _ in range(200):
        q, d = rng.randrange(256), edge if rng.random() < 0.3 else float(rng.randint(-2**40, 2**40))
        tx, ty = float(mp.cos(2 * mp.pi * q / 256)), float(mp.sin(2 * mp.pi * q / 256))
        u = d * d
        s = d * fma(u, fma(u, a * a * a * a * a / 120.0, -a * a * a / 6.0), a)
        m = u * fma(u, a * a * a * a / 24.0, -a * a / 2.0)
        cs, sn = fma(tx, m, fma(-ty, s, tx)), fma(ty, m, fma(tx, s, ty))
        th = 2 * mp.pi * (mp.mpf(q) / 256 + mp.mpf(d) / 2**49)
        assert abs(cs - mp.cos(th)) <= 1e-14 and abs(sn - mp.sin(th)) <= 1e-14
