"""The quick phase of hg_cr_pow (coolharm3d_b200/csrc/hg_crpow.h) where it can
go wrong: the ends of its table's intervals (the series' largest argument),
both sides of 1 and of powers of two, the ends of the exponent range.  Against
x^y in 60-digit decimal arithmetic rounded once; exact, as the function is."""
import numpy as np
import pytest

from test_crpow import _exact, _lib


@pytest.mark.parametrize("y", [2 / 3, -2 / 3, 1 / 3, -1 / 3, 5 / 3 - 1, 2.0, -1.9, 1e-3])
def test_quick_phase_rounds_correctly(y):
    p = _lib().or_cr_pow_raw
    rng = np.random.default_rng(11)
    i = rng.integers(0, 257, 240)
    xs = np.concatenate([
        (1 + i / 256) * (1 + rng.uniform(-1, 1, 240) * 10.0 ** rng.uniform(-16, -3, 240)) * 2.0 ** rng.integers(-30, 30, 240),
        1 + 10.0 ** rng.uniform(-15, -2, 60), 1 - 10.0 ** rng.uniform(-15, -2, 60),
        2.0 ** rng.integers(-1000, 1000, 40) * (1 - 2.0 ** -53),
        [2.0 ** -1022, np.nextafter(2.0 ** 1023, 0), np.nextafter(1, 2), np.nextafter(1, 0)],
    ])
    for x in xs:
        if x != 1 and abs(y * np.log(x)) < 690:
            assert p(float(x), y) == _exact(float(x), y), (float(x).hex(), y)
