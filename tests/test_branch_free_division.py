"""The divisions of the flux and inversion kernels that are rounded correctly
without a branch, with their way out where the operands are too small, too
large or of 53 ones: against the oracle, which divides as C does.  States over
many orders of magnitude, fields down to subnormal ones and exactly zero, with
strips of every length; bit for bit, as every division is correctly rounded on
both sides.  (The divisions on given operands: tests/test_device_functions.py;
against the kernels that take every entry: tests/test_known_zeros.py.)"""
import numpy as np
import pytest

import coolharm3d_b200 as hg
import fixtures
import harmtest as ht
from test_gpu_parity import engine_for

pytestmark = pytest.mark.gpu


def wide_state(f, lo, seed):
    """The fixture's state with fields scaled by 1 .. 10^lo, zone by zone, some
    zero, and densities by 1 .. 1e-6; the copies of a single zone alike."""
    rng = np.random.default_rng(seed)
    p = np.array(f["p0"])
    s = tuple(m if n > 1 else 1 for m, n in zip(p.shape, f["n"]))
    p[..., 5:] *= (10.0 ** rng.uniform(lo, 0, s) * (rng.random(s) > 0.2))[..., None]
    p[..., :2] *= (10.0 ** rng.uniform(-6, 0, s))[..., None]
    p[..., 2:5] *= (10.0 ** rng.uniform(lo, 0, s))[..., None]
    return p


@pytest.mark.parametrize("name", ["linwave_stress_10x8x6_s1", "linwave_vl_stress_8x8x8_s2", "balsara1_stress_n64_s1",
                                  "torus_24x16x8_s1", "torus_stress_16x24x6_s1"])
@pytest.mark.parametrize("lo", [-3, -100, -150, -160, -300, -323])
def test_wide_states_against_oracle(name, lo):
    f = fixtures.load(name)
    p0 = wide_state(f, lo, -lo)
    o = None
    for faces, x1 in ((1, 1), (2, 1), (3, 1), (3, 0)):
        e, cell6 = engine_for(f["n"], f["sw"], f, p0, f["t0"], f["dt0"])
        c = e.launch_config()
        c.strip_faces, c.strip_x1 = faces, x1
        e.set_launch_config(c)
        t, dt = e.step(2)
        p, gamma, fails = e.download(), e.gamma(), e.fail_counts()
        e.close()
        if o is None:
            o = ht.Oracle(f["n"], f["sw"], fixtures.geomd(f, cell6), lib=ht.CR_ORACLE)
            o.set_state(p0, f["t0"], f["dt0"])
            o.step(2)
            s = o.state()
        assert np.array_equal(p, s["p"], equal_nan=True), (faces, x1)
        assert fails.tolist() == s["nfailtot"].tolist()
