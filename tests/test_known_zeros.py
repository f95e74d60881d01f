"""The flux kernels that leave out the products with a geometry's known zeros
(flat space, axisymmetric tables) against the ones that take every entry: the
same numbers on every state, infinite, NaN and tiny ones included.  The second
engine gets the same geometry with one of its zeros negative, which the scan of
hg_set_geometry does not accept as known: every entry is then taken."""
import numpy as np
import pytest

import coolharm3d_b200 as hg
import fixtures
from test_gpu_parity import engine_for

pytestmark = pytest.mark.gpu

CASES = ["linwave_stress_10x8x6_s1", "linwave_vl_stress_8x8x8_s2", "balsara1_stress_n64_s1", "field_loop_24x24x1_s3",
         "torus_24x16x8_s1", "torus_stress_16x24x6_s1"]


def both(f, p0):
    out = []
    for general in (False, True):
        e, cell6 = engine_for(f["n"], f["sw"], f, p0, f["t0"], f["dt0"])
        if general:
            if f["sw"]["metric_dim"] == 0:
                geom, conn = hg.minkowski_tables(e.desc)[0].copy(), None
            else:
                geom, conn = np.array(f["geom"], float).copy(), f["conn"]
            geom.reshape(-1, hg.NGEOM)[:, 16 + 2] = -0.0  # gcov[0][2]
            e.set_geometry(geom, conn)
        t, dt = e.step(2)
        out.append(dict(p=e.download(), gamma=e.gamma(), pflag=e.pflag(), nfail=e.nfail(), t=np.array([t, dt]),
                        fails=e.fail_counts()))
        e.close()
    return out


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("wild", [None, np.inf, -np.inf, np.nan, 1e200, -1e160, 1e-310])
def test_known_zeros_change_nothing(name, wild):
    f = fixtures.load(name)
    p0 = np.array(f["p0"])
    if wild is not None:  # one zone of every variable's own
        rng = np.random.default_rng(3)
        for l in range(8):
            z = tuple(3 + int(rng.integers(m)) for m in f["n"])
            p0[z + (l,)] = wild
    a, b = both(f, p0)
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f"), k
