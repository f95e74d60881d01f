"""The flux kernels that leave out the products with a geometry's known zeros
(flat space, axisymmetric tables) against the ones that take every entry: the
same numbers on every state, infinite, NaN and tiny ones included.  The second
engine gets the same geometry with one of its zeros negative, which the scan of
hg_set_geometry does not accept as known: every entry is then taken.  With
strips of every length (a small grid's own is 1), the x1 faces in strips and
one to a thread.  The FMA and mixed forms, whose kernels round each in its own
way, on smooth states within their rounding."""
import numpy as np
import pytest

import coolharm3d_b200 as hg
import fixtures
from test_gpu_parity import engine_for
from test_mixed import fixture_engine, l1_rel

pytestmark = pytest.mark.gpu

CASES = ["linwave_stress_10x8x6_s1", "linwave_vl_stress_8x8x8_s2", "balsara1_stress_n64_s1", "field_loop_24x24x1_s3",
         "torus_24x16x8_s1", "torus_stress_16x24x6_s1"]


def every_entry(f, e):
    """The same geometry, not recognised: one of its zeros negative."""
    if f["sw"]["metric_dim"] == 0:
        geom, conn = hg.minkowski_tables(e.desc)[0].copy(), None
    else:
        geom, conn = np.array(f["geom"], float).copy(), f["conn"]
    geom.reshape(-1, hg.NGEOM)[:, 16 + 2] = -0.0  # gcov[0][2]
    e.set_geometry(geom, conn)


def both(f, p0, faces, x1):
    out = []
    for general in (False, True):
        e, cell6 = engine_for(f["n"], f["sw"], f, p0, f["t0"], f["dt0"])
        if general:
            every_entry(f, e)
        c = e.launch_config()
        c.strip_faces, c.strip_x1 = faces, x1
        e.set_launch_config(c)
        t, dt = e.step(2)
        out.append(dict(p=e.download(), gamma=e.gamma(), pflag=e.pflag(), nfail=e.nfail(), t=np.array([t, dt]),
                        fails=e.fail_counts()))
        e.close()
    return out


@pytest.mark.parametrize("faces,x1", [(1, 1), (2, 1), (3, 1), (3, 0)])
@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("wild", [None, np.inf, -np.inf, np.nan, 1e200, -1e160, 1e-310])
def test_known_zeros_change_nothing(name, wild, faces, x1):
    f = fixtures.load(name)
    p0 = np.array(f["p0"])
    if wild is not None:  # one zone of every variable's own
        rng = np.random.default_rng(3)
        for l in range(8):
            z = tuple(3 + int(rng.integers(m)) for m in f["n"])
            p0[z + (l,)] = wild
    a, b = both(f, p0, faces, x1)
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f"), k


@pytest.mark.parametrize("faces", [1, 3])
@pytest.mark.parametrize("name", ["linwave_12x10x8_s2", "field_loop_24x24x1_s3", "torus_24x16x8_s1"])
@pytest.mark.parametrize("precision,tol", [(hg.PREC_FP64_FMA, 1e-11), (hg.PREC_MIXED, 1e-5)])
def test_known_zeros_in_the_rounded_forms(name, precision, tol, faces):
    """relative L1 per variable: the FMA form's within 1e-11 (its distance from
    FP64 is 1e-13 .. 7e-12), the mixed form's within its own bound, 1e-5."""
    f = fixtures.load(name)
    p = []
    for general in (False, True):
        e = fixture_engine(f, precision)
        if general:
            every_entry(f, e)
        c = e.launch_config()
        c.strip_faces = faces
        e.set_launch_config(c)
        e.step(2)
        p.append(e.download())
        e.close()
    # a variable that is zero but for rounding (U3, B3 of the loop) is measured against the largest of its kind
    err = l1_rel(*p)
    for kind in (("U1", "U2", "U3"), ("B1", "B2", "B3")):
        size = {v: np.abs(p[1][3:-3, 3:-3, 3:-3, 2 + "U1 U2 U3 B1 B2 B3".split().index(v)]).sum() for v in kind}
        for v in kind:
            err[v] *= size[v] / max(size.values()) if max(size.values()) > 0 else 0
    assert max(err.values()) < tol, err
