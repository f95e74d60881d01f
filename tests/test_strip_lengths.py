"""The flux launch of all three directions: the same step whatever the strip
length, with and without x1 strips, and for block counts that leave a block
several strips; grids with remainders and with directions of one zone, and
every kind of face geometry the kernels are built for (known zeros and every
entry, flat and tables, with RESCALE_R and without, time-dependent).  FP64 bit
for bit; the FMA form, whose kernels the compiler contracts each in its own
way, to 1e-9 of each array's largest value (some 1e6 roundings), on smooth
states, where no rounding decides which branch of the inversion a zone takes."""
import numpy as np
import pytest

import coolharm3d_b200 as hg
import fixtures
from test_dynamic_metric import desc_of, metric_of

pytestmark = pytest.mark.gpu

KINDS = [("linwave_stress_10x8x6_s1", ""), ("linwave_vl_stress_8x8x8_s2", ""), ("balsara1_stress_n64_s1", ""),
         ("field_loop_24x24x1_s3", ""), ("field_loop_24x24x1_s3", "every"), ("linwave_12x10x8_s2", "rescale"),
         ("torus_24x16x8_s1", ""), ("torus_24x16x8_s1", "every"), ("torus_24x16x8_s1", "no rescale"),
         ("torus_24x16x8_s1", "every, no rescale"), ("torus_stress_16x24x6_s1", ""), ("torus_dynmink_12x10x6_s1", ""),
         ("torus_dynmink_12x10x6_s1", "no rescale")]


def grid(f, how, precision):
    sw = dict(f["sw"])
    if "rescale" in how:
        sw["rescale"] = int("no" not in how)
    d = desc_of(dict(f, sw=sw), precision)
    d.metric_dim = sw["metric_dim"]
    e = hg.Engine(d)
    cell6, rface = fixtures.cell6_of(f), f["rface"]
    if sw["metric_dim"] == 3:
        e.set_dynamic_metric(metric_of(f))
    else:
        if sw["metric_dim"] == 0:
            geom, cell6 = hg.minkowski_tables(d)
            conn = None
            if sw["rescale"]:  # radii away from zero for the scale factors
                cell6[..., 2:4] = 1.0 + 0.1 * np.arange(f["n"][0] + 6)[:, None, None, None]
                rface = 0.95 + 0.1 * np.arange(f["n"][0] + 6)
        else:
            geom, conn = f["geom"], f["conn"]
        geom = np.array(geom, float)
        if "every" in how:
            geom.reshape(-1, hg.NGEOM)[:, 16 + 2] = -0.0  # gcov[0][2]: not a known zero
        e.set_geometry(geom, conn)
    e.set_cell_data(cell6, rface if sw["rescale"] else None)
    if sw["cooling"]:
        e.set_cooling_tables(f["cool_omega"], f["cool_temp"])
    e.upload(f["p0"])
    e.set_time(f["t0"], f["dt0"])
    return e


@pytest.mark.parametrize("name,how,precision", [k + (hg.PREC_FP64,) for k in KINDS] +
                         [k + (hg.PREC_FP64_FMA,) for k in KINDS if "stress" not in k[0]])
def test_strip_length_changes_nothing(name, how, precision):
    f = fixtures.load(name)
    out = []
    for faces, x1, blocks in [(None, None, None), (1, 1, 1), (2, 1, 3), (3, 1, 2), (1, 0, 2), (2, 0, 5), (3, 0, 1000)]:
        e = grid(f, how, precision)
        if faces:
            c = e.launch_config()
            c.strip_faces, c.strip_x1, c.grid_flux = faces, x1, blocks
            e.set_launch_config(c)
        t, dt = e.step(2)
        out.append((e.download(), e.gamma(), e.nfail(), e.fail_counts(), np.array([t, dt])))
        e.close()
    assert np.isfinite(out[0][0]).all()
    for o in out[1:]:
        for a, b in zip(out[0], o):
            if precision == hg.PREC_FP64:
                assert np.array_equal(a, b)
            else:
                a, b = np.asarray(a, float), np.asarray(b, float)
                assert np.abs(a - b).max() <= 1e-9 * np.abs(a).max()
