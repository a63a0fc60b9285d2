"""Contacts where the longitude scale is unusual: beyond 90 degrees of latitude,
where it is negative, and close to a pole, where it is small beside its value at
the map's middle and beside the fixed-point unit."""
import numpy as np
import pytest

from glint_pipeline_gb300 import Configuration, DeviceBench
from oracle.bindings import Oracle, make_config
from test_gpu_parity import compare_meetings

pytestmark = pytest.mark.gpu

PI = 3.14159265  # the reference's (util/util.h:38)
METRES = 40076000.0 / 360.0  # a degree at the equator


def run(box, pts, steps, precision_mode, **args):
    args = dict(num_objects=len(pts), num_meeting_buckets=1 << 20, min_meet_time=1, **args)
    o = Oracle(make_config(**args), box, pts)
    g = DeviceBench(Configuration(precision_mode=precision_mode, **args), box, pts)
    far = pts.copy()  # last step: everyone apart, so that the contacts are reported
    far[:, 1] = box[1] + (box[3] - box[1]) * (np.arange(len(pts)) + 0.5) / len(pts)
    cross = contacts = 0
    for t in range(steps + 1):
        p = pts if t < steps else far
        o.step(p, t)
        st = g.step(p, t)
        c = o.counts()
        assert (st.checks, st.candidates, st.contacts) == (c.grid_check_counter, c.candidates, c.contacts), f"step {t}"
        compare_meetings(o.meetings(), g.meetings(), t)
        if t < steps:
            cross, contacts = max(cross, int(st.cross_checks)), max(contacts, int(st.contacts))
    g.close()
    o.close()
    return cross, contacts


@pytest.mark.parametrize("precision_mode", [0, 1])
def test_latitudes_beyond_ninety(precision_mode):
    """A map across 90 degrees; the objects lie about the boundary between two
    leaves that start above it."""
    rng = np.random.default_rng(90)
    n = 1200
    pts = np.empty((n, 2))
    pts[:, 0] = 0.5 + rng.uniform(-0.02, 0.02, n)
    pts[:, 1] = 90.3 + rng.uniform(-0.0005, 0.0005, n)
    pts[0], pts[1] = (0.01, 89.6), (0.99, 90.55)
    cross, contacts = run(np.array([0.0, 89.5, 1.0, 90.6]), pts, 3, precision_mode, grid_capacity=600)
    assert cross > 0 and contacts > 100


@pytest.mark.parametrize("precision_mode", [0, 1])
def test_pole_beside_a_lower_middle(precision_mode):
    """Pairs 4e-12 to 7.5e-12 of the reach inside it, 640 m from the pole on a
    map whose middle is 1.149 degrees away."""
    pairs, r = 60, 0.5
    x = 1.0e-4 + np.arange(pairs) * (2 * r / (METRES * 180 / PI))  # angles from the pole
    lat = 90.0 - x * 180 / PI
    delta = np.linspace(4.0e-12, 7.5e-12, pairs)
    dx = r * (1 - delta) / (np.sin((90.0 - lat) * (PI / 180)) * METRES)
    pts = np.empty((2 * pairs + 8, 2))
    pts[0:2 * pairs:2, 0] = 0.0
    pts[1:2 * pairs:2, 0] = dx
    pts[0:2 * pairs:2, 1] = pts[1:2 * pairs:2, 1] = lat
    mid = 90.0 - 0.02005 * 180 / PI
    box = np.array([0.0, 2 * mid - 89.999, 40.0, 89.999])
    pts[2 * pairs:, 0], pts[2 * pairs:, 1] = 39.0, box[1] + 0.1 * (1 + np.arange(8))
    _, contacts = run(box, pts, 3, precision_mode, grid_capacity=len(pts) - 4, reach_distance=r)
    assert contacts == pairs


@pytest.mark.parametrize("precision_mode", [0, 1])
def test_pole_of_a_whole_globe(precision_mode):
    """Pairs just beyond the reach, 1.7 m from the pole, where a latitude half a
    unit off in the globe's fixed-point frame is 1.5e-5 of the distance to the
    pole off."""
    pairs, r = 12, 10.0
    unit = 2.0 ** -31
    lat = 90.0 - (np.round(np.linspace(1.47e-5, 1.53e-5, pairs) / unit) + 0.5) * unit
    dx = r * (1 + np.linspace(1e-7, 2e-6, pairs)) / (np.sin((90.0 - lat) * (PI / 180)) * METRES)
    assert dx.max() < 355.0
    pts = np.empty((2 * pairs + 8, 2))
    pts[0:2 * pairs:2, 0] = -dx / 2
    pts[1:2 * pairs:2, 0] = dx / 2
    pts[0:2 * pairs:2, 1] = pts[1:2 * pairs:2, 1] = lat
    pts[2 * pairs:, 0], pts[2 * pairs:, 1] = 39.0, -0.1 * (1 + np.arange(8))
    _, contacts = run(np.array([-180.0, -90.0, 180.0, 90.0]), pts, 2, precision_mode, grid_capacity=len(pts) - 4,
                      reach_distance=r)
    assert contacts > 0
