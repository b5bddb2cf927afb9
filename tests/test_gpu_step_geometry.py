"""The forms of the geometry routines that only some steps take, on the states
and with the oracle of test_gpu_geometry_pin.py: howfar as a warp computes it
together (each lane an edge or a leaf), bit for bit; and hownear as an electron
step uses it, where a stand-in is allowed if the step comes out the same."""
import numpy as np
import pytest

import test_gpu_geometry_pin as pin

pytestmark = pytest.mark.gpu


class _Steps:
    """An engine whose geometry probe answers with howfar as the warp computes
    it, after a look at hownear as steps use it around the exact distance."""
    def __init__(self, engine):
        self.engine, self.stood_in, self.exact = engine, 0, 0

    def __getattr__(self, name):
        return getattr(self.engine, name)

    def probe_geometry(self, parts, t_in):
        one = self.engine.probe_geometry(parts, t_in)
        d = one["tperp"]
        rng = np.random.default_rng(len(parts))
        for off in (0.0, 1e-6, 1e-4, 1e-3, 5e-3, 0.1):
            # steps and ranges at the distance, and `off` (relative, and in cm) around it
            near = lambda: np.nextafter((d * (1 + off * rng.integers(-1, 2, len(d))) + off * rng.integers(-1, 2, len(d))
                                         ).astype(np.float32), np.float32(np.inf) * rng.choice([-1.0, 1.0], len(d)).astype(np.float32))
            t, limit = np.maximum(near(), 0), np.maximum(near(), 0)
            limit = np.maximum(limit, t)                                   # a step is no longer than the range
            limit = np.where(rng.integers(0, 2, len(d)) == 0, limit, -1).astype(np.float32)
            got = self.engine.probe_geometry(parts, t, limit)["tperp"]
            rejected = (limit >= 0) & (d >= limit)
            np.testing.assert_array_equal((limit >= 0) & (got >= limit), rejected)
            np.testing.assert_array_equal(np.minimum(got, t)[~rejected], np.minimum(d, t)[~rejected])
            np.testing.assert_array_equal((t <= got)[~rejected], (t <= d)[~rejected])
            self.stood_in += int((got != d).sum())
            self.exact += int((got == d).sum())
        got = self.engine.probe_geometry(parts, t_in, np.full(len(parts), -1, np.float32))
        return dict(got, tperp=d)


def test_the_reference_recordings(engine):
    steps = _Steps(engine)
    pin.test_device_geometry_equals_the_reference_recordings(steps)
    assert steps.stood_in > 1000 and steps.exact > 1000


@pytest.mark.parametrize("name", ["c1", "c3"])
def test_states_of_whole_transports(engine, name):
    pin.test_device_geometry_equals_the_oracle(_Steps(engine), name)


@pytest.mark.parametrize("offset", [0.0, 1e-6, 1e-4, 2e-3])
def test_polygon_vertices_and_edges(engine, offset):
    steps = _Steps(engine)
    pin.test_device_geometry_at_polygon_vertices_and_edges(steps, offset)
    assert steps.stood_in > 1000 and steps.exact > 1000
