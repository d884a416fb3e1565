"""Grid shapes that share a stream take their multiply and interleave in one launch: the results of each
stage in one launch for all shapes."""
import numpy as np
import pytest

import tild
from helpers import charged_system, small_diblock

pytestmark = pytest.mark.gpu


def _systems(fieldphase):
    shapes = [(16, 16, 16), (12, 14, 16), (20, 20, 20), (18, 16, 20), (15, 17, 19), (14, 14, 14), (24, 12, 12),
              (16, 20, 12), (22, 10, 14), (13, 16, 18), (16, 16, 16), (20, 16, 12)]
    systems = [small_diblock(3, 1, nx=n, box=tuple(0.5 * v for v in n), n_chains=40 + 5 * k, seed=80 + k)
               for k, n in enumerate(shapes)]
    systems[4:4] = [charged_system()]
    if fieldphase:
        systems[2].styles = systems[2].styles + [tild.Style(tild.STYLE_FIELDPHASE, 0, 1, 0.7, phase=0, dir=1, n_periods=2)]
    return systems


@pytest.mark.parametrize("fieldphase", [False, True])
@pytest.mark.parametrize("streams", [8, 3, 0])
def test_streams_of_several_shapes(streams, fieldphase):
    systems = _systems(fieldphase)
    out = []
    for pipeline in (0, 1):
        with tild.Batch(systems) as B:
            t = B.get_tune()
            assert t.fft_pipeline == 1 and t.fft_streams == 8   # the default of several shapes
            t.fft_pipeline, t.fft_streams = pipeline, streams
            B.set_tune(t)
            B.step(20)
            for k in (1, 4, 7):     # whole shapes at rest between others
                B.set_active(k, False)
            B.step(20)
            for k in (1, 4, 7):
                B.set_active(k, True)
            B.step(5)
            f = B.forces(3)
            out.append([B.get_state(i)[0] for i in range(len(systems))] + [B.density(i) for i in range(len(systems))] + [f])
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a, b), k


def test_large_batches_go_shape_by_shape():
    """Above 256 MB of spectra and force spectra each shape of a stream launches its own multiply and interleave."""
    shapes = [(120, 120, 120), (125, 120, 120), (120, 125, 120), (120, 120, 125), (125, 125, 120)]
    systems = [small_diblock(3, 1, nx=n, box=tuple(0.5 * v for v in n), n_chains=300, seed=k) for k, n in enumerate(shapes)]
    out = []
    for pipeline in (0, 1):
        with tild.Batch(systems) as B:
            t = B.get_tune()
            t.fft_pipeline, t.fft_streams = pipeline, 2
            B.set_tune(t)
            B.step(9)
            out.append([B.get_state(i)[0] for i in range(5)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
