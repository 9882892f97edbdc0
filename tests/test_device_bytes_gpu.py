"""Device memory of a catalogue as created: 64 bytes a pixel, and per sightline
the padding of its arrays."""
import numpy as np
import pytest

import tos_b200 as T
from test_gap_sweep_gpu import catalog

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_px", [1, 64, 500])
def test_bytes(engine, n_px):
    los, px = catalog([np.arange(3 * s, 3 * s + n_px) for s in range(400)])
    cat = T.Catalog(engine, los, px, 6)
    got = cat.device_bytes()
    cat.close()
    # 64 floats and 80 entries of 16 bytes of padding, two prefix entries, and
    # the sightline's own values (position, range, offset, count, cell: 100 at most)
    assert got <= 64 * len(px) + (64 * 4 + 80 * 16 + 24 + 100) * len(los) + 8192
