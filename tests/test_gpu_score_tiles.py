"""Plain f32 labels through FMA scores where a row meets several centre tiles (128
centres a pass, 16 to 128 of them a tile) and several feature slabs (64 features),
each kind of awkward data at each edge. The launches of a call say which form it
took, so that a shape the dispatch no longer sends to the scores fails here."""
import numpy as np
import pytest
import torch

from ferrolearn_gb300 import _native
from ferrolearn_gb300.kmeans import FittedKMeans
from oracle import oracle as O
from test_gpu_scores import _case

pytestmark = pytest.mark.gpu

# centres, rows, open rows, labels to 64 bits; the direct form: distances, labels
SCORED, DIRECT = 4, 2

# k = 128 / 129 / 257: one, two and three passes over tiles of 128, 80 and 96; k = 64, 72: tiles of 64
# and 80; d = 64 / 65 / 130: one, two and three slabs
SHAPES = [(39001, 64, 128), (39001, 65, 129), (39003, 130, 64), (5003, 257, 257), (52003, 65, 97), (67001, 63, 72)]


def _launches(call):
    before = _native.lib().fk_debug_launch_count()
    got = np.asarray(call())
    return got, _native.lib().fk_debug_launch_count() - before


@pytest.mark.parametrize("kind", ["blobs", "offset", "ties", "outlier", "nonfinite", "huge", "tiny"])
@pytest.mark.parametrize("n,d,k", SHAPES)
def test_scored_labels_over_tiles_and_slabs(n, d, k, kind):
    x, c = _case(kind, n, d, k, np.random.default_rng(n + k))
    model = FittedKMeans(c, None, 0.0, 0, "f32")
    want = O.predict(c, x)
    dev = torch.from_numpy(x).cuda()
    flat = torch.empty(n * d + 1, device="cuda")  # rows that start off a 16-byte boundary
    flat[1:] = dev.reshape(-1)
    for rows in (dev, flat[1:].reshape(n, d)):
        got, launches = _launches(lambda: model.predict(rows))
        assert launches == SCORED
        assert np.array_equal(got, want)


@pytest.mark.parametrize("n,d,k,form", [(520960, 16, 24, SCORED), (800, 999, 300, SCORED), (4001, 200, 257, SCORED),
                                        (521000, 15, 26, DIRECT), (600000, 16, 23, DIRECT),
                                        (24577, 64, 128, SCORED), (25000, 65, 129, SCORED),
                                        # row tiles of one wave: from d k = 12,500 on
                                        (0, 100, 124, DIRECT), (1, 100, 124, SCORED), (0, 125, 100, SCORED)])
def test_the_line_between_the_forms(n, d, k, form):
    n = n if n > 1 else n + 128 * torch.cuda.get_device_properties(0).multi_processor_count
    x, c = _case("blobs", n, d, k, np.random.default_rng(1))
    model = FittedKMeans(c, None, 0.0, 0, "f32")
    got, launches = _launches(lambda: model.predict(torch.from_numpy(x).cuda()))
    assert launches == form
    assert np.array_equal(got, O.predict(c, x))
