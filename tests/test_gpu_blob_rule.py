"""Blob flags at the cell and blob counts from which the cheap sum decides, against the oracle."""
import numpy as np
import pytest

from tests import _oracle as O
from tests.test_gpu_blob_flags import cells, flags

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 3, 4, 5])
@pytest.mark.parametrize("n", [3, (1 << 17) - 1, 1 << 17, (1 << 17) + 1])
def test_either_side_of_the_rule(ctx, n, k):
    rng = np.random.default_rng(k)
    cols = cells(n, k)
    blobs = np.concatenate([rng.uniform(0, 1, (k, 3)), rng.uniform(5, 300, (k, 1)), rng.uniform(0.5, 1.5, (k, 1))],
                           1).astype(np.float32)
    np.testing.assert_array_equal(flags(ctx, cols, blobs, 0.2, 0.5, 7), O.blob_flags(cols, blobs, 0.2, 0.5, 7))
