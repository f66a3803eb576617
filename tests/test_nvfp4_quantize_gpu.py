"""The NVFP4 activation quantizer at the row lengths where its work split changes, bit for bit against the NumPy restatement."""

import numpy as np
import pytest

from oracle import oracle_np as O
from tests.test_ref_quantize_gpu import dev, library_quantize, seeded_rows   # noqa: F401 (dev is a fixture)

pytestmark = pytest.mark.gpu


# less than a warp's blocks; two turns exactly full and with idle threads; three turns; the last row length held whole and one past it
@pytest.mark.parametrize("rows,k", [(9, 256), (8, 16384), (130, 5376), (9, 12288), (129, 17408), (8, 18432), (9, 18688)])
def test_quantizer_at_the_edges_of_its_split(dev, rows, k):   # noqa: F811
    x = seeded_rows(rows, k, rows + k)
    codes, scales, g = library_quantize(dev, x)
    np_codes, np_scales, np_g = O.quantize_activations(x, 2)
    assert np.array_equal(g.view(np.uint32), np_g.view(np.uint32))
    assert np.array_equal(scales, np_scales)
    assert np.array_equal(codes, np_codes)
