"""``svd_f32`` at the edges of the widths whose rows the spread Jacobi holds in registers,
held to the bars of the other wide sizes."""

import pytest

from test_gpu_svd_f32_wide import test_svd_f32_spread as spread

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [320, 321, 352, 353, 384, 385])
def test_width(q):
    spread(q + 700, q)
