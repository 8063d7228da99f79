"""Weights streamed to CTAs of more than 8 rows, for each ring the stream may use and with the targets
in shared memory or not, at layer widths that leave partly filled slots of the ring; against the
CPU oracle at the tolerances of the row-wise kernels' own test."""

import pytest

from tests.test_gpu_mlp_rows import test_rows_match_oracle as rows_match_oracle

pytestmark = pytest.mark.gpu

# n_in, width, depth, n_out, rows: 16 rows a CTA with four, one and two blocks a slot, the last two
# without staged targets (the first of them only in the fit), then 32 and 64 rows
SHAPES = [(6, 512, 2, 64, 1233), (6, 224, 2, 64, 1233), (6, 1024, 2, 512, 1233), (3, 1008, 2, 1000, 1233),
          (6, 320, 2, 64, 2450), (6, 256, 2, 64, 4900)]


@pytest.mark.parametrize("n_in,width,depth,n_out,rows", SHAPES)
def test_streamed_rows_match_oracle(n_in, width, depth, n_out, rows):
    rows_match_oracle(n_in, width, depth, n_out, rows)
