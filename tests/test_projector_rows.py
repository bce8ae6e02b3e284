"""The table projector where z-lines have no 16-byte alignment: one, two or four
rows a lane by the row count and the arithmetic, tiles of 32 and of 64 rows and
their remainders.  Comparison and reasons as in test_projector_shapes.py."""
import pytest

import test_projector_shapes as shapes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,NT,NP", [(21, 3, 9), (18, 5, 16), (20, 7, 12), (17, 9, 9), (23, 13, 20), (26, 15, 10), (19, 31, 10),
                                     (19, 42, 10), (16, 63, 9), (14, 62, 17), (15, 66, 8), (14, 97, 9)])
def test_rows_without_alignment(N, NT, NP):
    shapes.test_table_projector_equals_gather(N, NT, NP, 1, 1.0, 1.0, None)
