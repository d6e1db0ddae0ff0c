"""Encodes of many short rows, which share CTAs from 608 full ones on: row counts
on both sides of that and with rows left over, against the oracle."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,off", [(2, 0), (2, 1), (4, 1)])
@pytest.mark.parametrize("rows,logrow", [(1215, 6), (1216, 6), (1217, 8), (2435, 7), (4867, 5), (9735, 4), (19459, 3),
                                         (38919, 2), (65535, 1)])
def test_rows(ctx, oracle, rows, logrow, rate, off):
    x = rand_fe(np.random.default_rng(rows * 8 + rate), rows << logrow).reshape(rows, 1 << logrow, 2)
    assert np.array_equal(ctx.Encode(x, rate, off), oracle.encode_rows(x, rate, off))
