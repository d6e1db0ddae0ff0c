"""The device multiply at the words where its 32-bit columns carry: every
quadruple of edge words through gbz_field_ops, against integer arithmetic."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = (1 << 61) - 1
EDGES = [0, 1, 2, P - 1, P - 2, 1 << 60, (1 << 60) - 1, (1 << 32) - 1, 1 << 32, (1 << 32) + 1, (1 << 31) - 1,
         1 << 31, P - (1 << 32), P - (1 << 32) + 1, 0x1FFFFFFF00000000, 0x0000000100000001, 0x1FFFFFFE80000000]


@pytest.mark.parametrize("n", [1, 31, len(EDGES) ** 4])
def test_multiply_edges(gbz, ctx, n):
    q = np.array(list(itertools.product(EDGES, repeat=4)), dtype=np.uint64)[-n:]
    a, b = np.ascontiguousarray(q[:, :2]), np.ascontiguousarray(q[:, 2:])
    _, _, prod = ctx.field_ops(a, b)
    w = q.astype(object)
    re = (w[:, 0] * w[:, 2] - w[:, 1] * w[:, 3]) % P
    im = (w[:, 0] * w[:, 3] + w[:, 1] * w[:, 2]) % P
    assert np.array_equal(prod[:, 0], re.astype(np.uint64))
    assert np.array_equal(prod[:, 1], im.astype(np.uint64))
