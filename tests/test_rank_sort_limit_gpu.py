"""Streams of white noise whose windows and stores lie on both sides of the
15,360 keys that are sorted by rank: every prefix equals the one-shot result."""
import pytest

import cases
from test_pack_gpu import _noise
import test_stream_gpu as ts

pytestmark = pytest.mark.gpu
LIMIT = 15360


@pytest.mark.parametrize("dims,window_above,store_above", [([40, 30, 3], False, False), ([74, 50, 4], False, True),
                                                           ([88, 66, 4], True, True), ([11, 10, 9, 2], False, False),
                                                           ([14, 14, 15, 3], True, True)])
def test_both_sides(ctx, dims, window_above, store_above):
    case = cases.Case("noise", "regular", len(dims) - 1, cases.MULTI, _noise(dims, 9), 2.0 ** 20, dims)
    n = [len(ts.one_shot(ctx, case, t + 1, False).track_id) for t in range(dims[-1])]
    assert (max(b - a for a, b in zip(n, n[1:])) > LIMIT) == window_above
    assert (n[-1] > LIMIT) == store_above
    ts.stream_case(ctx, case, check_every=True)
