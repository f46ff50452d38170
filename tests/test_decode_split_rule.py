"""Keys per split of the decode attention: fewer where a head's splits then go in one launch, never more than by the number of requests."""

import pytest

from mini_infer_b200.parts.tuning import TUNING


@pytest.mark.parametrize("requests,by_requests", [(1, 128), (2, 128), (3, 256), (4, 256), (5, 512), (64, 512)])
@pytest.mark.parametrize("joined", [None, 128, 256, 512])
def test_never_more_keys_a_split(requests, by_requests, joined):
    split = TUNING.decode_split(requests, 512, joined)
    assert split == (by_requests if joined is None else min(joined, by_requests))
