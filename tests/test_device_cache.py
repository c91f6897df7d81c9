"""What the host asks a device once (csrc/brdc_device_cache.h): threads whose
handles ask first at the same time get one query and the same answer."""
import ctypes

import pytest


@pytest.mark.parametrize("device,queries", [(0, 1), (63, 1), (64, 0), (-1, 0)])
def test_one_query_for_all_threads(built_lib, device, queries):
    import build as b

    assert ctypes.CDLL(b.HOSTLIB).brdc_host_cache_queries(8, device) == queries
