"""A call that ran out of device memory reports it and leaves the context
usable: what it had begun is not taken for done by the next call."""
import pytest

import fake_runtime


@pytest.mark.parametrize("first,failing,again", [(100, 1000, 100), (100, 1000, 150), (64, 129, 1)])
def test_buffer_whose_growth_failed(first, failing, again):
    assert fake_runtime.runtime().L.buffer_recovers(first, failing, again) == 1
