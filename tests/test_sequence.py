"""Lists of calls that the library refuses before it issues anything."""
from array import array

import pytest

from cbm4gnn_b200 import _lib


@pytest.mark.parametrize("call,n_bases,message", [
    ([9] + [0] * 12, 1, "no known kind"),
    ([1, 3, 4, 0, 4, 0, 4, 1, 4, 4, 0, 0, 0], 2, "base that was not given"),
    ([0, 0, 0, 4, 1, 4, 4, 0, 0, 0, 0, 0, 0], 2, "plan"),
    ([0] * 13, 300, "bad arguments"),
])
def test_bad_lists_are_errors(call, n_bases, message):
    calls, bases = array("q", call), array("q", [0] * n_bases)
    rc = _lib.lib().cbm_b200_sequence(calls.buffer_info()[0], 1, bases.buffer_info()[0], n_bases, None)
    assert rc != 0
    with pytest.raises(Exception, match=message):
        _lib.check(rc)
