"""The flags of bounded waits, read and cleared through both libraries; raised here from the host, no wait is made to run out."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_flags_come_back_and_clear():
    from krasis_b200 import capi, seqops
    capi.load()
    seqops.load()
    seqops.check_waits()                         # nothing that ran before gave up
    for check, raise_flags, error in ((capi.check_waits, capi.load().kb2_wait_timeouts, capi.Kb2Error),
                                      (seqops.check_waits, seqops.load().kb2_seq_wait_timeouts, seqops.SeqOpsError)):
        was = C.c_int(-1)
        assert raise_flags(0, 1, C.byref(was)) == 0 and was.value == 0
        with pytest.raises(error, match="gave up"):
            check()
        check()
