"""A request whose transform's bounded waits run out reports it, whichever way it came
(device-resident, served alone, replayed or in a group), and the next one does not.
The waits run out because the barriers expect more bytes than the copies bring; the
kernels give up after their limit, and nothing faults.
"""
import pytest

from test_gpu_parity import native

pytestmark = pytest.mark.gpu


def test_requests_report_their_own_waits():
    nat = native()
    assert nat.selftest_request_waits() == 15
    assert nat.device_errors() == 0
    assert nat.selftest_wait_limit() is True
    assert nat.device_errors() == 0
