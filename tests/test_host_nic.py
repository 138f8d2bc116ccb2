"""The sending ends on the CPU, built with g++ over the library's headers in the enqueue trace's build: each
form that takes a slot at a time against the device frame by frame (Egress). tests/host_nic.cpp: the list
that a host with a warp of its own plays through its NIC (HostNic), whose traced enqueues had source and
destination swapped for a frame offered by a ScheduleNow'd event of its instant. tests/switch_port.cpp: a
switch port's slot staged in shared memory (sw_egress_staged)."""
import pytest

from test_sent_list import run_check


@pytest.mark.parametrize("form", ["host_nic", "switch_port"])
def test_sending_end_equals_egress(tmp_path, form):
    run_check(tmp_path, form)
