"""A host's sending end on the CPU: tests/host_nic.cpp, built with g++ over twins_b200/csrc/tb_tcp.cuh and
tb_egress.cuh in the enqueue trace's build. The list that a host with a warp of its own plays through its
NIC (HostNic) against the device frame by frame (Egress): frames sent and held, counters, and the traced
enqueues' endpoints, which a frame offered by a ScheduleNow'd event of its instant had swapped."""
from test_sent_list import run_check


def test_host_nic_equals_egress(tmp_path):
    run_check(tmp_path, "host_nic")
