"""The device arrays an RDMA batch keeps between its runs, on the CPU: tests/rdma_arrays.cpp over
twins_b200/csrc/tr_arrays.h and a model of the memory (tests/test_rdma_gpu.py runs a batch again on a B200)."""
from test_sent_list import run_check


def test_arrays_kept_between_runs(tmp_path):
    run_check(tmp_path, "rdma_arrays")
