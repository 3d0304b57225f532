"""The kernel table of the measurement program: a pass's products stand in one row, whichever kernels ran them."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402


def test_products_of_a_pass_share_a_row():
    work = {"dense_tc_kernel": ("tensor", 3.0e9, 1.0e15), "delta_scan_kernel": ("f32", 1.0e6, 1.0e12)}
    scan = {"delta_scan_kernel": (2.0, 1.0)}
    rows = bench.kernel_rows(dict(scan, dense_tc_kernel=(4.0, 2.0), dense_pair_kernel=(8.0, 5.0)), work)
    assert rows[0] == dict(kernel="dense_pair_kernel + dense_tc_kernel", us=12.0, launches=7.0, bound="tensor", frac=0.25)
    assert rows[1] == dict(kernel="delta_scan_kernel", us=2.0, launches=1.0, bound="f32", frac=0.5)
    assert bench.kernel_rows(dict(dense_pair_kernel=(6.0, 5.0)), work) == [
        dict(kernel="dense_pair_kernel", us=6.0, launches=5.0, bound="tensor", frac=0.5)]
    assert bench.kernel_rows(dict(dense_tc_kernel=(6.0, 5.0)), work)[0]["frac"] == 0.5
