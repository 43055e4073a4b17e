"""The bytes that the bench credits to a kernel's launch: the same for the main line and the
precision study, for every four-sweep kernel."""
import os
import re

import bench

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_four_sweep_kernels_are_credited_once_per_launch():
    with open(os.path.join(ROOT, "st_spix_gb300", "csrc", "kernels.h")) as f:
        names = re.findall(r"STSPIX_DECL_SWEEP\((kb_sweep4_\w+)\)", f.read())
    assert len(names) == 4
    # labels read and written and colours read once, however many sweeps, and the
    # statistics of four sweeps
    assert bench.SWEEP_LAUNCH_BYTES_PER_PX[4] == 4 + 12 + 4 + 16
    for n in names:
        assert bench.KERNEL_BYTES_PER_PX[n] == bench.SWEEP_LAUNCH_BYTES_PER_PX[4]
