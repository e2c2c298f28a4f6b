"""The DRAM traffic that bench.py prints comes from a committed profile: of
kernels that the sources still have, or none is printed."""
import glob
import os
import re

import pytest

import bench
import helpers as H


@pytest.mark.parametrize("workload", ["stokes65k", "star16k", "batch256"])
def test_traffic_is_of_kernels_that_exist(workload):
    traffic = bench.traffic_from_profile(workload)
    if traffic is None:
        return
    with open(os.path.join(H.ROOT, "profiles", "id_kernel_%s.txt" % workload)) as f:
        kernels = set(re.findall(r"\bid_\w+_kernel\b", f.read()))
    src = "".join(open(p).read() for p in
                  glob.glob(os.path.join(H.ROOT, "kern-interp-old_b200", "csrc", "*.cu")))
    assert kernels and all("%s(" % k in src for k in kernels)
    assert traffic > 0
