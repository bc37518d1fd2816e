"""A CTA may touch another CTA's shared memory only once that CTA runs, which a cluster barrier alone guarantees.  How
long CTAs take to start cannot be forced by a test, so the order is checked in the kernels' sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "qcmaquis_b200", "csrc")
# every source whose kernels address the shared memory of other CTAs of their cluster
SOURCES = ["jacobi_svd.cu", "qr_batched.cu"]


@pytest.mark.parametrize("name", SOURCES)
def test_barrier_before_any_access_to_other_ctas(name):
    src = open(os.path.join(CSRC, name)).read()
    kernels = re.findall(r"^__global__ .*?^}", src, flags=re.S | re.M)
    using = [k for k in kernels if "map_shared_rank" in k]
    assert using
    for k in using:
        # a statement of the kernel's own body (indented by four), taken by all threads of all CTAs
        barrier = re.search(r"^    cluster_sync\(\);", k, flags=re.M)
        assert barrier and barrier.start() < k.index("map_shared_rank")
