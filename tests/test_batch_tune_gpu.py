"""The batch tuner's candidates hold the untuned default: the item size by the batch's
size (256 elements on small ones, below the smallest fixed candidate)."""
import re

import pytest

from op2b.batch import AirfoilBatch

pytestmark = pytest.mark.gpu


def test_the_default_item_size_is_a_candidate(op2):
    b = AirfoilBatch([dict(I=40, J=20, mach=0.4, alpha=1.0, bump=0.05, seed=1)], fp32=False)
    rep = b.tune(iters=2)
    times = {tuple(m[:3]): float(m[3]) for m in
             re.findall(r"res_kernel=(\w+) block=(\d+) part_size=(\d+): ([\d.]+) ms/iter", rep)}
    assert {p for _, _, p in times} == {"0", "512", "8192"} and len(times) == 27
    chosen = re.search(r"chosen: res_kernel=(\w+) block=(\d+) part_size=(\d+)", rep).groups()
    assert times[chosen] == min(times.values())
    b.close()
