"""Schedule tables of other schedule sets: a table whose first line names the set of the
one-path-per-thread kernels (2), or an earlier or later one, is refused although its device and
entries are valid; this set's is taken."""
from __future__ import annotations

import ctypes as C

import pytest

from gemray_studio_b200 import GpuFrameRenderer, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule_set", [1, 2, abi.GR_SCHEDULE_SET, abi.GR_SCHEDULE_SET + 1])
def test_tables_of_other_kernels(engine_lib, tmp_path, schedule_set):
    r = GpuFrameRenderer()
    path = tmp_path / "schedules.txt"
    head = f"gemray-schedules {schedule_set} {r.lib.gr_device_label(r.ctx).decode()}"
    path.write_text(head + "\n0123456789abcdef 12 20 16 1.5\n")
    n, count = C.c_uint32(7), C.c_uint32()
    st = r.lib.gr_tuning_load(r.ctx, str(path).encode(), C.byref(n))
    assert r.lib.gr_tuning_count(r.ctx, C.byref(count)) == abi.GR_OK
    r.close()
    taken = schedule_set == abi.GR_SCHEDULE_SET and schedule_set > 2  # set 2 was timed on kernels that are gone
    assert (st == abi.GR_OK) == taken and n.value == count.value == (1 if taken else 0)
