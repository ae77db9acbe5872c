"""A memory access out of range, found by the kernels' own check: the error word
ends the launch within a few cycles, on grids of several blocks and where blocks
own their streams; the handle works on.

A run of 2,000,000 cycles of this design takes seconds when nothing ends it."""
import time

import numpy as np
import pytest

from tests import designlib as dl
from toucangpurt_gb300 import capi, sim

pytestmark = pytest.mark.gpu

CYCLES = 2_000_000
IN, OUT = 16, 64


@pytest.fixture()
def design(tmp_path, built):
    """Every cycle reads memory at the address in registers 0..7."""
    addr = [dl.MPart(top=[dl.top(0, 0, 0, IN + i) for i in range(8)], wbs=[dl.wb(32 + i, 120 + i) for i in range(8)])]
    zero = [dl.MPart(top=[], wbs=[dl.wb(0, OUT + i) for i in range(32)])]
    read = [dl.MPart(is_lut=False, mem_reads=[dl.mem_read(False, 8, 1, 120, OUT)])]
    p0 = dl.Part(vp_size=160, reg_reads=[(i, IN + i) for i in range(16)], levels=[zero, addr, read], exg_write=(0, OUT, 32))
    p1 = dl.Part(vp_size=64, exg_reads=[(i, 16 + i) for i in range(32)], levels=[], reg_write=(16, 16, 32))
    d = dl.Design(reg_pool=64, mem_pool=64, exg_pool=32, parts=[p0, p1], regions=[[0], [1]])
    paths = []
    for name, address in (("beyond", 0xF00), ("within", 0x3)):
        d.reg_init = bytes((address >> 4 * i) & 15 for i in range(8)) + bytes(56)
        paths.append(tmp_path / f"{name}.bin")
        d.write(paths[-1])
    return paths


@pytest.mark.parametrize("run,form", [("free", "resident programs"), ("batch", "own streams"), ("queue", "own streams")])
def test_error_ends_run(design, run, form):
    beyond, within = design
    with sim.Simulator(n_streams=24, groups_per_item=1) as s:
        s.init(0, beyond, None, False, False)
        st = s.design_stats()
        assert st["forms"][run] == form and st["launch_blocks"] == 3
        t = time.perf_counter()
        with pytest.raises(capi.TgsError) as e:
            if run == "free":
                s.eval_free_running(CYCLES)
            elif run == "batch":
                s.batch_run(np.full(24, CYCLES, np.uint32))
            else:
                s.batch_run(np.full(30, CYCLES, np.uint32), slots=24)
        t = time.perf_counter() - t
        assert e.value.code == capi.ERR_DEVICE_FAULT and "beyond memPool" in str(e.value)
        assert t < 0.5
        if run == "free":
            assert s.real_cycles() < 1000
        s.init(0, within, None, False, False)
        s.batch_run(np.full(24, 5, np.uint32))
        s.eval()
