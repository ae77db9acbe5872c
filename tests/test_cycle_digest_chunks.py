"""Per-cycle register digests: a warp sums a chunk of registers, and the chunk's
length follows from the number of registers (up to 64 chunks of 256, up to
128, more) and the grid.  Bit-exact on both sides of each line."""
import numpy as np
import pytest

from oracle import pyoracle
from toucangpurt_gb300 import sim, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(65_000, 64), (65_200, 65), (130_720, 128), (130_860, 129)],
                ids=lambda p: f"{p[1]}chunks")
def design(request, tmp_path_factory, built):
    ff, chunks = request.param
    d = tmp_path_factory.mktemp("chunks")
    dp, sp = d / "d.bin", d / "d.sym"
    info = sim.generate(dp, sp, **workloads.design_config("scale", n_lut=40_000, ff_bits=ff, luts_per_part=1_500, levels=9,
                                                          n_vec_ops=8, n_mems=2, mem_depth=64))
    assert (info["reg_pool"] + 255) // 256 == chunks
    return dp, sp, info


@pytest.mark.parametrize("streams", [1, 8, 19, 130])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("warps", [0, 2])  # grids with more warps than chunks and with fewer
def test_chunked_digests(design, streams, mode, warps):
    dp, sp, info = design
    cycles = np.full(streams, 6, np.uint32)
    stim = sim.StimulusSpec(11, info["pi_ids"], info["pi_bits"])
    ref = pyoracle.OracleDesign(dp, sp).run(cycles, stim, cycle_digests=True)
    with sim.Simulator(n_streams=streams, warps_per_block=warps, mode=mode) as s:
        s.init(0, dp, sp, False, False)
        got = s.batch_run(cycles, stim, cycle_digests=True)
    for k in ("cycle_digest", "rolling_digest", "final_reg_digest"):
        np.testing.assert_array_equal(getattr(got, k), ref[k], err_msg=k)
