"""Warp programs (the default source of exec levels): every warp reads its
records as one list, with a barrier entry of its own where it has no work
between two barriers.  Bit-exact against the oracle for one and many streams,
every group count, one warp (no barrier shared), more warps than a level has
units (barrier entries only) and pools in the design's own numbering, which
keep the other forms."""
import numpy as np
import pytest

from oracle import pyoracle
from toucangpurt_gb300 import sim, workloads

pytestmark = pytest.mark.gpu

DESIGNS = {
    # multiplexers, comparators, table ops and vector ops; memories and chains
    "mixed": workloads.design_config("learned", n_lut=9_000, n_mems=6, ff_bits=512, luts_per_part=1_500, levels=12),
    "palette": workloads.design_config("scale", n_lut=5_000, levels=9, ff_bits=300, n_vec_ops=8, n_mems=2,
                                       mem_depth=64, luts_per_part=700),
    "two_operand": workloads.design_config("small"),
}


@pytest.fixture(scope="module")
def designs(tmp_path_factory, built):
    d = tmp_path_factory.mktemp("programs")
    out = {}
    for name, cfg in DESIGNS.items():
        dp, sp = d / f"{name}.bin", d / f"{name}.sym"
        out[name] = dp, sp, sim.generate(dp, sp, **cfg)
    return out


@pytest.mark.parametrize("name", list(DESIGNS))
@pytest.mark.parametrize("streams,groups", [(1, 0), (8, 1), (9, 2), (37, 4), (64, 8), (70, 0)])
@pytest.mark.parametrize("warps", [0, 1, 5, 32])
@pytest.mark.parametrize("mode", [0, 1])
def test_programs_match_oracle(designs, name, streams, groups, warps, mode):
    dp, sp, info = designs[name]
    cycles = np.full(streams, 20, np.uint32)
    stim = sim.StimulusSpec(31, info["pi_ids"], info["pi_bits"])
    with sim.Simulator(n_streams=streams, groups_per_item=groups, warps_per_block=warps, mode=mode) as s:
        s.init(0, dp, sp, False, False)
        assert s.design_stats()["program_words"] > 0
        got = s.batch_run(cycles, stim, cycle_digests=True)
    ref = pyoracle.OracleDesign(dp, sp).run(cycles, stim, cycle_digests=True)
    np.testing.assert_array_equal(got.cycle_digest, ref["cycle_digest"])
    np.testing.assert_array_equal(got.final_reg_digest, ref["final_reg_digest"])
    np.testing.assert_array_equal(got.final_mem_digest, ref["final_mem_digest"])


def test_design_numbering_keeps_other_forms(designs):
    dp, sp, _ = designs["mixed"]
    with sim.Simulator(n_streams=16, value_pool=1) as s:
        s.init(0, dp, sp, False, False)
        st = s.design_stats()
    assert st["program_words"] == 0 and st["resident_words"] + st["stage_words"] > 0


@pytest.mark.parametrize("blocks_per_sm", [0, 1])
@pytest.mark.parametrize("warps", [2, 16, 17])  # 16 warps: the widest block that keeps its programs resident
def test_persistent_programs_resident_or_streamed(designs, blocks_per_sm, warps):
    """Persistent launches keep their programs in shared memory when every
    block's fit (up to 8 items of a region and 512 threads) and stream them
    otherwise; several items per block, memories, a stop design's tail lists."""
    dp, sp, info = designs["palette"]
    n = 8 * 40
    cycles = np.full(n, 12, np.uint32)
    stim = sim.StimulusSpec(7, info["pi_ids"], info["pi_bits"])
    with sim.Simulator(n_streams=n, groups_per_item=1, blocks_per_sm=blocks_per_sm, warps_per_block=warps, mode=0) as s:
        s.init(0, dp, sp, False, False)
        st = s.design_stats()
        got = s.batch_run(cycles, stim, cycle_digests=True)
    if blocks_per_sm:
        assert st["region_items"] > st["blocks"]  # several items of a region per block
    ref = pyoracle.OracleDesign(dp, sp).run(cycles, stim, cycle_digests=True)
    np.testing.assert_array_equal(got.cycle_digest, ref["cycle_digest"])
    np.testing.assert_array_equal(got.final_mem_digest, ref["final_mem_digest"])


@pytest.mark.parametrize("name,streams", [("palette", 1500), ("mixed", 2500)])
@pytest.mark.parametrize("groups", [1, 2, 4, 8])
@pytest.mark.parametrize("warps", [1, 5, 8])
@pytest.mark.parametrize("mode", [0, 1])
def test_teams_match_oracle(designs, name, streams, groups, warps, mode):
    """More than one block of work per SM: teams of warps in one block per SM,
    which look odd streams up in the nibble table; full and partial last rows
    of teams, stops and inputs, both forms, two runs (graph chunks replayed)."""
    dp, sp, info = designs[name]
    n = streams if groups < 8 else 2 * streams
    cycles = np.full(n, 5, np.uint32)
    stim = sim.StimulusSpec(13, info["pi_ids"], info["pi_bits"])
    with sim.Simulator(n_streams=n, groups_per_item=groups, warps_per_block=warps, mode=mode) as s:
        s.init(0, dp, sp, False, False)
        st = s.design_stats()
        assert st["blocks"] > 152
        got = s.batch_run(cycles, stim, cycle_digests=True)
        again = s.batch_run(cycles, stim, cycle_digests=True, stop_exit=True)
    ref = pyoracle.OracleDesign(dp, sp).run(cycles, stim, cycle_digests=True)
    for o in (got, again):
        np.testing.assert_array_equal(o.cycle_digest, ref["cycle_digest"])
        np.testing.assert_array_equal(o.final_reg_digest, ref["final_reg_digest"])
        np.testing.assert_array_equal(o.final_mem_digest, ref["final_mem_digest"])
