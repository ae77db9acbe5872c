"""Designs with one partition per region: blocks that own their streams retire
and admit queued streams on their own.  Against the oracle: queued lengths of
one cycle up, more slots than streams and fewer, partial last groups, stops
with and without the exit, resident runs with digests, tables and
continuation, every group count."""
import numpy as np
import pytest

from oracle import pyoracle
from toucangpurt_gb300 import sim, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def stop_design(tmp_path_factory, built):
    d = tmp_path_factory.mktemp("own")
    dp, sp = d / "d.bin", d / "s.bin"
    info = sim.generate(dp, sp, **workloads.design_config("small", seed=15, with_stop=2))
    assert info["partitions"] == 2
    return dp, sp, info


def _same(got, ref, stop_exit):
    keys = ["final_reg_digest", "final_mem_digest", "rolling_digest", "stop_cycle"]
    for k in keys:
        np.testing.assert_array_equal(getattr(got, k), ref[k], err_msg=k)


@pytest.mark.parametrize("n,slots", [(9, 8), (40, 16), (41, 24), (100, 40)])
@pytest.mark.parametrize("groups", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("stop_exit", [False, True])
def test_queued(stop_design, n, slots, groups, stop_exit):
    dp, sp, info = stop_design
    rng = np.random.default_rng(n)
    cyc = rng.integers(1, 40, n).astype(np.uint32)
    cyc[:3] = [1, 2, 1]
    stim = sim.StimulusSpec(5, info["pi_ids"], info["pi_bits"], workloads.toggles("batch", info["pi_bits"]))
    od = pyoracle.OracleDesign(dp, sp)
    lens = cyc
    if stop_exit:
        sc = od.run(cyc, stim)["stop_cycle"].astype(np.int64)
        lens = np.where(sc == 0xFFFFFFFF, cyc, np.minimum(sc + 1, cyc)).astype(np.uint32)
    ref = od.run(lens, stim, cycle_digests=True)
    with sim.Simulator(groups_per_item=groups) as s:
        s.init(0, dp, sp, False, False)
        got = s.batch_run(cyc, stim, slots=slots, stop_exit=stop_exit, cycle_digests=True)
        again = s.batch_run(cyc, stim, slots=slots, stop_exit=stop_exit, cycle_digests=True)
    _same(got, ref, stop_exit)
    _same(again, ref, stop_exit)
    for q in range(n):
        np.testing.assert_array_equal(got.cycle_digest[q, : lens[q]], ref["cycle_digest"][q, : lens[q]])


@pytest.mark.parametrize("n", [9, 16, 33])
@pytest.mark.parametrize("groups", [1, 2, 4])
@pytest.mark.parametrize("stop_exit", [False, True])
@pytest.mark.parametrize("table", [False, True])
def test_resident(stop_design, n, groups, stop_exit, table):
    dp, sp, info = stop_design
    ids, bits = info["pi_ids"], info["pi_bits"]
    stim = sim.StimulusSpec(5, ids, bits)
    if table:
        stim = sim.StimulusSpec(5, ids, bits, table=sim.stimulus_table(stim, n, 0, 30))
    od = pyoracle.OracleDesign(dp, sp)
    seeded = sim.StimulusSpec(5, ids, bits)
    cyc = np.full(n, 30, np.uint32)
    sc = od.run(cyc, seeded)["stop_cycle"].astype(np.int64)
    lens = np.where(sc == 0xFFFFFFFF, 30, np.minimum(sc + 1, 30)).astype(np.uint32) if stop_exit else cyc
    ref = od.run(lens, seeded, cycle_digests=True)
    with sim.Simulator(n_streams=n, groups_per_item=groups) as s:
        s.init(0, dp, sp, False, False)
        got = s.batch_run(cyc, stim, cycle_digests=True, stop_exit=stop_exit)
        _same(got, ref, stop_exit)
        for q in range(n):
            np.testing.assert_array_equal(got.cycle_digest[q, : lens[q]], ref["cycle_digest"][q, : lens[q]])
        if not table and not stop_exit:
            half = np.full(n, 15, np.uint32)
            s.batch_run(half, stim)
            got = s.batch_run(half, stim, continue_=True)
            _same(got, ref, stop_exit)
