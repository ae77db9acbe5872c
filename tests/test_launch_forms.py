"""The forms in which runs are launched, named by the design statistics, and each
against the oracle on designs whose streams stop: queued runs on grids of
several blocks and partitions (resident and streamed warp programs), blocks that
own their streams with every group count, teams with and without the exit."""
import numpy as np
import pytest

from oracle import pyoracle
from tests import designlib as dl
from toucangpurt_gb300 import capi, sim, workloads

pytestmark = pytest.mark.gpu

NO_STOP = 0xFFFFFFFF
SCALE = dict(seed=15, ff_bits=300, n_vec_ops=8, n_mems=2, mem_depth=64, with_stop=2, levels=9)
DESIGNS = {
    "one": ("small", dict(seed=15, with_stop=2)),  # one partition per region
    "four": ("scale", dict(SCALE, n_lut=5_000, luts_per_part=700)),
    "two": ("scale", dict(SCALE, n_lut=16_000, luts_per_part=4_000)),
}


@pytest.fixture(scope="module")
def designs(tmp_path_factory, built):
    d = tmp_path_factory.mktemp("forms")
    out = {}
    for name, (base, cfg) in DESIGNS.items():
        dp, sp = d / f"{name}.bin", d / f"{name}.sym"
        info = sim.generate(dp, sp, **workloads.design_config(base, **cfg))
        out[name] = dp, sp, info, pyoracle.OracleDesign(dp, sp)
    return out


def _expected(od, cyc, stim, stop_exit):
    """Lengths that the streams run and the oracle's results over them."""
    lens = cyc
    if stop_exit:
        sc = od.run(cyc, stim)["stop_cycle"].astype(np.int64)
        lens = np.where(sc == NO_STOP, cyc, np.minimum(sc + 1, cyc)).astype(np.uint32)
        assert (lens < cyc).any()
    return lens, od.run(lens, stim, cycle_digests=True)


def _same(got, lens, ref):
    for k in ("final_reg_digest", "final_mem_digest", "rolling_digest", "stop_cycle"):
        np.testing.assert_array_equal(getattr(got, k), ref[k], err_msg=k)
    for q in range(lens.size):
        np.testing.assert_array_equal(got.cycle_digest[q, :lens[q]], ref["cycle_digest"][q, :lens[q]])
        assert not got.cycle_digest[q, lens[q]:].any()


@pytest.mark.parametrize("name,streams,options,batch,queue,free", [
    ("one", 1, {}, "resident programs", "resident programs", "resident programs"),
    ("one", 9, {}, "own streams", "own streams", "resident programs"),
    ("one", 9, dict(mode=1), "programs", "programs", "programs"),
    # 152 and 153 blocks of one group, one per SM asked for
    ("one", 8 * 152, dict(groups_per_item=1, blocks_per_sm=1), "own streams", "own streams", "resident programs"),
    ("one", 8 * 153, dict(groups_per_item=1, blocks_per_sm=1), "resident programs", "resident programs", "resident programs"),
    ("one", 8 * 153, dict(groups_per_item=1), "own streams", "own streams", "resident programs"),
    ("four", 9, {}, "resident programs", "resident programs", "resident programs"),
    ("four", 9, dict(warps_per_block=17), "programs", "programs", "programs"),
    ("four", 9, dict(resident_netlist=1), "resident", "resident", "resident"),
    ("four", 9, dict(resident_netlist=2), "global", "global", "global"),
    ("four", 9, dict(resident_netlist=3), "staged", "staged", "staged"),
    ("two", 2500, dict(groups_per_item=4, warps_per_block=5), "teams", "programs", "teams"),
    # the graph form: teams where a region has more items than blocks
    ("two", 2500, dict(groups_per_item=4, warps_per_block=5, mode=1), "programs", "programs", "programs"),
    ("two", 2500, dict(groups_per_item=2, warps_per_block=5, blocks_per_sm=2, mode=1), "teams", "programs", "teams"),
])
def test_stats_name_the_launch(designs, name, streams, options, batch, queue, free):
    dp, sp = designs[name][:2]
    with sim.Simulator(n_streams=streams, **options) as s:
        s.init(0, dp, sp, False, False)
        st = s.design_stats()
    assert st["forms"] == {"batch": batch, "queue": queue, "free": free}
    assert st["launch_blocks"] == (152 if batch == "teams" else st["blocks"])
    assert not options.get("blocks_per_sm") or st["launch_blocks"] <= 152 * options["blocks_per_sm"]
    # the truth table and a value pool for every block of work in a launched block
    pools = -(-st["blocks"] // st["launch_blocks"])
    assert st["smem_per_block"] >= 4642 + pools * 4 * st["max_value_pool"] * st["groups_per_item"]


# (streams, slots): one group and one block per region, partial last groups, 25 groups
@pytest.mark.parametrize("n,slots", [(20, 8), (41, 24), (90, 64), (300, 200)])
@pytest.mark.parametrize("warps,form", [(0, "resident programs"), (17, "programs")])
@pytest.mark.parametrize("stop_exit", [False, True])
def test_queue_over_blocks(designs, n, slots, warps, form, stop_exit):
    dp, sp, info, od = designs["four"]
    cyc = np.random.default_rng(n).integers(1, 40, n).astype(np.uint32)
    cyc[:3] = [1, 2, 1]
    stim = sim.StimulusSpec(5, info["pi_ids"], info["pi_bits"])
    lens, ref = _expected(od, cyc, stim, stop_exit)
    with sim.Simulator(groups_per_item=1, warps_per_block=warps) as s:
        s.init(0, dp, sp, False, False)
        for _ in range(2):
            _same(s.batch_run(cyc, stim, slots=slots, stop_exit=stop_exit, cycle_digests=True), lens, ref)
        st = s.design_stats()
    assert st["forms"]["queue"] == form
    assert st["blocks"] == st["region_items"] >= 4 * (slots // 8)


# more slots than one group block holds, for every group count
@pytest.mark.parametrize("groups,n,slots", [(1, 41, 16), (2, 60, 32), (4, 100, 72), (8, 150, 136)])
@pytest.mark.parametrize("stop_exit", [False, True])
def test_own_streams_queue(designs, groups, n, slots, stop_exit):
    dp, sp, info, od = designs["one"]
    cyc = np.random.default_rng(n).integers(1, 40, n).astype(np.uint32)
    cyc[:3] = [1, 2, 1]
    stim = sim.StimulusSpec(5, info["pi_ids"], info["pi_bits"], workloads.toggles("batch", info["pi_bits"]))
    lens, ref = _expected(od, cyc, stim, stop_exit)
    with sim.Simulator(groups_per_item=groups) as s:
        s.init(0, dp, sp, False, False)
        _same(s.batch_run(cyc, stim, slots=slots, stop_exit=stop_exit, cycle_digests=True), lens, ref)
        st = s.design_stats()
    assert st["forms"]["queue"] == "own streams" and st["groups_per_item"] == groups and st["launch_blocks"] > 1


@pytest.mark.parametrize("groups,n", [(1, 17), (2, 39), (4, 72), (8, 131)])
@pytest.mark.parametrize("stop_exit", [False, True])
def test_own_streams_batch(designs, groups, n, stop_exit):
    dp, sp, info, od = designs["one"]
    cyc = np.full(n, 30, np.uint32)
    stim = sim.StimulusSpec(5, info["pi_ids"], info["pi_bits"])
    lens, ref = _expected(od, cyc, stim, stop_exit)
    with sim.Simulator(n_streams=n, groups_per_item=groups) as s:
        s.init(0, dp, sp, False, False)
        st = s.design_stats()
        assert st["forms"]["batch"] == "own streams" and st["groups_per_item"] == groups and st["launch_blocks"] > 1
        _same(s.batch_run(cyc, stim, stop_exit=stop_exit, cycle_digests=True), lens, ref)


# a full last row of teams, one with teams without work, more items than blocks
@pytest.mark.parametrize("name,n,options", [
    ("four", 1500, dict(groups_per_item=1, warps_per_block=5)),
    ("two", 2500, dict(groups_per_item=4, warps_per_block=5)),
    ("two", 2500, dict(groups_per_item=2, warps_per_block=5, blocks_per_sm=2)),
    ("two", 2500, dict(groups_per_item=2, warps_per_block=5, blocks_per_sm=2, mode=capi.MODE_GRAPH)),
])
@pytest.mark.parametrize("stop_exit", [False, True])
def test_teams_with_stops(designs, name, n, options, stop_exit):
    dp, sp, info, od = designs[name]
    cyc = np.full(n, 20, np.uint32)
    stim = sim.StimulusSpec(5, info["pi_ids"], info["pi_bits"])
    lens, ref = _expected(od, cyc, stim, stop_exit)
    with sim.Simulator(n_streams=n, **options) as s:
        s.init(0, dp, sp, False, False)
        assert s.design_stats()["forms"]["batch"] == "teams"
        for _ in range(2):
            _same(s.batch_run(cyc, stim, stop_exit=stop_exit, cycle_digests=True), lens, ref)


@pytest.mark.parametrize("n", [1, 19, 100])
@pytest.mark.parametrize("stop_exit", [False, True])
def test_resident_programs_with_stops(designs, n, stop_exit):
    dp, sp, info, od = designs["four"]
    cyc = np.full(n, 25, np.uint32)
    stim = sim.StimulusSpec(11, info["pi_ids"], info["pi_bits"])
    lens, ref = _expected(od, cyc, stim, stop_exit) if n > 1 else (cyc, od.run(cyc, stim, cycle_digests=True))
    if n == 1 and stop_exit:
        lens = np.minimum(cyc, ref["stop_cycle"].astype(np.int64) + 1).astype(np.uint32)
        ref = od.run(lens, stim, cycle_digests=True)
    with sim.Simulator(n_streams=n) as s:
        s.init(0, dp, sp, False, False)
        assert s.design_stats()["forms"]["batch"] == "resident programs"
        _same(s.batch_run(cyc, stim, stop_exit=stop_exit, cycle_digests=True), lens, ref)


# eval() takes its outcome from page-locked words, in which every block that
# owns its streams puts what it has seen; the graph form copies the stop flags
@pytest.mark.parametrize("groups,n", [(1, 17), (2, 40)])
def test_own_streams_eval_outcome(designs, groups, n):
    dp, sp, info, _ = designs["one"]
    stim = sim.StimulusSpec(5, info["pi_ids"], info["pi_bits"])
    table = sim.stimulus_table(stim, n, 0, 30)
    for only in (0, n // 2, n - 1):  # the stream that gets inputs, in the first, a middle and the last block
        out = []
        for mode in (capi.MODE_PERSISTENT, capi.MODE_GRAPH):
            with sim.Simulator(n_streams=n, groups_per_item=groups, mode=mode) as s:
                s.init(0, dp, sp, False, False)
                assert s.design_stats()["forms"]["batch"] == ("programs" if mode else "own streams")
                stops = []
                for c in range(30):
                    pool = s.reg_pool(only)
                    pool[info["pi_ids"]] = table[c, :, only]
                    s.write_reg_pool(pool, only)
                    stops.append(s.eval())
                out.append((stops, s.digest(only), s.eval_done()))
        assert out[0] == out[1]


# memories that hold bytes of 0x80 and above, whose digest terms carry out of
# the low byte; sizes off the 16 bytes that the retirements read at a time
@pytest.mark.parametrize("size", [40, 64, 77])
@pytest.mark.parametrize("mode,form", [(0, "own streams"), (1, "programs")])
def test_retired_memories_of_any_bytes(tmp_path, built, size, mode, form):
    zero = [dl.MPart(top=[], wbs=[dl.wb(0, 64 + i) for i in range(32)])]
    p0 = dl.Part(vp_size=160, reg_reads=[(i, 16 + i) for i in range(16)], levels=[zero], exg_write=(0, 64, 32))
    p1 = dl.Part(vp_size=64, exg_reads=[(i, 16 + i) for i in range(32)], levels=[], reg_write=(16, 16, 32))
    for fill in (np.arange(size) * 37 % 256, np.arange(size) % 128):
        d = dl.Design(reg_pool=64, mem_pool=size, exg_pool=32, parts=[p0, p1], regions=[[0], [1]],
                      mem_init=fill.astype(np.uint8).tobytes())
        d.write(tmp_path / "d.bin")
        with np.errstate(over="ignore"):
            want = sim.mix64(np.arange(size, dtype=np.uint64) << np.uint64(8) | fill.astype(np.uint64)).sum(dtype=np.uint64)
        with sim.Simulator(groups_per_item=1, mode=mode, validate=0) as s:  # the static checks want nibbles
            s.init(0, tmp_path / "d.bin", None, False, False)
            got = s.batch_run((np.arange(50) % 9 + 1).astype(np.uint32), slots=24)
            assert s.design_stats()["forms"]["queue"] == form
        np.testing.assert_array_equal(got.final_mem_digest, np.full(50, want, np.uint64))
