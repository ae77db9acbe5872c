"""Two simulators in one process whose launches take different amounts of shared
memory of the same kernel: loading the smaller one leaves the larger one's
launches as they were, in every form."""
import numpy as np
import pytest

from oracle import pyoracle
from toucangpurt_gb300 import capi, sim, workloads

pytestmark = pytest.mark.gpu

WIDE = dict(n_lut=60_000, levels=6, ff_bits=4_000, n_vec_ops=8, n_mems=2, mem_depth=64)
FORMS = {
    # (options, streams, the larger design, the smaller one)
    "staged": (dict(resident_netlist=3, groups_per_item=4), 40, ("scale", dict(WIDE, luts_per_part=6_000)),
               ("scale", dict(WIDE, n_lut=4_000, luts_per_part=300))),
    "resident": (dict(resident_netlist=1, groups_per_item=1), 1, ("small", dict(n_lut=4_096)), ("small", dict(n_lut=600))),
    "programs": (dict(mode=capi.MODE_GRAPH, groups_per_item=4), 40, ("scale", dict(WIDE, luts_per_part=6_000)),
                 ("scale", dict(WIDE, n_lut=4_000, luts_per_part=300))),
    "resident programs": (dict(mode=capi.MODE_PERSISTENT), 1, ("small", dict(n_lut=4_096)), ("small", dict(n_lut=600))),
    "own streams": (dict(mode=capi.MODE_PERSISTENT, groups_per_item=1), 24, ("small", dict(n_lut=4_096)),
                    ("small", dict(n_lut=600))),
    "teams": (dict(mode=capi.MODE_PERSISTENT, groups_per_item=4, warps_per_block=6), 2_600,
              ("scale", dict(WIDE, n_lut=30_000, luts_per_part=1_500)), ("scale", dict(WIDE, n_lut=10_000, luts_per_part=500))),
}


@pytest.mark.parametrize("form", list(FORMS))
def test_smaller_second_handle(tmp_path, built, form):
    options, n, big, small = FORMS[form]
    shown = min(n, 40)
    runs = []
    for i, (name, cfg) in enumerate((big, small)):
        dp, sp = tmp_path / f"{i}.bin", tmp_path / f"{i}.sym"
        info = sim.generate(dp, sp, **workloads.design_config(name, **cfg))
        stim = sim.StimulusSpec(3, info["pi_ids"], info["pi_bits"])
        od = pyoracle.OracleDesign(dp, sp)
        ref = {c: od.run(np.full(shown, c, np.uint32), stim)["final_reg_digest"] for c in (6, 7)}
        runs.append((sim.Simulator(n_streams=n, **options), dp, sp, stim, ref))

    def check(s, stim, ref, c):
        np.testing.assert_array_equal(s.batch_run(np.full(n, c, np.uint32), stim).final_reg_digest[:shown], ref[c])

    try:
        for s, dp, sp, stim, ref in runs:
            s.init(0, dp, sp, False, False)
            assert s.design_stats()["forms"]["batch"] == form
            check(s, stim, ref, 6)
        for s, dp, sp, stim, ref in runs:  # the larger one again, after the smaller one; other cycles: captured anew
            check(s, stim, ref, 6)
            check(s, stim, ref, 7)
    finally:
        for r in runs:
            r[0].cleanup()
