"""The mixed 4M- and the 16M-LUT benchmark designs, 64 streams: the graph form,
which the benchmark's helper no longer picks for them, gives the same per-cycle
digests and states as the persistent form, which the full-size fixtures pin."""
import numpy as np
import pytest

from toucangpurt_gb300 import sim, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,streams", [("learned", 256), ("largest", 64)])
def test_graph_form_at_full_size(tmp_path, built, name, streams):
    dp, sp = tmp_path / "d.bin", tmp_path / "d.sym"
    info = sim.generate(dp, sp, **workloads.design_config(name))
    stim = sim.StimulusSpec(17, info["pi_ids"], info["pi_bits"], workloads.toggles(name, info["pi_bits"]))
    cycles = np.full(streams, 3, np.uint32)
    out = []
    for mode in ("persistent", "graph"):
        s, _ = workloads.bench_simulator(name, dp, sp, streams=streams, schedule="greedy", mode=mode)
        assert s.design_stats()["forms"]["batch"] == "teams"
        out.append(s.batch_run(cycles, stim, cycle_digests=True))
        s.cleanup()
    for k in ("cycle_digest", "rolling_digest", "final_reg_digest", "final_mem_digest"):
        np.testing.assert_array_equal(getattr(out[0], k), getattr(out[1], k), err_msg=k)
