"""Stream groups per item where the option leaves them to the library: as many as
a block's shared memory has value pools for."""
import numpy as np
import pytest

from oracle import pyoracle
from toucangpurt_gb300 import capi, sim, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value_pool", [0, 1])
def test_large_value_pools(tmp_path, built, value_pool):
    """21,452 slots: the pools of four groups (348 KB) are more than a block
    can have, those of two (176 KB) are not; in the design's own numbering
    (64,128 slots) not even one group's."""
    dp, sp = tmp_path / "d.bin", tmp_path / "d.sym"
    info = sim.generate(dp, sp, **workloads.design_config("scale", seed=15, n_lut=150_000, luts_per_part=15_000, levels=4,
                                                          ff_bits=200_000, n_vec_ops=8, n_mems=2, mem_depth=64))
    n = 1000
    stim = sim.StimulusSpec(3, info["pi_ids"], info["pi_bits"])
    with sim.Simulator(n_streams=n, value_pool=value_pool) as s:
        if value_pool:
            with pytest.raises(capi.TgsError) as e:
                s.init(0, dp, sp, False, False)
            assert e.value.code == capi.ERR_RESOURCES
            return
        s.init(0, dp, sp, False, False)
        st = s.design_stats()
        assert st["groups_per_item"] == 2 and st["max_value_pool"] > 14_400
        got = s.batch_run(np.full(n, 3, np.uint32), stim)
        with pytest.raises(capi.TgsError):
            s.set_options(groups_per_item=4)
    ref = pyoracle.OracleDesign(dp, sp).run(np.full(24, 3, np.uint32), stim)
    np.testing.assert_array_equal(got.final_reg_digest[:24], ref["final_reg_digest"])


@pytest.fixture(scope="module")
def cones(tmp_path_factory, built):
    """Records of several levels, 18 partitions in a region."""
    d = tmp_path_factory.mktemp("cones")
    dp, sp = d / "d.bin", d / "d.sym"
    info = sim.generate(dp, sp, **workloads.design_config("scale", seed=15, n_lut=14_000, luts_per_part=400, levels=9,
                                                          ff_bits=2_000, n_vec_ops=8, n_mems=2, mem_depth=64,
                                                          cone_depth=3))
    return dp, sp, info


# both sides of two items of one group per SM and of three items of two groups
@pytest.mark.parametrize("mode", [0, 1])
def test_records_of_several_levels(cones, mode):
    dp, sp, info = cones
    stim = sim.StimulusSpec(3, info["pi_ids"], info["pi_bits"])
    ref = pyoracle.OracleDesign(dp, sp).run(np.full(40, 5, np.uint32), stim)["final_reg_digest"]
    seen = set()
    with sim.Simulator(mode=mode) as s:
        s.init(0, dp, sp, False, False)
        parts = s.design_stats()["region_items"]  # one stream: an item per partition
        for n in (40, 128, 136, 256, 400, 408, 520):
            groups = -(-n // 8)
            want = 4 if parts * -(-groups // 2) > 3 * 152 else 2 if parts * groups > 2 * 152 else 1
            if want == 2 and 6 * (groups + groups % 2) > 7 * groups:  # more padding than a sixth
                want = 1
            got = s.batch_run(np.full(n, 5, np.uint32), stim)
            assert s.design_stats()["groups_per_item"] == want, n
            seen.add(want)
            np.testing.assert_array_equal(got.final_reg_digest[:40], ref[:min(n, 40)])
    assert seen == {1, 2, 4}
