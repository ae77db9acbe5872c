"""Register writes are launched and not waited for: every other entry point
sees them, whether it works on the simulator's stream or past it."""
import numpy as np
import pytest

from toucangpurt_gb300 import sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("streams", [1, 9])
@pytest.mark.parametrize("mode", [0, 1])
def test_writes_are_seen(small_design, tmp_path, streams, mode):
    dp, sp, info = small_design
    with sim.Simulator(n_streams=streams, mode=mode) as s:
        s.init(0, dp, sp, False, False)
        ids = [i for i, _ in sim.symbol_registers(sp)["pi_0"]]
        last = streams - 1
        for v in (0x12345678, 0xFFFFFFFF, 0):
            s.set_register("pi_0", v, last)
            assert s.read_register("pi_0", last) == v
            s.set_register("pi_0", v ^ 5, last)
            pool = s.reg_pool(last)
            assert int("".join(f"{pool[i]:x}" for i in ids), 16) == v ^ 5
            s.set_register("pi_0", v, last)
            before = s.digest(last)[0]
            s.set_register("pi_0", v ^ 1, last)
            assert s.digest(last)[0] != before
        s.set_register("pi_0", 0xABCDEF01, last)
        s.dump_state(tmp_path / "state")
        s.set_register("pi_0", 3, last)
        s.load_state(tmp_path / "state")
        assert s.read_register("pi_0", last) == 0xABCDEF01
        s.set_register("pi_0", 7, last)
        s.reset_state()
        # a write between evaluations reaches the next one: two handles that
        # set the same inputs end alike, one that waits after every write
        with sim.Simulator(n_streams=streams, mode=mode) as t:
            t.init(0, dp, sp, False, False)
            for v in range(6):
                s.set_register("pi_0", v * 0x01234567, last)
                s.eval()
                t.set_register("pi_0", v * 0x01234567, last)
                t.read_register("pi_0", last)
                t.eval()
            np.testing.assert_array_equal(s.reg_pool(last), t.reg_pool(last))
