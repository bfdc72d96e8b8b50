"""A bounded grid barrier of the multigrid cycle's coarse levels that gives up is reported by the call
that ran the cycle, and the handle works on (the barrier's record is set by hand: no GPU waits)."""
import numpy as np
import pytest

from sysu_cfd_heat_gb300._lib import SysuError, lib
from sysu_cfd_heat_gb300.learned import LearnedPreconditioner
from test_gpu_resident_cg import seven_point

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_gnn", [False, True])
@pytest.mark.parametrize("call", ["fcg", "mg_apply", "add_pair"])
def test_a_barrier_that_gave_up_is_reported_once(call, use_gnn):
    rp, c, v, x, b = seven_point(24, 20, 18, seed=2)
    with LearnedPreconditioner(rp, c, v) as net:
        net.init_params(1)
        assert lib().sysu_gnn_mg_wait_selftest(net.h) == 1  # no cycle attached
        assert len(net.set_multigrid()) > 2
        run = {"fcg": lambda: net.fcg(b, use_gnn=use_gnn)[0], "mg_apply": lambda: net.mg_apply(b, use_gnn),
               "add_pair": lambda: net.add_pair(b, x)}[call]
        first = run()
        assert lib().sysu_gnn_mg_wait_selftest(net.h) == 0
        with pytest.raises(SysuError, match="timed out"):
            run()
        again = run()
        assert call == "add_pair" or np.array_equal(first, again)
