"""Droplets at positions that no box holds: every form refuses the call with the
same error, names the droplet and leaves it as it was."""
import numpy as np
import pytest

from pelemp_b200 import capi
from pelemp_b200 import workloads as W
from pelemp_b200.spray import SprayError, from_problem
from tests.gpu_util import device_sources, device_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("do_move", [0, 1])
@pytest.mark.parametrize("dim", [0, 1, 2])
@pytest.mark.parametrize("where,code", [(np.nan, capi.PMP_ERR_SOURCE_BOX), (np.inf, capi.PMP_ERR_STATE_BOX),
                                        (1e300, capi.PMP_ERR_STATE_BOX), (-1e300, capi.PMP_ERR_STATE_BOX)])
def test_every_form_refuses_alike(where, code, dim, do_move):
    prob = W.config2(n=3000, steps=1, ncells=(48, 48, 48), box=(16, 16, 16))
    b = 13  # the middle box, which no boundary touches
    part = prob.parts[b]
    i = int(np.argmax(part["rdata"][capi.PSTATE_DIA]))
    part["pos"][dim, i] = where
    for mode in (capi.PMP_MODE_FP64, capi.PMP_MODE_MIXED):
        sp = from_problem(prob, mode=mode)
        st_keep, st_v = device_state(prob)
        src, src_v = device_sources(prob)
        with pytest.raises(SprayError):
            sp.update_particles(st_v, src_v, prob.flow_dt, 0.0, prob.state_ghosts, prob.source_ghosts, 0, 0, do_move,
                                prob.spray_cfl_lev, 0)
        err = sp.last_error()
        assert (err.code, err.box, err.particle) == (code, b, i)
        got = sp.get_particles(b)
        for k in ("pos", "rdata", "id"):
            assert np.array_equal(got[k][..., i], part[k][..., i], equal_nan=k != "id")
        del st_keep
        sp.close()
