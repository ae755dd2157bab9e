"""The FP64 form in gas that holds fuel vapour, where part of the droplets take
up vapour (negative mass transfer number): the oracle's bits, and no second
evaluation of the droplets, which would show in the time."""
import numpy as np
import pytest

from pelemp_b200 import workloads as W
from pelemp_b200.spray import from_problem
from tests.gpu_util import assert_bitwise, device_sources, device_state, gpu_run, oracle_run

pytestmark = pytest.mark.gpu


def with_vapour(prob, share, spread=0.3, seed=2):
    """The gas with fuel vapour of about `share` of its mass, uneven from cell to cell."""
    rng = np.random.default_rng(seed)
    nf, ns = prob.nfuel, len(prob.species)
    for st in prob.state:
        f = share * (1.0 + spread * rng.random(st.shape[1:]))
        st[4] = 0.77 * (1.0 - f) * st[3]
        st[5] = 0.23 * (1.0 - f) * st[3]
        for k in range(nf):
            st[6 + k] = f / nf * st[3]
        for k in range(2 + nf, ns):
            st[4 + k] = 0.0
    return prob


@pytest.mark.parametrize("share", [0.02, 0.2, 0.5])
@pytest.mark.parametrize("nf", [1, 2])
def test_droplets_in_vapour_match_the_oracle(nf, share, oracle):
    prob = W.config1(n=4000, steps=2) if nf == 1 else W.config2(n=4000, steps=2, ncells=(16, 16, 16), box=(16, 16, 16))
    assert len(prob.boxes) == 1  # so that no grown boxes overlap
    prob = with_vapour(prob, share)
    pg, _, _ = gpu_run(prob, 2)
    po, _ = oracle_run(oracle, prob, 2)
    assert_bitwise(pg, po)


def test_condensation_costs_no_second_evaluation():
    """Measured 0.35 ms without vapour and 0.97 when every droplet was evaluated twice."""
    ms = {}
    for share in (0.0, 0.3):
        prob = with_vapour(W.config2(n=300_000, steps=1, ncells=(32, 32, 32), box=(32, 32, 32)), share)
        sp = from_problem(prob, set_droplets=False)
        st_keep, st_v = device_state(prob)
        src, src_v = device_sources(prob)
        times = []
        for _ in range(6):
            for b, p in enumerate(prob.parts):
                sp.set_particles(b, p["pos"], p["rdata"], p["id"])
            sp.update_particles(st_v, src_v, prob.flow_dt, 0.0, prob.state_ghosts, prob.source_ghosts, 0, 0, 1,
                                prob.spray_cfl_lev, 0)
            times.append(sp.stats().kernel_ms)
        ms[share] = min(times[1:])
        del st_keep
        sp.close()
    print("update without and with vapour: %.3f and %.3f ms" % (ms[0.0], ms[0.3]))
    assert ms[0.3] < 1.7 * ms[0.0]
