"""The droplet store (pmp_store.cu) where a call's own kernels, another stream
or memory could be in its way: droplets handed over and packed on streams that
do not order one another."""
import ctypes as C

import numpy as np
import pytest

from pelemp_b200 import capi, spray
from pelemp_b200.spray import from_problem
from tests.test_gpu_handover import droplets, level

pytestmark = pytest.mark.gpu

HOLD = 200_000_000  # clock cycles for which a stream is held, 0.1 s


def filled(prob, counts, nf=2, seed=3):
    """A container with `counts` droplets handed over, and the droplets."""
    rng = np.random.default_rng(seed)
    sp = from_problem(prob, set_droplets=False)
    drs = [droplets(rng, n, nf, lo, hi, prob.dx[0]) for n, (lo, hi) in zip(counts, prob.boxes)]
    for b, d in enumerate(drs):
        sp.set_particles(b, *d)
    return sp, drs


def expected_dt(prob, drs):
    v = np.concatenate([d[1][:3] for d in drs], axis=1)
    return np.min(0.5 / np.max(np.abs(v) * (1.0 / prob.dx)[:, None], axis=0))


def check(sp, drs):
    for b, d in enumerate(drs):
        got = sp.get_particles(b)
        for have, want in zip((got["pos"], got["rdata"], got["id"]), d):
            assert np.array_equal(have, want)


def refuse(sp, box, n):
    """A hand-over of n droplets that is refused."""
    p = capi.Particles()
    p.layout, p.where, p.n = 7, capi.PMP_WHERE_DEVICE, n
    assert spray.lib().pmp_spray_set_particles(sp._h, box, C.byref(p)) == capi.PMP_ERR_INVALID


@pytest.mark.parametrize("counts", [(3000, 2000), (60_000, 50_000)])
@pytest.mark.parametrize("case", ["packed", "staged", "refused"])
def test_emptied_box_and_another_stream(case, counts):
    """A box is handed over empty while the stream of the hand-over's kernels is held, and the next
    operation runs on a stream that does not wait for that one."""
    import torch
    prob = level(2)
    sp, drs = filled(prob, counts)
    if case != "staged":
        sp.est_timestep(0.5)  # packs: the hand-over then unpacks the other box
    empty = droplets(np.random.default_rng(0), 0, 2, *prob.boxes[0], prob.dx[0])
    side = torch.cuda.Stream()
    torch.cuda._sleep(HOLD)
    if case == "refused":
        refuse(sp, 0, 5)  # unpacks, and is refused
    sp.set_particles(0, *empty)
    drs[0] = empty
    assert sp.est_timestep(0.5, stream=side.cuda_stream) == expected_dt(prob, drs)
    torch.cuda.synchronize()
    check(sp, drs)
