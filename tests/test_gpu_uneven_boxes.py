"""A level whose boxes differ in size: the gas records' pass covers each box's
cells and no more."""
import numpy as np
import pytest

from pelemp_b200 import capi
from pelemp_b200 import workloads as W
from pelemp_b200.spray import from_problem, views
from tests.gpu_util import assert_bitwise, gpu_run, host_run, oracle_run

pytestmark = pytest.mark.gpu

MODES = [capi.PMP_MODE_FP64, capi.PMP_MODE_MIXED]


def split(prob, cuts):
    """The one-box problem `prob` with its domain cut at `cuts` (per direction) into boxes of its state
    and droplets."""
    (lo, hi), = prob.boxes
    g = prob.state_ghosts
    st, = prob.state
    part, = prob.parts
    cell = np.floor(part["pos"] / prob.dx[:, None]).astype(int)
    edges = [[lo[d], *cuts[d], hi[d] + 1] for d in range(3)]
    prob.boxes, prob.state, prob.parts = [], [], []
    for k in range(len(edges[2]) - 1):
        for j in range(len(edges[1]) - 1):
            for i in range(len(edges[0]) - 1):
                a = [edges[d][c] for d, c in enumerate((i, j, k))]
                e = [edges[d][c + 1] for d, c in enumerate((i, j, k))]
                inside = np.all([(cell[d] >= a[d]) & (cell[d] < e[d]) for d in range(3)], axis=0)
                prob.boxes.append((tuple(a), tuple(v - 1 for v in e)))
                prob.state.append(np.ascontiguousarray(st[:, a[2]:e[2] + 2 * g, a[1]:e[1] + 2 * g, a[0]:e[0] + 2 * g]))
                prob.parts.append({key: np.ascontiguousarray(v[..., inside]) for key, v in part.items()})
    return prob


# 1, 2, 8, 32, 33 and 1331 boxes: none, one and more looks of 32, the last of them ragged
CUTS = [([], [], []), ([1], [], []), ([20], [3], [29]), ([5, 8, 24], [4, 9, 30], [16]), (list(range(2, 22, 2)), [1, 30], []),
        (list(range(3, 33, 3))[:10],) * 3]


@pytest.mark.parametrize("cuts", CUTS, ids=lambda c: str(np.prod([len(v) + 1 for v in c])))
@pytest.mark.parametrize("run", [gpu_run, host_run])
def test_boxes_of_every_size_match_the_oracle(cuts, run, oracle):
    prob = split(W.config1(n=3000, steps=1), cuts)
    pg, _, _ = run(prob, 1)
    po, _ = oracle_run(oracle, prob, 1)
    assert_bitwise(pg, po)
    pm, _, _ = run(prob, 1, mode=capi.PMP_MODE_MIXED)
    for a, b in zip(pm, po):
        for row in (capi.PSTATE_T, capi.PSTATE_DIA):
            assert np.all(np.abs(a["rdata"][row] / b["rdata"][row] - 1) <= 1e-4)


@pytest.mark.parametrize("mode", MODES)
def test_small_boxes_beside_a_large_one(mode):
    """One box of 96^3 and 400 of 8^3 (400 x 11 + 4156 CTAs of records) take little more time than the one;
    with a row of 4156 CTAs a box, 20 times as much (3.4 and 0.25 ms beside 128^3)."""
    import torch

    def update_ms(small):
        prob = W.config1(n=10, steps=1)
        prob.boxes = [((0, 0, 0), (95, 95, 95))]
        prob.boxes += [((96 + 8 * (i % 20), 8 * (i // 20), 0), (103 + 8 * (i % 20), 8 * (i // 20) + 7, 7)) for i in range(small)]
        prob.domain_hi = (255, 159, 95)
        prob.phi = prob.dx * np.array([256, 160, 96])
        sp = from_problem(prob, mode=mode, set_droplets=False)
        keep, los, slos = [], [], []
        for b, (lo, hi) in enumerate(prob.boxes):
            shape = tuple(hi[d] - lo[d] + 1 for d in (2, 1, 0))
            st = torch.zeros((9,) + tuple(n + 6 for n in shape), dtype=torch.float64, device="cuda")
            st[3], st[4], st[5], st[7], st[8] = 0.4, 0.4 * 0.77, 0.4 * 0.23, 1e5, 900.0
            keep.append((st, torch.zeros((6,) + tuple(n + 4 for n in shape), dtype=torch.float64, device="cuda")))
            los.append([v - 3 for v in lo])
            slos.append([v - 2 for v in lo])
            pos = np.array([[lo[d] + 0.5 + 0.3 * i for i in range(4)] for d in range(3)]) * prob.dx[0]
            rd = np.zeros((11, 4))
            rd[3], rd[4], rd[5], rd[6] = 300.0, 2e-5, 1.0, 1.0
            sp.set_particles(b, pos, rd, np.arange(1, 5, dtype=np.int32))
        sv, srv = views([k[0] for k in keep], los), views([k[1] for k in keep], slos)
        ms = []
        for _ in range(6):
            sp.update_particles(sv, srv, 1e-7, 0.0, 3, 2, 0, 0, 0, 0.1, 0)
            ms.append(sp.stats().kernel_ms)
        sp.close()
        return min(ms[1:])

    one, many = update_ms(0), update_ms(400)
    print("update of one box of 96^3, and with 400 of 8^3: %.3f and %.3f ms" % (one, many))
    assert many < 4 * one
