"""Hand-over and write-back of droplets (pmp_store.cu): bytes in, bytes out.

Every layout and place (records or component arrays, host or device memory,
device memory the kernels cannot take directly), counts around the kernels'
128-droplet tiles, one and two fuels, before and after packing, and a box
handed over again while the others are packed.  The droplets come back
exactly; the packed order is by cell, stable in the caller's order.
"""
import ctypes as C

import numpy as np
import pytest

from pelemp_b200 import capi, spray
from pelemp_b200 import workloads as W
from pelemp_b200.spray import from_problem

pytestmark = pytest.mark.gpu


def droplets(rng, n, nf, lo, hi, dx):
    pos = (np.asarray(lo)[:, None] + rng.random((3, n)) * (np.asarray(hi) - lo + 1)[:, None]) * dx
    rd = rng.standard_normal((10 + nf, n))
    rd[4] = 2e-5
    return pos, rd, rng.integers(1, 1 << 30, n, dtype=np.int32)


def level(nf):
    return W.config1(n=10, steps=1) if nf == 1 else W.config2(n=10, steps=1, ncells=(32, 16, 16), box=(16, 16, 16))


def records(pos, rd, ids):
    rec = np.empty((ids.size, 4 + rd.shape[0]))
    rec[:, :3], rec[:, 3:-1] = pos.T, rd.T
    tail = rec.view(np.int32)
    tail[:, -2], tail[:, -1] = ids, 7  # cpu: not kept
    return rec


def particles(layout, where, n, arrays):
    """pmp_particles over numpy arrays or (address, row bytes) of device memory"""
    p = capi.Particles()
    p.layout, p.where, p.n = layout, where, n
    if layout == capi.PMP_LAYOUT_AOS:
        p.aos = arrays[0]
    else:
        pos, rd, ids, nr = arrays
        for d in range(3):
            p.pos[d] = pos + 8 * n * d
        for r in range(nr):
            p.rdata[r] = rd + 8 * n * r
        p.id = ids
    return p


class Buffers:
    """The droplets' arrays in host or device memory, `shift` bytes past the start of a buffer."""

    def __init__(self, where, layout, n, nf, shift=0, data=None):
        import torch
        self.where, self.layout, self.n, self.nf, self.shift = where, layout, n, nf, shift
        nw = (4 + 10 + nf) * 8 * n
        dev = "cuda" if where == capi.PMP_WHERE_DEVICE else "cpu"
        self.t = torch.zeros(nw + 64, dtype=torch.uint8, device=dev)
        if data is not None:
            raw = b"".join(np.ascontiguousarray(a).tobytes() for a in data)
            if raw:
                self.t[shift:shift + len(raw)] = torch.frombuffer(bytearray(raw), dtype=torch.uint8).to(dev)

    def struct(self):
        a = self.t.data_ptr() + self.shift
        nr = 10 + self.nf
        if self.layout == capi.PMP_LAYOUT_AOS:
            return particles(self.layout, self.where, self.n, (a,))
        return particles(self.layout, self.where, self.n, (a, a + 24 * self.n, a + 8 * (3 + nr) * self.n, nr))

    def read(self):
        raw = self.t.cpu().numpy()[self.shift:].tobytes()
        n, nr = self.n, 10 + self.nf
        if self.layout == capi.PMP_LAYOUT_AOS:
            rec = np.frombuffer(raw[:8 * (4 + nr) * n]).reshape(n, 4 + nr)
            tail = rec.view(np.int32)
            assert np.all(tail[:, -1] == 0)
            return rec[:, :3].T, rec[:, 3:-1].T, tail[:, -2]
        d = np.frombuffer(raw[:8 * (3 + nr) * n]).reshape(3 + nr, n)
        return d[:3], d[3:], np.frombuffer(raw[8 * (3 + nr) * n:8 * (3 + nr) * n + 4 * n], dtype=np.int32)


def hand_over(sp, box, layout, where, nf, dr, shift=0):
    data = (records(*dr),) if layout == capi.PMP_LAYOUT_AOS else dr
    b = Buffers(where, layout, dr[2].size, nf, shift, data)
    rc = spray.lib().pmp_spray_set_particles(sp._h, box, C.byref(b.struct()))
    assert rc == capi.PMP_OK
    b.t.fill_(255)  # the library holds its own copy once the call returned


def check_box(sp, box, dr, nf, layout, where, shift=0):
    b = Buffers(where, layout, dr[2].size, nf, shift)
    rc = spray.lib().pmp_spray_get_particles(sp._h, box, C.byref(b.struct()))
    assert rc == capi.PMP_OK
    for got, want in zip(b.read(), dr):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("nf", [1, 2])
@pytest.mark.parametrize("layout", [capi.PMP_LAYOUT_AOS, capi.PMP_LAYOUT_SOA])
@pytest.mark.parametrize("where,shift", [(capi.PMP_WHERE_DEVICE, 0), (capi.PMP_WHERE_DEVICE, 8),
                                         (capi.PMP_WHERE_DEVICE, 4), (capi.PMP_WHERE_HOST, 0)])
def test_round_trip(nf, layout, where, shift):
    prob = level(nf)
    rng = np.random.default_rng(11)
    sp = from_problem(prob, set_droplets=False)
    nb = len(prob.boxes)
    for n in (1, 127, 128, 129, 1000, 3):
        drs = []
        for b, (lo, hi) in enumerate(prob.boxes):
            drs.append(droplets(rng, 0 if n == 3 and b else n + 17 * b, nf, lo, hi, prob.dx[0]))
            hand_over(sp, b, layout, where, nf, drs[b], shift)
        for b in range(nb):
            check_box(sp, b, drs[b], nf, layout, where, shift)  # still staged
        sp.est_timestep(0.5)  # packs
        for b in range(nb):
            check_box(sp, b, drs[b], nf, layout, where, shift)
        # one box again, then twice more before anything packs
        for m in (5, n + 40, 2):
            drs[-1] = droplets(rng, m, nf, *prob.boxes[-1], prob.dx[0])
            hand_over(sp, nb - 1, layout, where, nf, drs[-1], shift)
        for b in range(nb):
            check_box(sp, b, drs[b], nf, layout, where, shift)
        sp.est_timestep(0.5)
        for b in range(nb):
            check_box(sp, b, drs[b], nf, layout, where, shift)


def test_packed_order_is_stable_by_cell():
    prob = level(2)
    rng = np.random.default_rng(2)
    sp = from_problem(prob, set_droplets=False)
    drs = [droplets(rng, 5000 + b, 2, lo, hi, prob.dx[0]) for b, (lo, hi) in enumerate(prob.boxes)]
    for b, d in enumerate(drs):
        sp.set_particles(b, *d)
    sp.redistribute()  # nothing moved: each box in its packed order
    for b, (d, (lo, hi)) in enumerate(zip(drs, prob.boxes)):
        c = np.floor(d[0] * (1.0 / prob.dx)[:, None]).astype(np.int64) - np.asarray(lo)[:, None]
        order = np.argsort((c[2] * 16 + c[1]) * 16 + c[0], kind="stable")
        got = sp.get_particles(b)
        assert np.array_equal(got["id"], d[2][order]) and np.array_equal(got["rdata"], d[1][:, order])


@pytest.mark.parametrize("counts,crowd,again", [
    ((2048, 2048), 0, None),  # as many as one launch sorts
    ((2048, 2049), 0, None),  # one more, the first box too few to expect it
    ((2049, 2048), 0, None),  # counted
    ((2049, 0), 0, None),  # counted, and too few of them in the end
    ((40000, 1), 0, None),
    ((9000, 3000), 64, None),  # the fullest cell that is sorted by counting
    ((9000, 3000), 65, None),
    ((9000, 3000), 9000, None),  # one cell holds a box
    ((100, 9000), 0, None),  # staging rows exchanged with ranks in them
    ((3000, 5000), 0, (0, 4000)),  # rows given up
    ((3000, 5000), 0, (1, 4000)),  # rows given up at the end
    ((200000, 150000), 0, None),  # a CTA's cells hold more than its tile
])
def test_sorted_by_cell_and_stable(counts, crowd, again):
    """Packed, then re-binned: by new box, then by cell, in the order handed over.  Droplets lie in
    either box and are dead or alive."""
    prob = level(2)
    rng = np.random.default_rng(5)
    sp = from_problem(prob, set_droplets=False)
    dx = prob.dx[0]
    (lo, _), (_, hi) = prob.boxes
    drs = [droplets(rng, n, 2, lo, hi, dx) for n in counts]
    if crowd:
        # one cell with `crowd` droplets of box 0, and no others
        pos = drs[0][0]
        cell = np.floor(pos / dx).astype(int)
        pos[0, np.all(cell == [[3], [4], [5]], axis=0)] += dx
        pos[:, rng.permutation(counts[0])[:crowd]] = (np.array([[3], [4], [5]]) + rng.random((3, crowd))) * dx
        if crowd < counts[0]:
            cell = np.floor(drs[1][0] / dx).astype(int)
            drs[1][0][0, np.all(cell == [[3], [4], [5]], axis=0)] += dx
    for d in drs:
        if d[2].size > 1:
            d[2][rng.random(d[2].size) < 0.1] *= -1
    for _ in range(2):
        for b, d in enumerate(drs):
            sp.set_particles(b, *d)
        if again:
            drs[again[0]] = droplets(rng, again[1], 2, lo, hi, dx)
            sp.set_particles(again[0], *drs[again[0]])
        sp.est_timestep(0.5)
        for b, d in enumerate(drs):
            got = sp.get_particles(b)
            assert np.array_equal(got["id"], d[2]) and np.array_equal(got["rdata"], d[1])
        pos, rd = (np.concatenate([d[i] for d in drs], axis=1) for i in (0, 1))
        ids = np.concatenate([d[2] for d in drs])
        c = np.floor(pos * (1.0 / prob.dx)[:, None]).astype(np.int64)
        key = ((c[0] // 16 * 16 + c[2]) * 16 + c[1]) * 16 + c[0] % 16
        key[ids <= 0] = 1 << 20
        order = np.argsort(key, kind="stable")[:np.count_nonzero(ids > 0)]
        assert sp.redistribute() == np.count_nonzero(ids <= 0)
        split = np.count_nonzero(key[order] < 4096)
        for b, sel in enumerate((order[:split], order[split:])):
            got = sp.get_particles(b)
            assert np.array_equal(got["id"], ids[sel]) and np.array_equal(got["rdata"], rd[:, sel])


def test_refused():
    prob = level(1)
    sp = from_problem(prob, set_droplets=False)
    L, h = spray.lib(), sp._h
    p = capi.Particles()
    p.n, p.where = 4, capi.PMP_WHERE_DEVICE
    for layout in (capi.PMP_LAYOUT_AOS, capi.PMP_LAYOUT_SOA, 5):
        p.layout = layout  # no arrays
        assert L.pmp_spray_set_particles(h, 0, C.byref(p)) != capi.PMP_OK
    with pytest.raises(spray.SprayError):
        sp.est_timestep(0.5)  # the box has no droplets yet
    sp.set_particles(0, *droplets(np.random.default_rng(0), 4, 1, *prob.boxes[0], prob.dx[0]))
    p.layout, p.n = capi.PMP_LAYOUT_SOA, 3
    assert L.pmp_spray_get_particles(h, 0, C.byref(p)) == capi.PMP_ERR_INVALID  # another count


def test_wide_keys():
    """Boxes whose cells and count need more than 31 key bits together (64-bit keys)."""
    prob = level(1)
    n = 512
    prob.boxes = [((n * i, 0, 0), (n * i + n - 1, n - 1, n - 1)) for i in range(20)]
    prob.domain_hi = (20 * n - 1, n - 1, n - 1)
    prob.phi = prob.dx * np.array([20 * n, n, n])
    sp = from_problem(prob, set_droplets=False)
    rng = np.random.default_rng(8)
    drs = [droplets(rng, 300 + b, 1, lo, hi, prob.dx[0]) for b, (lo, hi) in enumerate(prob.boxes)]
    for b, d in enumerate(drs):
        sp.set_particles(b, *d)
    sp.est_timestep(0.5)
    drs[3] = droplets(rng, 50, 1, *prob.boxes[3], prob.dx[0])
    sp.set_particles(3, *drs[3])  # the others keep their order
    v = np.concatenate([d[1][:3] for d in drs], axis=1)
    assert sp.est_timestep(0.5) == np.min(0.5 / np.max(np.abs(v) * (1.0 / prob.dx)[:, None], axis=0))
    for b, d in enumerate(drs):
        check_box(sp, b, d, 1, capi.PMP_LAYOUT_SOA, capi.PMP_WHERE_DEVICE)
