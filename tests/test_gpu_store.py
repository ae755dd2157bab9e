"""The droplet store (pmp_store.cu) where a call's own kernels, another stream
or memory could be in its way: droplets handed over and packed on streams that
do not order one another."""
import ctypes as C

import numpy as np
import pytest

from pelemp_b200 import capi, spray
from pelemp_b200 import workloads as W
from pelemp_b200.spray import from_problem
from tests.gpu_util import assert_bitwise, device_sources, device_state, gpu_run
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


@pytest.mark.parametrize("mode", [capi.PMP_MODE_FP64, capi.PMP_MODE_MIXED])
def test_update_after_a_refused_one_on_another_stream(mode):
    """An update is refused after it packed the droplets on a held stream; the next one runs on another."""
    import torch
    prob = W.config2(n=20_000, steps=1, ncells=(32, 16, 16), box=(16, 16, 16))
    want, _, ref = gpu_run(prob, 1, mode=mode)
    sp = from_problem(prob, mode=mode)
    st_keep, st_v = device_state(prob)
    held, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(held):
        torch.cuda._sleep(HOLD)
    for do_move in (1, 0):
        src, src_v = device_sources(prob)
        torch.cuda.current_stream().synchronize()
        if do_move:
            with pytest.raises(spray.SprayError):  # the views do not cover this many ghost cells
                sp.update_particles(st_v, src_v, prob.flow_dt, 0.0, prob.state_ghosts + 1, prob.source_ghosts, 0, 0,
                                    1, prob.spray_cfl_lev, held.cuda_stream)
        sp.update_particles(st_v, src_v, prob.flow_dt, 0.0, prob.state_ghosts, prob.source_ghosts, 0, 0, do_move,
                            prob.spray_cfl_lev, other.cuda_stream)
    assert_bitwise([sp.get_particles(b) for b in range(len(prob.boxes))], want)
    del st_keep, ref


def fail_alloc(sp, k):
    assert spray.lib().pmp_spray_debug_fail_alloc(sp._h, k) == capi.PMP_OK


def by_cell(prob, drs):
    """The droplets of `drs` by new box, then by cell, in their order (boxes of 16^3 cells along x)."""
    pos, rd, ids = (np.concatenate([d[i] for d in drs], axis=-1) for i in range(3))
    c = np.floor(pos * (1.0 / prob.dx)[:, None]).astype(np.int64)
    key = ((c[0] // 16 * 16 + c[2]) * 16 + c[1]) * 16 + c[0] % 16
    order = np.argsort(key, kind="stable")
    return [(pos[:, o], rd[:, o], ids[o]) for o in (order[key[order] // 4096 == b] for b in range(len(prob.boxes)))]


@pytest.mark.parametrize("n", [100, 60_000])
@pytest.mark.parametrize("call", ["set", "pack", "redistribute"])
def test_allocation_fails(call, n):
    """Each allocation of a call fails in turn, on a held stream: the call succeeds without it or reports
    an error, and after that the droplets are handed over again, packed and re-binned as if nothing had
    happened."""
    import torch
    prob = level(2)
    (lo, _), (_, hi) = prob.boxes
    side = torch.cuda.Stream()
    failed = 0
    for k in range(1, 12):
        rng = np.random.default_rng(k)
        sp = from_problem(prob, set_droplets=False)
        # box 0 is given droplets of both boxes, so that re-binning changes the boxes' counts
        drs = [droplets(rng, n, 2, lo, hi, prob.dx[0]), droplets(rng, 0, 2, lo, hi, prob.dx[0])]
        if call == "set":
            fail_alloc(sp, k)
        try:
            for b, d in enumerate(drs):
                sp.set_particles(b, *d)
        except spray.SprayError:
            failed += 1
            fail_alloc(sp, 0)
            for b, d in enumerate(drs):
                sp.set_particles(b, *d)
        fail_alloc(sp, k if call == "pack" else 0)
        if call == "pack":
            with torch.cuda.stream(side):
                torch.cuda._sleep(HOLD // 10)
            try:
                sp.est_timestep(0.5, stream=side.cuda_stream)
            except spray.SprayError:
                failed += 1
                fail_alloc(sp, 0)
                drs[0] = droplets(rng, n, 2, lo, hi, prob.dx[0])
                sp.set_particles(0, *drs[0])
        check(sp, drs)
        if call == "redistribute":
            sp.est_timestep(0.5)
        fail_alloc(sp, k if call == "redistribute" else 0)
        try:
            sp.redistribute(stream=side.cuda_stream)
        except spray.SprayError:
            assert call == "redistribute"
            failed += 1
            fail_alloc(sp, 0)
            assert sp.est_timestep(0.5) == expected_dt(prob, drs)
            sp.redistribute()
        fail_alloc(sp, 0)
        check(sp, by_cell(prob, drs))
        assert sp.est_timestep(0.5, stream=side.cuda_stream) == expected_dt(prob, drs)
        sp.close()
    assert failed > 0


def on_device(d):
    import torch
    return tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in d)


@pytest.mark.parametrize("call,k,counts", [
    ("set", 3, (60_000, 40)),  # the counts, after the rows and their keys
    ("pack", 3, (60_000, 40)),  # the passes' arrays, after the store and the caller's indices
    ("redistribute", 1, (40, 60_000)),  # not counted before: the passes' arrays,
    ("redistribute", 2, (40, 60_000)),  # the counts
])
def test_no_memory_to_count_with(call, k, counts):
    """The sort by counting is a choice: a call for whose counts or passes there is no memory sorts
    without them."""
    prob = level(2)
    rng = np.random.default_rng(1)
    drs = [droplets(rng, n, 2, lo, hi, prob.dx[0]) for n, (lo, hi) in zip(counts, prob.boxes)]
    sp = from_problem(prob, set_droplets=False)
    for _ in range(2):
        fail_alloc(sp, k if call == "set" else 0)
        for b, d in enumerate(drs):
            sp.set_particles(b, *on_device(d))
        fail_alloc(sp, k if call == "pack" else 0)
        assert sp.est_timestep(0.5) == expected_dt(prob, drs)
        check(sp, drs)
        fail_alloc(sp, k if call == "redistribute" else 0)
        assert sp.redistribute() == 0
        check(sp, by_cell(prob, drs))


def held_mib():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # what earlier tests left to torch
    free, total = torch.cuda.mem_get_info()
    return (total - free) / 2**20


def boxes_of(side, nb):
    """A level of nb[0] x nb[1] x nb[2] boxes of side^3 cells, one fuel, without droplets."""
    prob = W.config1(n=10, steps=1)
    prob.boxes = [(tuple(side * c for c in (i, j, k)), tuple(side * c + side - 1 for c in (i, j, k)))
                  for k in range(nb[2]) for j in range(nb[1]) for i in range(nb[0])]
    prob.domain_hi = tuple(side * n - 1 for n in nb)
    prob.phi = prob.dx * side * np.array(nb)
    return prob


def test_memory_of_a_dense_first_box():
    """Droplets nearly all in the first of many large boxes.  What 326k droplets need: rows and keys
    (136 bytes, for up to twice as many), store, indices and lists (120 + 24), a sort (under 64):
    155 MB; a cell counted for each place of 512 padded boxes: 1 GB."""
    prob = boxes_of(64, (8, 8, 8))
    rng = np.random.default_rng(6)
    counts = [300_000] + [50] * 511
    drs = [droplets(rng, n, 1, lo, hi, prob.dx[0]) for n, (lo, hi) in zip(counts, prob.boxes)]
    sp = from_problem(prob, set_droplets=False)
    for b, d in enumerate(drs):
        sp.set_particles(b, *on_device((d[0][:, :1], d[1][:, :1], d[2][:1])))
    sp.est_timestep(0.5)  # the kernels are loaded
    sp.close()
    sp = from_problem(prob, set_droplets=False)
    before = held_mib()
    dev = [on_device(d) for d in drs]
    own = held_mib() - before
    for _ in range(3):
        for b, d in enumerate(dev):
            sp.set_particles(b, *d)
        assert sp.est_timestep(0.5) == expected_dt(prob, drs)
        assert held_mib() - before - own < 300
        sp.set_grids(prob.boxes)


def store_counts(sp):
    """(allocations of the store, sorts by counting) so far"""
    a, s = C.c_longlong(), C.c_longlong()
    assert spray.lib().pmp_spray_debug_store(sp._h, C.byref(a), C.byref(s)) == capi.PMP_OK
    return a.value, s.value


def allocs(sp):
    return store_counts(sp)[0]


def cell_sorts(sp, call):
    """Sorts by counting that a call runs."""
    before = store_counts(sp)[1]
    call()
    return store_counts(sp)[1] - before


def test_crowded_cells_are_not_counted_again():
    """A level with an injector: a third of the droplets in two cells for 20 passes, then spread, then
    crowded again.  The order is right every time; a sort that follows a crowded one does not count, and
    once the droplets have spread counting comes back."""
    prob = level(2)
    rng = np.random.default_rng(9)
    n = 9000
    sp = from_problem(prob, set_droplets=False)
    counted = []
    for i in range(60):
        drs = [droplets(rng, n, 2, lo, hi, prob.dx[0]) for lo, hi in prob.boxes]
        if i < 20 or i >= 50:
            drs[0][0][:, :n // 3] = (np.array([[3], [4], [5]]) + rng.random((3, n // 3))) * prob.dx[0]
            drs[0][0][0, :n // 6] += 4 * prob.dx[0]
        sp.set_grids(prob.boxes)
        for b, d in enumerate(drs):
            sp.set_particles(b, *d)
        counted.append((cell_sorts(sp, lambda: sp.est_timestep(0.5)), cell_sorts(sp, sp.redistribute)))
        check(sp, by_cell(prob, drs))
    # while two cells are crowded a packing never sorts by counting, and of the 16 sorts after a crowded one
    # at most the last tries (a re-binning finds out by running it); once spread, within 8 passes, all do
    assert all(c[0] == 0 for c in counted[:20] + counted[50:])
    assert sum(c[1] for c in counted[:20]) <= 2 and sum(c[1] for c in counted[50:]) <= 2
    assert all(c == (1, 1) for c in counted[28:50])


def test_memory_after_a_large_hand_over():
    """8M droplets, then 8000, by a handle that lives on.  What stays of the large one are buffers of up to
    256 MB each: the caller's indices, the update's list and the sort's arrays (8, 8 and under 32 bytes a
    droplet: 384 MB)."""
    import torch
    prob = boxes_of(64, (2, 2, 2))
    big = 1_000_000
    dx = prob.dx[0]
    lo = torch.tensor([b[0] for b in prob.boxes], device="cuda", dtype=torch.float64)
    pos = (torch.rand((3, big), device="cuda", dtype=torch.float64) * 64)
    rd = torch.rand((11, big), device="cuda", dtype=torch.float64)
    ids = torch.arange(1, big + 1, device="cuda", dtype=torch.int32)
    at = torch.empty_like(pos)
    sp = from_problem(prob, set_droplets=False)
    torch.cuda.synchronize()
    before = held_mib()
    held = []
    for n in (big, 1000, 1000, big):
        sp.set_grids(prob.boxes)
        for b in range(8):
            at.copy_((pos + lo[b][:, None]) * dx)
            sp.set_particles(b, at[:, :n].contiguous(), rd[:, :n].contiguous(), ids[:n].contiguous())
        assert sp.est_timestep(0.5) == float((0.5 / ((rd[:3, :n] * (1.0 / prob.dx[0])).amax(0))).min())
        held.append(held_mib() - before)
    print("MiB held after 8M, 8k, 8k, 8M droplets:", [round(v) for v in held])
    assert held[0] > 1500 and max(held[1:3]) < 512 and held[3] < held[0] + 64


def test_allocations_of_repeated_hand_overs():
    """64 boxes of 300 droplets: handed over, then again box by box without new grids, then with them.  A
    pass allocates a few buffers at most (rows and keys are exchanged as they double), then none."""
    prob = boxes_of(8, (4, 4, 4))
    rng = np.random.default_rng(2)
    drs = [droplets(rng, 300, 1, lo, hi, prob.dx[0]) for lo, hi in prob.boxes]
    dev = [on_device(d) for d in drs]
    sp = from_problem(prob, set_droplets=False)
    made = []
    for i in range(7):
        if i > 3:
            sp.set_grids(prob.boxes)
        before = allocs(sp)
        for b, d in enumerate(dev):
            sp.set_particles(b, *d)
        assert sp.est_timestep(0.5) == expected_dt(prob, drs)
        made.append(allocs(sp) - before)
    check(sp, drs)
    print("allocations of the passes:", made)
    # the first: 8 exchanges of two buffers, counts, and one each of store, indices, sort, map and list;
    # the second: two exchanges while the boxes give their rows up, and the sort's
    assert made[0] <= 22 and made[1] <= 6 and made[3:] == [0] * 4


@pytest.mark.parametrize("per_cell,staged,rebinned", [(12, True, True), (20, False, True), (30, False, False)])
def test_dense_levels_are_not_counted(per_cell, staged, rebinned):
    """Which sort a level of evenly dense cells takes, and that its order is right."""
    prob = level(2)
    rng = np.random.default_rng(per_cell)
    drs = [droplets(rng, per_cell * 4096, 2, lo, hi, prob.dx[0]) for lo, hi in prob.boxes]
    dev = [on_device(d) for d in drs]
    sp = from_problem(prob, set_droplets=False)
    for _ in range(2):
        sp.set_grids(prob.boxes)
        for b, d in enumerate(dev):
            sp.set_particles(b, *d)
        assert cell_sorts(sp, lambda: sp.est_timestep(0.5)) == staged
        assert cell_sorts(sp, sp.redistribute) == rebinned
        check(sp, by_cell(prob, drs))


@pytest.mark.parametrize("each", [17, 40, 64])
def test_dense_layer_is_counted(each):
    """Two layers of cells with up to 64 droplets each and none elsewhere: more in a block's 256 cells than
    its tile holds, counted all the same."""
    prob = level(2)
    rng = np.random.default_rng(each)
    drs = []
    for lo, hi in prob.boxes:
        pos, rd, ids = droplets(rng, 512 * each, 2, lo, hi, prob.dx[0])
        cell = rng.permutation(np.repeat(np.arange(512), each))
        pos = (np.stack([cell % 16 + lo[0], cell // 16 % 16, cell // 256]) + rng.random(pos.shape)) * prob.dx[0]
        drs.append((pos, rd, ids))
    dev = [on_device(d) for d in drs]
    sp = from_problem(prob, set_droplets=False)
    for b, d in enumerate(dev):
        sp.set_particles(b, *d)
    assert cell_sorts(sp, lambda: sp.est_timestep(0.5)) == 1 and cell_sorts(sp, sp.redistribute) == 1
    check(sp, by_cell(prob, drs))


@pytest.mark.parametrize("refused", [False, True])
def test_capture_after_an_update_on_another_stream(refused):
    """The droplets are packed by an update on one stream, which only the caller has waited for, and the
    next update is captured on another (captures in which calls that wait are not allowed)."""
    import torch
    prob = W.config2(n=20_000, steps=2, ncells=(32, 16, 16), box=(16, 16, 16))
    st_keep, st_v = device_state(prob)
    src, src_v = device_sources(prob)
    side = torch.cuda.Stream()

    def update(sp, do_move, stream, ghosts=prob.source_ghosts):
        sp.update_particles(st_v, src_v, prob.flow_dt, 0.0, prob.state_ghosts, ghosts, 0, 0, do_move,
                            prob.spray_cfl_lev, stream.cuda_stream, sync=False)

    warm = from_problem(prob)  # the buffers that an update keeps are the handle's own, the kernels are loaded
    update(warm, 0, side)
    want = from_problem(prob)
    for do_move in ((0, 1) if not refused else (1,)):
        update(want, do_move, side)
    want.sync()
    sp = from_problem(prob)
    update(sp, 0, side)
    sp.sync()
    for b, p in enumerate(prob.parts):
        sp.set_particles(b, p["pos"], p["rdata"], p["id"])
    torch.cuda.synchronize()
    if refused:
        with pytest.raises(spray.SprayError):  # the source views do not cover this many ghost cells
            update(sp, 0, side, prob.source_ghosts + 1)
    else:
        update(sp, 0, side)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        update(sp, 1, torch.cuda.current_stream())
    g.replay()
    torch.cuda.synchronize()
    sp.sync()
    assert_bitwise([sp.get_particles(b) for b in range(len(prob.boxes))],
                   [want.get_particles(b) for b in range(len(prob.boxes))])
    del g, st_keep
    warm.close()


@pytest.mark.parametrize("sizes", ["like", "growing", "shrinking"])
def test_rows_of_a_first_hand_over(sizes):
    """What a level's first hand-over takes for its staging rows: exactly the rows of like boxes, a quarter
    more at most than those of growing ones, exchanged a few times."""
    prob = boxes_of(32, (4, 2, 2))
    like = 60_000
    counts = {"like": [like] * 16, "growing": [8_000 * (b + 1) for b in range(16)],
              "shrinking": [8_000 * (16 - b) for b in range(16)]}[sizes]
    rng = np.random.default_rng(4)
    big = [on_device(d) for d in (droplets(rng, max(counts), 1, lo, hi, prob.dx[0]) for lo, hi in prob.boxes)]
    warm, _ = filled(boxes_of(32, (4, 2, 2)), [100] * 16, nf=1)
    warm.est_timestep(0.5)
    warm.close()
    sp = from_problem(prob, set_droplets=False)
    before, made = held_mib(), allocs(sp)
    for b, (d, n) in enumerate(zip(big, counts)):
        sp.set_particles(b, d[0][:, :n].contiguous(), d[1][:, :n].contiguous(), d[2][:n].contiguous())
    held, made = held_mib() - before, allocs(sp) - made
    need = 136 * sum(counts) / 2**20
    print("%s: %d allocations, %.0f MiB held for %.0f of rows and keys" % (sizes, made, held, need))
    # the counts (4 MB), and the driver's granules of 2 MB
    assert held < {"like": 1.02, "growing": 1.27, "shrinking": 2.02}[sizes] * need + 12 and made <= 15
