"""Register caps of the FP64 update over the handle's own map (grid, 128
threads): 128 is the default, 96 another kernel with the same results, and an
autotuner's file of earlier kernels is not read back."""
import numpy as np
import pytest

from pelemp_b200 import capi
from pelemp_b200 import workloads as W
from pelemp_b200.spray import from_problem
from tests.gpu_util import assert_bitwise, device_sources, device_state, gpu_run, host_run
from tests.test_gpu_batched import close_sources, small_config3

pytestmark = pytest.mark.gpu


def kernels_of(call):
    """Names of the update kernels that a call launches (the profiler now and then misses a short call)."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    for _ in range(5):
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            call()
            torch.cuda.synchronize()
        names = [e.key for e in prof.key_averages() if "spray_update_fp64" in e.key]
        if names:
            return names
    pytest.skip("no kernel records from the profiler")


def update_kernels(prob, setup):
    import torch
    sp = from_problem(prob)
    setup(sp)
    st_keep, st_v = device_state(prob)
    src, src_v = device_sources(prob)

    def update():
        sp.update_particles(st_v, src_v, prob.flow_dt, 0.0, prob.state_ghosts, prob.source_ghosts, 0, 0, 0,
                            prob.spray_cfl_lev, torch.cuda.current_stream().cuda_stream)

    update()
    names = kernels_of(update)
    cfg = sp.launch()
    del st_keep
    sp.close()
    return names, (cfg.kind, cfg.block, cfg.regs)


def test_cap_of_96_is_a_kernel_of_its_own():
    prob = small_config3(30_000)
    default, cfg = update_kernels(prob, lambda sp: None)
    again, _ = update_kernels(prob, lambda sp: sp.set_launch())
    low, cfg96 = update_kernels(prob, lambda sp: sp.set_launch(regs=96))
    assert cfg == (capi.PMP_LAUNCH_GRID, 128, 128) and cfg96 == (capi.PMP_LAUNCH_GRID, 128, 96)
    assert len(default) == 1 and again == default and len(low) == 1 and low != default


@pytest.mark.parametrize("run", [gpu_run, host_run])
def test_results_of_both_caps(run):
    prob = small_config3(60_000)
    p0, s0, _ = run(prob, prob.steps)
    p1, s1, _ = run(prob, prob.steps, setup=lambda sp: sp.set_launch(regs=96))
    assert_bitwise(p1, p0)
    close_sources(s1, s0)


def test_cache_of_earlier_kernels_is_not_read(tmp_path):
    prob = W.config1(n=20_000, steps=1)
    cache = tmp_path / "tune.txt"
    st_keep, st_v = device_state(prob)
    src, src_v = device_sources(prob)

    def tune():
        sp = from_problem(prob)
        rep = sp.autotune(st_v, src_v, prob.flow_dt, prob.state_ghosts, prob.source_ghosts, 0, 0, prob.spray_cfl_lev,
                          cache_path=str(cache))
        sp.close()
        return rep.cached

    assert tune() == 0 and tune() == 1
    key, times = cache.read_text().splitlines()[-1].split("\t")
    head, rev = key.rsplit("|rev=", 1)
    for old in (head, head + "|rev=%d" % (int(rev) - 1)):
        cache.write_text(old + "\t" + times + "\n")
        assert tune() == 0
    del st_keep
