"""The autotuner against the layout choice: what it times is what a batch of
that many instances runs, and its choice, made for that many, does not take
the layouts that spread an instance over the chip from single plans."""
import pytest

import cuopo_b200 as cu
from cuopo_b200 import sweep

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(autouse=True)
def _reset():
    cu.autotune_reset()
    yield
    cu.autotune_reset()


def base_for(n_t):
    return cu.derive_params(sweep.cw_base_inputs(n_t=n_t, n_z=20, n_thr=3.0, r_percent=95.0))[0]


@pytest.mark.parametrize("n_t,count", [(8192, 6), (16384, 6), (32768, 4)])
def test_tuned_time_is_that_of_a_batch(n_t, count):
    """A few instances run spread over 16 CTAs, at half the time of the general
    kernels or less; the tuner's time must be near the batch's (within 30 %)."""
    p, n_rt = base_for(n_t), 40
    insts = [dict(n_t=n_t, ap0=p.ap0, Rs=p.Rs, delta=p.delta, gdd=p.gdd, seed=k) for k in range(count)]
    with cu.Batch(p, insts) as b:
        b.seed_noise(1e-15)
        times = []
        for _ in range(3):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            b.reset()
            e0.record()
            b.step(n_rt, n_rt, 0.0)
            b.wait()
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
    r = cu.autotune(p, cu.F32, count=count, n_rt=n_rt)
    assert 0 < r["ms"] < 1.3 * min(times), (r, times)


@pytest.mark.parametrize("n_t", [8192, 16384, 32768])
def test_plans_keep_their_layout(n_t):
    p = base_for(n_t)
    with cu.Plan(p) as plan:
        alone = plan.config
    default = cu.kernel_config(n_t)
    r = cu.autotune(p, cu.F32, count=120, n_rt=1)
    with cu.Plan(p) as plan:
        assert plan.config == alone, r
    # a choice made by hand holds for plans as well
    m, cl = {8192: (8192, 1), 16384: (8192, 2), 32768: (8192, 4)}[n_t]
    cu.kernel_select(n_t, m, cl)
    with cu.Plan(p) as plan:
        assert (plan.config.cluster, plan.config.threads) == (cl, m // 16)
    cu.kernel_select(n_t, *default)
    with cu.Plan(p) as plan:
        assert plan.config == alone
