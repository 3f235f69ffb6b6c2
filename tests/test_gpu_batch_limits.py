"""A step whose round-trip limit lies at or below what the instances have
already run: none has a round trip left, so each ends with flag 2, its
round trips and power as they were and its fields untouched.  The kernels
reach the end of such an instance without a round trip's barriers in between:
every CTA and warp must have read the instance's state before the leader
writes it, on each kind of layout (one CTA, a cluster, an instance spread over
a cluster)."""
import numpy as np
import pytest

import cuopo_b200 as cu
from tests.helpers import params_2eq, params_3eq

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def signal(b, dtype):
    out = np.zeros(b.total, dtype)
    b.get_signal(out)
    torch.cuda.synchronize()
    return out


# instances: spread over a cluster, a few CTAs each, one CTA (or the decomposition's cluster) each
@pytest.mark.parametrize("neq,n_t,prec,count", [
    (2, 512, cu.F32, 1), (2, 4096, cu.F32, 1), (2, 4096, cu.F32, 25), (2, 4096, cu.F32, 140), (2, 4096, cu.F32, 310),
    (2, 8192, cu.F32, 1), (2, 8192, cu.F32, 70), (2, 16384, cu.F32, 40), (2, 32768, cu.F32, 3),
    (2, 32768, cu.F32, 25), (2, 65536, cu.F32, 2), (3, 512, cu.F32, 900), (3, 65536, cu.F32, 2),
    (3, 4096, cu.F32, 200), (2, 4096, cu.F64, 150), (2, 16384, cu.F64, 20), (3, 16384, cu.F64, 2)])
@pytest.mark.parametrize("limit", [1, 2])
def test_step_below_the_round_trips_already_run(neq, n_t, prec, count, limit):
    p = (params_2eq if neq == 2 else params_3eq)(n_t=n_t, n_z=2, regime=cu.CW)
    dtype = np.complex64 if prec == cu.F32 else np.complex128
    rng = np.random.default_rng(count)
    start = (0.3 * (rng.standard_normal(n_t) + 1j * rng.standard_normal(n_t))).astype(dtype)
    insts = [dict(n_t=n_t, ap0=p.ap0, Rs=0.97, delta=0.05, gdd=0.0, seed=0)] * count
    with cu.Batch(p, insts, precision=prec) as b:
        b.set_signal(np.tile(start, count))
        b.reset()
        b.step(2, 10, 0.0)
        ps0, rts0, flags0 = b.results()
        assert (rts0 == 2).all() and (flags0 == 0).all()
        before = signal(b, dtype)
        b.step(5, limit, 0.0)
        ps, rts, flags = b.results()
        assert (flags == 2).all() and (rts == 2).all() and np.array_equal(ps, ps0)
        assert np.array_equal(signal(b, dtype), before)
        assert b.pending() == 0
