"""A wait between the CTAs of an instance that runs out (about 1 s, through
cuopo_batch_hold, which keeps an instance's first CTA from ever seeing an
exchange complete): the instance ends with flag 4, the CTAs that ran it take
no other one, and what they have not taken is as it was, so that the next step
finishes it with the results of an undisturbed run."""
import numpy as np
import pytest

import cuopo_b200 as cu
from cuopo_b200._lib import check, load
from tests.helpers import params_2eq, params_3eq

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def signal(b, dtype):
    out = np.zeros(b.total, dtype)
    b.get_signal(out)
    torch.cuda.synchronize()
    return out.reshape(b.count, -1)


# the last two: more instances than clusters are resident, so that some are left when every cluster has given up
@pytest.mark.parametrize("neq,n_t,prec,count,some_left", [(2, 8192, cu.F32, 12, False), (3, 16384, cu.F64, 20, True),
                                                          (2, 16384, cu.F64, 40, True)])
def test_a_wait_that_runs_out_ends_its_instance_only(neq, n_t, prec, count, some_left):
    p = (params_2eq if neq == 2 else params_3eq)(n_t=n_t, n_z=3, regime=cu.CW)
    rng = np.random.default_rng(count)
    insts = [dict(n_t=n_t, ap0=p.ap0, Rs=0.97, delta=0.01 * k, gdd=1e-4, seed=0) for k in range(count)]
    dtype = np.complex64 if prec == cu.F32 else np.complex128
    start = (0.3 * (rng.standard_normal((count, n_t)) + 1j * rng.standard_normal((count, n_t)))).astype(dtype)
    with cu.Batch(p, insts, precision=prec) as ref, cu.Batch(p, insts, precision=prec) as b:
        ref.set_signal(start.reshape(-1))
        ref.run(4, 0.0)
        ps_ref, _, flags_ref = ref.results()
        assert (flags_ref == 2).all()
        want = signal(ref, dtype)
        b.set_signal(start.reshape(-1))
        b.reset()
        check(load().cuopo_batch_hold(b._h, 1))
        b.step(4, 4, 0.0)
        _, rts, flags = b.results()
        gone, left = flags == 4, flags == 0
        assert (gone | left).all() and gone.any() and left.any() == some_left, flags
        assert (rts[gone] == 1).all() and (rts[left] == 0).all()
        assert np.array_equal(signal(b, dtype)[left], start[left])
        assert b.pending() == left.sum()
        check(load().cuopo_batch_hold(b._h, 0))
        b.step(4, 4, 0.0)
        ps, rts, flags = b.results()
        assert (flags[gone] == 4).all() and (flags[left] == 2).all() and (rts[left] == 4).all()
        assert np.array_equal(ps[left], ps_ref[left])
        assert np.array_equal(signal(b, dtype)[left], want[left])
