"""GDD round trips on the one-CTA kernels.  With the fields of an instance in
one CTA's shared memory no barrier lies between the element-wise pass before
the GDD step, where every warp reads the pass's staged coefficients, and the
GDD step itself, so the GDD step must not write them: a warp that reads late
would run the closing half step of that round trip without coupling.  Whether
a run shows such a write is up to the warps' timing; many instances and
many short round trips (2 slices and a GDD step each) give it the most chances.

Every instance of a batch and the same instance alone (on another layout of
the same arithmetic) must agree bit for bit."""
import numpy as np
import pytest

import cuopo_b200 as cu
from tests.helpers import params_2eq, params_3eq

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N_RT = 40


def run(p, start, prec, count):
    insts = [dict(n_t=p.n_t, ap0=p.ap0, Rs=0.97, delta=0.05, gdd=-2e-4, seed=0)] * count
    with cu.Batch(p, insts, precision=prec) as b:
        b.set_signal(np.tile(start, count))
        b.run(N_RT, 0.0)
        ps, rts, _ = b.results()
        out = np.zeros(b.total, start.dtype)
        b.get_signal(out)
        torch.cuda.synchronize()
    assert (rts == N_RT).all()
    return out.reshape(count, p.n_t), ps


@pytest.mark.parametrize("neq,n_t,prec,counts", [
    (2, 512, cu.F32, (600,)), (2, 1024, cu.F32, (600,)), (2, 2048, cu.F32, (290,)), (2, 4096, cu.F32, (140, 290)),
    (3, 512, cu.F32, (880,)), (3, 4096, cu.F32, (148, 290)),
    (2, 512, cu.F64, (1100,)), (2, 4096, cu.F64, (148,)), (3, 2048, cu.F64, (148,)), (3, 4096, cu.F64, (148,))])
def test_gdd_round_trips_of_every_instance_agree(neq, n_t, prec, counts):
    p = (params_2eq if neq == 2 else params_3eq)(n_t=n_t, n_z=2, regime=cu.CW)
    rng = np.random.default_rng(n_t + neq)
    start = 0.3 * (rng.standard_normal(n_t) + 1j * rng.standard_normal(n_t))
    start = start.astype(np.complex64 if prec == cu.F32 else np.complex128)
    ref, ps_ref = run(p, start, prec, 1)
    assert np.isfinite(ps_ref[0]) and ps_ref[0] > 0
    for count in counts:
        got, ps = run(p, start, prec, count)
        assert (got == ref[0]).all(), count
        assert (ps == ps_ref[0]).all(), count
