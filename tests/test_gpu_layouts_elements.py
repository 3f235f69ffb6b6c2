"""Layouts of one arithmetic with the cavity elements that a CW signal alone
does not show: nanosecond pump windows, the modulator on signal and idler,
and the seeded idler.  Batches of one and of many instances run
on different layouts; instance for instance the signals and power histories
must be equal bit for bit.  From the second round trip on the signal depends
on the pump window's place, the idler and its modulator."""
import numpy as np
import pytest

import cuopo_b200 as cu

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def inputs(neq, n_t, regime, n_rt=3, eom=1):
    if neq == 2:
        return cu.default_inputs(crystal=cu.PPLN, n_eqs=2, regime=regime, n_t=n_t, n_z=3, n_rt=n_rt, lp_nm=532.0,
                                 lambda_um=6.970206862971646, n_thr=4.0, r_percent=98.0, delta=0.05, gdd_percent=40.0,
                                 lcr_mm=5.0, use_eom=eom, mod_depth_pi=0.6, freq_det_mhz=4.0)
    return cu.default_inputs(crystal=cu.SPPLT, n_eqs=3, regime=regime, n_t=n_t, n_z=3, n_rt=n_rt, lp_nm=532.0,
                             ls_nm=1550.0, lambda_um=8.719670871908674, n_thr=3.0, r_percent=98.0, delta=0.05,
                             gdd_percent=40.0, lcr_mm=20.0, use_eom=eom, mod_depth_pi=0.6, freq_det_mhz=4.0)


def signals(b):
    out = np.zeros(b.total, np.complex64)
    b.get_signal(out)
    torch.cuda.synchronize()
    offs = np.concatenate([[0], np.cumsum(b.n_t)])
    return [out[offs[k]:offs[k + 1]] for k in range(b.count)]


@pytest.mark.parametrize("neq,n_t,regime,count", [
    (3, 512, cu.NS, 300), (3, 2048, cu.NS, 40), (3, 4096, cu.NS, 40), (3, 4096, cu.NS, 160), (3, 8192, cu.NS, 20),
    (3, 16384, cu.NS, 12), (2, 1024, cu.NS, 160), (2, 4096, cu.NS, 30), (2, 4096, cu.CW, 150), (2, 8192, cu.CW, 40),
    (2, 32768, cu.NS, 9)])
def test_elements_do_not_depend_on_the_number_of_instances(neq, n_t, regime, count):
    inp, n_rt = inputs(neq, n_t, regime), 3
    with cu.Batch(None, [inp], seeds=[7]) as b:
        b.seed_noise(0.1)
        b.run(n_rt, 0.0)
        want, (ps, _, _) = signals(b)[0], b.results()
        hist = b.history(0, n_rt) if regime == cu.NS else None
    assert np.isfinite(ps[0]) and ps[0] > 0
    with cu.Batch(None, [inp] * count, seeds=[7] * count) as b:
        b.seed_noise(0.1)
        b.run(n_rt, 0.0)
        got, (psm, _, _) = signals(b), b.results()
        assert all(np.array_equal(g, want) for g in got) and (psm == ps[0]).all()
        if hist is not None:
            assert np.array_equal(b.history(count - 1, n_rt), hist)


def test_batch_noise_of_two_fields_and_of_mixed_batches():
    """Instances with two fields have no idler stream, alone (the idler buffer is absent) or beside instances with
    three; the idler of those is stream 1: a round trip from it equals the plan's from host-seeded fields."""
    ins = [inputs(2, 512, cu.CW, eom=0), inputs(3, 1024, cu.CW, eom=0), inputs(2, 2048, cu.CW, eom=0),
           inputs(3, 512, cu.CW, eom=0)]
    seeds = [5, 2 ** 35 + 1, 2 ** 64 - 2, 9]
    for sel in ([0, 2], [0, 1, 2, 3]):
        with cu.Batch(None, [ins[k] for k in sel], seeds=[seeds[k] for k in sel]) as b:
            b.seed_noise(1e-2)
            for k, s in zip(sel, signals(b)):
                assert np.array_equal(s, cu.noise_host(ins[k].n_t, 1e-2, seeds[k], 0)), k
            b.run(1, 0.0)
            after = dict(zip(sel, signals(b)))
        for k in sel:
            p, _ = cu.derive_params(ins[k])
            f = [torch.zeros(p.n_t, dtype=torch.complex64, device="cuda"),
                 torch.from_numpy(cu.noise_host(p.n_t, 1e-2, seeds[k], 0).copy()).cuda(),
                 torch.from_numpy(cu.noise_host(p.n_t, 1e-2, seeds[k], 1).copy()).cuda() if p.n_eqs == 3 else None]
            with cu.Plan(p) as plan:
                plan.round_trips(*f, None, 0, 0, 1)
                torch.cuda.synchronize()
            assert np.array_equal(f[1].cpu().numpy(), after[k]), k
