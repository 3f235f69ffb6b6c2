"""Layouts of one arithmetic: single instances and batches of any size run the
same operations on other thread and cluster layouts (up to 16 CTAs per
instance, four threads per 16-point transform, two instances per SM), chosen
by the number of instances.  The results must not depend on the choice: equal
bit for bit, and within the oracle's bounds (F64 1e-10, F32 5e-5 over round
trips, as for the other layouts).

Counts are chosen to cross every rung: one instance, one and two waves of the
16-CTA clusters, the 4-, 2- and 1-CTA layouts, one CTA per SM, two per SM."""
import numpy as np
import pytest

import cuopo_b200 as cu
from oracle import binding as ob
from tests.helpers import params_2eq, params_3eq, rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def run(neq, n_t, prec, count, n_rt=2):
    """count instances with equal starts and GDD on; instance 0's cavity and the last one's differ from the rest."""
    p = (params_2eq if neq == 2 else params_3eq)(n_t=n_t, n_z=3, regime=cu.CW, delta=0.05)
    insts = [dict(n_t=n_t, ap0=p.ap0, Rs=0.97, delta=0.05 if k else -0.1, gdd=-2e-4, seed=0) for k in range(count)]
    rng = np.random.default_rng(n_t + neq)
    s0 = 0.3 * (rng.standard_normal(n_t) + 1j * rng.standard_normal(n_t))
    s0 = s0.astype(np.complex64 if prec == cu.F32 else np.complex128)
    with cu.Batch(p, insts, precision=prec) as b:
        b.set_signal(np.tile(s0, count))
        b.run(n_rt, 0.0)
        ps, rts, flags = b.results()
        out = np.zeros(b.total, s0.dtype)
        b.get_signal(out)
        torch.cuda.synchronize()
    assert (rts == n_rt).all() and (flags == 2).all()
    return p, insts, s0, out.reshape(count, n_t), ps


CASES = [(2, n, cu.F32, (1, 2, 40, 150, 300)) for n in (512, 1024, 2048)] + \
        [(2, 4096, cu.F32, (1, 12, 30, 70, 100, 200)), (2, 8192, cu.F32, (1, 10, 30, 50, 80)),
         (2, 16384, cu.F32, (1, 10, 22, 40)), (2, 32768, cu.F32, (1, 10, 20)), (3, 512, cu.F32, (1, 200)), (3, 1024, cu.F32, (1, 60, 140)),
         (3, 2048, cu.F32, (1, 20, 60, 140)), (3, 4096, cu.F32, (1, 30, 70, 140, 160)), (3, 8192, cu.F32, (1, 12, 30, 80)),
         (3, 16384, cu.F32, (1, 12, 30, 40)), (3, 32768, cu.F32, (1, 10, 17)), (3, 65536, cu.F32, (1, 9)),
         (2, 512, cu.F64, (1, 100, 200)), (2, 1024, cu.F64, (1, 60, 140)), (2, 2048, cu.F64, (1, 60, 140)),
         (2, 4096, cu.F64, (1, 30, 70, 140)), (2, 8192, cu.F64, (1, 12, 30, 60)), (2, 16384, cu.F64, (1, 12, 30)),
         (2, 32768, cu.F64, (1, 9)), (3, 1024, cu.F64, (1, 60, 140)), (3, 2048, cu.F64, (1, 30, 60, 140)),
         (3, 4096, cu.F64, (1, 30, 70)), (3, 8192, cu.F64, (1, 12, 30)), (3, 16384, cu.F64, (1, 12)),
         (3, 32768, cu.F64, (1, 9))]


@pytest.mark.parametrize("neq,n_t,prec,counts", CASES)
def test_results_do_not_depend_on_the_number_of_instances(neq, n_t, prec, counts):
    p, insts, s0, ref, ps_ref = run(neq, n_t, prec, counts[0])
    for c in counts[1:]:
        _, _, _, got, ps = run(neq, n_t, prec, c)
        assert np.array_equal(got[0], ref[0]) and ps[0] == ps_ref[0], c
        assert all(np.array_equal(got[k], got[1]) for k in range(1, c)) and (ps[1:] == ps[1]).all(), c
    # instance 0 against the FP64 oracle
    q = cu.Params(**p.to_dict())
    q.Rs, q.delta, q.gdd = 0.97, -0.1, -2e-4
    T, w = cu.make_grids(n_t, q.t_rt)
    A = [np.zeros(n_t, np.complex128), s0.astype(np.complex128),
         np.zeros(n_t, np.complex128) if neq == 3 else None]
    pump = np.full(n_t, np.float32(q.ap0) if prec == cu.F32 else q.ap0, np.complex128)
    ob.round_trips(q, w.astype(np.float64), T.astype(np.float64), A[0], A[1], A[2], pump, 2, 0, 2)
    assert rel_l2(ref[0], A[1]) < (5e-5 if prec == cu.F32 else 1e-10)


def test_single_plan_equals_batch_of_every_layout():
    """The plan entry point (one instance) against instance 1 of batches on the other layouts."""
    n_t = 4096
    for count in (2, 30, 70, 200):
        p, insts, s0, got, ps = run(2, n_t, cu.F32, count)
        q = cu.Params(**p.to_dict())
        q.Rs, q.delta, q.gdd = 0.97, 0.05, -2e-4
        with cu.Plan(q) as plan:
            Ap = torch.zeros(n_t, dtype=torch.complex64, device="cuda")
            As = torch.from_numpy(s0.copy()).cuda()
            h = torch.zeros(2, dtype=torch.float64, device="cuda")
            plan.round_trips(Ap, As, None, None, 0, 0, 2, ps_hist=h)
            torch.cuda.synchronize()
        assert np.array_equal(As.cpu().numpy(), got[1]) and h[-1].item() == ps[1]


@pytest.mark.parametrize("count", [3, 16, 40])
def test_mixed_grids_equal_uniform_batches(count):
    """Groups that share the chip get other layouts than groups alone; the results stay."""
    sizes = (1024, 4096, 8192, 16384)
    p = params_2eq(n_t=1024, n_z=3, delta=0.05)
    rng = np.random.default_rng(count)
    nts = [int(n) for n in rng.choice(sizes, count)]
    starts = [(0.3 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))).astype(np.complex64) for n in nts]
    mk = lambda idx: [dict(n_t=nts[k], ap0=p.ap0, Rs=0.97, delta=0.01 * k, gdd=1e-4, seed=0) for k in idx]

    def solve(idx):
        with cu.Batch(p, mk(idx)) as b:
            b.set_signal(np.concatenate([starts[k] for k in idx]))
            b.run(2, 0.0)
            out = np.zeros(b.total, np.complex64)
            b.get_signal(out)
            torch.cuda.synchronize()
        offs = np.concatenate([[0], np.cumsum([nts[k] for k in idx])])
        return {k: out[offs[i]:offs[i + 1]] for i, k in enumerate(idx)}

    mixed = solve(list(range(count)))
    for n in sizes:
        idx = [k for k in range(count) if nts[k] == n]
        if idx:
            alone = solve(idx)
            assert all(np.array_equal(alone[k], mixed[k]) for k in idx)


def test_batch_noise_equals_the_host_generator():
    """One launch seeds every instance: sizes that fill no block, 2 and 3 fields, seeds beyond 32 bits."""
    p = params_3eq(n_t=512, n_z=2, regime=cu.CW)
    nts = [512, 1024, 2048, 512, 4096]
    seeds = [0, 7, 2 ** 40 + 3, 123, 2 ** 63 + 1]
    insts = [dict(n_t=n, ap0=p.ap0, Rs=0.9, delta=0.0, gdd=0.0, seed=s) for n, s in zip(nts, seeds)]
    with cu.Batch(p, insts) as b:
        b.seed_noise(1e-3)
        out = np.zeros(b.total, np.complex64)
        b.get_signal(out)
        torch.cuda.synchronize()
    offs = np.concatenate([[0], np.cumsum(nts)])
    for k, (n, s) in enumerate(zip(nts, seeds)):
        assert np.array_equal(out[offs[k]:offs[k + 1]], cu.noise_host(n, 1e-3, s, 0)), k


@pytest.mark.parametrize("n,f64,batch", [(8192, False, 149), (8192, False, 300), (4096, True, 149), (4096, True, 297),
                                         (4096, False, 1190)])
@pytest.mark.parametrize("in_place", [False, True])
def test_fft_persistent_grid(n, f64, batch, in_place):
    """Batches beyond one transform per CTA, in place too (the next transform is loaded before this one is stored).
    Bounds: four stages of about ten roundings each, sqrt(40) u = 4e-7 (F32), 7e-16 (F64)."""
    rng = np.random.default_rng(batch)
    x = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(np.complex128 if f64 else np.complex64)
    d = torch.from_numpy(x).cuda()
    got = cu.fft_c2c(d, -1, out=d if in_place else None).cpu().numpy()
    ref = np.fft.fft(x.astype(np.complex128), axis=-1)
    assert rel_l2(got, ref) < (1e-14 if f64 else 5e-7)


@pytest.mark.parametrize("n_t", [256, 512, 2048, 8192, 32768])
def test_bands_against_fp64_sum(n_t):
    """Field synthesis from band rows against the FP64 sum over the modes (from the smallest grid, two
    points n1 per instance, on).  Bound: FP32 products and a 128-point transform, 1e-6 relative L2."""
    from cuopo_b200 import warmstart as ws
    rng = np.random.default_rng(n_t)
    count = 5
    q0 = rng.integers(64, n_t // 2 - 63, count)
    y = np.zeros((count, 512), np.float32)
    y[:, :256] = rng.uniform(-0.2, 1.0, (count, 256))       # negative magnitudes count as zero
    phi = rng.uniform(-np.pi, np.pi, count)
    y[:, 256:320], y[:, 320:384] = np.cos(phi)[:, None], np.sin(phi)[:, None]
    y[:, 384:448] = ws.centre_code(q0, n_t)[:, None]
    y[:, 448:512] = rng.uniform(-2, 0, count)[:, None]
    f, _ = ws.WarmStartModel(None, 1.0, {"kind": "band"}).fields(torch.from_numpy(y).cuda(), n_t)
    f = f.cpu().numpy()
    Y = y.astype(np.float64)
    for i in range(count):
        a = np.maximum(Y[i, :256], 0)
        c = a * np.sqrt(10 ** Y[i, 448:512].mean() / np.sum(a * a))
        c = c * np.exp(0.5j * np.arctan2(Y[i, 320:384].mean(), Y[i, 256:320].mean()))
        k = np.arange(128) - 64
        spec = np.zeros(n_t, np.complex128)
        np.add.at(spec, (q0[i] + k) % n_t, c[:128])
        np.add.at(spec, (-q0[i] + k) % n_t, c[128:])
        assert rel_l2(f[i], np.fft.ifft(spec) * n_t) < 1e-6


@pytest.mark.parametrize("n_in,width,depth,n_out,batch", [(64, 128, 1, 128, 1), (4, 512, 2, 512, 1300),
                                                           (4, 512, 2, 512, 2400), (5, 256, 2, 1024, 257),
                                                           (3, 1152, 1, 128, 130)])
def test_network_tile_widths_and_ragged_batches(n_in, width, depth, n_out, batch):
    """Forward and gradients where the tile width changes, with rows that fill no tile, a full 64-wide
    input and layers wider than the first; an unaligned output goes through the network's own buffer.
    Bounds as in test_gpu_mlp.py (forward 2e-3, gradients 2e-2 relative L2)."""
    import ctypes as C

    from cuopo_b200 import warmstart as ws
    from cuopo_b200._lib import check, load
    from oracle import mlp_oracle as mo
    mlp = ws.MLP(n_in, width, depth, n_out, max_batch=batch, seed=3)
    rng = np.random.default_rng(batch)
    x = rng.uniform(-1, 1, (batch, n_in)).astype(np.float32)
    t = (0.5 * rng.standard_normal((batch, n_out))).astype(np.float32)
    X = torch.from_numpy(x).cuda()
    y = mlp.forward(X)
    buf = torch.zeros(batch * n_out + 1, device="cuda")
    check(load().cuopo_mlp_forward(mlp._h, X.data_ptr(), buf.data_ptr() + 4, batch,
                                   torch.cuda.current_stream().cuda_stream))
    loss, g = mlp.gradients(X, torch.from_numpy(t).cuda())
    p = mlp.get_params().astype(np.float64)
    mlp.close()
    dims = mo.layer_dims(n_in, width, depth, n_out)
    y_ref, _ = mo.forward(p, x, dims, emulate_bf16=True)
    loss_ref, g_ref = mo.loss_and_grads(p, x, t, dims, emulate_bf16=True)
    assert rel_l2(y.cpu().numpy(), y_ref) < 2e-3
    assert torch.equal(buf[1:].reshape(batch, n_out), y)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    o = 0
    for n, k in dims:
        for size in (n * k, n):
            assert rel_l2(g[o:o + size], g_ref[o:o + size]) < 2e-2
            o += size
