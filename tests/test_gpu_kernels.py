"""Kernels at the sizes where their tiling can go wrong: prime factors of the
transform lengths, remainders and alignments of the point measurement."""

import math

import numpy as np
import pytest

from oracle import bldfm_oracle as O

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def ragged_kw(nx, ny, halo_cells, footprint, n=6):
    """A solve whose extended grid is (nx, ny) + 2 halo_cells with unit cells."""
    z, p = O.vertical_profiles(n, 6.0, (2.0, -1.5), ustar=0.3, mol=-40.0)
    rng = np.random.default_rng(nx * 1000 + ny)
    src = np.zeros((ny, nx)) if footprint else rng.uniform(0.0, 1.0, (ny, nx))
    return dict(srf_flx=src, z=z, profiles=p, domain=(float(nx), float(ny)), levels=n, modes=(nx & ~1, ny & ~1),
                meas_pt=(3.0, 2.0), footprint=footprint, halo=halo_cells + 0.5, precision="double")


@pytest.mark.parametrize("nx,ny,halo,footprint", [
    (14, 22, 0, True), (14, 22, 0, False),     # 2 x 7, 2 x 11: the smallest generic factors
    (10, 26, 13, False),                       # 36 and 52 = 4 x 13
    (59, 129, 129, True),                      # output lines 316 = 4 x 79 and 386 = 2 x 193
    (30, 34, 114, False),                      # 258 = 2 x 3 x 43 and 262 = 2 x 131
    (98, 50, 0, False),                        # 2 x 7 x 7: two generic stages
])
def test_generic_radix_lengths(nx, ny, halo, footprint):
    """FP64 solves on lines with large prime factors against the oracle (numpy's
    FFT): the bar of the FP64 path, 1e-10."""
    from bldfm_gb300 import steady_state_transport_solver

    kw = ragged_kw(nx, ny, halo, footprint)
    _, c, f = steady_state_transport_solver(**kw)
    _, oc, of = O.steady_state_transport_solver(**kw)
    assert relerr(c, oc) <= 1e-10 and relerr(f, of) <= 1e-10
    _, c32, f32 = steady_state_transport_solver(**kw, mode="fp32")
    assert relerr(c32, oc) <= 1e-4 and relerr(f32, of) <= 1e-4


@pytest.mark.parametrize("count,n", [(1, 1), (1, 2), (3, 1023), (2, 1024), (5, 4095), (3, 4097), (2, 70001),
                                     (700, 33), (3, 65536), (3, 65537), (1, 1300003)])
@pytest.mark.parametrize("phase", [0, 1])
def test_point_measurement_remainders(count, n, phase):
    """Every remainder and both 8-byte phases against math.fsum of the exact
    products' roundings: a few eps of the sum of magnitudes."""
    import torch

    from bldfm_gb300.utils import point_measurement_batch

    rng = np.random.default_rng(n)
    F = rng.standard_normal(count * n + 1)
    G = rng.standard_normal(count * n + 1)
    f = torch.from_numpy(F).cuda()[phase:phase + count * n].view(count, n)
    g = torch.from_numpy(G).cuda()[phase:phase + count * n].view(count, n)
    out = point_measurement_batch(f, g).cpu().numpy()
    for b in range(0, count, max(1, count // 7)):
        a = F[phase + b * n:phase + (b + 1) * n] * G[phase + b * n:phase + (b + 1) * n]
        assert abs(out[b] - math.fsum(a)) <= 4 * 2.0**-52 * math.fsum(np.abs(a))


@pytest.mark.parametrize("n,offset", [(256, 0), (768, 1), (4352, 0), (39168, 2)])
def test_training_step_tiles(n, offset):
    """The training step at its smallest batch, at fewer stages than CTAs, and
    with a second round of tiles, on inputs at any 4-byte address: every
    parameter block's gradient within 2e-3 of the FP64 oracle (the bar of the
    MLP tests: BF16 operands), the loss within 1e-3, the same bits twice."""
    import torch

    from bldfm_gb300.mlp import MLP, param_slices
    from oracle import mlp_oracle as MO

    rng = np.random.default_rng(n)
    X = rng.uniform(-1, 1, (n, 8)).astype(np.float32)
    T = rng.standard_normal((n, 4)).astype(np.float32)
    w = rng.uniform(0.5, 1.5, (n, 4)).astype(np.float32)

    def dev(a):
        buf = torch.empty(a.size + offset, dtype=torch.float32, device="cuda")
        t = buf[offset:].view(a.shape)
        t.copy_(torch.from_numpy(a))
        return t

    net = MLP(batch=n, seed=5)
    p = net.params()
    args = [dev(a) for a in (X, T, w)]
    net.train_step(*args, 0.0)
    g, loss = net.grads()
    net.train_step(*args, 0.0)
    g2, loss2 = net.grads()
    assert np.array_equal(g, g2) and loss == loss2
    _, lo, go = MO.forward_backward(p, X, T, w)
    assert abs(loss - lo) <= 1e-3 * lo
    for name, (a, b) in param_slices().items():
        assert relerr(g[a:b], go[a:b]) <= 2e-3, name


@pytest.mark.parametrize("nx,ny,footprint,levels", [
    (501, 533, True, 8),            # odd mode counts (clamped), pairs of modes per thread
    (512, 560, True, 8),            # even, with the unpaired Nyquist row and column
    (460, 512, False, [0, 3, 8]),   # a source spectrum and several output levels
    (20, 6, False, [0, 3, 8]),      # one mode per thread, fewer modes than a block
    (97, 101, True, 8),             # four lanes per mode, a last warp partly filled
    (120, 140, False, [0, 3, 8]),   # ... two warps of them a scheduler
    (3, 2, True, 4),                # the smallest grids
])
def test_fp64_sweep_items(nx, ny, footprint, levels):
    """Both FP64 sweeps over every mode of grids with odd and even mode counts,
    above and below the size where a thread takes two modes: 1e-10 against the
    oracle (reference rounding), 1e-11 against its invariant imbedding."""
    from bldfm_gb300 import steady_state_transport_solver

    z, p = O.vertical_profiles(8, 6.0, (2.0, -1.5), ustar=0.3, mol=-40.0)
    rng = np.random.default_rng(nx)
    src = np.zeros((ny, nx)) if footprint else rng.uniform(0.0, 1.0, (ny, nx))
    kw = dict(srf_flx=src, z=z, profiles=p, domain=(4.0 * nx, 4.0 * ny), levels=levels,
              modes=(2 * nx, 2 * ny) if footprint else (nx, ny), meas_pt=(3.0, 2.0), footprint=footprint, halo=0.0,
              precision="double")
    _, c, f = steady_state_transport_solver(**kw)
    _, oc, of = O.steady_state_transport_solver(**kw)
    assert relerr(c, oc) <= 1e-10 and relerr(f, of) <= 1e-10
    _, c, f = steady_state_transport_solver(**kw, mode="fp64r")
    _, oc, of = O.steady_state_transport_solver(**kw, sweep="riccati")
    assert relerr(c, oc) <= 1e-11 and relerr(f, of) <= 1e-11


def test_batch_of_more_sources_than_a_grid_row():
    """The forward passes take cases by the grid's y, which ends at 65,535: the
    cases on both sides of it give what a batch of three gives (the same FP32
    operations per case: a few ulp)."""
    from bldfm_gb300.batch import solve_batch

    three = [dict(ragged_kw(4, 2, 0, False), precision="single") for _ in range(3)]
    for k, kw in enumerate(three):
        kw["srf_flx"] = kw["srf_flx"] + k
    ref = solve_batch(three)
    res = solve_batch([three[k % 3] for k in range(65537)])
    for k in (0, 1, 65533, 65534, 65535, 65536):
        for a, b in zip(res[k][1:], ref[k % 3][1:]):
            assert relerr(a, b) <= 16 * 2.0**-24


@pytest.mark.parametrize("sizes", [
    [(4, 2)],                              # one line per block, fewer lines than blocks
    [(64, 48), (4, 2), (150, 302)],        # several cases: the grid is the largest case's
    [(512, 640), (20, 6)],                 # more lines than two blocks an SM: several per block
])
def test_batch_forward_passes(sizes):
    """Dispersion cases of one batch share the launches of the forward transform
    and of the k = 0 values: every case, beside a footprint, against the oracle
    at the bar of the FP32 path, 1e-4."""
    from bldfm_gb300.batch import solve_batch

    z, p = O.vertical_profiles(8, 6.0, (2.0, -1.5), ustar=0.3, mol=-40.0)
    cases = []
    for i, (nx, ny) in enumerate(sizes + [(32, 24)]):
        fp = i == len(sizes)
        src = np.zeros((ny, nx)) if fp else np.random.default_rng(nx).uniform(0.0, 1.0, (ny, nx))
        cases.append(dict(srf_flx=src, z=z, profiles=p, domain=(4.0 * nx, 4.0 * ny), levels=[2, 8],
                          modes=(nx, ny), meas_pt=(3.0, 2.0), footprint=fp, halo=8.0, precision="double"))
    for kw, (_, c, f) in zip(cases, solve_batch(cases)):
        _, oc, of = O.steady_state_transport_solver(**kw)
        assert relerr(c.cpu().numpy() if hasattr(c, "cpu") else c, oc) <= 1e-4
        assert relerr(f.cpu().numpy() if hasattr(f, "cpu") else f, of) <= 1e-4


def test_solve_batch_in_parts(monkeypatch):
    """A batch that goes back in parts gives the bits of the whole batch, with its
    error statements, status word and refusals."""
    from bldfm_gb300 import batch as B

    z, p = O.vertical_profiles(8, 6.0, (2.0, -1.5), ustar=0.3, mol=-40.0)
    cases = [dict(srf_flx=np.full((ny, nx), 0.5), z=z, profiles=p, domain=(4.0 * nx, 4.0 * ny), levels=lv,
                  modes=(nx, ny), meas_pt=(3.0, 2.0), footprint=fp, halo=8.0, precision="double")
             for nx, ny, lv, fp in [(64, 48, 8, True), (40, 30, [0, 8], False), (128, 96, 8, True), (6, 4, 8, False),
                                    (64, 48, [2, 4, 8], False)]]
    whole, s = B.solve_batch(cases), B.BatchSolver()
    monkeypatch.setattr(B, "PART_BYTES", 1 << 16)
    assert len(B._split_batch([B._output_bound(kw) for kw in cases])) > 2
    for _ in range(3):
        got = B.solve_batch(cases, solver=s)
        assert s.status() == 0
        # sums of 32 positive FP32 samples added atomically, in any order
        np.testing.assert_allclose(got.error_estimates, whole.error_estimates, rtol=32 * 2.0**-23)
        np.testing.assert_array_equal(s.error_estimates(len(cases)), got.error_estimates)
        for (_, c0, f0), (_, c1, f1) in zip(whole, got):
            np.testing.assert_array_equal(c0, c1)
            np.testing.assert_array_equal(f0, f1)
        with pytest.raises(ValueError):
            B.solve_batch(cases[:-1] + [dict(cases[-1], modes=(5, 4))], solver=s)


@pytest.mark.parametrize("count,size", [(1, 10), (130, 32), (3, 200)])
def test_serving_tiles(count, size):
    """The fused serving kernel with fewer tiles than SMs, with a new case at
    every tile of a block, and with several tiles of a case per block: the batch
    gives the single footprints (the bar of the batched serving test)."""
    from bldfm_gb300.surrogate import Surrogate, load

    net, _, _ = load()
    sur = Surrogate(net, spot_every=0)
    dom = (3.9 * size, 3.9 * size)
    items = [dict(n=128, zm=20.0, wind=(3.0 * math.cos(i), 3.0 * math.sin(i)), srf_shape=(size, size), domain=dom,
                  modes=(size, size), meas_pt=(0.5 * dom[0], 0.4 * dom[1]), ustar=0.3, mol=-50.0 - i)
             for i in range(count)]
    outs = [(c.cpu().numpy(), f.cpu().numpy()) for c, f in sur.solve_batch_prepared(sur.prepare_batch(items))]
    assert sur.status() == 0
    for i in range(0, count, 13):
        c, f = sur.solve_prepared(sur.prepare(**items[i]))
        assert relerr(outs[i][0], c.cpu().numpy()) < 1e-6 and relerr(outs[i][1], f.cpu().numpy()) < 1e-6


@pytest.mark.parametrize("bad", ["modes", "profile"])
def test_refused_parts_leave_the_last_batch(monkeypatch, bad):
    """A large batch whose last case is refused, by its description or by its
    profiles, is refused before anything runs: outputs on the device, status word
    and error statements stay the last batch's."""
    from bldfm_gb300 import batch as B

    z, p = O.vertical_profiles(8, 6.0, (2.0, -1.5), ustar=0.3, mol=-40.0)
    cases = [dict(srf_flx=np.full((48, 64), 0.5 + i), z=z, profiles=p, domain=(256.0, 192.0), levels=8, modes=(64, 48),
                  meas_pt=(3.0, 2.0 + i), footprint=i % 2 == 0, halo=8.0, precision="double") for i in range(6)]
    s = B.BatchSolver()
    outs = [t for pair in s.solve(cases) for t in pair]
    want, est = [t.cpu() for t in outs], s.error_estimates(6)
    monkeypatch.setattr(B, "PART_BYTES", 1 << 16)
    assert len(B._split_batch([B._output_bound(kw) for kw in cases])) > 2
    neg = tuple(-a for a in p)
    last = dict(cases[0], modes=(5, 4)) if bad == "modes" else dict(cases[0], profiles=neg)
    with pytest.raises(ValueError):
        B.solve_batch(cases[:0:-1] + [last], solver=s)
    s.stream.synchronize()
    for a, b in zip(want, outs):
        np.testing.assert_array_equal(a, b.cpu())
    assert s.status() == 0
    np.testing.assert_array_equal(s.error_estimates(6), est)


def test_failure_between_parts_keeps_what_ran(monkeypatch):
    """A part that fails after the first has run: the solver's last batch is the
    parts that ran, and the next batch is as good as ever."""
    from bldfm_gb300 import batch as B

    z, p = O.vertical_profiles(8, 6.0, (2.0, -1.5), ustar=0.3, mol=-40.0)
    cases = [dict(srf_flx=np.zeros((48, 64)), z=z, profiles=p, domain=(256.0, 192.0), levels=8, modes=(64, 48),
                  meas_pt=(3.0, 2.0 + i), footprint=True, halo=8.0, precision="double") for i in range(6)]
    s = B.BatchSolver()
    whole = B.solve_batch(cases, solver=s)
    monkeypatch.setattr(B, "PART_BYTES", 1 << 16)
    cuts = B._split_batch([B._output_bound(kw) for kw in cases])
    run, calls = s._run, []

    def failing(prepared, ws):
        calls.append(len(prepared[0]))
        if len(calls) == 2:
            raise RuntimeError("second part")
        return run(prepared, ws)

    monkeypatch.setattr(s, "_run", failing)
    with pytest.raises(RuntimeError, match="second part"):
        B.solve_batch(cases, solver=s)
    monkeypatch.undo()
    assert s._parts == [cuts[1]] and s.status() == 0
    np.testing.assert_allclose(s.error_estimates(cuts[1]), whole.error_estimates[: cuts[1]], rtol=32 * 2.0**-23)
    for (_, c0, f0), (_, c1, f1) in zip(whole, B.solve_batch(cases, solver=s)):
        np.testing.assert_array_equal(c0, c1)
        np.testing.assert_array_equal(f0, f1)


@pytest.mark.parametrize("at", [2, 5])
def test_status_of_every_part(monkeypatch, at):
    """A non-finite source in a middle or the last part: the call reports it, the
    solver's status word too, and the next batch is clean."""
    from bldfm_gb300 import _lib
    from bldfm_gb300 import batch as B

    z, p = O.vertical_profiles(8, 6.0, (2.0, -1.5), ustar=0.3, mol=-40.0)
    cases = [dict(srf_flx=np.full((48, 64), 0.5), z=z, profiles=p, domain=(256.0, 192.0), levels=8, modes=(64, 48),
                  meas_pt=(3.0, 2.0), footprint=False, halo=8.0, precision="double") for _ in range(6)]
    monkeypatch.setattr(B, "PART_BYTES", 1 << 16)
    cuts = B._split_batch([B._output_bound(kw) for kw in cases])
    assert len(cuts) == 5 and cuts[1] <= 2 and cuts[-2] <= 5
    bad = [dict(kw) for kw in cases]
    bad[at]["srf_flx"] = bad[at]["srf_flx"].copy()
    bad[at]["srf_flx"][3, 5] = np.nan
    s = B.BatchSolver()
    for _ in range(2):
        with pytest.raises(FloatingPointError):
            B.solve_batch(bad, solver=s)
        assert s.status() == _lib.ERR_NONFINITE
        B.solve_batch(cases, solver=s)
        assert s.status() == 0


@pytest.mark.parametrize("mode", ["fp64", "fp64r"])
@pytest.mark.parametrize("nx,ny,levels", [(64, 48, 8), (7, 5, [2, 8]), (512, 400, [0, 8])])
def test_single_solve_outputs_own_their_memory(mode, nx, ny, levels):
    """A caller that keeps one output of a single solve keeps no memory of the
    other: each array's memory is its own and no larger."""
    from bldfm_gb300 import steady_state_transport_solver

    z, p = O.vertical_profiles(8, 6.0, (2.0, -1.5), ustar=0.3, mol=-40.0)
    _, c, f = steady_state_transport_solver(np.zeros((ny, nx)), z, p, (4.0 * nx, 4.0 * ny), levels,
                                            modes=(nx & ~1, ny & ~1), footprint=True, halo=8.0, precision="double",
                                            mode=mode)
    owners = [a if a.base is None else a.base for a in (c, f)]
    assert owners[0] is not owners[1]
    assert all(o.base is None and o.nbytes == a.nbytes for o, a in zip(owners, (c, f)))


@pytest.mark.parametrize("n", [65536, 4_000_000])  # one cluster; partial sums of the whole device
@pytest.mark.parametrize("phase", [0, 1])
@pytest.mark.parametrize("values", ["absorbed", "cancelling"])
def test_point_measurement_worst_case(n, phase, values):
    """Products that a plain addition loses, where a thread's chain of eight FMAs,
    the join of its two chains and the sums over threads each meet them, and
    sums that cancel within a thread's 16 points.  Bound in u = 2^-53 of the sum
    of magnitudes: 8 for the chain, 1 for the join, 2 for the compensated sum, 1
    for the result (13 for a compensated sum per point and a plain tree over 256
    threads: product 1, sum 2, tree 8, partials 2)."""
    import torch

    from bldfm_gb300.utils import point_measurement_batch

    lead = phase  # a field at an odd 8-byte phase has one leading point, then pairs
    a = np.zeros(n)
    pairs = a[lead:lead + 2 * ((n - lead) // 2)].reshape(-1, 2)
    if values == "absorbed":
        d = 0.99 * 2.0**-53
        pairs[0] = 1.0, d                   # thread 0's chains; the second is lost in their join
        pairs[256:2048:256, 0] = d          # ... and the first chain's seven further FMAs
        pairs[[16, 8, 4, 2, 1], 0] = d      # the lanes a tree over the warp adds to lane 0
        pairs[32:256:32, 0] = d             # ... and over the warps
    else:
        rng = np.random.default_rng(n)
        m = len(pairs) // 512  # a thread's consecutive pairs are 256 apart
        big = 10.0 ** rng.uniform(6, 9, (m, 1, 256, 1))
        pairs[: 512 * m].reshape(m, 2, 256, 2)[:] = big * np.array([1.0, -1.0]).reshape(1, 2, 1, 1)
        pairs += rng.uniform(-1, 1, pairs.shape)
    f = torch.ones(n + 1, dtype=torch.float64, device="cuda")[phase:phase + n].view(1, n)
    g = torch.empty(n + 1, dtype=torch.float64, device="cuda")[phase:phase + n].view(1, n)
    g.copy_(torch.from_numpy(a).view(1, n))
    out = float(point_measurement_batch(f, g)[0])
    assert abs(out - math.fsum(a)) <= 12 * 2.0**-53 * math.fsum(np.abs(a))


def test_parts_of_any_sequence(monkeypatch):
    """A large batch in a sequence that has no slices goes in parts as a list does."""
    from collections import deque

    from bldfm_gb300 import batch as B

    z, p = O.vertical_profiles(8, 6.0, (2.0, -1.5), ustar=0.3, mol=-40.0)
    cases = [dict(srf_flx=np.zeros((48, 64)), z=z, profiles=p, domain=(256.0, 192.0), levels=8, modes=(64, 48),
                  meas_pt=(3.0, 2.0 + i), footprint=True, halo=8.0, precision="double") for i in range(6)]
    whole = B.solve_batch(cases)
    monkeypatch.setattr(B, "PART_BYTES", 1 << 16)
    assert len(B._split_batch([B._output_bound(kw) for kw in cases])) > 2
    for (_, c0, f0), (_, c1, f1) in zip(whole, B.solve_batch(deque(cases))):
        np.testing.assert_array_equal(c0, c1)
        np.testing.assert_array_equal(f0, f1)
