"""Sizes at which the kernels change form -- squares a lane holds, lanes a
square gets, registers against cell lists, groups of proposals -- against the
FP64 oracle or the one-at-a-time annealer."""
from __future__ import annotations


import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 96, 97, 128, 161, 193, 224, 225, 256, 257, 512, 1000, 1024])
def test_sat_energy_at_form_changes(ctx, oracle, n):
    """FP32 energies within 1e-5 of the oracle's, candidate counts equal, and
    all but a few gradients (an axis within rounding of another may win)
    within 1e-4; crowded configurations (many hits a square) included."""
    from sqs import sat
    from sqs.workloads import sat_microbench

    x, L = sat_microbench(configs=5, n=n, seed=n)
    if n > 1:
        x[3, :, :2] *= 0.5                      # four times the density
        x[4, :, :2] = 0.3 + 0.2 * x[4, :, :2] / L[4] * min(L[4], 3.0)  # one crowded corner
    x32, L32 = x.astype(np.float32), L.astype(np.float32)
    e, g, c = sat.energy(x32, L32, ctx=ctx, grad=True, count=True)
    eo, go, co = oracle.total_batch(x32.astype(np.float64), L32.astype(np.float64))
    np.testing.assert_allclose(e, eo, rtol=1e-5, atol=1e-6)
    assert np.all(np.abs(c.astype(np.int64) - co) <= np.maximum(1, 1e-5 * co))
    off = np.abs(g - go) - 1e-4 * (1 + np.abs(go))
    assert np.mean(off > 0) <= 2e-3


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 128, 129, 255, 256, 257, 511, 512, 513, 1000])
def test_fp64_energy_at_form_changes(ctx, oracle, n):
    """Energy within 1e-12 relative and gradient within 1e-12 of the oracle's,
    also where a square has more partners than a neighbour list holds and where
    squares lie far outside the box."""
    from sqs.sat import energy_fp64
    from sqs.workloads import sat_microbench

    states, sides = [], []
    for k, (shrink, stray) in enumerate([(1.0, 0), (0.4, 0), (1.0, 3)]):
        x, L = sat_microbench(configs=1, n=n, seed=70 + k, density_side=1.02)
        x[0, :, :2] *= shrink
        if stray and n > stray:
            x[0, :stray, :2] += [[60.0, -35.0]]
        states.append(x[0])
        sides.append(L[0] * 0.98)
    e, g = energy_fp64(states, np.array(sides), ctx=ctx)
    for k, (x, L) in enumerate(zip(states, sides)):
        eo, go = oracle.total_smooth(x, L)
        assert e[k] == pytest.approx(eo, rel=1e-12, abs=1e-300), k
        np.testing.assert_allclose(g[k], go, rtol=0, atol=1e-12 * max(1.0, np.abs(go).max()))


@pytest.mark.parametrize("n", [1, 2, 11, 12, 13, 24, 31, 32, 33, 41, 60, 90, 120, 180])
def test_proposal_forms_equal_one_at_a_time(ctx, n):
    """Registers, groups of two and of four give the one-at-a-time trajectory:
    every replica's final state, energy and counts, from the grid and from a
    crowded start (three quarters of the pitch)."""
    from sqs.anneal import AnnealJob, anneal_batch, jittered_grid

    xya, side = jittered_grid(n, seed=n)
    crowded = xya.copy()
    crowded[:, :2] = 0.5 + 0.75 * (crowded[:, :2] - 0.5)
    for k, start in enumerate((xya, crowded)):
        args = dict(L0=side, replicas=8, sweeps=max(20, 3000 // n), exchange_every=10, tmin=1e-3, tmax=1.0,
                    sigma_xy=0.05, seed=9 + k, polish_iters=0)
        a, b = (anneal_batch([AnnealJob(start, serial=s, **args)], ctx=ctx, trace=True)[0] for s in (False, True))
        for key in ("proposals", "accepted", "exchange_attempts", "exchange_accepts", "L_cert", "shrinks"):
            assert a[key] == b[key], key
        assert a["proposals"] == 8 * n * args["sweeps"]
        assert a["launch"]["overflows"] == b["launch"]["overflows"]
        for key in ("xya", "energy", "energy_full", "rung"):
            np.testing.assert_array_equal(a["trace"][key], b["trace"][key], err_msg=key)
        np.testing.assert_array_equal(a["trace"]["energy"], a["trace"]["energy_full"])


@pytest.mark.parametrize("n", [2, 33, 65, 256, 257, 1000])
@pytest.mark.parametrize("stray", [1, 2, 5])
def test_sat_energy_of_squares_far_outside(ctx, oracle, n, stray):
    """Wall terms have no bound: squares 1e4 outside the box (1e8 of energy
    each) within the same tolerances as any others."""
    from sqs import sat
    from sqs.workloads import sat_microbench

    stray = min(stray, n)
    x, L = sat_microbench(configs=3, n=n, seed=900 + n)
    x[:, :stray, :2] += [[9.0e3, -1.1e4]]
    x32, L32 = x.astype(np.float32), L.astype(np.float32)
    e, g, _ = sat.energy(x32, L32, ctx=ctx, grad=True)
    eo, go, _ = oracle.total_batch(x32.astype(np.float64), L32.astype(np.float64))
    np.testing.assert_allclose(e, eo, rtol=1e-5)
    off = np.abs(g - go) - 1e-4 * (1 + np.abs(go))
    assert np.mean(off > 0) <= 2e-3


@pytest.mark.parametrize("n", [2, 33, 256, 257, 512, 1024])
def test_sat_energy_of_the_smallest_overlaps(ctx, n):
    """One pair overlapping by 2^-22 .. 2^-18 in an otherwise separated lattice:
    every value is exact in FP32, so the energy is the overlap's square."""
    from sqs import sat

    gaps = [2.0 ** -k for k in range(18, 23)]
    x = np.zeros((len(gaps), n, 3))
    i = np.arange(n)
    x[:, :, 0], x[:, :, 1] = 1.0 + 1.25 * (i % 32), 1.0 + 1.25 * (i // 32)
    for k, gap in enumerate(gaps):
        x[k, 0, 0] = x[k, 1, 0] - 1.0 + gap
    e, _, _ = sat.energy(x.astype(np.float32), np.float32(48.0), ctx=ctx)
    np.testing.assert_array_equal(e, [np.float32(gap * gap) for gap in gaps])


def _device_batch(ctx, x32, L32):
    from sqs import sat

    configs, n, _ = x32.shape
    bufs = [ctx.alloc(x32.shape, np.float32).upload(x32), ctx.alloc((configs,), np.float32).upload(L32),
            ctx.alloc((configs,), np.float32), ctx.alloc(x32.shape, np.float32), ctx.alloc((configs,), np.uint32)]
    return bufs, lambda threads: sat.energy_device(ctx, configs, n, *bufs, threads=threads)


@pytest.mark.parametrize("threads", [32, 64, 128, 256])
def test_cta_form_at_squares_a_thread(ctx, oracle, threads):
    """Every CTA width at the sizes where the squares a thread holds change
    their bound, 1 to 1024 squares."""
    from sqs.workloads import sat_microbench

    edges = {1, 2, 1023, 1024}
    npt = 1
    while threads * npt < 1024:
        edges |= {threads * npt - 1, threads * npt, threads * npt + 1}
        npt *= 2
    for n in sorted(edges):
        x, L = sat_microbench(configs=2, n=n, seed=n)
        x32, L32 = x.astype(np.float32), L.astype(np.float32)
        bufs, run = _device_batch(ctx, x32, L32)
        run(threads)
        e, g, c = (b.download() for b in bufs[2:])
        for b in bufs:
            b.free()
        eo, go, co = oracle.total_batch(x32.astype(np.float64), L32.astype(np.float64))
        np.testing.assert_allclose(e, eo, rtol=1e-5, atol=1e-6)
        assert np.all(np.abs(c.astype(np.int64) - co) <= np.maximum(1, 1e-5 * co))
        off = np.abs(g - go) - 1e-4 * (1 + np.abs(go))
        assert np.mean(off > 0) <= 2e-3


def test_narrow_ctas_pay_off_for_small_configurations(ctx):
    """8,192 configurations of 17 squares leave all but one warp of a wide CTA
    without work, so CTAs of 32 threads take well under the time of 256."""
    import time

    from sqs.workloads import sat_microbench

    x, L = sat_microbench(configs=8192, n=17, seed=1)
    bufs, run = _device_batch(ctx, x.astype(np.float32), L.astype(np.float32))
    took = {32: [], 256: []}
    for _ in range(7):
        for threads, ts in took.items():
            run(threads)
            ctx.sync()
            t0 = time.perf_counter()
            for _ in range(50):
                run(threads)
            ctx.sync()
            ts.append(time.perf_counter() - t0)
    for b in bufs:
        b.free()
    assert min(took[32]) < 0.7 * min(took[256]), took
