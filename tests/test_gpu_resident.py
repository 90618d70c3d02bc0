"""The on-chip solvers (tiles that fit the chip, both precisions) at the sizes
where their split can go wrong: single rows and columns, items exactly filled
and one pixel over, groups with idle members, ragged last levels, the largest
tiles they take and the first one they leave to the streaming solver.  FP64 is
compared with the CPU oracle bit for bit; mixed precision with FP64, within
the bounds of the mixed mode elsewhere: 1e-3 rad RMS of the continuous
solution and 1e-4 of the cycles, with the floor of 3 that a handful of
half-cycle pixels needs."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from cuphu_b200 import synthetic as S
from cuphu_b200._lib import (CuPhuScene, CuPhuSolveStats, check, default_params,
                             default_solve_options, lib)
from tests.devbuf import dptr, empty, to_dev, to_host
from tests.test_gpu_laplace import gpu_solve

pytestmark = pytest.mark.gpu


def scene(nr, nc, seed, blocked=False):
    """(costs, phase): arc variances from a smooth coherence, and with
    ``blocked`` a band of arcs that carry no weight."""
    ig, g, _, _ = S.bumps(nr, nc, seed=seed, nbumps=3, amp_range=(5.0, 25.0),
                          sigma_range=(8.0, 60.0))
    ph = np.mod(np.angle(ig), 2 * np.pi).astype(np.float32)
    rng = np.random.default_rng(seed)
    narcs = (nr - 1) * nc + nr * (nc - 1)
    costs = np.zeros((max(narcs, 1), 2), np.int16)
    nra = (nr - 1) * nc
    costs[:nra, 1] = (1 + 80 * (1 - g[:-1].reshape(-1))).astype(np.int16)
    costs[nra:narcs, 1] = (1 + 80 * (1 - g[:, 1:].reshape(-1))).astype(np.int16)
    if blocked and narcs > 40:
        a = int(rng.integers(0, narcs // 2))
        costs[a:a + narcs // 7, 1] = 32000
    return costs, ph


@pytest.mark.parametrize("shape,blocked", [
    ((1, 1), False), ((1, 70), False), ((70, 1), False), ((2, 64), False), ((16, 64), True),
    ((17, 65), False), ((15, 1037), True), ((1025, 63), False), ((255, 1030), False),
    ((512, 512), True), ((967, 961), False), ((1000, 1102), True), ((270, 1030), True),
    ((1536, 1536), False), ((1540, 1537), False)])
def test_on_chip_solve_matches_fp64(torch_cuda, shape, blocked):
    costs, ph = scene(*shape, seed=shape[0] + 3 * shape[1], blocked=blocked)
    _, k64, c64, s64 = gpu_solve(torch_cuda, costs, ph, precision=1, n_irls=2)
    _, k32, c32, s32 = gpu_solve(torch_cuda, costs, ph, precision=0, n_irls=2)
    rms = float(np.sqrt(np.mean((c32.astype(np.float64) - c64) ** 2)))
    assert rms < 1e-3, rms
    assert int(np.sum(k32 != k64)) <= max(3, int(1e-4 * k64.size))
    assert abs(s32.total_iters - s64.total_iters) <= 3 + s64.total_iters // 50


def test_batch_of_on_chip_and_streamed_tiles(torch_cuda):
    """One job whose tiles go both ways, some sharing the chip side by side:
    every scene's outputs equal those of its own call."""
    shapes = [(60, 50), (1500, 1530), (300, 340), (1, 90), (512, 512)]
    p = default_params()
    o = default_solve_options(precision=0, n_irls=1, max_iter=120)
    data = []
    for i, sh in enumerate(shapes):
        ig, g, _, _ = S.bumps(*sh, seed=70 + i, nbumps=2, amp_range=(5, 20), sigma_range=(8, 20))
        ph = np.mod(np.angle(ig), 2 * np.pi).astype(np.float32)
        data.append((to_dev(ph), to_dev(g)))

    def call(which):
        scenes = (CuPhuScene * len(which))()
        out = []
        for j, i in enumerate(which):
            du = empty(shapes[i], torch_cuda.float32)
            dc = empty(shapes[i], torch_cuda.int32)
            out.append((du, dc))
            scenes[j] = CuPhuScene(None, data[i][0].data_ptr(), data[i][1].data_ptr(), None, None,
                                   shapes[i][0], shapes[i][1], 1, 1, 0, 0, 5.0, du.data_ptr(),
                                   dc.data_ptr())
        st = CuPhuSolveStats()
        check(lib().cuphu_unwrap_batch_device(scenes, len(which), 0, C.byref(p), C.byref(o),
                                              C.byref(st), None))
        return [(to_host(u), to_host(c)) for u, c in out], st

    got, st = call(range(len(shapes)))
    assert st.ntiles == len(shapes)
    longest = 0
    for i in range(len(shapes)):
        want, one = call([i])
        longest = max(longest, one.max_iters_pass)
        assert np.array_equal(got[i][0].view(np.int32), want[0][0].view(np.int32))
        assert np.array_equal(got[i][1], want[0][1])
    assert st.max_iters_pass == longest


@pytest.mark.parametrize("shape,blocked", [
    ((1, 1), False), ((1, 70), False), ((70, 1), False), ((16, 64), True), ((17, 65), False),
    ((15, 1037), True), ((1025, 63), False), ((500, 333), True), ((1024, 1024), False)])
def test_fp64_on_chip_solve_bit_exact_vs_oracle(torch_cuda, shape, blocked):
    costs, ph = scene(*shape, seed=5 + shape[0] + 3 * shape[1], blocked=blocked)
    x, k, unw, iters = O.laplace_f64(costs, ph, O.lap_opts(n_irls=1, max_iter=60))
    gu, gk, gc, st = gpu_solve(torch_cuda, costs, ph, precision=1, n_irls=1, max_iter=60)
    assert st.total_iters == int(iters.sum())
    assert np.array_equal(gk, k)
    assert np.array_equal(gu.view(np.int32), unw.view(np.int32))
    assert np.array_equal(gc, (x + (float(ph[0, 0]) - x[0, 0])).astype(np.float32))


def test_fp64_division_outside_the_correction_range(torch_cuda):
    """Weights of 2^60 and 2^120: the diagonals of the first allow the
    correction steps, those of the second take the IEEE division.  Everything
    scales by powers of two (eps is far below both), so the solutions agree
    bit for bit."""
    from cuphu_b200.autograd import wls_solve
    t = torch_cuda
    g = t.Generator(device="cuda")
    g.manual_seed(3)
    gd, gr, w = (t.rand((90, 75), generator=g, device="cuda") for _ in range(3))
    w = (w * 3 + 0.5)
    out = [wls_solve(gd, gr, w * 2.0 ** e, w.flip(0).contiguous() * 2.0 ** e, max_iter=40)
           for e in (60, 120)]
    assert t.isfinite(out[0]).all() and float(out[0].abs().max()) > 0
    assert t.equal(out[0], out[1])


@pytest.mark.parametrize("tiny", [-930, -980])
def test_fp64_residuals_outside_the_correction_range(torch_cuda, tiny):
    """A warm start of one pixel of 1 and, far from it, one of 2^tiny, without targets: residuals
    of the second lie below the range of the correction steps and take the IEEE division.  The
    same scaled by 2^150 stays inside the range; the problem is linear, so the solutions agree bit
    for bit."""
    from cuphu_b200.autograd import wls_solve
    t = torch_cuda
    g = t.Generator(device="cuda")
    g.manual_seed(4)
    wd, wr = (t.rand((100, 140), generator=g, device="cuda") + 0.5 for _ in range(2))
    none = t.zeros_like(wd)
    u0 = t.zeros((100, 140), dtype=t.float64, device="cuda")
    u0[20, 20], u0[70, 110] = 1.0, 2.0 ** tiny
    out = [wls_solve(none, none, wd, wr, u0=u0 * s, max_iter=20) / s for s in (1.0, 2.0 ** 150)]
    assert 0.0 < float(out[0][70, 110]) < 2.0 ** tiny
    assert float(out[0][71, 110]) > 0.0
    assert t.equal(out[0], out[1])
