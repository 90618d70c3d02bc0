"""The streaming solver (k_solve), which runs the tiles that do not fit the chip, at sizes where
many items need few pixels: long strips a fraction of an item wide, alone and in jobs whose other
tiles stay on the chip.  FP64 is compared bit for bit, with the CPU oracle and between jobs; mixed
precision with FP64 within the bounds of the mixed mode (1e-3 rad RMS of the continuous solution,
1e-4 of the cycles with a floor of 3)."""
import ctypes as C

import numpy as np
import pytest

import cuphu_b200
import oracle as O
from cuphu_b200 import synthetic as S
from cuphu_b200._lib import (CuPhuScene, CuPhuSolveStats, check, default_params,
                             default_solve_options, lib)
from tests.devbuf import dptr, empty, to_dev, to_host
from tests.test_gpu_laplace import gpu_solve
from tests.test_gpu_resident import scene
from tests.test_solver_plan import solver_plan

pytestmark = pytest.mark.gpu

TIMEOUT = -5
# per precision: scenes of one job, and which of them are streamed
JOBS = {0: ([(37920, 20), (60, 50), (18960, 70), (1, 70), (300, 66)], [1, 0, 1, 0, 0]),
        1: ([(16483, 20), (90, 75), (8300, 70), (1, 70), (300, 66)], [1, 0, 1, 0, 0])}


def streamed(shapes, precision):
    sms = cuphu_b200.gpu_info(0)["sm_count"]
    return [1 - int(t[0]) for t in solver_plan(shapes, precision, sms)[0]]


@pytest.fixture(scope="module")
def inputs():
    def make(precision):
        out = []
        for i, sh in enumerate(JOBS[precision][0]):
            ig, g, _, _ = S.bumps(*sh, seed=70 + i, nbumps=2, amp_range=(5, 20), sigma_range=(8, 20))
            out.append((to_dev(np.mod(np.angle(ig), 2 * np.pi).astype(np.float32)), to_dev(g)))
        return out
    return {p: make(p) for p in JOBS}


def solve(torch, data, precision, stats=True, **opts):
    """The scenes of `data` in one job: (status, [(unw, labels)], statistics)."""
    scenes = (CuPhuScene * len(data))()
    out = []
    for j, (ph, g) in enumerate(data):
        nr, nc = ph.shape
        out.append((empty((nr, nc), torch.float32), empty((nr, nc), torch.int32)))
        scenes[j] = CuPhuScene(None, ph.data_ptr(), g.data_ptr(), None, None, nr, nc, 1, 1, 0, 0,
                               5.0, out[j][0].data_ptr(), out[j][1].data_ptr())
    p = default_params()
    o = default_solve_options(precision=precision, **{**dict(n_irls=1, max_iter=60), **opts})
    st = CuPhuSolveStats()
    rc = lib().cuphu_unwrap_batch_device(scenes, len(data), 0, C.byref(p), C.byref(o),
                                         C.byref(st) if stats else None, None)
    torch.cuda.synchronize()
    return rc, [(to_host(u), to_host(c)) for u, c in out], st


def same(a, b):
    return np.array_equal(a[0].view(np.int32), b[0].view(np.int32)) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("shape,blocked", [((16483, 20), False), ((8300, 70), True)])
def test_streamed_fp64_bit_exact_vs_oracle(torch_cuda, shape, blocked):
    assert streamed([shape], 1) == [1]
    costs, ph = scene(*shape, seed=5, blocked=blocked)
    x, k, unw, iters = O.laplace_f64(costs, ph, O.lap_opts(n_irls=1, max_iter=40))
    gu, gk, gc, st = gpu_solve(torch_cuda, costs, ph, precision=1, n_irls=1, max_iter=40)
    assert st.total_iters == int(iters.sum())
    assert np.array_equal(gk, k)
    assert np.array_equal(gu.view(np.int32), unw.view(np.int32))
    assert np.array_equal(gc, (x + (float(ph[0, 0]) - x[0, 0])).astype(np.float32))


@pytest.mark.parametrize("replace_every", [50, 1, 3, 7, 0])
def test_streamed_mixed_close_to_fp64(torch_cuda, replace_every):
    """The true residual in place of the recursive one every 50, 1, 3 and 7 iterations, and never."""
    shape = (18960, 70)
    assert streamed([shape], 0) == [1]
    costs, ph = scene(*shape, seed=6, blocked=True)
    _, k64, c64, s64 = gpu_solve(torch_cuda, costs, ph, precision=1, n_irls=1, max_iter=60)
    dcost, dph = to_dev(costs), to_dev(ph)
    du, dc = (empty(shape, torch_cuda.float32) for _ in range(2))
    dk = empty(shape, torch_cuda.int32)
    o = default_solve_options(precision=0, n_irls=1, max_iter=60, replace_every=replace_every)
    st = CuPhuSolveStats()
    check(lib().cuphu_laplace_solve_device(dptr(dcost), costs.shape[1], dptr(dph), *shape,
                                           C.byref(o), dptr(du), dptr(dk), dptr(dc), C.byref(st),
                                           None))
    rms = float(np.sqrt(np.mean((to_host(dc).astype(np.float64) - c64) ** 2)))
    assert rms < 1e-3, rms
    assert int(np.sum(to_host(dk) != k64)) <= max(3, int(1e-4 * k64.size))
    assert abs(st.total_iters - s64.total_iters) <= 3 + s64.total_iters // 50


@pytest.mark.parametrize("precision", [0, 1])
def test_job_of_streamed_and_on_chip_tiles(torch_cuda, inputs, precision):
    """Every scene against its own call: FP64 sums and those of the streaming solver do not depend
    on the job, so they agree bit for bit; the order of the on-chip mixed sums may depend on it."""
    shapes, kinds = JOBS[precision]
    assert streamed(shapes, precision) == kinds
    rc, got, st = solve(torch_cuda, inputs[precision], precision)
    check(rc)
    assert st.ntiles == len(shapes)
    longest, work = 0, 0.0
    for i, sh in enumerate(shapes):
        rc, (want,), one = solve(torch_cuda, [inputs[precision][i]], precision)
        check(rc)
        longest = max(longest, one.max_iters_pass)
        work += one.px_iters
        if precision == 1 or kinds[i]:
            assert same(got[i], want)
        else:
            cycles = np.rint((got[i][0].astype(np.float64) - want[0]) / (2 * np.pi))
            assert np.count_nonzero(cycles) <= max(3, int(1e-4 * sh[0] * sh[1]))
    assert st.max_iters_pass == longest
    if precision == 1:
        assert st.px_iters == work


@pytest.mark.parametrize("precision,nshape", [(0, 3), (1, 2)])
def test_launch_shapes_give_identical_streamed_results(torch_cuda, inputs, precision, nshape):
    """Every depth of the shared-memory ring and number of blocks per SM, over several tiles and
    slices of a few items."""
    outs = []
    for v in range(nshape):
        check(lib().cuphu_test_force_solve_shape(v))
        try:
            rc, out, _ = solve(torch_cuda, inputs[precision], precision, n_irls=2)
        finally:
            check(lib().cuphu_test_force_solve_shape(-1))
        check(rc)
        outs.append(out)
    for out in outs[1:]:
        assert all(same(a, b) for a, b in zip(out, outs[0]))


def test_autotune_keeps_streamed_results(torch_cuda, inputs):
    shape = JOBS[0][0][2]
    data = [inputs[0][2]]
    rc, want, _ = solve(torch_cuda, data, 0)
    check(rc)
    ig, g, _, _ = S.bumps(*shape, seed=72, nbumps=2, amp_range=(5, 20), sigma_range=(8, 20))
    ch = cuphu_b200.autotune(ig, g, 5.0)
    assert (ch["solver_stages"], ch["solver_blocks_per_sm"]) in ((3, 2), (2, 2), (6, 1))
    rc, got, _ = solve(torch_cuda, data, 0)
    check(rc)
    assert same(got[0], want[0])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("which", [[0], [0, 1, 2]])
def test_skipped_barrier_of_a_streamed_job(torch_cuda, inputs, precision, which):
    """A block that does not arrive at its first barrier, in a job of the streaming solver alone and
    in one that runs the on-chip solver first; the next call is normal."""
    data = [inputs[precision][i] for i in which]
    rc, want, _ = solve(torch_cuda, data, precision)
    check(rc)
    for stats in (False, True):
        check(lib().cuphu_test_skip_barrier_once(0, 1))
        rc, _, _ = solve(torch_cuda, data, precision, stats=stats, timeout_ms=20)
        assert rc == (TIMEOUT if stats else 0)
        assert lib().cuphu_last_status(0) == TIMEOUT
    rc, got, _ = solve(torch_cuda, data, precision)
    check(rc)
    assert lib().cuphu_last_status(0) == 0
    assert all(same(a, b) for a, b in zip(got, want))


def test_jobs_of_more_than_1024_tiles(torch_cuda, inputs):
    """Refused where more than 1024 tiles are streamed, before any work is enqueued, and accepted
    otherwise; the next call is not disturbed."""
    t = torch_cuda
    g = t.Generator(device="cuda")
    g.manual_seed(8)

    def data(nr, nc):
        return (t.rand((nr, nc), generator=g, device="cuda") * 6.28,
                t.rand((nr, nc), generator=g, device="cuda") * 0.5 + 0.4)

    long, short = data(16401, 1), data(20, 30)
    assert streamed([long[0].shape, short[0].shape], 1) == [1, 0]
    scenes = (CuPhuScene * 1027)()
    out = [(empty(d[0].shape, t.float32), empty(d[0].shape, t.int32)) for d in (long, short)]
    for j in range(1027):
        k = 0 if j < 1025 else 1
        ph, c = (long, short)[k]
        scenes[j] = CuPhuScene(None, ph.data_ptr(), c.data_ptr(), None, None, *ph.shape, 1, 1, 0, 0,
                               5.0, out[k][0].data_ptr(), out[k][1].data_ptr())
    p, o = default_params(), default_solve_options(precision=1, n_irls=0)
    assert lib().cuphu_unwrap_batch_device(scenes, 1027, 0, C.byref(p), C.byref(o), None, None) == -2
    rc, (want,), _ = solve(t, [short], 1)
    check(rc)
    rc, got, st = solve(t, [short] * 1100, 1)
    check(rc)
    assert st.ntiles == 1100
    assert all(same(u, want) for u in got)
