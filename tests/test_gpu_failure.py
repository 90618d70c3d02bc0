"""Bounded device waits: a solver block that never arrives at a grid barrier
(cuphu_test_skip_barrier_once) makes every other block's wait run out after
the configured limit; the kernel returns, the call reports CUPHU_ERR_TIMEOUT,
and the next call on the same device runs normally.  The failure is made on
the host side of the barrier protocol: no fault, trap or unbounded wait."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from cuphu_b200 import synthetic as S
from cuphu_b200._lib import (CuPhuError, CuPhuScene, CuPhuSolveStats, check, default_params,
                             default_solve_options, default_tile_params, lib)
from tests.devbuf import dptr, empty, to_dev, to_host

pytestmark = pytest.mark.gpu

TIMEOUT = -5


def _run(torch, ph, g, precision, timeout_ms, stats):
    nr, nc = ph.shape
    dph, dg = to_dev(ph), to_dev(g)
    du = empty((nr, nc), torch.float32)
    dc = empty((nr, nc), torch.int32)
    p = default_params(nlooks=5.0, ncorrlooks=5.0)
    t = default_tile_params(ntilerow=2, ntilecol=2, rowovrlp=12, colovrlp=12)
    o = default_solve_options(precision=precision, n_irls=2, timeout_ms=timeout_ms)
    st = CuPhuSolveStats()
    rc = lib().cuphu_unwrap_device(None, dptr(dph), dptr(dg), None, None, nr, nc, 0, C.byref(p),
                                   C.byref(t), C.byref(o), dptr(du), dptr(dc), None,
                                   C.byref(st) if stats else None, None)
    torch.cuda.synchronize()
    return rc, to_host(du)


@pytest.mark.parametrize("precision", [0, 1])
def test_skipped_barrier_times_out_and_device_recovers(torch_cuda, precision):
    ig, g, _, _ = S.bumps(120, 140, seed=51, nbumps=2)
    ph = O.phase_from_igram(ig)
    rc0, want = _run(torch_cuda, ph, g, precision, 5000, stats=True)
    check(rc0)
    # asynchronous call: enqueue succeeds, the device status carries the timeout
    check(lib().cuphu_test_skip_barrier_once(0, 0))
    rc, _ = _run(torch_cuda, ph, g, precision, 20, stats=False)
    assert rc == 0
    assert lib().cuphu_last_status(0) == TIMEOUT
    # a call that waits for its statistics returns the timeout itself
    check(lib().cuphu_test_skip_barrier_once(0, 1))
    rc, _ = _run(torch_cuda, ph, g, precision, 20, stats=True)
    assert rc == TIMEOUT
    with pytest.raises(CuPhuError):
        check(rc)
    # the switch is one-shot: the next call is normal and bit-identical
    rc, got = _run(torch_cuda, ph, g, precision, 5000, stats=True)
    check(rc)
    assert lib().cuphu_last_status(0) == 0
    assert np.array_equal(got.view(np.int32), want.view(np.int32))


@pytest.mark.parametrize("precision,replace,side", [(0, 1, 1000), (0, 50, 1000), (1, 0, 700)])
def test_waiting_for_another_tile_is_not_a_timeout(torch_cuda, precision, replace, side):
    """Three equal scenes of which two run side by side: the remaining blocks wait for the third
    scene's partners far longer than the limit (about 15 ms with a replacement in every
    iteration), but those make progress, so the call succeeds."""
    scenes = (CuPhuScene * 3)()
    keep = []
    for i in range(3):
        ig, g, _, _ = S.bumps(side, side, seed=9 + i, nbumps=3, amp_range=(20, 40),
                              sigma_range=(30, 90))
        ph = np.mod(np.angle(ig), 2 * np.pi).astype(np.float32)
        bufs = (to_dev(ph), to_dev(g), empty((side, side), torch_cuda.float32),
                empty((side, side), torch_cuda.int32))
        keep.append(bufs)
        scenes[i] = CuPhuScene(None, bufs[0].data_ptr(), bufs[1].data_ptr(), None, None, side,
                               side, 1, 1, 0, 0, 5.0, bufs[2].data_ptr(), bufs[3].data_ptr())
    p = default_params()
    o = default_solve_options(precision=precision, n_irls=0, max_iter=400, timeout_ms=5,
                              replace_every=replace)
    st = CuPhuSolveStats()
    check(lib().cuphu_unwrap_batch_device(scenes, 3, 0, C.byref(p), C.byref(o), C.byref(st), None))
    assert st.total_iters == 400


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("block", [0, 2, 40, 147, 100000])
def test_skipped_barrier_of_any_block_number(torch_cuda, precision, block):
    """A small scene's solve launches a few blocks; a number beyond them is taken modulo their
    number, so the hook always does what it says."""
    ig, g, _, _ = S.bumps(70, 90, seed=52, nbumps=2)
    ph = O.phase_from_igram(ig)
    check(lib().cuphu_test_skip_barrier_once(0, block))
    rc, _ = _run(torch_cuda, ph, g, precision, 20, stats=True)
    assert rc == TIMEOUT
    rc, _ = _run(torch_cuda, ph, g, precision, 5000, stats=True)
    check(rc)
