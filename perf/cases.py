"""Performance cases of the unwrapping path: what users have the library do, over the range of
sizes, options and entry points, with seeded synthetic inputs made on the GPU.

Every case names an operation (``op``):

* ``host``    -- ``cuphu_b200.unwrap`` on NumPy arrays: the drop-in call, host phase, uploads and
                 downloads included;
* ``device``  -- ``cuphu_unwrap_device``: the same pipeline on device-resident data;
* ``batch``   -- ``cuphu_unwrap_batch_device``: a stack of uneven interferograms in one call;
* ``adjoint`` -- ``autograd.irls_solve`` forward and backward (gradients of a loss on the
                 continuous solution with respect to arc targets and arc weights);
* ``costs``   -- ``cuphu_build_costs_device``: the statistical-cost build of a network-flow run,
                 with its residues;
* ``labels``  -- ``cuphu_b200.regrow_conncomp``: connected components of an unwrapped phase.

The scenes follow the recipes of ``cuphu_b200.synthetic`` (Gaussian bumps plus a ramp, power-law
topography, smooth coherence, a low-coherence water blob, Cramer-Rao phase noise).
"""
import ctypes as C
import math

import numpy as np
import torch

import cuphu_b200
from cuphu_b200._lib import (CuPhuScene, check, default_params, default_solve_options,
                             default_tile_params, lib)
from cuphu_b200._unwrap import _auto_ntiles_by_target_size
from cuphu_b200.autograd import irls_solve

MODE = {"smooth": 0, "defo": 1, "topo": 2}
PRECISION = {"mixed": 0, "fp64": 1}
OVERLAP = 64
TARGET = 1024


def _case(name, op, rows, cols, scene="bumps", cost="defo", nlooks=5.0, precision="mixed",
          n_irls=16, mask=False, post=False, count=1):
    c = {"op": op, "rows": rows, "cols": cols, "scene": scene, "cost": cost, "nlooks": nlooks,
         "precision": precision, "n_irls": n_irls, "mask": mask, "post": post, "count": count}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a chip around one building or crater: latency of the whole call counts
        _case("host_96x128", "host", 96, 128, cost="smooth"),
        # the standard small scene, through the drop-in call with its default precision
        _case("host_512_defo", "host", 512, 512),
        # the same scene at full precision, device to device
        _case("device_512_fp64", "device", 512, 512, precision="fp64"),
        # one burst subset, ragged, with a water mask that is grown by the call
        _case("host_901x1250_masked", "host", 901, 1250, scene="water", cost="smooth", nlooks=9.0,
              mask=True),
        # a topographic scene that tiles itself 2 x 2 or so, with both clean-up passes
        _case("device_2051x1537_topo", "device", 2051, 1537, scene="topo", cost="topo",
              nlooks=20.0, post=True),
        # the large scene with water, three reweighting passes
        _case("device_4096_smooth", "device", 4096, 4096, scene="water", cost="smooth",
              nlooks=9.0, n_irls=3),
        # a short time series of uneven interferograms in one call
        _case("batch_8_uneven", "batch", 1024, 1024, count=8),
        # gradients through the solve: a patch in a training loop, and the full scene
        _case("adjoint_256", "adjoint", 256, 256, precision="fp64", n_irls=5),
        _case("adjoint_2048", "adjoint", 2048, 2048, precision="fp64", n_irls=5),
        # cost arrays for a network-flow run: a ragged subset and a full frame
        _case("costs_1000x1531_smooth", "costs", 1000, 1531, cost="smooth", nlooks=9.0),
        _case("costs_8192_topo", "costs", 8192, 8192, scene="topo", cost="topo", nlooks=20.0),
        # components regrown from an unwrapped phase after a user's own edits
        _case("labels_2048", "labels", 2048, 2048, scene="water", nlooks=9.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["host", "host", "host", "device", "device", "device", "batch", "adjoint",
                     "costs", "labels"])
    nlooks = rng.choice([3.0, 5.0, 9.0, 20.0])
    scene = rng.choice(["bumps", "water", "topo"])
    cost = rng.choice(["smooth", "defo", "topo"])
    if op == "host":
        return _case(None, op, _log(rng, 64, 1430), _log(rng, 64, 1430), scene, cost, nlooks,
                     rng.choice(["mixed", "mixed", "mixed", "fp64"]), rng.choice([3, 8, 16]),
                     mask=rng.random() < 0.4)
    if op == "device":
        rows = _log(rng, 300, 2400)
        cols = _log(rng, 300, 2400)
        return _case(None, op, rows, cols, scene, cost, nlooks,
                     "fp64" if rows * cols < 1200000 and rng.random() < 0.4 else "mixed",
                     rng.choice([3, 8]) if rows * cols > 1500000 else rng.choice([8, 16]),
                     mask=rng.random() < 0.3, post=rng.random() < 0.3)
    if op == "batch":
        side = _log(rng, 400, 1100)
        return _case(None, op, side, _log(rng, 400, 1100), nlooks=nlooks, n_irls=8,
                     count=rng.randint(3, 8))
    if op == "adjoint":
        return _case(None, op, _log(rng, 100, 1500), _log(rng, 100, 1500), precision="fp64",
                     nlooks=nlooks, n_irls=rng.choice([2, 5]))
    if op == "costs":
        return _case(None, op, _log(rng, 200, 8000), _log(rng, 200, 8000), scene, cost, nlooks)
    return _case(None, op, _log(rng, 150, 3000), _log(rng, 150, 3000), scene, cost, nlooks)


# ── scenes ────────────────────────────────────────────────────────────────

def _field(g, rows, cols, sigma):
    """Uniform noise low-passed by a Gaussian of ``sigma`` pixels, rescaled to [0, 1]."""
    u = torch.rand((rows, cols), generator=g, device="cuda")
    ky = torch.fft.fftfreq(rows, device="cuda")[:, None]
    kx = torch.fft.rfftfreq(cols, device="cuda")[None, :]
    h = torch.exp(-2.0 * (math.pi * sigma) ** 2 * (ky * ky + kx * kx))
    f = torch.fft.irfft2(torch.fft.rfft2(u - u.mean()) * h, s=(rows, cols))
    return (f - f.min()) / (f.max() - f.min()).clamp_min(1e-12)


def _scene(case, seed, rows=None, cols=None):
    """(igram complex64, coherence, true phase, valid mask) on the GPU, from the seed alone."""
    rows, cols = rows or case["rows"], cols or case["cols"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def uni(lo, hi):
        return lo + (hi - lo) * float(torch.rand((), generator=g, device="cuda"))

    amp = None
    lo, hi = (0.2, 0.9) if case["scene"] == "topo" else (0.3, 0.95)
    if case["scene"] == "topo":
        ky = torch.fft.fftfreq(rows, device="cuda")[:, None]
        kx = torch.fft.rfftfreq(cols, device="cuda")[None, :]
        k2 = ky * ky + kx * kx
        k2[0, 0] = 1.0
        a = k2 ** (-0.75)
        a[0, 0] = 0.0
        w = torch.randn((rows, cols), generator=g, device="cuda")
        h = torch.fft.irfft2(torch.fft.rfft2(w) * a, s=(rows, cols))
        # 0 to 2500 m over the 8192-pixel scene's geometry; smaller scenes see less relief
        top = 40.3 * max(rows, cols) / 8192.0
        truth = (h - h.min()) / (h.max() - h.min()) * max(top, 6.0)
        amp = torch.empty((rows, cols), device="cuda").exponential_(1.0, generator=g)
    else:
        rr = torch.arange(rows, device="cuda", dtype=torch.float32)[:, None]
        cc = torch.arange(cols, device="cuda", dtype=torch.float32)[None, :]
        truth = 0.05 * cc + 0.0 * rr
        small = min(1.0, min(rows, cols) / 400.0)
        for _ in range(6 if rows * cols > 4000000 else 3):
            s = uni(30.0, 90.0) * max(small, 0.2)
            h = uni(10.0, 40.0) * max(small, 0.2) * (1.0 if uni(-1.0, 1.0) > 0 else -1.0)
            r0, c0 = uni(0.0, rows), uni(0.0, cols)
            truth = truth + h * torch.exp(-((rr - r0) ** 2 + (cc - c0) ** 2) / (2.0 * s * s))
    gamma = lo + (hi - lo) * _field(g, rows, cols, 20.0)
    valid = torch.ones((rows, cols), dtype=torch.bool, device="cuda")
    if case["scene"] == "water":
        blob = _field(g, rows, cols, max(rows, cols) / 40.0)
        step = max(1, rows // 512), max(1, cols // 512)
        valid = blob <= torch.quantile(blob[::step[0], ::step[1]].reshape(-1), 0.85)
        low = 0.02 + 0.08 * torch.rand((rows, cols), generator=g, device="cuda")
        gamma = torch.where(valid, gamma, low)
    sd = torch.sqrt((1.0 - gamma * gamma) / (2.0 * case["nlooks"] * gamma * gamma))
    re = torch.cos(truth) + sd * torch.randn((rows, cols), generator=g, device="cuda")
    im = torch.sin(truth) + sd * torch.randn((rows, cols), generator=g, device="cuda")
    ig = torch.complex(re, im)
    if amp is not None:
        ig = ig * amp
    return ig.contiguous(), gamma.contiguous(), truth, valid


def _phase(ig):
    p = torch.angle(ig)
    return torch.where(p < 0, p + 2.0 * math.pi, p).to(torch.float32).contiguous()


def _wrapped_arcs(ig):
    """Wrapped phase differences on the two arc planes (unused last row / column zero)."""
    gd, gr = torch.zeros(ig.shape, device="cuda"), torch.zeros(ig.shape, device="cuda")
    gd[:-1] = torch.angle(ig[1:] * ig[:-1].conj())
    gr[:, :-1] = torch.angle(ig[:, 1:] * ig[:, :-1].conj())
    return gd, gr


def _arc_weights(gamma):
    """Per-arc weights of a training program: inverse phase variance of the arcs' mean coherence."""
    def weight(a, b):
        m = (0.5 * (a + b)).clamp(0.05, 0.98)
        return m * m / (1.0 - m * m)
    wd, wr = torch.zeros_like(gamma), torch.zeros_like(gamma)
    wd[:-1] = weight(gamma[1:], gamma[:-1])
    wr[:, :-1] = weight(gamma[:, 1:], gamma[:, :-1])
    return wd, wr


def _sides(case):
    """Uneven sides of a batch's interferograms: full, half and three-quarter extents."""
    part = [(1.0, 1.0), (0.5, 1.0), (1.0, 0.5), (0.5, 0.5), (0.75, 1.0), (0.5, 0.75), (1.0, 0.75),
            (0.75, 0.5)]
    return [(max(64, int(case["rows"] * a)), max(64, int(case["cols"] * b)))
            for a, b in part[:case["count"]]]


# ── what a program has in hand, and one pass ──────────────────────────────

def prepare(case, seed):
    op = case["op"]
    st = {"case": case}
    if op == "batch":
        st["params"] = default_params(nlooks=case["nlooks"], ncorrlooks=case["nlooks"])
        st["opts"] = default_solve_options(precision=PRECISION[case["precision"]],
                                           n_irls=case["n_irls"])
        sides = _sides(case)
        st["scenes"] = (CuPhuScene * len(sides))()
        st["bufs"] = []
        for k, (r, c) in enumerate(sides):
            ig, gamma, _, _ = _scene(case, seed * 64 + k, r, c)
            unw = torch.empty((r, c), device="cuda")
            cc = torch.empty((r, c), dtype=torch.int32, device="cuda")
            st["bufs"].append((ig, gamma, unw, cc))
            nt = _auto_ntiles_by_target_size(r, c, TARGET, OVERLAP, OVERLAP)
            st["scenes"][k] = CuPhuScene(ig.data_ptr(), None, gamma.data_ptr(), None, None, r, c,
                                         nt[0], nt[1], OVERLAP, OVERLAP, case["nlooks"],
                                         unw.data_ptr(), cc.data_ptr())
        return st
    ig, gamma, truth, valid = _scene(case, seed)
    rows, cols = case["rows"], case["cols"]
    if op == "host":
        st["igram"], st["corr"] = ig.cpu().numpy(), gamma.cpu().numpy()
        st["mask"] = valid.cpu().numpy() if case["mask"] else None
    elif op == "device":
        nt = _auto_ntiles_by_target_size(rows, cols, TARGET, OVERLAP, OVERLAP)
        st["igram"], st["corr"] = ig, gamma
        st["mask"] = valid.to(torch.uint8).contiguous() if case["mask"] else None
        st["params"] = default_params(nlooks=case["nlooks"], ncorrlooks=case["nlooks"])
        st["tile"] = default_tile_params(ntilerow=nt[0], ntilecol=nt[1], rowovrlp=OVERLAP,
                                         colovrlp=OVERLAP,
                                         laplace_neighbor_feedback=int(case["post"]),
                                         fix_cycle_spikes=int(case["post"]))
        st["opts"] = default_solve_options(precision=PRECISION[case["precision"]],
                                           n_irls=case["n_irls"])
        st["unw"] = torch.empty((rows, cols), device="cuda")
        st["cc"] = torch.empty((rows, cols), dtype=torch.int32, device="cuda")
    elif op == "adjoint":
        st["arcs"] = _wrapped_arcs(ig) + _arc_weights(gamma)
        st["truth"] = (truth - truth.mean()).to(torch.float64)
    elif op == "costs":
        narcs = (rows - 1) * cols + rows * (cols - 1)
        st["phase"], st["corr"] = _phase(ig), gamma
        st["params"] = default_params(nlooks=case["nlooks"], ncorrlooks=case["nlooks"])
        st["costs"] = torch.empty((narcs, 2 if case["cost"] == "smooth" else 4),
                                  dtype=torch.int16, device="cuda")
        st["residues"] = torch.empty((rows - 1, cols - 1), dtype=torch.int8, device="cuda")
    else:
        st["unw"] = (_phase(ig) + 2.0 * math.pi *
                     torch.round((truth - _phase(ig)) / (2.0 * math.pi))).cpu().numpy()
        st["corr"] = gamma.cpu().numpy()
    return st


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _loss(u, truth):
    return (u - u.mean() - truth).square().mean()


def run(st):
    case = st["case"]
    op, rows, cols = case["op"], case["rows"], case["cols"]
    if op == "host":
        pad = {"mask": st["mask"], "mask_pad_distance": 2} if case["mask"] else {}
        return cuphu_b200.unwrap(st["igram"], st["corr"], case["nlooks"], cost=case["cost"],
                                 init="laplace", precision=case["precision"],
                                 n_irls=case["n_irls"], **pad)
    if op == "device":
        check(lib().cuphu_unwrap_device(_ptr(st["igram"]), None, _ptr(st["corr"]),
                                        _ptr(st["mask"]), None, rows, cols, MODE[case["cost"]],
                                        C.byref(st["params"]), C.byref(st["tile"]),
                                        C.byref(st["opts"]), _ptr(st["unw"]), _ptr(st["cc"]),
                                        None, None, _stream()))
        return st["unw"], st["cc"]
    if op == "batch":
        check(lib().cuphu_unwrap_batch_device(st["scenes"], len(st["bufs"]), MODE[case["cost"]],
                                              C.byref(st["params"]), C.byref(st["opts"]), None,
                                              _stream()))
        return [(b[2], b[3]) for b in st["bufs"]]
    if op == "adjoint":
        leaves = [t.detach().requires_grad_(True) for t in st["arcs"]]
        u = irls_solve(*leaves, n_irls=case["n_irls"], precision=case["precision"])
        _loss(u, st["truth"]).backward()
        return [u.detach()] + [t.grad for t in leaves]
    if op == "costs":
        check(lib().cuphu_build_costs_device(_ptr(st["phase"]), _ptr(st["corr"]), None, rows, cols,
                                             MODE[case["cost"]], C.byref(st["params"]),
                                             _ptr(st["costs"]), _ptr(st["residues"]), _stream()))
        return st["costs"], st["residues"]
    return cuphu_b200.regrow_conncomp(st["unw"], st["corr"])


# ── what a pass cannot do without ─────────────────────────────────────────

def work(case):
    n = case["rows"] * case["cols"]
    if case["op"] == "batch":
        n = sum(r * c for r, c in _sides(case))
    if case["op"] == "costs":
        narcs = 2 * n - case["rows"] - case["cols"]
        return {"bytes": 8.0 * n + n + (4 if case["cost"] == "smooth" else 8) * narcs,
                "flops": 60.0 * narcs}
    if case["op"] == "labels":
        return {"bytes": 12.0 * n, "flops": 4.0 * n}
    # conjugate-gradient steps: about as many per solve as the scene has pixels along a tile's
    # edge, some 25 operations per pixel each
    edge = min(math.sqrt(n / case["count"]), float(TARGET))
    steps = (case["n_irls"] + 1) * edge
    if case["op"] == "adjoint":
        # four arc planes and the truth in, the solution and four gradients out
        return {"bytes": (16.0 + 8.0 + 8.0 + 16.0) * n, "flops": 2.0 * steps * 25.0 * n}
    return {"bytes": 20.0 * n + (n if case["mask"] else 0), "flops": steps * 25.0 * n}


# ── the same results in 64 bits ───────────────────────────────────────────

EPS = 1e-12


def _apply(x, wd, wr):
    y = EPS * x
    f = wd[:-1] * (x[:-1] - x[1:])
    y[:-1] += f
    y[1:] -= f
    f = wr[:, :-1] * (x[:, :-1] - x[:, 1:])
    y[:, :-1] += f
    y[:, 1:] -= f
    return y


def _diag(wd, wr):
    d = torch.full_like(wd, EPS)
    d[:-1] += wd[:-1]
    d[1:] += wd[:-1]
    d[:, :-1] += wr[:, :-1]
    d[:, 1:] += wr[:, :-1]
    return d


def _rhs(gd, gr, wd, wr):
    b = torch.zeros_like(gd)
    f = wd[:-1] * gd[:-1]
    b[:-1] -= f
    b[1:] += f
    f = wr[:, :-1] * gr[:, :-1]
    b[:, :-1] -= f
    b[:, 1:] += f
    return b


def _pcg(b, wd, wr, x=None, max_iter=1000, tol=1e-3):
    """Jacobi-preconditioned conjugate gradients with the solver's stopping rule."""
    d = _diag(wd, wr)
    r = b.clone() if x is None else b - _apply(x, wd, wr)
    x = torch.zeros_like(b) if x is None else x.clone()
    z = r / d
    rz = float((r * z).sum())
    stop = float(np.float32(tol)) ** 2 * rz
    p = z.clone()
    for _ in range(max_iter if rz > 0 else 0):
        q = _apply(p, wd, wr)
        pq = float((p * q).sum())
        if pq <= 0:
            break
        alpha = rz / pq
        x += alpha * p
        r -= alpha * q
        z = r / d
        new = float((r * z).sum())
        if new < stop:
            break
        p = z + (new / rz) * p
        rz = new
    return x


def _reweight(w0d, w0r, ed, er, k, floor=0.01, start=0.5):
    delta = max(floor, start * 0.5 ** k)
    return (w0d / torch.sqrt(ed * ed + delta * delta), w0r / torch.sqrt(er * er + delta * delta))


def _arc_diff(u):
    dd, dr = torch.zeros_like(u), torch.zeros_like(u)
    dd[:-1] = u[1:] - u[:-1]
    dr[:, :-1] = u[:, 1:] - u[:, :-1]
    return dd, dr


class _Exact(torch.autograd.Function):
    """One solve with its adjoint, in 64 bits."""

    @staticmethod
    def forward(ctx, gd, gr, wd, wr, u0):
        u = _pcg(_rhs(gd, gr, wd, wr), wd, wr, u0)
        ctx.save_for_backward(gd, gr, wd, wr, u)
        return u

    @staticmethod
    def backward(ctx, ubar):
        gd, gr, wd, wr, u = ctx.saved_tensors
        dd, dr = _arc_diff(_pcg(ubar - ubar.mean(), wd, wr))
        ud, ur = _arc_diff(u)
        return wd * dd, wr * dr, dd * (gd - ud), dr * (gr - ur), None


def _variance(gamma, other, case):
    """SNAPHU's quantised phase variance of an arc from its two coherences."""
    p = default_params(nlooks=case["nlooks"], ncorrlooks=case["nlooks"])
    rho0 = p.rhosconst1 / p.ncorrlooks + p.rhosconst2
    power = 2.0 * p.cstd1 + p.cstd2 * math.log(p.ncorrlooks) + p.cstd3 * p.ncorrlooks
    rho = 0.5 * (gamma + other)
    rho = torch.where(rho < p.defothreshfactor * rho0, torch.zeros_like(rho), rho)
    v = (torch.pow(1.0 - rho, power) / 6.0 + p.sigsqcorr) * p.nshortcycle ** 2 / p.costscale
    return torch.floor(v).clamp_min(float(p.sigsqshortmin))


def _exact_unwrap(case, seed):
    ig, gamma, _, valid = _scene(case, seed)
    ph = torch.angle(ig.to(torch.complex128))
    ph = torch.where(ph < 0, ph + 2.0 * math.pi, ph)
    gamma = gamma.to(torch.float64)
    if not case["mask"]:
        valid = torch.ones_like(valid)
    elif case["op"] == "host":
        for _ in range(2):  # the call grows the mask by two pixels
            m = valid.clone()
            m[1:] |= valid[:-1]
            m[:-1] |= valid[1:]
            m[:, 1:] |= valid[:, :-1]
            m[:, :-1] |= valid[:, 1:]
            valid = m
    w0d, w0r = torch.zeros_like(ph), torch.zeros_like(ph)
    w0d[:-1] = (valid[1:] & valid[:-1]) / _variance(gamma[:-1], gamma[1:], case)
    w0r[:, :-1] = (valid[:, 1:] & valid[:, :-1]) / _variance(gamma[:, :-1], gamma[:, 1:], case)
    gd, gr = _arc_diff(ph)
    gd -= 2.0 * math.pi * torch.round(gd / (2.0 * math.pi))
    gr -= 2.0 * math.pi * torch.round(gr / (2.0 * math.pi))
    x = _pcg(_rhs(gd, gr, w0d, w0r), w0d, w0r)
    for k in range(case["n_irls"]):
        dd, dr = _arc_diff(x)
        wd, wr = _reweight(w0d, w0r, dd - gd, dr - gr, k)
        x = _pcg(_rhs(gd, gr, wd, wr), wd, wr, x)
    u = x + (ph[0, 0] - x[0, 0])
    return ph + 2.0 * math.pi * torch.round((u - ph) / (2.0 * math.pi))


def exact(case, seed):
    op, n = case["op"], case["rows"] * case["cols"]
    if op in ("host", "device"):
        nt = _auto_ntiles_by_target_size(case["rows"], case["cols"], TARGET, OVERLAP, OVERLAP)
        if nt != (1, 1) or case["post"]:
            return None  # the stitched scene is a set of cycle decisions, not one solve
        u = _exact_unwrap(case, seed)
        return (u.cpu().numpy() if op == "host" else u, None)
    if op == "adjoint" and n <= 4500000:
        ig, gamma, truth, _ = _scene(case, seed)
        leaves = [t.to(torch.float64).requires_grad_(True)
                  for t in _wrapped_arcs(ig) + _arc_weights(gamma)]
        gd, gr, w0d, w0r = leaves
        u = _Exact.apply(gd, gr, w0d, w0r, None)
        for k in range(case["n_irls"]):
            dd, dr = _arc_diff(u)
            wd, wr = _reweight(w0d, w0r, dd - gd, dr - gr, k)
            u = _Exact.apply(gd, gr, wd, wr, u.detach())
        _loss(u, (truth - truth.mean()).to(torch.float64)).backward()
        return [u.detach()] + [t.grad for t in leaves]
    return None  # whole numbers: costs, residues and labels, and the batch's stitched scenes
