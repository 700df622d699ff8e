"""h2g_calcrk_noalloc: CalcRK! for callers that cannot allocate device memory (their memory
belongs to a pool such as CUDA.jl's, or they run a loop that must not stall on cudaMalloc /
cudaFree).  The entry point allocates nothing; its
reduction scratch is a fixed array inside the library.  It must return the same residual as the
handle-based h2g_calcrk, on two calls in a row (the shared scratch keeps the last call's
contents), and refuse grids larger than its scratch.

This file is collected last so that a failure here does not hide any other test's result."""
import ctypes as C

import numpy as np
import pytest

import h2_b200
from h2_b200 import _lib as L
from conftest import mode3_model

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a.ravel(order="F"))).cuda()


@pytest.mark.parametrize("case", [dict(NX=40), dict(NX=41, NY=37), dict(NX=40, is_steady=False, dt=1e-4)],
                         ids=["mode3", "odd", "transient"])
def test_calcrk_noalloc_matches_calcrk(oracle, case):
    import torch
    prob = mode3_model(oracle, **case)
    w = prob.wk
    rng = np.random.default_rng(5)
    w["theta"][1:-1, 1:-1, 1:-1] += rng.standard_normal(tuple(n - 2 for n in prob.shape))
    steady = prob.is_steady
    # the existing entry point (handle based)
    s = h2_b200.Solver(*prob.shape)
    s.set_grid(prob.ZC, prob.dZ, prob.dx, prob.dy, prob.dt, prob.HC, steady)
    s.set_fields(w["lam"], w["mask"], None if steady else w["rho"], None if steady else w["cp"])
    s.set_rhs(w["b"])
    s.set_theta(w["theta"])
    r_ref, res_ref = s.calc_rk()
    s.close()
    # the allocation-free entry point on device arrays the caller owns
    lib = L.load()
    d = {n: _dev(torch, w[n]) for n in ("theta", "b", "lam", "mask", "rho", "cp")}
    zc = torch.from_numpy(prob.ZC.copy()).cuda()
    dz = torch.from_numpy(prob.dZ.copy()).cuda()
    r = torch.zeros_like(d["theta"])
    HC = np.ascontiguousarray(prob.HC, dtype=np.float64)
    torch.cuda.synchronize()
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    for call in range(2):
        if call == 1:
            r.fill_(123.0)  # stale values must be overwritten on the interior
            torch.cuda.synchronize()
        res = C.c_double(0.0)
        st = lib.h2g_calcrk_noalloc(*prob.shape, ptr(d["theta"]), ptr(d["b"]), ptr(d["lam"]), ptr(d["mask"]),
                                    ptr(d["rho"]), ptr(d["cp"]), ptr(zc), ptr(dz), prob.dx, prob.dy, prob.dt,
                                    HC.ctypes.data_as(C.POINTER(C.c_double)), int(steady), ptr(r), C.byref(res),
                                    None)
        assert st == 0
        got = r.cpu().numpy().reshape(prob.shape, order="F")
        assert np.array_equal(got[1:-1, 1:-1, 1:-1], r_ref[1:-1, 1:-1, 1:-1])
        assert abs(res.value - res_ref) <= 1e-13 * res_ref


def test_calcrk_noalloc_rejects_oversized_grid():
    lib = L.load()
    HC = np.zeros(6)
    res = C.c_double(-1.0)
    one = C.c_void_p(16)  # never dereferenced: the size check comes first
    st = lib.h2g_calcrk_noalloc(10, 1002, 102, one, one, one, one, one, one, one, one, 1e-5, 1e-5, 1.0,
                                HC.ctypes.data_as(C.POINTER(C.c_double)), 1, one, C.byref(res), None)
    assert st == L.H2G_BAD_ARG and res.value == -1.0


class _Call:
    """A problem's arrays on the device and its call; the handle's residual and norm to compare with."""

    def __init__(self, prob, stream=None):
        import torch
        w = prob.wk
        self.prob = prob
        s = h2_b200.Solver(*prob.shape)
        s.set_grid(prob.ZC, prob.dZ, prob.dx, prob.dy, prob.dt, prob.HC, prob.is_steady)
        s.set_fields(w["lam"], w["mask"], *((None, None) if prob.is_steady else (w["rho"], w["cp"])))
        s.set_rhs(w["b"])
        s.set_theta(w["theta"])
        self.r_ref, self.res_ref = s.calc_rk()
        s.close()
        self.d = [_dev(torch, w[n]) for n in ("theta", "b", "lam", "mask", "rho", "cp")]
        self.z = [torch.from_numpy(a.copy()).cuda() for a in (prob.ZC, prob.dZ)]
        self.r = torch.zeros_like(self.d[0])
        self.HC = np.ascontiguousarray(prob.HC, dtype=np.float64)
        self.stream = stream
        torch.cuda.synchronize()

    def __call__(self):
        p = self.prob
        res = C.c_double(0.0)
        st = L.load().h2g_calcrk_noalloc(*p.shape, *(C.c_void_p(t.data_ptr()) for t in self.d + self.z), p.dx, p.dy,
                                         p.dt, self.HC.ctypes.data_as(C.POINTER(C.c_double)), int(p.is_steady),
                                         C.c_void_p(self.r.data_ptr()), C.byref(res),
                                         C.c_void_p(self.stream.cuda_stream) if self.stream else None)
        assert st == 0
        return res.value

    def residual(self):
        return self.r.cpu().numpy().reshape(self.prob.shape, order="F")[1:-1, 1:-1, 1:-1]


def test_calcrk_noalloc_calls_from_several_threads(oracle):
    """Calls on grids with different numbers of blocks, from threads with a stream each and from threads that
    share one: every call returns its own norm, and so do the calls after them."""
    import threading

    import torch
    shared = torch.cuda.Stream()
    sizes = [(41, 37, 30), (120, 90, 30), (24, 20, 30), (64, 130, 30)]
    calls = [_Call(mode3_model(oracle, *n), stream)
             for n, stream in zip(sizes, (shared, shared, torch.cuda.Stream(), None))]
    alone = [c() for c in calls]
    got = [[] for _ in calls]

    def work(q):
        for _ in range(100):
            got[q].append(calls[q]())

    ts = [threading.Thread(target=work, args=(q,)) for q in range(len(calls))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for q, c in enumerate(calls):
        assert got[q] == [alone[q]] * 100
        assert c() == alone[q] and abs(alone[q] - c.res_ref) <= 1e-13 * c.res_ref
        assert np.array_equal(c.residual(), c.r_ref[1:-1, 1:-1, 1:-1])


@pytest.mark.parametrize("transient", [False, True], ids=["steady", "transient"])
@pytest.mark.parametrize("n", [(1, 7, 3), (33, 1, 5), (128, 8, 2), (129, 9, 4), (257, 7, 3), (31, 17, 1), (96, 16, 30)],
                         ids=lambda n: "x".join(map(str, n)))
def test_calcrk_noalloc_shapes(oracle, n, transient):
    """Remainders of the blocks of 8 rows and 128 positions, one cell wide and one row, with five materials, masked
    cells inside and all boundary types: the oracle's residual to the bit, the norm, and again after a call on a
    grid with another number of blocks."""
    from test_gpu_boxes import box_problem
    prob = box_problem(oracle, *n, seed=sum(n), transient=transient)
    rng = np.random.default_rng(sum(n))
    inner = (slice(1, -1),) * 3
    m = prob.wk["mask"]
    m[inner] = np.where(rng.uniform(size=m[inner].shape) < 0.1, 0.0, 1.0)
    prob.wk["theta"][inner] += rng.standard_normal(m[inner].shape)
    r_ref, res_ref = oracle.calc_rk(prob)
    call, other = _Call(prob), _Call(mode3_model(oracle, 24, 20))
    want = other()
    for _ in range(2):
        res = call()
        assert np.array_equal(call.residual(), r_ref[inner])
        assert abs(res - res_ref) <= 1e-13 * res_ref
        assert other() == want
