"""The resident preconditioner (k_resident: Krylov update, 10 colour passes and CalcAX with its inner
products in one cooperative launch) against the oracle and against the separate launches.

It must give exactly the bits of the separate launches: the preconditioner is compared with
`array_equal` to the oracle for every number of rows per tile, planes per warp, ragged and one-tile
grids, masked cells and every boundary type; whole PBiCGSTAB and CG solves equal the colour-pass solves
(a forced launch shape selects those) bit for bit, residual history included.  A zero wait budget ends
the solve with H2G_TIMEOUT and the handle keeps working."""
import ctypes
import threading

import numpy as np
import pytest

import h2_b200
from h2_b200 import _lib as L
from conftest import mode3_model
from test_gpu_boxes import GRIDS, box_problem
from test_gpu_kernels import make_solver, random_interior

pytestmark = pytest.mark.gpu

# NX = 198..201 needs 4 tiles along the positions, so 37 tiles of rows: R = ceil(NY / 37)
SIZES = [(40, 40, 30), (41, 37, 30), (62, 63, 30), (200, 74, 30), (199, 100, 30), (201, 140, 30), (198, 181, 30),
         (200, 222, 30), (200, 230, 30), (254, 259, 30), (190, 290, 30), (126, 74, 60), (125, 147, 60), (129, 147, 60),
         (126, 290, 60)]


def launches_of(s, itr):
    return 2 + 3 * itr


@pytest.mark.parametrize("n", SIZES, ids=["x".join(map(str, n)) for n in SIZES])
def test_preconditioner_bit_exact(oracle, n):
    prob = mode3_model(oracle, n[0], n[1], n[2])
    s = make_solver(prob)
    bb = random_interior(prob.shape, sum(n))
    assert np.array_equal(s.preconditioner(bb, "gs"), oracle.preconditioner(prob, bb, "gs"))
    # quotients outside the range of the reciprocal steps: zeros, tiny, huge and subnormal numerators
    bb *= np.random.default_rng(1).choice([0.0, -0.0, 1e-150, 1e-310, 1e150, 1.0], prob.shape)
    assert np.array_equal(s.preconditioner(bb, "gs"), oracle.preconditioner(prob, bb, "gs"))
    s.close()


@pytest.mark.parametrize("grid", GRIDS, ids=["x".join(map(str, g)) for g in GRIDS])
def test_preconditioner_boxes(oracle, grid):
    prob = box_problem(oracle, *grid, seed=sum(grid) + 3)
    s = make_solver(prob)
    bb = random_interior(prob.shape, 5)
    assert np.array_equal(s.preconditioner(bb, "gs"), oracle.preconditioner(prob, bb, "gs"))
    s.close()


def test_preconditioner_masked_cells(oracle):
    prob = box_problem(oracle, 33, 31, 9, seed=22)
    m = prob.wk["mask"]
    inner = (slice(1, -1),) * 3
    m[inner] = np.where(np.random.default_rng(5).uniform(size=m[inner].shape) < 0.1, 0.0, 1.0)
    s = make_solver(prob)
    bb = random_interior(prob.shape, 6)
    assert np.array_equal(s.preconditioner(bb, "gs"), oracle.preconditioner(prob, bb, "gs"))
    s.close()


@pytest.mark.parametrize("n", [(41, 37, 30), (121, 70, 30), (198, 181, 30)], ids=lambda n: "x".join(map(str, n)))
def test_transient_grid(oracle, n):
    """a_p0 in the class table: the preconditioner gives the oracle's bits, a solve those of the colour passes,
    and a grid with more (key, rho cp) pairs than a class holds keeps the colour passes."""
    prob = mode3_model(oracle, n[0], n[1], n[2], is_steady=False, dt=1e-4)
    s = make_solver(prob)
    bb = random_interior(prob.shape, 8)
    assert np.array_equal(s.preconditioner(bb, "gs"), oracle.preconditioner(prob, bb, "gs"))
    s.snapshot()
    st, res = s.solve("pbicgstab", tol=1e-8, maxItr=100, smoother="gs")
    th = s.get_theta()
    assert res.launches == launches_of(s, res.itr)
    s.snapshot(restore=True)
    s.set_tuning(8, 2)
    assert s.solve("pbicgstab", tol=1e-8, maxItr=100, smoother="gs")[1].itr == res.itr
    assert np.array_equal(s.get_theta(), th)
    s.set_tuning(0)
    prob.wk["rho"][1:-1, 1:-1, 1:-1] *= 1.0 + 0.01 * np.random.default_rng(3).integers(0, 40, (n[0], n[1], n[2]))
    s.set_fields(prob.wk["lam"], prob.wk["mask"], prob.wk["rho"], prob.wk["cp"])
    assert np.array_equal(s.preconditioner(bb, "gs"), oracle.preconditioner(prob, bb, "gs"))
    st, res = s.solve("pbicgstab", tol=1e-8, maxItr=100, smoother="gs")
    assert res.launches != launches_of(s, res.itr)
    s.close()


@pytest.mark.parametrize("method", ["pbicgstab", "cg"])
@pytest.mark.parametrize("n", [(24, 20, 30), (41, 37, 30), (121, 117, 30), (200, 230, 30), (124, 140, 60)],
                         ids=lambda n: "x".join(map(str, n)))
def test_solve_identical(oracle, method, n):
    prob = mode3_model(oracle, n[0], n[1], n[2])
    cap = 20000 if n[0] < 150 else 60
    out = []
    for resident in (True, False):
        s = make_solver(prob)
        if not resident:
            s.set_tuning(8, 2)
        hist = np.zeros(cap)
        st, res = s.solve(method, tol=1e-8, maxItr=cap, smoother="gs", hist=hist)
        out.append((st, res.itr, res.res0, res.res, hist[:res.itr].copy(), s.get_theta()))
        per = (3, 2) if method == "pbicgstab" else (5, 4)
        assert (res.launches == per[1] + per[0] * res.itr) == resident
        s.close()
    assert out[0][:4] == out[1][:4]
    assert np.array_equal(out[0][4], out[1][4]) and np.array_equal(out[0][5], out[1][5])


def test_timeout_is_reported(oracle):
    prob = mode3_model(oracle, 40)
    ref = make_solver(prob)
    st, rr = ref.solve("pbicgstab", tol=1e-8, maxItr=20000, smoother="gs")
    assert st == 0 and rr.launches == launches_of(ref, rr.itr)
    s = make_solver(prob)
    s.snapshot()
    for _ in range(2):
        s.set_wait_limit(0)
        res = L.Result()
        st = L.load().h2g_pbicgstab(s.h, 1e-8, 200, 1, 0, None, ctypes.byref(res))
        assert st == L.H2G_TIMEOUT and res.status == L.H2G_TIMEOUT and not res.isconverged
        with pytest.raises(h2_b200.H2GError) as e:
            s.preconditioner(random_interior(prob.shape, 1), "gs")
        assert e.value.status == L.H2G_TIMEOUT
        s.set_wait_limit(2_000_000_000)
        s.snapshot(restore=True)
        st, res = s.solve("pbicgstab", tol=1e-8, maxItr=20000, smoother="gs")
        assert st == 0 and (res.itr, res.res) == (rr.itr, rr.res)
        assert np.array_equal(s.get_theta(), ref.get_theta())
    s.close()
    ref.close()


def test_two_threads(oracle):
    """Two host threads solving on their own handles and streams: the calls share the SMs in turn and
    each gives its lone solve's bits."""
    import torch
    prob = mode3_model(oracle, 62, 63)
    ref = make_solver(prob)
    _, rr = ref.solve("pbicgstab", tol=1e-8, maxItr=20000, smoother="gs")
    th = ref.get_theta()
    ref.close()
    got = [None, None]

    def work(q):
        stream = torch.cuda.Stream()
        s = make_solver(prob)
        L.check(s.lib.h2g_set_stream(s.h, ctypes.c_void_p(stream.cuda_stream)))
        s.snapshot()
        for _ in range(4):
            s.snapshot(restore=True)
            st, res = s.solve("pbicgstab", tol=1e-8, maxItr=20000, smoother="gs")
        got[q] = (st, res.itr, res.res, s.get_theta())
        s.close()

    ts = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for g in got:
        assert g[0] == 0 and g[1:3] == (rr.itr, rr.res)
        assert np.array_equal(g[3], th)


@pytest.mark.parametrize("threads", [2, 3])
def test_batch_shares(oracle, threads):
    """h2g_batch_solve: members on a share of the SMs beside each other, members that need them all, and one
    without a split; the handles alternate between a share and all SMs.  Always the lone solve's bits."""
    sizes = [(62, 63, 30), (200, 222, 30), (62, 63, 30), (121, 117, 30), (260, 40, 30), (41, 37, 30)]
    hs = [make_solver(mode3_model(oracle, *n)) for n in sizes]
    for s in hs:
        s.snapshot()
    ptr = (ctypes.c_void_p * len(hs))(*[s.h.value for s in hs])
    lone = None
    for _ in range(2):
        got = []
        for s in hs:
            s.snapshot(restore=True)
            st, res = s.solve("pbicgstab", tol=1e-8, maxItr=60, smoother="gs")
            got.append((res.itr, res.res, s.get_theta()))
            s.snapshot(restore=True)
        lone = lone or got
        outs = (L.Result * len(hs))()
        L.load().h2g_batch_solve(len(hs), ptr, 0, 1e-8, 60, 1, threads, outs)
        got += [(o.itr, o.res, s.get_theta()) for o, s in zip(outs, hs)]
        for q, g in enumerate(got):
            ref = lone[q % len(hs)]
            assert g[:2] == ref[:2] and np.array_equal(g[2], ref[2])
    for s in hs:
        s.close()


@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
def test_sor_identical(oracle, n):
    """solveSOR! with theta on the chip: field and residual history of the separate passes, bit for bit, for
    passes within a launch, a whole launch and more, and where the last test ends the solve."""
    prob = mode3_model(oracle, *n)
    s, ref = make_solver(prob), make_solver(prob)
    ref.set_tuning(8, 2)
    for omega, passes, tol in ((1.5, 1, 0.0), (1.0, 32, 0.0), (1.5, 71, 0.0), (1.0, 60, 0.5)):
        out = []
        for q in (s, ref):
            q.set_theta(prob.wk["theta"])
            hist = np.zeros(passes)
            st, res = q.sor(omega=omega, tol=tol, maxItr=passes, hist=hist)
            out.append((st, res.itr, res.res0, res.res, hist, q.get_theta()))
        assert res.launches == 2 + 2 * res.itr
        assert out[0][:4] == out[1][:4]
        assert np.array_equal(out[0][4], out[1][4]) and np.array_equal(out[0][5], out[1][5])
    s.set_wait_limit(0)
    res = L.Result()
    assert L.load().h2g_sor(s.h, 1.0, 0.0, 20, 0, None, ctypes.byref(res)) == L.H2G_TIMEOUT
    s.set_wait_limit(2_000_000_000)
    s.set_theta(prob.wk["theta"])
    s.sor(omega=1.0, tol=0.5, maxItr=60)
    assert np.array_equal(s.get_theta(), out[0][5])
    s.close()
    ref.close()


@pytest.mark.parametrize("grid", GRIDS, ids=["x".join(map(str, g)) for g in GRIDS])
def test_sor_boxes(oracle, grid):
    prob = box_problem(oracle, *grid, seed=sum(grid) + 3)
    s, ref = make_solver(prob), make_solver(prob)
    ref.set_tuning(8, 2)
    out = []
    for q in (s, ref):
        hist = np.zeros(40)
        st, res = q.sor(omega=1.3, tol=0.0, maxItr=40, hist=hist)
        out.append((res.itr, hist, q.get_theta()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1], equal_nan=True) and np.array_equal(out[0][2], out[1][2], equal_nan=True)
    s.close()
    ref.close()


@pytest.mark.parametrize("n", [(41, 37, 30), (198, 181, 30), (200, 222, 30), (129, 147, 60), (126, 290, 60)],
                         ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_preconditioner_reads_only_updated_cells(oracle, n, bad):
    """Guards and masked cells of bb may hold anything, as in the separate passes, which never read them; and
    what is not finite in an updated cell stays out of the masked ones."""
    prob = mode3_model(oracle, n[0], n[1], n[2])
    rng = np.random.default_rng(3)
    masked = np.zeros(prob.shape, dtype=bool)
    masked[1:-1, 1:-1, 1:-1] = rng.uniform(size=(n[0], n[1], n[2])) < 0.0005
    prob.wk["mask"][masked] = 0.0
    guards = np.ones(prob.shape, dtype=bool)
    guards[1:-1, 1:-1, 1:-1] = False
    clean = random_interior(prob.shape, 4)
    clean[masked] = 0.0
    dirty = clean.copy(order="F")
    dirty[guards | masked] = bad
    inside = clean.copy(order="F")
    inside[n[0] // 2, n[1] // 2, n[2] // 2] = bad
    s, ref = make_solver(prob), make_solver(prob)
    ref.set_tuning(8, 2)
    want = ref.preconditioner(clean, "gs")
    assert np.isfinite(want).all()
    assert np.array_equal(s.preconditioner(clean, "gs"), want)
    assert np.array_equal(s.preconditioner(dirty, "gs"), want)
    assert np.array_equal(s.preconditioner(inside, "gs"), ref.preconditioner(inside, "gs"), equal_nan=True)
    s.close()
    ref.close()


class _FilledDevice:
    """Takes the device's free memory but for about `leave` bytes."""

    def __init__(self, leave):
        import torch
        torch.cuda.empty_cache()
        self.rt = ctypes.CDLL("libcudart.so.12")
        self.held = []
        for chunk in (1 << 30, 1 << 26, 1 << 21):
            while torch.cuda.mem_get_info()[0] > leave + chunk:
                p = ctypes.c_void_p()
                if self.rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(chunk)):
                    self.rt.cudaGetLastError()
                    break
                self.held.append(p)

    def release(self):
        for p in self.held:
            self.rt.cudaFree(p)
        self.held = []


def test_without_memory_for_the_buffers(oracle, monkeypatch):
    """A device without room for the messages of the tiles: the solve takes the separate passes, again on the next
    call, and the resident form once there is room."""
    import torch
    prob = mode3_model(oracle, 254, 296)
    s = make_solver(prob)
    s.snapshot()
    monkeypatch.setenv("H2G_RB_COOP", "0")  # the separate passes: tuned and captured
    st, ref = s.solve("pbicgstab", tol=1e-8, maxItr=8, smoother="gs")
    th = s.get_theta()
    monkeypatch.delenv("H2G_RB_COOP")
    held = _FilledDevice(12 << 20)
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        s.snapshot(restore=True)
        st2, res = s.solve("pbicgstab", tol=1e-8, maxItr=8, smoother="gs")
        assert (st2, res.itr, res.res) == (st, ref.itr, ref.res) and res.launches == ref.launches
        assert np.array_equal(s.get_theta(), th)
    assert free < 15 << 20 and torch.cuda.mem_get_info()[0] >= free - (2 << 20)  # no buffer is kept
    held.release()
    s.snapshot(restore=True)
    st2, res = s.solve("pbicgstab", tol=1e-8, maxItr=8, smoother="gs")
    assert (st2, res.itr, res.res) == (st, ref.itr, ref.res) and res.launches == launches_of(s, res.itr)
    assert np.array_equal(s.get_theta(), th)
    s.close()


def test_fields_on_a_full_device(oracle):
    """h2g_set_fields of a transient grid on a device with little or no memory left either works, without what
    there is no room for, or reports the failed allocation; once there is room the same handle works in full."""
    prob = mode3_model(oracle, 200, 190, is_steady=False, dt=1e-4)
    w = prob.wk
    bb = random_interior(prob.shape, 2)
    want = oracle.preconditioner(prob, bb, "gs")
    for leave in (0, 4, 10, 16, 24, 40):
        s = h2_b200.Solver(*prob.shape)
        s.set_grid(prob.ZC, prob.dZ, prob.dx, prob.dy, prob.dt, prob.HC, False)
        full = _FilledDevice(leave << 20)
        try:
            s.set_fields(w["lam"], w["mask"], w["rho"], w["cp"])
        except h2_b200.H2GError as e:
            assert e.status == L.H2G_CUDA_ERROR
        full.release()
        s.set_fields(w["lam"], w["mask"], w["rho"], w["cp"])
        assert np.array_equal(s.preconditioner(bb, "gs"), want), leave
        s.close()


# grids of uniform layers: (NX, NY, NZ), then whether PBiCGSTAB, CG and SOR are resident
ROUTES = [((240, 240, 14), (0, 0, 1)), ((240, 240, 15), (1, 0, 1)), ((240, 240, 17), (1, 1, 1)),
          ((240, 240, 2), (0, 0, 0)), ((180, 180, 7), (0, 0, 0)), ((180, 180, 8), (1, 0, 1)),
          ((90, 212, 3), (0, 0, 0)), ((90, 212, 4), (1, 0, 1)), ((90, 212, 10), (1, 1, 1)),
          ((124, 140, 1), (1, 1, 1)), ((180, 180, 31), (0, 0, 1)), ((180, 180, 33), (1, 0, 1)),
          ((120, 120, 32), (0, 0, 1)), ((120, 120, 35), (1, 1, 1)), ((70, 70, 33), (1, 1, 1)), ((60, 60, 45), (0, 0, 0)),
          ((63, 148, 30), (1, 1, 1)), ((127, 120, 29), (1, 1, 1)), ((254, 290, 27), (1, 1, 1)),
          ((127, 147, 57), (1, 0, 1))]


@pytest.mark.parametrize("n,resident", ROUTES, ids=["x".join(map(str, r[0])) for r in ROUTES])
def test_routes(oracle, n, resident):
    """Both sides of the rule by rows and planes, odd numbers of planes beyond 30 and tiles along the positions whose
    last one holds nothing but a guard: the route, and the separate passes' bits."""
    prob = box_problem(oracle, *n, seed=1)
    w = prob.wk
    w["lam"][...] = np.array([0.4, 1.5, 50.0, 149.0])[np.arange(prob.shape[2]) // 2 % 4][None, None, :]
    s, ref = make_solver(prob), make_solver(prob)
    ref.set_tuning(8, 2)
    bb = random_interior(prob.shape, 7)
    assert np.array_equal(s.preconditioner(bb, "gs"), ref.preconditioner(bb, "gs"))
    for method, route in zip(("pbicgstab", "cg", "sor"), resident):
        got = []
        for q in (s, ref):
            q.set_theta(w["theta"])
            hist = np.zeros(6)
            if method == "sor":
                st, res = q.sor(omega=1.2, tol=0.0, maxItr=6, hist=hist)
            else:
                st, res = q.solve(method, tol=0.0, maxItr=6, smoother="gs", hist=hist)
            got.append((st, res.itr, hist, q.get_theta(), res.launches))
        assert got[0][:2] == got[1][:2]
        assert np.array_equal(got[0][2], got[1][2]) and np.array_equal(got[0][3], got[1][3])
        assert (got[0][4] != got[1][4]) == bool(route), method
    s.close()
    ref.close()


@pytest.mark.parametrize("passes,resident", [(1, False), (2, False), (5, False), (6, True), (33, True)])
def test_sor_of_few_passes(oracle, passes, resident):
    """A call of up to 5 passes does not pay for the tiles' set-up: it takes the separate passes."""
    prob = mode3_model(oracle, 41, 37)
    s, ref = make_solver(prob), make_solver(prob)
    ref.set_tuning(8, 2)
    got = [q.sor(omega=1.3, tol=0.0, maxItr=passes) + (q.get_theta(),) for q in (s, ref)]
    assert got[0][0] == got[1][0] and got[0][1].res == got[1][1].res and got[0][1].itr == passes
    assert np.array_equal(got[0][2], got[1][2])
    assert got[1][1].launches == 2 + 2 * passes
    assert got[0][1].launches == (2 + (passes + 31) // 32 if resident else 2 + 2 * passes)
    s.close()
    ref.close()


@pytest.mark.parametrize("method", [0, 1, 2], ids=["pbicgstab", "cg", "sor"])
def test_batch_parts(oracle, method):
    """Eight threads: parts of the SMs for up to 4 (CG 8) members at a time, all of them in turn, or the separate
    passes where those are faster beside each other (SOR of more than 4, CG that needs all SMs).  Twice, so that
    the splits of a handle alternate; always the lone call's bits."""
    sizes = [(62, 63), (200, 222), (121, 117), (41, 37), (62, 63), (121, 117), (24, 20), (41, 37)]
    hs = [make_solver(mode3_model(oracle, *n)) for n in sizes]
    ptr = (ctypes.c_void_p * len(hs))(*[s.h.value for s in hs])
    lone = []
    for s in hs:
        s.snapshot()
        res = s.solve("cg" if method else "pbicgstab", tol=1e-8, maxItr=40)[1] if method < 2 else \
            s.sor(tol=1e-8, maxItr=40)[1]
        lone.append((res.itr, res.res, s.get_theta(), res.launches))
    for _ in range(2):
        for s in hs:
            s.snapshot(restore=True)
        outs = (L.Result * len(hs))()
        L.load().h2g_batch_solve(len(hs), ptr, method, 1e-8, 40, 1, 8, outs)
        for q, (o, s) in enumerate(zip(outs, hs)):
            assert (o.itr, o.res) == lone[q][:2] and np.array_equal(s.get_theta(), lone[q][2])
            separate = method == 2 or (method == 1 and sizes[q] == (200, 222))
            assert (o.launches != lone[q][3]) == separate
    for s in hs:
        s.close()


def test_threads_on_parts(oracle):
    """Host threads on streams of their own get parts of the SMs, threads that share the default stream take all of
    them in turn; a thread's split changes with what is in flight.  Each call gives its lone call's bits."""
    import torch
    sizes = [(62, 63), (41, 37), (121, 117), (62, 63), (24, 20), (121, 117)]
    probs = [mode3_model(oracle, *n) for n in sizes]
    lone, got = [], [[] for _ in sizes]

    def call(s):
        s.snapshot(restore=True)
        st, res = s.solve("pbicgstab", tol=1e-8, maxItr=50, smoother="gs")
        out = (st, res.itr, res.res)
        th = s.get_theta()
        st, res = s.sor(tol=0.0, maxItr=20)
        return out + (res.res, th, s.get_theta())

    for p in probs:
        s = make_solver(p)
        s.snapshot()
        lone.append(call(s))
        s.close()

    def work(q):
        s = make_solver(probs[q])
        if q < 4:
            stream = torch.cuda.Stream()
            L.check(s.lib.h2g_set_stream(s.h, ctypes.c_void_p(stream.cuda_stream)))
        s.snapshot()
        for _ in range(6):
            got[q].append(call(s))
        s.close()

    ts = [threading.Thread(target=work, args=(q,)) for q in range(len(sizes))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for ref, out in zip(lone, got):
        assert len(out) == 6
        for g in out:
            assert g[:4] == ref[:4] and np.array_equal(g[4], ref[4]) and np.array_equal(g[5], ref[5])


def test_transient_grid_with_another_step(oracle):
    """h2g_set_grid with another time step keeps the (key, rho cp) pairs of the fields and makes the classes anew;
    h2g_set_fields finds the pairs again, too many of them included."""
    prob = mode3_model(oracle, 41, 37, is_steady=False, dt=1e-4)
    w = prob.wk
    s = make_solver(prob)
    bb = random_interior(prob.shape, 9)
    rng = np.random.default_rng(4)
    for scale, many, resident in ((1.0, False, True), (1.7, False, True), (1.7, True, False), (0.6, False, True)):
        w["rho"][1:-1, 1:-1, 1:-1] *= scale * (1.0 + 0.01 * rng.integers(0, 40, (41, 37, 30)) if many else scale)
        if not many:
            w["rho"][...] = np.round(w["rho"], -2) + 100.0
            w["cp"][...] = np.round(w["cp"], -3) + 1000.0
            w["rho"][1:-1, 1:-1, 1:-1] = np.where(w["lam"][1:-1, 1:-1, 1:-1] > 1.0, 8000.0 * scale, 2000.0)
        s.set_fields(w["lam"], w["mask"], w["rho"], w["cp"])
        for dt in (1e-4, 3e-5, 2e-3):
            prob.dt = dt
            s.set_grid(prob.ZC, prob.dZ, prob.dx, prob.dy, dt, prob.HC, False)
            assert np.array_equal(s.preconditioner(bb, "gs"), oracle.preconditioner(prob, bb, "gs")), (scale, many, dt)
            s.set_theta(w["theta"])
            st, res = s.solve("pbicgstab", tol=0.0, maxItr=3, smoother="gs")
            assert (res.launches == launches_of(s, res.itr)) == resident
    s.close()


def test_switches(oracle, monkeypatch):
    """What turns the resident form off, and back: the calls and the variables that ask for a variant of the
    separate passes, as include/h2g.h lists them."""
    prob = mode3_model(oracle, 41, 37)
    s = make_solver(prob)
    s.snapshot()

    def forms():
        out = []
        for method, launches in (("pbicgstab", 2 + 3 * 5), ("sor", 2 + 1)):
            s.snapshot(restore=True)
            res = s.sor(tol=0.0, maxItr=6)[1] if method == "sor" else s.solve(method, tol=0.0, maxItr=5)[1]
            out.append(res.launches == launches)
        assert out[0] == out[1]
        return out[0]

    assert forms()
    for off, back in ((lambda: s.set_tuning(8, 2), lambda: s.set_tuning(0)),
                      (lambda: s.set_sweep(0), lambda: s.set_sweep(-1)),
                      (lambda: s.set_sweep(1, 2), lambda: s.set_sweep(-1)),
                      (lambda: s.set_coop(0), lambda: s.set_coop(-1)), (lambda: s.set_coop(1), lambda: s.set_coop(-1))):
        off()
        assert not forms()
        back()
        assert forms()
    for name in ("H2G_RB_ROWS", "H2G_RB_PLANES", "H2G_RB_DD", "H2G_AX_DD", "H2G_RB_FUSED", "H2G_SW_CHUNKS", "H2G_SW_DD",
                 "H2G_RB_COOP"):
        monkeypatch.setenv(name, "0")
        assert not forms(), name
        monkeypatch.delenv(name)
    s.autotune(), s.sweep(), s.coop()  # asking turns nothing off
    assert forms()
    s.close()


def test_messages_are_counted_anew(oracle):
    """Calls that may take so many iterations that the messages' numbers are counted anew every few of them, with
    both Krylov methods, SOR and the preconditioner between: always the first call's bits."""
    prob = mode3_model(oracle, 24, 20)
    s = make_solver(prob)
    s.snapshot()
    bb = random_interior(prob.shape, 3)
    first = None
    for _ in range(9):
        got = []
        for method in ("pbicgstab", "cg"):
            s.snapshot(restore=True)
            st, res = s.solve(method, tol=1e-4, maxItr=10_000_000, smoother="gs")
            got += [st, res.itr, res.res, s.get_theta()]
        s.snapshot(restore=True)
        st, res = s.sor(tol=0.5, maxItr=10_000_000)
        got += [st, res.itr, res.res, s.get_theta(), s.preconditioner(bb, "gs")]
        first = first or got
        assert all(np.array_equal(a, b) for a, b in zip(first, got))
    s.close()
