"""Runs of steps with the blocks resident in shared memory (AUTO, from a few
steps per call on, any uniform grid) against the one-CTA-per-block kernel, bit
for bit: one block that is its own neighbour, block counts that are no power
of two, tumour outside the anatomy (empty blocks whose cells react by
themselves), values below 0 and above 1, tissue fractions below 0.1 (cells
that read p_w and p_g), every launch shape and the fallback of grids whose
blocks do not fit."""
import threading

import numpy as np
import pytest

from gliomasolver_b200 import BlockPool, GbfkError
from gliomasolver_b200.anatomy import make_case
from gliomasolver_b200.schedule import make_schedule

pytestmark = pytest.mark.gpu


def _fields(n, seed, prec):
    R = np.float64 if prec == "f64" else np.float32
    pw, pg, c0, _ = make_case(n, seed)
    rng = np.random.default_rng(seed + 50)
    c0 = np.maximum(c0, rng.uniform(0, 1, c0.shape) * (rng.uniform(0, 1, c0.shape) < 0.03))
    c0[0, 0, :] = 1.7
    c0[1, :, 2] = -0.3
    pw[n // 2, :, : n // 3] = 0.0
    pg[n // 2, :, : n // 3] = 0.0
    thin = rng.uniform(0, 1, c0.shape) < 0.02
    pw[thin] *= 0.08
    pg[thin] *= 0.08
    return [a.astype(R) for a in (pw, pg, c0)]


def _pool(n, prec, fields, stream=None):
    pool = BlockPool((n // 8) ** 3, prec, stream=stream)
    pool.set_uniform(n // 8)
    for name, a in zip(("p_w", "p_g", "phi"), fields):
        pool.upload_dense(name, a)
    return pool


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n,seed,steps", [(8, 3, 7), (16, 2, 30), (24, 1, 4), (72, 5, 9), (128, 1, 40), (168, 2, 5)])
def test_resident_run_equals_block_steps(gbfk_lib, prec, n, seed, steps):
    fields = _fields(n, seed, prec)
    s = make_schedule(0.3, 0.2, 300.0, 25.6, n // 8, prec)
    with _pool(n, prec, fields) as a, _pool(n, prec, fields) as b:
        b.step_kernel = "block"
        # the second call starts from a clamped state, the third from an
        # uploaded one again; the face phase goes on from call to call
        for k, again in ((steps, False), (steps + 3, False), (steps, True)):
            for p in (a, b):
                if again:
                    p.upload_dense("phi", fields[2])
                p.rd_step(s.Dw, s.Dg, s.rho, s.dt, k, check_nan=True)
            assert np.array_equal(a.download_dense("phi"), b.download_dense("phi"))
        # 168^3 in FP64 has more heavy blocks than the SMs hold
        if (n, prec) != (168, "f64") and steps > 6:
            assert a.step_kernel == "run"


def test_steps_that_leave_out_the_empty_blocks(gbfk_lib):
    """256^3 does not fit: launches over the blocks with tissue, the empty
    blocks' steps (some hold tumour) in one launch, odd and even step counts."""
    n, prec = 256, "f32"
    fields = _fields(n, 4, prec)
    s = make_schedule(0.3, 0.2, 300.0, 25.6, n // 8, prec)
    with _pool(n, prec, fields) as a, _pool(n, prec, fields) as b:
        b.step_kernel = "block"
        for k in (4, 3, 5):
            for p in (a, b):
                p.rd_step(s.Dw, s.Dg, s.rho, s.dt, k, check_nan=True)
            assert np.array_equal(a.download_dense("phi"), b.download_dense("phi"))


@pytest.mark.parametrize("n", [32, 56])
def test_nan_in_a_resident_run_is_reported(gbfk_lib, n):
    fields = _fields(n, 1, "f32")
    fields[2][n // 2, n // 2, n // 2] = np.nan
    s = make_schedule(0.2, 0.05, 300.0, 25.6, n // 8, "f32")
    with _pool(n, "f32", fields) as pool:
        with pytest.raises(GbfkError) as e:
            pool.rd_step(s.Dw, s.Dg, s.rho, s.dt, 20, check_nan=True)
        assert e.value.code == 4


def test_resident_run_replayed_from_a_graph(gbfk_lib):
    """A run captured in a CUDA graph and replayed, with runs outside the
    graph in between: the state count on the device keeps the face phase."""
    import torch

    n, prec = 48, "f32"
    fields = _fields(n, 6, prec)
    s = make_schedule(0.2, 0.05, 300.0, 25.6, n // 8, prec)
    st = torch.cuda.Stream()
    with _pool(n, prec, fields, st.cuda_stream) as a, _pool(n, prec, fields) as b:
        b.step_kernel = "block"
        a.rd_step(s.Dw, s.Dg, s.rho, s.dt, 8)
        a.sync()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            a.rd_step(s.Dw, s.Dg, s.rho, s.dt, 7)
        total = 8
        for _ in range(3):
            with torch.cuda.stream(st):
                g.replay()
            a.rd_step(s.Dw, s.Dg, s.rho, s.dt, 9)
            total += 16
        b.rd_step(s.Dw, s.Dg, s.rho, s.dt, total)
        a.sync()
        assert np.array_equal(a.download_dense("phi"), b.download_dense("phi"))
        del g


def test_two_pools_from_two_threads(gbfk_lib):
    """Two contexts stepped from two threads at once, each in many runs."""
    cases = [(64, "f32", 3), (96, "f64", 4)]
    want, got, errors = {}, {}, []

    def go(n, prec, seed, kind, out):
        try:
            fields = _fields(n, seed, prec)
            s = make_schedule(0.2, 0.05, 300.0, 25.6, n // 8, prec)
            with _pool(n, prec, fields) as pool:
                pool.step_kernel = kind
                for _ in range(25):
                    pool.rd_step(s.Dw, s.Dg, s.rho, s.dt, 20)
                pool.sync()
                out[n] = pool.download_dense("phi")
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    for c in cases:
        go(*c, "block", want)
    threads = [threading.Thread(target=go, args=(*c, "auto", got)) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for n, _, _ in cases:
        assert np.array_equal(got[n], want[n])


@pytest.mark.parametrize("prec,bpd,samples", [("f64", 5, 9), ("f32", 12, 3), ("f32", 3, 40)])
def test_stage_of_resident_runs_equals_steps_by_launches(gbfk_lib, prec, bpd, samples):
    """A stage by teams of CTAs (block counts that are no power of two, two
    anatomies per team, both initial conditions, horizons from 0 steps on)
    against the per-block kernel, twice on one batch."""
    from gliomasolver_b200.tmcmc import Batch, sample_stage, to_gbfk_samples

    R = np.float64 if prec == "f64" else np.float32
    n = 8 * bpd
    anat = [make_case(n, seed)[:2] for seed in (0, 5)]
    anat[1] = tuple(a * 0.9 for a in anat[1])
    stage = sample_stage(samples, anat[0][0], seed=2, tend_range=(1.0, 60.0))
    recs, _ = to_gbfk_samples(stage, bpd, prec, anatomy=[i % 2 for i in range(samples)])
    for i, r in enumerate(recs):
        r.nsteps = min(r.nsteps, 60) * (i != 1)
        r.ic = i % 3 == 2
    with Batch(bpd, samples, prec, max_anatomies=2) as b:
        for i, (pw, pg) in enumerate(anat):
            b.set_anatomy(i, pw.astype(R), pg.astype(R))
        for _ in range(2):
            b.set_samples(recs)
            b.run(1)
            want = [b.download(i) for i in range(samples)]
            b.set_samples(recs)
            b.run(0)
            assert b.samples_per_cta == -1 and b.graph_count == 1
            for i in range(samples):
                assert np.array_equal(b.download(i), want[i]), i
            for r in recs:  # other step counts and horizons the second time
                r.nsteps += 3
    assert max(w.max() for w in want) > 0.1


@pytest.mark.parametrize("prec,n", [("f32", 176), ("f64", 144), ("f64", 160)])
def test_steps_over_the_heavy_blocks_equal_the_block_kernel(gbfk_lib, prec, n):
    """Grids whose heavy blocks do not fit the SMs: calls too short for their own tables, odd and even step counts, an
    unclamped first state, tumour in empty blocks, cells of every class, and new coefficients on the same pool."""
    pw, pg, c0, _ = make_case(n, 3)
    rng = np.random.default_rng(n)
    c0 = np.maximum(c0, rng.uniform(0, 1, c0.shape) * (rng.uniform(0, 1, c0.shape) < 0.03))
    c0[0, 0, :], c0[1, :, 2] = 1.7, -0.3
    sel = rng.uniform(0, 1, c0.shape) < 0.02
    pw[sel] *= 0.08
    pg[sel] *= 0.08
    R = np.float64 if prec == "f64" else np.float32
    pw, pg, c0 = (a.astype(R) for a in (pw, pg, c0))
    out = {}
    for kind in ("block", "auto"):
        with _pool(n, prec, (pw, pg, c0)) as pool:
            pool.step_kernel = kind
            got = []
            for Dw, steps in ((0.3, 7), (0.3, 4), (0.3, 2), (0.15, 7)):
                s = make_schedule(Dw, 0.2, 300.0, 25.6, n // 8, prec)
                pool.rd_step(s.Dw, s.Dg, s.rho, s.dt, steps, check_nan=True)
                got.append(pool.download_dense("phi"))
                if steps > 3:
                    assert pool.step_kernel == ("block" if kind == "block" else "pipelined")
        out[kind] = got
    for a, b in zip(out["auto"], out["block"]):
        assert np.array_equal(a, b)


def _ball_value(R, x, centre):
    """The smoothed ball's value at a cell with the centre's y and z, formed in
    Real as the reference does."""
    p = R(R(x) - R(centre))
    psi = R(R(np.sqrt(R(p * p)) - R(0.005)) * R(64))
    return R(0.5 * (float(R(R(1) - psi)) - np.sin(np.pi * float(psi)) / np.pi))


@pytest.mark.parametrize("prec,bpd", [("f32", 8), ("f64", 8), ("f32", 6), ("f32", 12)])
def test_stage_of_balls_with_a_negative_value_at_a_block_face(gbfk_lib, prec, bpd):
    """The ball's profile rounds below 0 where psi is next to 1; the first cell
    of a block is such a one, and its sign crosses the face like any other's."""
    from gliomasolver_b200.tmcmc import Batch, StageSample, to_gbfk_samples

    R = np.float64 if prec == "f64" else np.float32
    n = 8 * bpd
    spacing = 1 / (8 << int(np.ceil(np.log2(bpd))))
    centres, x = [], R(16 * spacing + 0.005 + 1 / 64)
    for _ in range(4000):
        if _ball_value(R, 16 * spacing, x) < 0:
            centres.append(float(x))
        x = np.nextafter(x, R(0))
    y = 12 * spacing
    stage = [StageSample(0.2, 0.1, 20.0, (c, y, y)) for c in (centres[0], centres[-1])]
    stage += [StageSample(0.1, 0.05, 9.0, (0.4, 0.3, 0.3)), stage[0]]
    recs, _ = to_gbfk_samples(stage, bpd, prec, ic="ball")
    pw = np.full((n, n, n), 0.7, dtype=R)
    with Batch(bpd, len(recs), prec, max_anatomies=1) as b:
        b.set_anatomy(0, pw, (1 - pw).astype(R))
        for nsteps in ((0, 0, 0, 0), (1, 6, 9, 0), (2, 1, 0, 5)):
            for r, k in zip(recs, nsteps):
                r.nsteps = k
            out = []
            for kind in (1, 0):
                b.set_samples(recs)
                b.run(kind)
                out.append([b.download(i) for i in range(len(recs))])
            assert b.samples_per_cta == -1 or max(nsteps) == 0
            if max(nsteps) == 0:
                assert out[0][0][12, 12, 16] < 0 and out[0][0][12, 12, 15] == 0
            for i, (want, got) in enumerate(zip(*out)):
                assert np.array_equal(got, want), (nsteps, i)


@pytest.mark.parametrize("prec,n", [("f32", 64), ("f64", 72), ("f32", 152)])
def test_new_coefficients_keep_the_lists_and_a_new_anatomy_does_not(gbfk_lib, prec, n):
    """Calls with other coefficients, then with another anatomy too, resident
    and over the heavy blocks, against the block kernel."""
    fields, other = _fields(n, 3, prec), _fields(n, 8, prec)
    other[0][: n // 3] = 0
    other[1][: n // 3] = 0
    with _pool(n, prec, fields) as a, _pool(n, prec, fields) as b:
        b.step_kernel = "block"
        for k, Dw in enumerate((0.3, 0.1, 0.1, 0.22, 0.05)):
            s = make_schedule(Dw, 0.2, 300.0, 25.6, n // 8, prec)
            for p in (a, b):
                if k == 3:
                    p.upload_dense("p_w", other[0])
                    p.upload_dense("p_g", other[1])
                p.rd_step(s.Dw, s.Dg, s.rho, s.dt, 9, check_nan=True)
            assert np.array_equal(a.download_dense("phi"), b.download_dense("phi")), k


@pytest.mark.parametrize("n", [64, 72])
def test_new_coefficients_do_not_block_the_host(gbfk_lib, n):
    """A call with new coefficients on a known anatomy is enqueued behind 0.2 s
    of other work on the stream without waiting for it."""
    import time

    import torch

    fields = _fields(n, 1, "f32")
    st = torch.cuda.Stream()
    with _pool(n, "f32", fields, st.cuda_stream) as pool:
        def step(Dw):
            s = make_schedule(Dw, 0.1, 100.0, 25.6, n // 8, "f32")
            pool.rd_step(s.Dw, s.Dg, s.rho, s.dt, 12)

        step(0.2)
        step(0.2)
        pool.sync()
        done = torch.cuda.Event()
        t0 = time.perf_counter()
        with torch.cuda.stream(st):
            torch.cuda._sleep(400_000_000)  # cycles: at least 0.2 s
        step(0.1)
        step(0.15)
        returned = time.perf_counter() - t0
        done.record(st)
        pending = not done.query()
        pool.sync()
        assert pending and returned < 0.1 < time.perf_counter() - t0
        assert pool.step_kernel == "run"


def test_a_short_call_on_a_new_anatomy_builds_no_lists(gbfk_lib):
    """Grids that are no power of two: the block kernel needs no lists, and a
    few steps do not pay for them; where they are there, they are used."""
    n = 72
    fields = _fields(n, 2, "f32")
    s = make_schedule(0.2, 0.1, 300.0, 25.6, n // 8, "f32")
    with _pool(n, "f32", fields) as pool:
        for upload, steps, kernel in ((False, 5, "block"), (False, 9, "run"), (False, 4, "run"), (True, 5, "block"),
                                      (True, 12, "run"), (False, 3, "run")):
            if upload:
                pool.upload_dense("p_w", fields[0])
            pool.rd_step(s.Dw, s.Dg, s.rho, s.dt, steps)
            assert pool.step_kernel == kernel


class _FullDevice:
    """Every byte of device memory that cudaMalloc still gives, down to its
    smallest pieces, held until the end of the block."""

    def __enter__(self):
        import ctypes

        self.rt = ctypes.CDLL("libcudart.so.12")
        self.held, size = [], 1 << 36
        while size >= 256:
            p = ctypes.c_void_p()
            if len(self.held) < 20000 and self.rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
                self.held.append(p)
            else:
                self.rt.cudaGetLastError()
                size //= 2
        return self

    def __exit__(self, *exc):
        for p in self.held:
            self.rt.cudaFree(p)


def test_runs_without_room_for_their_tables_take_the_launches(gbfk_lib):
    """No device memory left: a call of several steps on a grid that is no
    power of two (its lists), and a gradient whose sweep got longer (its
    pointer table), run with a launch per step, which need neither."""
    n = 72
    fields = _fields(n, 2, "f32")
    s = make_schedule(0.2, 0.1, 300.0, 25.6, n // 8, "f32")
    g = 32
    gf = _fields(g, 2, "f32")
    gf[2] = np.clip(gf[2], 0, 1) * (gf[0] + gf[1] > 0)
    gs = make_schedule(0.2, 0.1, 300.0, 25.6, g // 8, "f32")
    masks = (gf[2] > 0.2).astype(float), (gf[2] > 0.1).astype(float)

    def gradient(pool, steps, kind):
        pool.step_kernel = kind
        return pool.forward_adjoint(gs.Dw, gs.Dg, gs.rho, 0.2 * gs.dt, steps, sigma=0.0, nsnapshots=4, grad_c0=True,
                                    t1_uc=0.7, t2_uc=0.25, slope=2.0)

    with _pool(n, "f32", fields) as warm, _pool(n, "f32", fields) as pool, _pool(g, "f32", gf) as grad:
        grad.set_observations(*masks)
        want_g = gradient(grad, 150, "pipelined")
        gradient(grad, 8, "auto")  # the runs' buffers, a short table
        warm.rd_step(s.Dw, s.Dg, s.rho, s.dt, 20)
        assert warm.step_kernel == "run"
        warm.step_kernel = "block"
        warm.upload_dense("phi", fields[2])
        warm.rd_step(s.Dw, s.Dg, s.rho, s.dt, 21)
        want = warm.download_dense("phi")
        pool.rd_step(s.Dw, s.Dg, s.rho, s.dt, 1)  # the coefficients, no lists
        pool.sync()
        with _FullDevice():
            pool.rd_step(s.Dw, s.Dg, s.rho, s.dt, 20)
            pool.sync()
            kernel = pool.step_kernel
            got_g = gradient(grad, 150, "auto")
        assert kernel == "block"
        assert np.array_equal(pool.download_dense("phi"), want)
        again = gradient(grad, 150, "auto")
    for got in (got_g, again):
        assert np.array_equal(got["grad_c0"], want_g["grad_c0"]) and got["loss"] == want_g["loss"]


@pytest.mark.parametrize("n", [64, 72, 176])
def test_a_runs_tables_leave_another_threads_capture_alone(gbfk_lib, n):
    """The first call of several steps on a pool (lists, exchange buffers,
    images), made while another thread captures a stream in the global mode."""
    import torch

    fields = _fields(n, 3, "f32")
    s = make_schedule(0.2, 0.1, 300.0, 25.6, n // 8, "f32")
    x = torch.zeros(100, device="cuda")
    with _pool(n, "f32", fields) as a, _pool(n, "f32", fields) as b:
        b.step_kernel = "block"
        a.rd_step(s.Dw, s.Dg, s.rho, s.dt, 1)
        a.sync()
        errors, graph = [], torch.cuda.CUDAGraph()

        def steps():
            try:
                a.rd_step(s.Dw, s.Dg, s.rho, s.dt, 12)
            except GbfkError as e:
                errors.append(e)

        with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
            x.add_(1)
            thread = threading.Thread(target=steps)
            thread.start()
            thread.join()
        graph.replay()
        b.rd_step(s.Dw, s.Dg, s.rho, s.dt, 13)
        assert not errors and float(x.sum()) == 100
        assert a.step_kernel == ("pipelined" if n == 176 else "run")
        assert np.array_equal(a.download_dense("phi"), b.download_dense("phi"))
