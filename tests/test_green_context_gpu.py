"""Contexts on a stream of a green context (a part of the GPU's SMs): kernels
whose CTAs wait for one another are launched with as many as fit there, and
every call gives the bits it gives on the whole GPU."""
import numpy as np
import pytest

from gliomasolver_b200 import BlockPool
from gliomasolver_b200.anatomy import make_case
from gliomasolver_b200.schedule import make_schedule

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def part(gbfk_lib):
    """A stream of a green context with 64 of the SMs."""
    cu = pytest.importorskip("cuda.bindings.driver")
    import torch

    torch.zeros(1, device="cuda")

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r
        return r[1]

    dev = ok(cu.cuDeviceGet(torch.cuda.current_device()))
    every = ok(cu.cuDeviceGetDevResource(dev, cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups = ok(cu.cuDevSmResourceSplitByCount(1, every, 0, 64))
    ctx = ok(cu.cuGreenCtxCreate(ok(cu.cuDevResourceGenerateDesc([groups[0]], 1)), dev,
                                 cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(cu.cuGreenCtxStreamCreate(ctx, cu.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(stream)
    cu.cuStreamDestroy(stream)
    cu.cuGreenCtxDestroy(ctx)


def _pool(n, prec, stream):
    R = np.float64 if prec == "f64" else np.float32
    pw, pg, c0, _ = make_case(n, 1)
    pool = BlockPool((n // 8) ** 3, prec, stream=stream)
    pool.set_uniform(n // 8)
    for name, a in (("p_w", pw), ("p_g", pg), ("phi", c0)):
        pool.upload_dense(name, a.astype(R))
    return pool


@pytest.mark.parametrize("n,prec", [(64, "f32"), (72, "f64"), (128, "f32"), (128, "f64")])
def test_steps_on_a_part_of_the_gpu(part, n, prec):
    """Runs on 64 SMs, and (128^3) grids that fit the GPU's SMs but not these."""
    s = make_schedule(0.2, 0.1, 300.0, 25.6, n // 8, prec)
    out = []
    for stream in (None, part):
        with _pool(n, prec, stream) as pool:
            for steps in (20, 9):
                pool.rd_step(s.Dw, s.Dg, s.rho, s.dt, steps, check_nan=True)
                out.append(pool.download_dense("phi"))
            assert pool.step_kernel == ("pipelined" if stream and n == 128 else "run")
    assert np.array_equal(out[0], out[2]) and np.array_equal(out[1], out[3])


def test_gradient_on_a_part_of_the_gpu(part):
    n = 64
    s = make_schedule(0.2, 0.1, 100.0, 25.6, n // 8, "f64")
    out = []
    for stream in (None, part):
        with _pool(n, "f64", stream) as pool:
            c0 = pool.download_dense("phi")
            pool.set_observations((c0 > 0.2).astype(float), (c0 > 0.1).astype(float))
            out.append(pool.forward_adjoint(s.Dw, s.Dg, s.rho, s.dt, 30, sigma=0.0, nsnapshots=8, grad_c0=True,
                                            t1_uc=0.7, t2_uc=0.25, slope=2.0))
    assert np.array_equal(out[0]["grad_c0"], out[1]["grad_c0"]) and out[0]["loss"] == out[1]["loss"]


def test_stage_on_a_part_of_the_gpu(part):
    from gliomasolver_b200.tmcmc import Batch, sample_stage, to_gbfk_samples

    n = 64
    pw, pg, _, _ = make_case(n, 1)
    recs, _ = to_gbfk_samples(sample_stage(6, pw, seed=2, tend_range=(5.0, 20.0)), n // 8, "f32")
    out = []
    for stream in (None, part):
        with Batch(n // 8, 6, "f32", max_anatomies=1, stream=stream) as b:
            b.set_anatomy(0, pw.astype(np.float32), pg.astype(np.float32))
            b.set_samples(recs)
            b.run(0)
            out.append([b.download(i) for i in range(6)])
    for want, got in zip(*out):
        assert np.array_equal(got, want)


def test_ghost_list_steps_on_a_part_of_the_gpu(part):
    from topology_util import uniform_topology

    bpd, n = 8, 64
    pw, pg, c0, _ = make_case(n, 1)
    blocks, csr = uniform_topology(bpd, np.arange(bpd ** 3))
    s = make_schedule(0.2, 0.1, 300.0, 25.6, bpd, "f32")
    out = []
    for stream in (None, part):
        with BlockPool(bpd ** 3, "f32", stream=stream) as pool:
            pool.set_topology(blocks, csr)
            for name, a in (("p_w", pw), ("p_g", pg), ("phi", c0)):
                v = a.astype(np.float32).reshape(bpd, 8, bpd, 8, bpd, 8).transpose(0, 2, 4, 1, 3, 5)
                pool.upload(name, np.ascontiguousarray(v).ravel())
            pool.rd_step(s.Dw, s.Dg, s.rho, s.dt, 12, check_nan=True)
            out.append(pool.download("phi", bpd ** 3 * 512))
            assert pool.step_kernel == "run"
    assert np.array_equal(out[0], out[1])
