"""Where a NaN goes: every way of taking several steps leaves it in the same
cells as the one-CTA-per-block kernel, which evaluates the domain test
p_w + p_g + phi > 0 of every cell as it is written: a CSF cell at +0 is outside
the domain and keeps its +0 next to a NaN, one with phi > 0 is inside and
becomes NaN through a coefficient of 0."""
import numpy as np
import pytest

from gliomasolver_b200 import BlockPool, GbfkError
from gliomasolver_b200.schedule import make_schedule

pytestmark = pytest.mark.gpu


def layered(n, seed, prec, thin=False):
    """p_w, p_g, phi: tissue cut into rooms by CSF sheets one to three cells
    thick, a corner of CSF (empty blocks in it from 32^3 on), phi in the
    tissue only, NaN in tissue cells of one room in front of a sheet; with
    `thin` also cells whose p_w + p_g is below 0.1."""
    R = np.float64 if prec == "f64" else np.float32
    rng = np.random.default_rng(seed)
    tissue = np.ones((n, n, n), dtype=bool)
    at = 5
    for k in range(n):
        width = 1 + k % 3
        if at + width + 3 > n:
            break
        tissue[:, :, at:at + width] = False
        tissue[at:at + width, :, :] &= rng.random((width, n, n)) < 0.5
        at += width + 6
    tissue[: 3 * n // 4, : 3 * n // 4, : 3 * n // 4] = False
    pw = np.where(tissue, rng.uniform(0.3, 0.7, tissue.shape), 0.0)
    pg = np.where(tissue, 1.0 - pw, 0.0)
    if thin:
        few = rng.random(tissue.shape) < 0.02
        pw, pg = np.where(few, 0.06 * pw, pw), np.where(few, 0.06 * pg, pg)
    phi = np.where(tissue & (rng.random(tissue.shape) < 0.4), rng.uniform(0, 1, tissue.shape), 0.0)
    spot = np.argwhere(tissue[:, :, 4])[:: max(1, n)][:4]
    for z, y in spot:
        phi[z, y, 4] = np.nan
    return [a.astype(R) for a in (pw, pg, phi)]


def _pool(n, prec, fields):
    pool = BlockPool((n // 8) ** 3, prec)
    pool.set_uniform(n // 8)
    for name, a in zip(("p_w", "p_g", "phi"), fields):
        pool.upload_dense(name, a)
    return pool


def same_as_block_steps(n, prec, fields, calls, used):
    s = make_schedule(0.3, 0.2, 300.0, 25.6, n // 8, prec)
    with _pool(n, prec, fields) as a, _pool(n, prec, fields) as b:
        b.step_kernel = "block"
        for steps in calls:
            for p in (a, b):
                p.rd_step(s.Dw, s.Dg, s.rho, s.dt, steps)
            got, want = a.download_dense("phi"), b.download_dense("phi")
            assert a.step_kernel == used
            assert np.array_equal(got, want, equal_nan=True), (steps, np.isnan(got).sum(), np.isnan(want).sum())
        assert 0 < np.isnan(want).sum() < want.size
        for p in (a, b):
            with pytest.raises(GbfkError) as e:
                p.rd_step(s.Dw, s.Dg, s.rho, s.dt, 8, check_nan=True)
            assert e.value.code == 4


@pytest.mark.parametrize("thin", [False, True])
@pytest.mark.parametrize("prec,n", [("f32", 24), ("f64", 32), ("f32", 64), ("f32", 104), ("f64", 72)])
def test_nan_beside_csf_in_a_resident_run(gbfk_lib, prec, n, thin):
    same_as_block_steps(n, prec, layered(n, n, prec, thin), (8, 13, 40), "run")


@pytest.mark.parametrize("prec,n", [("f32", 152), ("f64", 120)])
def test_nan_beside_csf_in_steps_over_the_heavy_blocks(gbfk_lib, prec, n):
    same_as_block_steps(n, prec, layered(n, n, prec), (8, 13), "pipelined")


def outside(fields, kind, seed=0):
    """The same with values in the CSF too, whole blocks of it among them:
    positive ones ("positive"), a NaN at the border of an empty block and of
    the CSF block beside it, each with a positive neighbour across ("nan"),
    both, or one NaN inside an empty block that is +0 else ("alone")."""
    pw, pg, phi = (f.copy() for f in fields)
    rng = np.random.default_rng(seed)
    csf = pw + pg == 0
    if kind == "alone":
        phi = np.nan_to_num(phi)
        phi[12, 12, 12] = np.nan
        return pw, pg, phi
    if kind != "nan":
        phi[csf & (rng.random(phi.shape) < 0.7)] = 0.37
    if kind != "positive":
        phi[8, 8, 8], phi[8, 8, 7], phi[8, 8, 9] = np.nan, 0.2, 0.2
        phi[7, 12, 12], phi[8, 12, 12], phi[9, 12, 12] = np.nan, 0.2, 0.2
    if kind == "nan":
        phi[~csf] = np.nan_to_num(phi[~csf])
    return pw, pg, phi


@pytest.mark.parametrize("kind", ["positive", "nan", "both"])
@pytest.mark.parametrize("prec,n", [("f32", 32), ("f64", 48), ("f32", 104), ("f64", 72)])
def test_nan_and_tumour_in_empty_blocks_of_a_resident_run(gbfk_lib, prec, n, kind):
    """A NaN crosses between an empty block and its neighbours through the
    cells that are inside the domain (phi > 0), both ways."""
    same_as_block_steps(n, prec, outside(layered(n, n, prec), kind), (8, 13, 40), "run")


@pytest.mark.parametrize("kind", ["positive", "nan", "both"])
@pytest.mark.parametrize("prec,n", [("f32", 152), ("f64", 120)])
def test_nan_and_tumour_in_empty_blocks_of_streamed_steps(gbfk_lib, prec, n, kind):
    same_as_block_steps(n, prec, outside(layered(n, n, prec), kind), (8, 13), "pipelined")


@pytest.mark.parametrize("n,used", [(32, "run"), (152, "pipelined")])
def test_nan_that_arises_in_a_run_with_tumour_in_empty_blocks(gbfk_lib, n, used):
    """Coefficients whose sum over six faces overflows: a cell with six tissue
    neighbours falls to 0 in the first step and to inf * 0 in the second."""
    pw, pg, phi = layered(n, n, "f32")
    tissue = pw + pg > 0
    pw, pg = tissue.astype(np.float32), np.zeros_like(pg)
    phi = np.where(tissue, np.float32(0.5), np.float32(0.37))
    with _pool(n, "f32", (pw, pg, phi)) as a, _pool(n, "f32", (pw, pg, phi)) as b:
        b.step_kernel = "block"
        for steps in (1, 1, 8, 9):
            for p in (a, b):
                p.upload_dense("phi", phi)
                p.rd_step(6.2e37, 6.2e36, 0.05, 1e-3, steps)
            got, want = a.download_dense("phi"), b.download_dense("phi")
            assert np.array_equal(got, want, equal_nan=True), steps
            assert np.isnan(want).any() == (steps > 1)
        assert a.step_kernel == used


@pytest.mark.parametrize("kind", ["nan", "both", "alone"])
def test_gradient_with_nan_in_an_empty_block(gbfk_lib, kind):
    """A step keeps such a NaN: the states, the loss and lambda_0 are those of
    the block kernel whatever the call before was (its buffers' empty blocks
    may be known to hold +0), with the same coefficients and new ones."""
    n, steps = 32, 10
    pw, pg, phi = outside(layered(n, 3, "f32"), kind)
    clean = np.where(pw + pg > 0, np.nan_to_num(phi), 0).astype(np.float32)
    rng = np.random.default_rng(1)
    t1, fl = ((rng.random(pw.shape) < f).astype(float) for f in (0.05, 0.1))
    with _pool(n, "f32", (pw, pg, phi)) as pool:
        pool.set_observations(t1, fl)
        for Dw, before in ((0.2, None), (0.2, clean), (0.1, clean), (0.15, None)):
            s = make_schedule(Dw, 0.1, 100.0, 25.6, n // 8, "f32")
            out = {}
            for k in ("block", "pipelined", "auto"):
                pool.step_kernel = k
                for field in (before, phi):
                    if field is None:
                        continue
                    pool.upload_dense("phi", field)
                    out[k] = pool.forward_adjoint(s.Dw, s.Dg, s.rho, min(s.dt, 0.2), steps, sigma=0.0, nsnapshots=4,
                                                  grad_c0=True, t1_uc=0.7, t2_uc=0.25, slope=2.0)
            for k in ("pipelined", "auto"):
                assert np.array_equal(out[k]["grad_c0"], out["block"]["grad_c0"], equal_nan=True), (Dw, k)
                assert out[k]["loss"] == out["block"]["loss"], (Dw, k)


@pytest.mark.parametrize("prec,bpd", [("f32", 4), ("f64", 3), ("f32", 12)])
def test_nan_beside_csf_in_a_stage(gbfk_lib, prec, bpd):
    """Initial conditions that are NaN: everywhere in the tissue (a NaN
    origin), or at the origin alone (0 / 0 with a width whose square is 0)."""
    from gliomasolver_b200.tmcmc import Batch, sample_stage, to_gbfk_samples

    n = 8 * bpd
    pw, pg, _ = layered(n, 7, prec)
    recs, _ = to_gbfk_samples(sample_stage(4, pw, seed=2, tend_range=(5.0, 30.0)), bpd, prec)
    for i, r in enumerate(recs):
        r.nsteps = 9 + 4 * i
    recs[1].x0[0] = np.nan
    z, y = np.argwhere(pw[:, :, 4] > 0)[n]
    recs[2].x0[0], recs[2].x0[1], recs[2].x0[2] = 4 / n, y / n, z / n
    recs[2].sigma = 1e-200
    with Batch(bpd, 4, prec, max_anatomies=1) as b:
        b.set_anatomy(0, pw, pg)
        out = []
        for kind in (1, 0):
            b.set_samples(recs)
            with pytest.raises(GbfkError) as e:
                b.run(kind)
            assert e.value.code == 4
            out.append([b.download(i) for i in range(4)])
    for i, (want, got) in enumerate(zip(*out)):
        assert np.array_equal(got, want, equal_nan=True), i
        assert np.isnan(want).any() == (i in (1, 2))


@pytest.mark.parametrize("prec,bpd", [("f64", 4), ("f32", 8)])
def test_nan_beside_csf_in_a_resident_sweep(gbfk_lib, prec, bpd):
    """The gradient with NaN in the initial field: the same cells of lambda_0
    as with a launch per step."""
    n, steps = 8 * bpd, 14
    pw, pg, phi = layered(n, 3, prec, thin=True)
    rng = np.random.default_rng(1)
    t1, fl = ((rng.random(pw.shape) < f).astype(float) for f in (0.05, 0.1))
    s = make_schedule(0.2, 0.1, 100.0, 25.6, bpd, prec)
    out = {}
    with _pool(n, prec, (pw, pg, phi)) as pool:
        pool.set_observations(t1, fl)
        for kind in ("pipelined", "auto"):
            pool.step_kernel = kind
            out[kind] = pool.forward_adjoint(s.Dw, s.Dg, s.rho, min(s.dt, 0.2), steps, sigma=0.0, nsnapshots=4,
                                             grad_c0=True, term_magnitudes=True, t1_uc=0.7, t2_uc=0.25, slope=2.0)
    a, b = out["auto"], out["pipelined"]
    assert np.array_equal(a["grad_c0"], b["grad_c0"], equal_nan=True)
    assert np.isnan(a["loss"]) == np.isnan(b["loss"])
    for key in ("dDw", "drho", "dDw_abs", "drho_abs"):
        scale = b[key.replace("_abs", "") + "_abs"]
        assert np.isnan(a[key]) == np.isnan(b[key]), key
        assert np.isnan(b[key]) or abs(a[key] - b[key]) <= 1e-14 * scale + 1e-13 * abs(b[key]), key


@pytest.mark.parametrize("steps,ck", [(1, 1), (2, 4), (3, 1), (9, 3)])
@pytest.mark.parametrize("prec,bpd", [("f64", 4), ("f32", 8)])
def test_gradient_with_nan_that_arises_in_few_steps(gbfk_lib, prec, bpd, steps, ck):
    """An infinite tissue fraction: its faces' coefficients are NaN, also those
    toward CSF, and the states after the first, whether the forward steps are
    a run or (few) a launch each."""
    n = 8 * bpd
    pw, pg, phi = layered(n, 3, prec)
    phi[np.isnan(phi)] = 0.1
    for z, y in np.argwhere(pw[:, :, 4] > 0)[:: n][:5]:
        pw[z, y, 4] = np.inf
    rng = np.random.default_rng(1)
    t1, fl = ((rng.random(pw.shape) < f).astype(float) for f in (0.05, 0.1))
    s = make_schedule(0.2, 0.1, 100.0, 25.6, bpd, prec)
    out = {}
    with _pool(n, prec, (pw, pg, phi)) as pool:
        pool.set_observations(t1, fl)
        for kind in ("pipelined", "auto"):
            pool.step_kernel = kind
            out[kind] = pool.forward_adjoint(s.Dw, s.Dg, s.rho, min(s.dt, 0.2), steps, sigma=0.0, nsnapshots=ck,
                                             grad_c0=True, term_magnitudes=True, t1_uc=0.7, t2_uc=0.25, slope=2.0)
    a, b = out["auto"], out["pipelined"]
    assert np.isnan(b["grad_c0"]).any()
    assert np.array_equal(a["grad_c0"], b["grad_c0"], equal_nan=True) and a["loss"] == b["loss"]
    for key in ("dDw", "drho", "dDw_abs", "drho_abs"):
        assert a[key] == b[key] or np.isnan(a[key]) and np.isnan(b[key]), key
