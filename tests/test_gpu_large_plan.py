"""The iteration with one W and d in two kernels, as plans of complex data and
those whose image vectors would take more than 32 GB run it, on real data."""
import numpy as np
import pytest

import oracle as O
from helpers import noise_floor, relerr
from test_gpu_step import SHAPES, problem
from tval3g import capi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1e-5, 0.55, 1.0])   # steps accepted, shortened, restarted
@pytest.mark.parametrize("tv", [0, 1])
def test_real_instance_beside_a_complex_one(tv, c, torch_cuda):
    """A plan with one complex instance runs the two kernels for all: the real one follows the oracle (the tolerance is
    test_gpu_step's)."""
    torch = torch_cuda
    rng = np.random.default_rng(5)
    Ac = (rng.standard_normal((20, 36)) + 1j * rng.standard_normal((20, 36))).astype(np.complex64)
    bc = Ac @ (rng.standard_normal(36) + 1j * rng.standard_normal(36))
    bc = torch.tensor(np.stack([bc.real, bc.imag], 1).astype(np.float32).ravel(), device="cuda")
    for k, shape in enumerate(SHAPES):
        m, n, rowptr, colind, val, A, b = problem(shape, 10 * k + tv)
        opts = W.options(2.0 ** 6, 2.0 ** 4, 1e-9, 4, tv_norm=tv, tol_inn=1e-9, c=c)
        solve = lambda extra: O.solve(A, b.astype(np.float64), shape, dict(opts, **extra), record=True)  # noqa: E731
        r = solve({})
        specs = [capi.csr_problem(shape, m, n, rowptr, colind, val), capi.dense_problem((6, 6), Ac)]
        plan = capi.Plan(specs, [opts, opts], graph=True, trace=True)
        dU = [torch.empty(n, device="cuda"), torch.empty(72, device="cuda")]
        info = plan.solve([torch.tensor(b, device="cuda"), bc], dU)[0]
        tr = plan.trace(0)
        plan.close()
        assert info["status"] == 0
        assert [int(t[3]) for t in tr] == [int(x[3]) for x in r.iters], shape
        e, tol = relerr(dU[0].cpu().numpy().reshape(shape), r.U), 16 * noise_floor(solve, r.U) + 2.0 ** -23
        assert e < tol, (shape, e, tol)


@pytest.mark.parametrize("tv", [0, 1])
def test_plan_above_32_gb(tv, torch_cuda):
    """A thin volume of 3.2e8 voxels with its rays in one corner solves as the corner alone does (the rest stays zero),
    in the memory of 23 image vectors and the index."""
    torch = torch_cuda
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 80 GB of free device memory")
    rng = np.random.default_rng(7)
    E, R, corner, large = 128, 100, (96, 96, 1), (9800, 32767, 1)
    p0, p1 = (np.stack([np.zeros(k, int), rng.integers(8, 72, k), rng.integers(8, 72, k)], 1) for k in (E, R))
    u = np.zeros(corner)
    u[20:50, 30:60] = 1.0
    i, j = np.divmod(np.arange(E * R), R)
    off, pix = W.bresenham_csr_3d(p0[i], p1[j], corner[2], corner[1])
    scale = 1 / 64
    b = np.add.reduceat(u.ravel()[pix], off[:-1]) * scale
    opts = W.options(2.0 ** 8, 2.0 ** 5, 1e-9, 4, tv_norm=tv, tol_inn=1e-9)
    db = [torch.tensor(b.astype(np.float32), device="cuda")]

    def solve(shape):
        g = dict(numMPs=1, numPaths=E * R, E=E, R=R, use_path=np.arange(1, E * R + 1), rv_x=shape[2], rv_y=shape[1],
                 rv_z=shape[0], scale=scale, xe=p0[:, 0], ye=p0[:, 1], ze=p0[:, 2], xr=p1[:, 0], yr=p1[:, 1], zr=p1[:, 2])
        spec = capi.ray3d_problem(shape, g)
        plan = capi.Plan([spec], [opts], graph=True, trace=True)
        U = torch.full((spec.n,), 7.0, device="cuda")
        info = plan.solve(db, [U])[0]
        tr, bytes_ = plan.trace(0), plan.stats()["device_bytes"]
        plan.close()
        assert info["status"] == 0 and info["total_iters"] == 4
        return U.view(shape), [int(t[3]) for t in tr], bytes_
    Us, bts, _ = solve(corner)
    Ul, btl, bytes_ = solve(large)
    part = Ul[:corner[0], :corner[1]]
    assert btl == bts
    # the same arithmetic per element, the scalars from FP64 sums in another order
    assert relerr(part.cpu().numpy(), Us.cpu().numpy()) < 1e-5
    assert int(torch.count_nonzero(Ul)) == int(torch.count_nonzero(part)) > 1000
    # the index of a brick of 8 x 8 x 4: its voxels' order (256), eight word offsets (32), its place among the empty ones (4)
    bricks = -(-large[0] // 4) * -(-large[1] // 8)
    assert bytes_ < 23 * 4 * np.prod(large, dtype=np.int64) + 292 * bricks + (64 << 20)
    del Ul, part
    torch.cuda.empty_cache()
    capi.trim_memory()


def test_time_step(torch_cuda):
    """The iteration's one kernel is timed where the plan runs it, and 0 elsewhere; the next solve starts afresh."""
    torch = torch_cuda
    m, n, rowptr, colind, val, A, b = problem((23, 31), 1)
    opts = W.options(2.0 ** 6, 2.0 ** 4, 1e-9, 4)
    spec = capi.csr_problem((23, 31), m, n, rowptr, colind, val)
    plan = capi.Plan([spec], [opts])
    db, u1, u2 = [torch.tensor(b, device="cuda")], [torch.empty(n, device="cuda")], [torch.empty(n, device="cuda")]
    plan.solve(db, u1)
    assert plan.time_step(5) > 0
    plan.solve(db, u2)
    assert torch.equal(u1[0], u2[0])
    plan.close()
    cplx = capi.Plan([capi.csr_problem((23, 31), m, n, rowptr, colind, val.astype(np.complex64))], [opts])
    assert cplx.time_step(5) == 0
    cplx.close()
