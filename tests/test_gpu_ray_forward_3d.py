"""The 3D ray forward on both sides of the line between its forms (56 K rays, a
fifth of the voxels up to 40 K, a fourteenth of them): the same sums, bit for
bit; and volumes of a batch, whose launch takes the other form than each alone,
solve to the same bits."""
import numpy as np
import pytest

from tval3g import capi
from tval3g import workloads as W
from test_gpu_ray_forward import _apply, _points, _sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,ny,nx", [(1, 1, 70), (9, 17, 33), (16, 40, 8), (30, 20, 25)])
@pytest.mark.parametrize("below", [1, 0])
def test_both_forms_give_the_same_sums(nz, ny, nx, below, torch_cuda):
    rng = np.random.default_rng(nz)
    n = nz * ny * nx
    R = 56 * 1024 + min(n // 5, 40 * 1024) + n // 14 - below
    e, r = _points(rng, 1, (nx, ny, nz)), _points(rng, R, (nx, ny, nz))
    g = dict(numMPs=1, numPaths=R, E=1, R=R, use_path=1 + rng.permutation(R), rv_x=nx, rv_y=ny, rv_z=nz, scale=0.3,
             xe=e[:, 0], ye=e[:, 1], ze=e[:, 2], xr=r[:, 0], yr=r[:, 1], zr=r[:, 2])
    x = rng.standard_normal(n).astype(np.float32)
    off, pix = W.bresenham_csr_3d(np.repeat(e, R, 0), r, nx, ny)
    want = np.empty(R, np.float32)
    want[g["use_path"] - 1] = _sums(off, pix, x, 0.3)
    y = _apply(torch_cuda, capi.ray3d_problem((nz, ny, nx), g), x)
    assert np.array_equal(y, want)


def test_volumes_of_a_batch_solve_as_each_alone(torch_cuda):
    torch = torch_cuda
    specs, bs = [], []
    for k, side in enumerate((16, 20, 23, 18, 16, 21)):   # 12800 rays each: 76800 in the launch
        g = W.hemisphere_geometry(side, 160, 80, (side - 1) / 2.0 - 0.5, np.random.default_rng(k))
        g["scale"] = 0.02
        specs.append(capi.ray3d_problem((side,) * 3, g))
        op = capi.Operator(specs[-1])
        u = torch.zeros((side,) * 3, device="cuda")
        u[side // 4:side // 2, side // 3:, side // 4:3 * side // 4] = 1.0
        bs.append(op.apply(u.reshape(-1), torch.empty(op.rows, device="cuda")).clone())
        op.close()
    opts = W.options(2.0 ** 8, 2.0 ** 5, 1e-9, 6, tv_norm=0)

    def solve(idx):
        plan = capi.Plan([specs[i] for i in idx], [opts] * len(idx))
        U = [torch.empty(specs[i].n, device="cuda") for i in idx]
        plan.solve([bs[i] for i in idx], U)
        plan.close()
        return U
    together = solve(range(6))
    for i in range(6):
        assert torch.equal(together[i], solve([i])[0])
