"""3D ray operators at the ends of what they accept: a volume one voxel thick
with more than 2^24 bricks, and volumes that cover part of the image."""
import numpy as np
import pytest

from tval3g import capi
from tval3g import workloads as W

pytestmark = pytest.mark.gpu


def _geometry(p0, p1, rv):
    E, R = len(p0), len(p1)
    g = dict(numMPs=1, numPaths=E * R, E=E, R=R, use_path=np.arange(1, E * R + 1), rv_x=rv[2], rv_y=rv[1], rv_z=rv[0],
             scale=1.0, xe=p0[:, 0], ye=p0[:, 1], ze=p0[:, 2], xr=p1[:, 0], yr=p1[:, 1], zr=p1[:, 2])
    i, j = np.divmod(np.arange(E * R), R)
    return g, W.bresenham_csr_3d(p0[i], p1[j], rv[2], rv[1])


def test_adjoint_more_than_2_24_bricks(torch_cuda):
    """1 x 32767 x 32767 voxels are 2^25 bricks; the rays lie in those from 2^24 on and below."""
    torch = torch_cuda
    rv = (32767, 32767, 1)
    p0 = np.array([[0, 5, 32760], [0, 32766, 16390]])
    p1 = np.array([[0, 32766, 32766], [0, 0, 0], [0, 32000, 32766]])
    g, (off, pix) = _geometry(p0, p1, rv)
    y = np.arange(1, 7, dtype=np.float32)   # whole numbers: every sum is exact
    op = capi.Operator(capi.ray3d_problem(rv, g))
    out = torch.full((op.cols,), 7.0, device="cuda")
    op.apply(torch.tensor(y, device="cuda"), out, trans=True)
    at, inv = np.unique(np.asarray(pix, np.int64), return_inverse=True)
    want = np.bincount(inv, np.repeat(y, np.diff(off)))
    assert np.array_equal(out[torch.tensor(at, device="cuda")].cpu().numpy(), want.astype(np.float32))
    assert int(torch.count_nonzero(out)) == len(at)
    op.close()


@pytest.mark.parametrize("shape,rv", [((5, 5, 5), (5, 4, 4)), ((7, 9, 10), (5, 11, 11)), ((3, 40, 41), (5, 31, 31)),
                                      ((13, 13, 13), (1, 40, 54))])
def test_adjoint_of_a_volume_smaller_than_the_image(shape, rv, torch_cuda):
    """Nothing is written past the image, although the last layer of bricks reaches beyond it; between the volume's end
    and the image's lie zeros, in the adjoint and in the normal product."""
    torch = torch_cuda
    rng = np.random.default_rng(sum(shape))
    n, guard = int(np.prod(shape)), 8192
    assert n > np.prod(rv)
    p0, p1 = (np.stack([rng.integers(0, s, k) for s in (rv[2], rv[1], rv[0])], 1) for k in (6, 9))
    g, (off, pix) = _geometry(p0, p1, rv)
    y = rng.integers(-9, 10, 54).astype(np.float32)
    op = capi.Operator(capi.ray3d_problem(shape, g))
    buf = torch.full((n + guard,), 7.0, device="cuda")
    op.apply(torch.tensor(y, device="cuda"), buf[:n], trans=True)
    out = buf.cpu().numpy()
    assert np.array_equal(out[:np.prod(rv)], np.bincount(pix, np.repeat(y, np.diff(off)), np.prod(rv)).astype(np.float32))
    assert np.all(out[n:] == 7.0)
    assert np.all(out[np.prod(rv):n] == 0)
    x = torch.tensor(rng.integers(-9, 10, n).astype(np.float32), device="cuda")
    Ax, want = torch.empty(54, device="cuda"), torch.full((n,), 7.0, device="cuda")
    op.apply(x, Ax)
    op.apply(Ax, want, trans=True)
    buf.fill_(7.0)
    op.apply(x, buf[:n], trans=2)
    assert torch.equal(buf[:n], want) and torch.all(buf[n:] == 7.0)
    op.close()
