"""What a ray operator keeps on the device for its tiled adjoint."""
import numpy as np
import pytest

from tval3g import capi
from tval3g import workloads as W

pytestmark = pytest.mark.gpu


def test_large_image_with_few_rays(torch_cuda):
    """8192^2, no tile cut: per tile its pixels' order (256 bytes), eight word offsets (32) and its place in the launch
    list (4).  Sixteen parts' offsets would be 480 bytes more per tile.  Besides: 27 image vectors, the transposed image,
    the launches' tile maps and partial sums (together below 64 MB)."""
    torch = torch_cuda
    side, tiles = 8192, 512 * 512
    rng = np.random.default_rng(1)
    p = rng.integers(0, side, (4, 3))
    g = dict(use_path=np.ones(9), xe=p[0], ye=p[1], xr=p[2], yr=p[3], ld=side, scale=1.0)
    spec = capi.ray2d_problem((side, side), g)
    op = capi.Operator(spec)
    y = np.arange(1, 10, dtype=np.float32)
    out = op.apply(torch.tensor(y, device="cuda"), torch.full((side * side,), 7.0, device="cuda"), trans=True)
    assert float(out.double().sum()) == sum(v * (1 + max(abs(int(p[0][e]) - int(p[2][r])), abs(int(p[1][e]) - int(p[3][r]))))
                                            for (e, r), v in zip(np.ndindex(3, 3), y))
    op.close()
    plan = capi.Plan([spec], [W.options(1.0, 1.0, 1e-6, 2)])
    bytes_ = plan.stats()["device_bytes"]
    plan.close()
    assert 28 * 4 * side * side + 256 * tiles < bytes_ < 28 * 4 * side * side + 292 * tiles + (64 << 20)
