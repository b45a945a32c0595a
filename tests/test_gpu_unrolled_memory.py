"""What a checkpoint of the unrolled solve takes: U, the two multipliers of D U
and d over the image, delta over the measurements with entries."""
import numpy as np
import pytest

from tval3g import capi
from tval3g import workloads as W

pytestmark = pytest.mark.gpu


def test_bytes_per_checkpoint(torch_cuda):
    torch = torch_cuda
    side, T = 32, 512
    g = W.ring_geometry(side, T)
    spec = capi.ray2d_problem((side, side), g)
    m = int(np.count_nonzero(g["use_path"]))
    assert m > 100 * side * side

    def used(K):
        torch.cuda.synchronize()
        capi.trim_memory()
        before = torch.cuda.mem_get_info()[0]
        h = capi.Unrolled(spec, 1, W.options(2 ** 8, 2 ** 5, 1e-4, K), K, ckpt=1)
        torch.cuda.synchronize()
        capi.trim_memory()
        after = torch.cuda.mem_get_info()[0]
        h.close()
        return before - after
    used(2)   # (code)
    few, many = used(8), used(88)
    # 80 checkpoints and the reverse steps' partial sums (7 doubles of up to 1184 blocks each); 2 MB per allocation
    per = 8 * (4 * side * side + m) + 7 * 8 * 1184
    assert 0.9 * 80 * per < many - few < 80 * per + (16 << 20)
