"""Products of one operator must not overlap on the device; where they did, the
products after them are right all the same (the tiles' part counts are back at
zero)."""
import numpy as np
import pytest

from helpers import relerr
from tval3g import capi
from tval3g import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,T", [(33, 256), (64, 512), (128, 512)])
def test_adjoint_after_overlapping_adjoints(side, T, torch_cuda):
    torch = torch_cuda
    g = W.ring_geometry(side, T)
    op = capi.Operator(capi.ray2d_problem((side, side), g))
    y = torch.tensor(np.random.default_rng(side).standard_normal(op.rows).astype(np.float32), device="cuda")
    want = op.apply(y, torch.empty(op.cols, device="cuda"), trans=True).clone()
    a = W.ray2d_csr(g, side * side)
    host = np.bincount(a["colind"], np.repeat(y.double().cpu().numpy(), np.diff(a["rowptr"])) * g["scale"], side * side)
    assert relerr(want.cpu().numpy(), host) < 1e-6
    streams = [torch.cuda.Stream() for _ in range(3)]
    out = [torch.empty(op.cols, device="cuda") for _ in streams]
    torch.cuda.synchronize()
    for _ in range(20):
        for s, o in zip(streams, out):
            op.apply_n(y, o, 5, trans=True, stream=s.cuda_stream)
    torch.cuda.synchronize()
    got = torch.full((op.cols,), float("nan"), device="cuda")
    assert torch.equal(op.apply(y, got, trans=True), want)
    op.close()
