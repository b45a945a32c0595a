"""The dense forward of several right-hand sides: the forms that launches of few
and of many rows take, over row lengths on both sides of every line between
them (aligned and not, one and two chunks of shared memory, remainders), give
the same bits as one right-hand side alone, and each is the FP64 product
rounded once."""
import numpy as np
import pytest

from tval3g import capi
from tval3g import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,h,w,layers", [(9, 1, 5, 200), (9, 1, 8, 200), (190, 25, 25, 16), (400, 41, 41, 4),
                                          (700, 23, 89, 3), (600, 32, 64, 4), (667, 47, 47, 5), (520, 1, 4095, 5),
                                          (900, 64, 64, 8), (900, 17, 241, 3), (1300, 81, 81, 3), (500, 1, 6144, 7),
                                          (500, 1, 6147, 7), (300, 127, 127, 20), (300, 128, 128, 20)])
def test_layers_equal_one_right_hand_side(m, h, w, layers, torch_cuda):
    torch = torch_cuda
    n = h * w
    assert m <= 1024 + n / 4 < m * layers   # few rows alone, many together
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((m, n), generator=g, device="cuda")
    x = torch.randn((layers, n), generator=g, device="cuda")
    one = capi.Operator(capi.dense_problem((h, w), A, device_ptr=A.data_ptr()), device_inputs=True)
    many = capi.Operator(capi.dense_problem((h * layers, w), A, layers=layers, device_ptr=A.data_ptr()),
                         device_inputs=True, tensor=False)
    y = torch.full((layers, m), float("nan"), device="cuda")
    many.apply(x.reshape(-1), y)
    y1 = torch.empty(m, device="cuda")
    for k in range(layers):
        xk = x[k].clone()   # (aligned, as a vector of its own)
        assert torch.equal(one.apply(xk, y1), y[k])
    want, mag = x.double() @ A.double().T, x.double().abs() @ A.double().abs().T
    assert bool(((y.double() - want).abs() <= 2.0 ** -24 * mag).all())   # FP64 sums, one rounding
    xb = torch.empty(layers * n + 1, device="cuda")   # x not 16-byte aligned
    xb[1:] = x.reshape(-1)
    assert torch.equal(many.apply(xb[1:], torch.empty_like(y)), y)
    one.close()
    many.close()


@pytest.mark.parametrize("m,h,w", [(20000, 16, 32), (20001, 16, 32), (90000, 4, 4), (30000, 63, 65), (30000, 64, 64)])
def test_normal_product_of_many_short_rows(m, h, w, torch_cuda):
    """Both sides of the line from which it is two products (rows of fewer than 4096 columns)."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(m)
    A = torch.randn((m, h * w), generator=g, device="cuda") / 64
    x = torch.randn(h * w, generator=g, device="cuda")
    op = capi.Operator(capi.dense_problem((h, w), A, device_ptr=A.data_ptr()), device_inputs=True)
    y = op.apply(x, torch.full((h * w,), 7.0, device="cuda"), trans=2)
    A64, B64 = A.double(), A.double().abs()
    want = A64.T @ (A64 @ x.double())
    # A x rounded (by rows: eight products in FP32 first), float partials of row chunks, one rounding
    assert bool(((y.double() - want).abs() <= 16 * 2.0 ** -24 * (B64.T @ (B64 @ x.double().abs()))).all())
    assert float((y.double() - want).norm() / want.norm()) < 3e-7
    op.close()


def test_matrix_not_16_byte_aligned(torch_cuda):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(3)
    for m, h, w, layers in ((300, 64, 64, 1), (300, 64, 64, 9), (300, 16, 64, 9), (40, 16, 64, 1)):
        buf = torch.randn(m * h * w + 1, generator=g, device="cuda")
        A = buf[1:].view(m, h * w)
        x = torch.randn((layers, h * w), generator=g, device="cuda")
        op = capi.Operator(capi.dense_problem((h * layers, w), A, layers=layers, device_ptr=A.data_ptr()),
                           device_inputs=True, tensor=False)
        y = op.apply(x.reshape(-1), torch.empty((layers, m), device="cuda"))
        want, mag = x.double() @ A.double().T, x.double().abs() @ A.double().abs().T
        assert bool(((y.double() - want).abs() <= 2.0 ** -24 * mag).all())
        op.close()


def test_many_small_matrices_in_a_batch_equal_each_alone(torch_cuda):
    """Twelve unaligned matrices are many rows to a launch, one is few."""
    torch = torch_cuda
    ws = [W.dense2d(seed=s, side=25, sampling=0.3, tv_norm=s % 2, maxit=6, tol=1e-9) for s in range(12)]
    specs = [capi.dense_problem(w["shape"], w["A"]) for w in ws]
    bs = [torch.tensor(w["b"], device="cuda") for w in ws]

    def solve(idx):
        plan = capi.Plan([specs[i] for i in idx], [ws[i]["opts"] for i in idx])
        U = [torch.empty(specs[i].n, device="cuda") for i in idx]
        plan.solve([bs[i] for i in idx], U)
        plan.close()
        return [u.cpu().numpy() for u in U]
    together = solve(range(12))
    for i in range(12):
        assert np.array_equal(together[i], solve([i])[0])
