"""The dense forward at the longest row an image can have."""
import pytest

from tval3g import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2 ** 31 - 1, 2 ** 31 - 2048, 2 ** 31 - 2049])
def test_forward_of_one_long_row(n, torch_cuda):
    """n near 2^31: the last chunk's end does not fit an int.  Ones times zeros and whole numbers: an exact sum."""
    torch = torch_cuda
    A = torch.ones(n, device="cuda")
    x = torch.zeros(n, device="cuda")
    x[:3] = 1.0
    x[-5000:] = 2.0
    op = capi.Operator(capi.dense_problem((1, n), A.view(1, n), device_ptr=A.data_ptr()), device_inputs=True)
    y = torch.empty(1, device="cuda")
    op.apply(x, y)
    assert float(y) == 10003.0
    op.close()
