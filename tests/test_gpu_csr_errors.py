"""Host CSR arrays that an operator refuses, wherever in them the fault lies."""
import numpy as np
import pytest

from tval3g import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", [0, 1, 1234, -1])
@pytest.mark.parametrize("what,message", [(-1, "column index out of range"), (50 * 40, "column index out of range"),
                                          (-2 ** 31, "column index out of range"), (None, "not monotone")])
def test_refused(where, what, message, torch_cuda):
    m, n, per = 600, 50 * 40, 4
    rng = np.random.default_rng(3)
    rowptr, colind = np.arange(m + 1) * per, rng.integers(0, n, m * per)
    val = np.ones(m * per, np.float32)
    capi.Operator(capi.csr_problem((50, 40), m, n, rowptr, colind, val)).close()
    if what is None:
        row = where % (m - 1) + 1
        rowptr[row] = rowptr[row + 1] + 1
    else:
        colind[where] = what
    with pytest.raises(Exception) as e:
        capi.Operator(capi.csr_problem((50, 40), m, n, rowptr, colind, val))
    assert message in str(e.value)
