"""Row pointers that do not cover the columns exactly are refused by the direct-solve replacement before a kernel reads
through them."""
import pytest
import torch

from jspsr import ext

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("ptr", [[5, 6, 7], [1, 2, 3], [-1, 0, 1], [0, 1, 3], [0, 1, 1], [0, 3, 2], [0, -1, 2], [0, 2],
                                 [0, 1, 1, 2]])
def test_row_pointers(ptr, dtype):
    cols, vals, b = torch.tensor([0, 1], device=DEV), torch.ones(2, device=DEV), torch.ones(2, device=DEV)
    assert torch.allclose(ext.solve_cusparse(torch.tensor([0, 1, 2], dtype=dtype, device=DEV), cols, vals, b, 1e-12), b)
    with pytest.raises(ValueError):
        ext.solve_cusparse(torch.tensor(ptr, dtype=dtype, device=DEV), cols, vals, b, 1e-12)
