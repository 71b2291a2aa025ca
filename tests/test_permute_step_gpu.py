"""The tiled transpose whose steps are two or four large tiles (512 or 1024 elements) with few axes left:
one tile, a last step with fewer tiles than the others, several steps per block, extents left that are
no powers of two, and the most axes left that it takes and one more. Bit-exact against a
plain transpose of a tensor that holds its own indices."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,ptup", [
    ([32, 32], [1, 0]), ([96, 160], [1, 0]), ([64, 64, 257], [2, 0, 1]), ([1728, 1728], [1, 0]), ([2048, 4096], [1, 0]),
    ([16, 5, 16, 2], [2, 0, 1, 3]), ([16, 37, 16, 2], [2, 0, 1, 3]), ([16, 3001, 16, 2], [2, 0, 1, 3]),
    ([2] * 13, list(range(13))[::-1]), ([2] * 22, list(range(22))[::-1]),
    ([32, 3, 2, 3, 2, 3, 2, 3, 32], [8, 1, 3, 2, 5, 4, 7, 6, 0]),
    ([32] + [2, 3] * 6 + [32], [13, 2, 1, 4, 3, 6, 5, 8, 7, 10, 9, 12, 11, 0]),
    ([32] + [2] * 13 + [32], [14, 2, 1, 4, 3, 6, 5, 8, 7, 10, 9, 12, 11, 13, 0])])
def test_few_large_tiles_per_step(dims, ptup):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    n = int(np.prod(dims))
    x = torch.arange(n, dtype=torch.float64, device="cuda")
    x = torch.complex(x, -0.5 * x)
    out = q.permute(x, dims, ptup)
    ref = x.reshape(dims).permute([ptup.index(i) for i in range(len(dims))]).reshape(-1)
    assert torch.equal(torch.view_as_real(out), torch.view_as_real(ref))
