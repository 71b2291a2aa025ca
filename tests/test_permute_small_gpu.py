"""Tiled transposes of one step per block, whose tile bases are decoded in step, and the sizes where
blocks get a second one: a single tile and a few, of powers of two and of other sizes; tiles of 32 to
1024 elements, one to several per step; a last step with fewer tiles. Bit-exact against a plain
transpose of a tensor that holds its own indices."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu

SMALL = [([2] * n, [int(v) for v in np.random.default_rng(7 * n + s).permutation(n)]) for n in (7, 9, 12, 16, 17, 18, 19)
         for s in (0, 1)]
PLAIN = [([a, b], [1, 0]) for a, b in ((2, 32), (2, 33), (32, 64), (33, 32), (100, 32), (256, 33), (300, 33), (16, 33),
                                       (64, 1000), (100, 1024), (17, 1024), (1000, 7), (37, 2048), (4096, 64), (4864, 64),
                                       (9729, 32), (32, 4096), (64, 4096), (152, 2048), (155648, 4))]


@pytest.mark.parametrize("dims,ptup", SMALL + PLAIN + [([3] * 4, [1, 2, 3, 0]), ([3] * 8, [1, 2, 0, 4, 7, 6, 3, 5]),
                                                       ([3] * 11, [9, 7, 4, 8, 0, 1, 2, 10, 6, 3, 5]),
                                                       ([2, 2**15, 2], [2, 1, 0]), ([5] * 6, [3, 0, 2, 5, 4, 1])])
def test_small_transposes(dims, ptup):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    x = torch.arange(int(np.prod(dims)), dtype=torch.float64, device="cuda")
    x = torch.complex(x, -0.5 * x)
    out = q.permute(x, dims, ptup)
    ref = x.reshape(dims).permute([ptup.index(i) for i in range(len(dims))]).reshape(-1)
    assert torch.equal(torch.view_as_real(out), torch.view_as_real(ref))
