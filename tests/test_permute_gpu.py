"""The tiled transpose on extents that are not powers of two: several tiles of odd size per step,
a last step with fewer, several steps per block (the next step's bases are decoded a step
ahead), and the smallest tensors that take a tile. Bit-exact against numpy's transpose of a
tensor that holds its own indices."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import qtnh_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[33, 31], [3] * 7, [3] * 11, [3] * 13, [5] * 9, [6] * 7, [7] * 7, [2, 3] * 6,
                                  [3, 64, 5, 32, 7, 9], [2] * 18, [11, 13, 17, 19, 23]])
@pytest.mark.parametrize("seed", range(3))
def test_tiled_permute_any_extents(dims, seed):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng = np.random.default_rng(seed + 10 * len(dims))
    ptup = [int(x) for x in rng.permutation(len(dims))]
    if seed == 0:
        ptup = list(range(len(dims)))[::-1]
    a = np.arange(int(np.prod(dims)), dtype=np.float64).reshape(dims)
    a = a - 0.5j * a
    out = q.permute(torch.from_numpy(a.reshape(-1)).cuda(), dims, ptup)
    torch.cuda.synchronize()
    ref = np.transpose(a, np.argsort(ptup))  # axis i goes to position ptup[i]
    assert np.array_equal(out.cpu().numpy(), ref.reshape(-1))
