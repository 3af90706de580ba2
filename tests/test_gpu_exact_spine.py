"""The exact scan's walk over tiles with special elements: tiles with more of them
than are kept among tiles with a few, as many as the walk stages and more, at the
ends of the array.  Specials are made by ties: while the sum lies in [1/2, 1), an
odd multiple of 2^-54 is half a unit in its last place."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.gpu_util import dev, empty

pytestmark = pytest.mark.gpu

TILE = 2048


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


# (tiles, overflowing tiles, [first, end) of tiles with `k` ties each)
CASES = [
    (40, [0, 1, 39], (5, 38), 3),      # the array's ends
    (300, [290], (5, 255), 4),         # 1000 specials in 250 tiles
    (300, [150, 151, 299], (20, 140), 8),
    (300, [3], (10, 260), 2),          # the last tiles that are staged
    (600, [270, 500], (10, 580), 2),   # more than are staged
    (300, [200], (10, 40), 60),        # more specials than are staged
    (33, [], (1, 33), 31),             # 32 x 31 + the tiles' own two
]


@pytest.mark.parametrize("sch", [0, 1, 3])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_against_oracle(capi, sch, case):
    tiles, over, (a, b), k = CASES[case]
    rng = np.random.default_rng(case)
    N = tiles * TILE - 7
    w = rng.lognormal(size=N)
    w[0] = 1.5 * w.sum()  # the sum is in [1/2, 1) from the first element on
    w /= w.sum()
    at = [t * TILE + np.arange(1, TILE - 7) for t in over]
    at += [t * TILE + rng.choice(TILE - 7, size=k, replace=False) for t in range(a, b)]
    at = np.concatenate(at)
    at = at[at > 0]
    w[at] = (np.round(w[at] * 2.0 ** 54).astype(np.int64) | 1) * 2.0 ** -54
    ref_rep, ref_cf, ref_words = O.resample(sch, w, 9, 1)[:3]
    rep, cf = empty(N, torch.int32), empty(N, torch.int32)
    nb = capi.resample_workspace_size(N)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    wd = dev(w)
    words = capi.resample(sch, N, wd.data_ptr(), capi.threefry_state(9, offset=1),
                          rep.data_ptr(), cf.data_ptr(), ws.data_ptr(), nb)
    assert words == ref_words
    assert np.array_equal(rep.cpu().numpy(), ref_rep)
    assert np.array_equal(cf.cpu().numpy(), ref_cf)
