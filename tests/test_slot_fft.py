"""The special FFT of fides_encode / fides_decode at every split of its stages: the last
min(log2 n, 7) run on contiguous blocks and the others on strided sub-problems, each two a round
with a single one left over when their number is odd.  The FP64 error of a radix-2 FFT of 2^15
unit-range slots is below 16 stages * 2^-52 * sqrt(n) of the slots; the rounding of a coefficient
adds at most sqrt(N) / 2 at the scale, so 1e-9 at scale 2^45 leaves the FFT room and no
wrong stage any."""
import numpy as np
import pytest

import oracle as O
from ckks_host import encode, xrng
from test_encode import check_encoded

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C(fides):
    from fides_b200 import params as P
    prm = P.config_c(4)
    return prm, O.Oracle(prm.logN, prm.q, prm.p, prm.dnum), fides.Context(prm.logN, prm.q, prm.p, prm.dnum)


@pytest.mark.parametrize("logn", [0, 1, 2, 5, 6, 7, 8, 9, 11, 14, 15])
def test_every_split_of_the_stages(fides, C, logn):
    import torch
    prm, o, ctx = C
    N, n = prm.N, 1 << logn
    rng = xrng(2500 + logn)
    z = rng.uniform(-1, 1, (2, n)) + 1j * rng.uniform(-1, 1, (2, n))
    pts = ctx.encode(torch.from_numpy(z), 2.0 ** 45, 2)
    for i in range(2):
        ref = np.zeros(N)
        ref[::N // (2 * n)] = encode(z[i], 2 * n, 2.0 ** 45)
        check_encoded(fides, o, ctx, pts[i], ref, prm.q, 2)
    back = ctx.decode(pts, 2.0 ** 45, n_slots=n).cpu().numpy()
    assert np.abs(back - z).max() < 1e-9
