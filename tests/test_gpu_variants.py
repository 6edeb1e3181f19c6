"""GPU tests of the kernels chosen by size, at the edges of their ranges."""
import numpy as np
import pytest

from oracle import oracle as O
from projects_b200 import gridrec as G
from projects_b200 import phantom as ph

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n,a,S,group", [(16, 5, 1, 4), (32, 40, 3, 4), (64, 45, 7, 4),
                                         (128, 33, 5, 3), (256, 21, 2, 1)])
def test_fbp_groups_same_bits_and_oracle(n, a, S, group):
    """Slices backprojected in groups of 4, 2 and 1 (every remainder of the call and of the
    plan's slice count): the bits of one slice at a time, whose row filter packs the same
    rows, and the oracle's image."""
    th = np.linspace(0.0, 179.0, a).astype(np.float32)
    rng = np.random.default_rng(n + S)
    sinos = rng.uniform(-1.0, 6.0, (S, a, n)).astype(np.float32)  # values beyond 5 are gated
    f = G.FBP(n, a, th, max_slices=group)
    got = f.reconstruct(_dev(sinos)).cpu().numpy()
    f.close()
    one = G.FBP(n, a, th, max_slices=1)
    for s in range(S):
        alone = one.reconstruct(_dev(sinos[s:s + 1])).cpu().numpy()[0]
        np.testing.assert_array_equal(got[s], alone)
        ref = O.port_optimized_fbp(sinos[s], th)
        assert ph.rel_l2(got[s], ref) < 1e-5
    one.close()
