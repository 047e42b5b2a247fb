"""Element sites where an element is hundreds of times larger than the cutoff
(positions along it are then too long for single precision to tell which sites
are in reach), against the CPU restatement, entry for entry."""
import numpy as np
import pytest

from cac_b200 import gen

pytestmark = pytest.mark.gpu

CUT, SKIN = 95.0, 5.0


def large_element(length, seed):
    """One element 1.8 box lengths long in its third direction, and an atom
    beside each of its sites, just inside the list cutoff and square to that
    direction."""
    rng = np.random.default_rng(seed)
    hi = np.full(3, length)
    edges = np.array([[120.0, 2400.0, 0.0], [-90.0, 60.0, 2400.0], [1.8 * length, 130.0, 70.0]])
    origin = 0.5 * hi - 0.5 * edges.sum(axis=0)
    nodex = origin + (gen.HEX_CORNERS / 8.0) @ edges
    i, j, k = np.meshgrid(*[np.arange(9) / 8.0] * 3, indexing="ij")
    sites = origin + np.stack([i, j, k], axis=-1).reshape(-1, 3) @ edges
    along = edges[2] / np.linalg.norm(edges[2])
    side = rng.normal(size=sites.shape)
    side -= (side @ along)[:, None] * along
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    x = sites + side * (CUT + SKIN - 10.0 ** rng.uniform(-5.0, -2.0, (len(sites), 1)))
    s = gen.System(boxlo=np.zeros(3), boxhi=hi, x=x, v=np.zeros_like(x), nodex=nodex[None], nodev=np.zeros((1, 8, 3)))
    gen.wrap_into_box(s)
    return s


@pytest.mark.parametrize("length", [8000.0, 25000.0])
def test_sites_of_a_large_element(length, oracle_mod):
    from cac_b200.api import Engine
    s = large_element(length, 3)
    st = oracle_mod.OracleState(s)
    want = oracle_mod.build_list(st, CUT + SKIN, False).canonical(s.natoms)
    assert (want[:, 1] == 1).sum() >= 729
    e = Engine(0)
    e.upload(s)
    e.pair_lj(0.4093, 60.0, CUT)
    e.neighbor(SKIN, 10)
    e.build_lists()
    assert np.array_equal(e.neighbor_list(), want)
    e.close()
