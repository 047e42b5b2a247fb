"""Atom lists in boxes thousands of A long, where 32 consecutive sorted atoms
(a chunk of the build) stand far apart in one row of cells, against the CPU
restatement, entry for entry."""
import numpy as np
import pytest

from cac_b200 import gen

pytestmark = pytest.mark.gpu


def long_box(length, gaps, fill, seed):
    """Groups of eight atoms in some rows of cells, `gaps` A apart in x, and
    `fill` more anywhere."""
    rng = np.random.default_rng(seed)
    hi = np.array([length, 60.0, 60.0])
    x = [rng.uniform(0.0, 1.0, (fill, 3)) * hi]
    for row in range(6):
        y = 3.4 + 9.0 * row
        for gap in gaps:
            x.append(np.array([40.0 + gap, y, y]) + rng.uniform(-3.0, 3.0, (8, 3)))
    x = np.concatenate(x)
    none = np.zeros((0, 8, 3))
    return gen.System(boxlo=np.zeros(3), boxhi=hi, x=x, v=np.zeros_like(x), nodex=none, nodev=none.copy())


# 2,048 and 4,096 A are where fixed-point positions of 2^-20 A from the first
# atom's cell would change sign and repeat; above 38,000 atoms a chunk takes one
# warp, below four
@pytest.mark.parametrize("length,gaps,fill", [(2500.0, (0.0, 2048.0), 0), (4200.0, (0.0, 4096.0), 0),
                                              (9000.0, (0.0, 2045.0, 4096.0, 6144.0, 8191.0), 0),
                                              (9000.0, (0.0, 1500.0, 3548.0, 4096.0), 40000)])
def test_groups_far_apart_in_a_row(length, gaps, fill, oracle_mod):
    from cac_b200.api import Engine
    s = long_box(length, gaps, fill, 5)
    st = oracle_mod.OracleState(s)
    e = Engine(0)
    e.upload(s)
    e.pair_lj(0.4093, 2.338, 5.5)
    e.neighbor(1.0, 10)
    for half in (False, True):
        e.build_lists(half=half)
        want = oracle_mod.build_list(st, 6.5, False).canonical(s.natoms)
        assert len(want) > 300
        assert np.array_equal(e.neighbor_list(), want)
        if half:
            assert np.array_equal(e.neighbor_list(half=True), oracle_mod.build_list(st, 6.5, True).canonical(s.natoms))
    e.close()


def test_cells_wider_than_the_fixed_point_screen_covers(oracle_mod):
    """A cutoff of 700 A (two cells of 750 A in each direction)."""
    from cac_b200.api import Engine
    rng = np.random.default_rng(6)
    hi = np.full(3, 1500.0)
    x = rng.uniform(0.0, 1.0, (200, 3)) * hi
    none = np.zeros((0, 8, 3))
    s = gen.System(boxlo=np.zeros(3), boxhi=hi, x=x, v=np.zeros_like(x), nodex=none, nodev=none.copy())
    st = oracle_mod.OracleState(s)
    e = Engine(0)
    e.upload(s)
    e.pair_lj(0.4093, 300.0, 700.0)
    e.neighbor(20.0, 10)
    e.build_lists(half=True)
    assert np.array_equal(e.neighbor_list(), oracle_mod.build_list(st, 720.0, False).canonical(s.natoms))
    assert np.array_equal(e.neighbor_list(half=True), oracle_mod.build_list(st, 720.0, True).canonical(s.natoms))
    e.close()


@pytest.mark.parametrize("boxes", [3, 4, -3])
@pytest.mark.parametrize("axes", [(2,), (0, 1, 2)])
def test_positions_boxes_away_are_refused(boxes, axes):
    """Atoms without elements whose positions are given several box lengths
    away, where one wrap leaves them outside: their neighbours stand under
    images that list entries cannot hold, and the build says so."""
    from cac_b200.api import CacB200Error, Engine
    s = gen.build_slab(3, 1, 1, 6, temperature=10.0, seed=1)
    s.nodex, s.nodev = s.nodex[:0], s.nodev[:0]
    for d in axes:
        s.x[:, d] += boxes * (s.boxhi - s.boxlo)[d]
    e = Engine(0)
    e.upload(s)
    e.pair_lj(0.4093, 2.338, 5.5)
    e.neighbor(1.0, 10)
    with pytest.raises(CacB200Error, match="image"):
        e.build_lists()
    e.close()
