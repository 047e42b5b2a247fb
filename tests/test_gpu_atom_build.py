"""The atom list build (masks of 32 candidates, one warp or four per chunk of
32 sorted atoms) against the CPU restatement, entry for entry: chunk
remainders, cells holding more candidates than one round of masks, a single
cell along an axis' neighbourhood, positions on the box faces, and sizes on
both sides of the line between the four-warp and one-warp forms."""
import numpy as np
import pytest

from cac_b200 import gen
from helpers import SKIN

pytestmark = pytest.mark.gpu

# (nx, ny, le, la, strain, cutoff, atoms dropped from the end)
SHAPES = [(3, 1, 1, 3, 0.0, 5.5, 0), (3, 1, 1, 3, 0.0, 5.5, 17), (3, 1, 1, 3, 0.0, 5.5, 18), (3, 1, 1, 3, 0.02, 5.5, 1457),
          (3, 1, 1, 6, 0.0, 11.0, 5), (4, 2, 1, 9, -0.05, 8.0, 3), (3, 1, 1, 3, 0.0, 2.0, 0),
          (6, 4, 1, 12, 0.01, 5.0, 7), (7, 4, 1, 9, 0.0, 9.0, 1)]


@pytest.mark.parametrize("shape", SHAPES)
def test_lists_equal_the_restatement(shape, oracle_mod):
    from cac_b200.api import Engine
    nx, ny, le, la, strain, cut, drop = shape
    s = gen.build_slab(nx, ny, le, la, temperature=300.0, strain=strain, seed=sum(shape[:4]))
    n = s.natoms - drop
    s.x, s.v = s.x[:n].copy(), s.v[:n].copy()
    # some atoms on the lower faces of the box, and just inside the upper ones
    for d in range(3):
        s.x[d::97, d] = s.boxlo[d]
        s.x[d + 3::89, d] = np.nextafter(s.boxhi[d], s.boxlo[d])
    st = oracle_mod.OracleState(s)
    want = {half: oracle_mod.build_list(st, cut + SKIN, half).canonical(s.natoms) for half in (False, True)}
    e = Engine(0)
    e.upload(s)
    e.pair_lj(0.4093, 2.338, cut)
    e.neighbor(SKIN, 10)
    for queue in (True, False):
        e.work_queue(queue)
        e.build_lists()
        assert np.array_equal(e.neighbor_list(), want[False])
    e.build_lists(half=True)
    assert np.array_equal(e.neighbor_list(), want[False])
    assert np.array_equal(e.neighbor_list(half=True), want[True])
    e.close()


@pytest.mark.parametrize("copies,na", [(1, 1458), (6, 1458), (6, 0), (6, 40000)])
def test_element_walk_with_crowded_cells(copies, na, oracle_mod):
    """Elements lying over one another, so that an element cell holds more than
    32 of them (36 with six copies), for both forms of the element walk (eight
    atoms to a warp below 30,000 queries)."""
    from cac_b200.api import Engine
    s = gen.build_slab(3, 1, 1, 3, temperature=300.0, seed=4)
    rng = np.random.default_rng(9)
    s.nodex = np.concatenate([s.nodex + rng.uniform(-0.5, 0.5, (1, 1, 3)) for _ in range(copies)])
    s.nodev = np.concatenate([s.nodev] * copies)
    if na > s.natoms:      # more atoms, anywhere
        s.x = np.concatenate([s.x, rng.uniform(s.boxlo, s.boxhi, (na - s.natoms, 3))])
        s.v = np.zeros_like(s.x)
    s.x, s.v = s.x[:na].copy(), s.v[:na].copy()
    gen.wrap_into_box(s)
    cut = 3.0 if na < 40000 else 0.6
    st = oracle_mod.OracleState(s)
    want = oracle_mod.build_list(st, cut + 0.4, False).canonical(s.natoms)
    e = Engine(0)
    e.upload(s)
    e.pair_lj(0.4093, 2.338, cut)
    e.neighbor(0.4, 10)
    e.build_lists()
    assert np.array_equal(e.neighbor_list(), want)
    e.close()
