"""The element sites of the lists (single-precision maps, row by row, the close
calls exactly; entries turned into pair-table indices 32 queries at a time)
against the CPU restatement, entry for entry: distorted and sheared elements,
more elements in reach than are staged at once, lists longer than one turn of
the conversion, and query counts around its blocks."""
import numpy as np
import pytest

from cac_b200 import gen

pytestmark = pytest.mark.gpu

# (copies of the elements, displacement of each node, shear, cutoff, atoms kept, half)
CASES = [(1, 0.0, 0.0, 9.5, 1458, True), (1, 1.2, 0.0, 5.0, 1458, False), (1, 0.8, 0.15, 7.0, 33, True),
         (1, 0.3, -0.1, 2.0, 31, False), (3, 0.5, 0.05, 4.0, 0, True), (20, 0.2, 0.0, 2.0, 32, False),
         (20, 0.4, 0.02, 1.2, 1, True)]


@pytest.mark.parametrize("case", CASES)
def test_element_sites_equal_the_restatement(case, oracle_mod):
    from cac_b200.api import Engine
    copies, amp, shear, cut, na, half = case
    s = gen.build_slab(3, 1, 1, 3, temperature=300.0, seed=6)
    rng = np.random.default_rng(17)
    nx = np.concatenate([s.nodex + rng.uniform(-0.4, 0.4, (1, 1, 3)) * (c > 0) for c in range(copies)])
    rel = nx - nx.mean(axis=1, keepdims=True)
    nx[..., 0] += shear * rel[..., 1]
    nx[..., 2] += shear * rel[..., 0]
    s.nodex = nx + rng.uniform(-amp, amp, nx.shape)
    s.nodev = np.concatenate([s.nodev] * copies)
    s.x, s.v = s.x[s.natoms - na:].copy(), s.v[s.natoms - na:].copy()
    gen.wrap_into_box(s)
    st = oracle_mod.OracleState(s)
    e = Engine(0)
    e.upload(s)
    e.pair_lj(0.4093, 2.338, cut)
    e.neighbor(0.5, 10)
    e.build_lists(half=half)
    assert np.array_equal(e.neighbor_list(), oracle_mod.build_list(st, cut + 0.5, False).canonical(s.natoms))
    if half:
        assert np.array_equal(e.neighbor_list(half=True), oracle_mod.build_list(st, cut + 0.5, True).canonical(s.natoms))
    e.close()


@pytest.mark.parametrize("na,ne,scale", [(9, 12, 1.0), (0, 1, 2.5), (700, 3, 3.0), (31000, 2, 2.0), (31003, 12, 1.5)])
def test_scattered_queries_equal_the_restatement(na, ne, scale, oracle_mod):
    """Atoms and elements far apart, so that the queries of a warp stand in
    many places (eight or 32 of them to a warp, below and above 30,000)."""
    from cac_b200.api import Engine
    s = gen.build_slab(3, 1, 1, 3, temperature=300.0, seed=8)
    rng = np.random.default_rng(23)
    s.boxhi = s.boxlo + scale * (s.boxhi - s.boxlo)
    s.nodex = s.nodex[:ne] - s.nodex[:ne].mean(axis=1, keepdims=True) + rng.uniform(s.boxlo, s.boxhi, (ne, 1, 3))
    s.nodev = s.nodev[:ne].copy()
    s.x = rng.uniform(s.boxlo, s.boxhi, (na, 3))
    s.v = np.zeros_like(s.x)
    gen.wrap_into_box(s)
    cut = 2.5 if na < 31000 else 0.8
    st = oracle_mod.OracleState(s)
    e = Engine(0)
    e.upload(s)
    e.pair_lj(0.4093, 2.338, cut)
    e.neighbor(0.5, 10)
    e.build_lists()
    assert np.array_equal(e.neighbor_list(), oracle_mod.build_list(st, cut + 0.5, False).canonical(s.natoms))
    e.close()
