"""The FP64 pair passes: two or four lanes per site by the size (a replica's
forces must not depend on which), and the knot lookup at the ends of the
spline tables, against the CPU restatement."""
import numpy as np
import pytest

from cac_b200 import gen
from helpers import LJ, SKIN, rel_err

pytestmark = pytest.mark.gpu


def engine(systems, pair, setfl=None):
    from cac_b200.api import Engine
    e = Engine(0)
    e.upload_batch(systems) if isinstance(systems, list) else e.upload(systems)
    e.pair_lj(*LJ) if pair == "lj" else e.pair_eam(setfl)
    e.neighbor(SKIN, 10)
    return e


@pytest.mark.parametrize("nr,cut_scale", [(10000, 1.0), (2000, 1.0), (500, 1.01), (500, 0.97)])
def test_knots_at_the_ends_of_the_tables(nr, cut_scale, oracle_mod, tmp_path):
    """cut_scale > 1: pairs beyond the last knot; < 1: a table longer than the
    cutoff.  The bar is the FP64 parity bar."""
    p = gen.EamParams(nr=nr)
    path = str(tmp_path / "t.setfl")
    gen.write_setfl(p, path)
    lines = open(path).read().split("\n")
    w = lines[4].split()
    lines[4] = " ".join(w[:4] + [repr(float(w[4]) * cut_scale)])
    open(path, "w").write("\n".join(lines))
    s = gen.build_slab(3, 1, 2, 6, temperature=300.0, disp=0.4, seed=21)
    e = engine(s, "eam", path)
    e.compute()
    st = oracle_mod.OracleState(s)
    L = oracle_mod.build_list(st, 5.0 * cut_scale + SKIN, True)
    oracle_mod.eam_forces(st, L, oracle_mod.Eam(path))
    f, nf, _ = e.forces()
    assert rel_err(f, st.f) < 1e-10 and rel_err(nf, st.nodef) < 1e-10
    e.close()


@pytest.mark.parametrize("pair", ["lj", "eam"])
@pytest.mark.parametrize("other", [(4, 3, 1, 9), (8, 5, 1, 18)])
def test_forces_do_not_depend_on_lanes_per_site(pair, other, tmp_path):
    """The same replica alone (four lanes a site) and in batches of 19 k and
    120 k sites (four and two): equal bit for bit, with and without tallies."""
    path = str(tmp_path / "cu.setfl")
    gen.write_setfl(gen.EamParams(), path)
    s = gen.replica(2500, 50, temperature=300.0, strain=0.01, seed=77)
    alone = engine(s, pair, path)
    batch = engine([gen.build_slab(*other, temperature=300.0, seed=3), s], pair, path)
    for e in (alone, batch):
        e.setup()
        e.run_nve(11, 0.001)
    for tally in (False, True):
        if tally:
            alone.compute()
            batch.compute()
            assert np.array_equal(batch.energy()["eatom"][-s.natoms:], alone.energy()["eatom"])
        f, nf, gf = alone.forces()
        F, NF, GF = batch.forces()
        assert np.array_equal(F[-s.natoms:], f)
        assert np.array_equal(NF[-s.nelements:], nf) and np.array_equal(GF[-s.nelements:], gf)
    alone.close()
    batch.close()
