"""The mixed form's pair passes: one, two or four lanes per site by the size
(a replica's forces must not depend on which), and the EAM terms as cubics in
r^2 where the splines are smooth, as the splines themselves where they are
not (few, wide knot intervals) and at the edges of the fitted range."""
import numpy as np
import pytest

from cac_b200 import gen
from helpers import LJ, SKIN, rel_err

pytestmark = pytest.mark.gpu


def tables(kind):
    # "kinked": wide knot intervals, whose jumps in curvature no cubic across
    # them follows
    p = gen.EamParams(nr={"coarse": 2000, "kinked": 250}.get(kind, 10000))
    frho, rhor, z2r = p.tables()
    if kind == "smooth":      # taken to zero at the cutoff
        s = ((p.cut - np.arange(p.nr) * p.dr).clip(0.0) / 0.5) ** 4
        rhor, z2r = rhor * s / (1.0 + s), z2r * s / (1.0 + s)
    return dict(nrho=p.nrho, drho=p.drho, nr=p.nr, dr=p.dr, cut=p.cut, mass=p.mass, frho=frho, rhor=rhor, z2r=z2r)


def engine(systems, pair, form, kind="smooth"):
    from cac_b200.api import Engine
    e = Engine(0)
    e.upload_batch(systems) if isinstance(systems, list) else e.upload(systems)
    e.pair_lj(*LJ) if pair == "lj" else e.pair_eam(tables(kind))
    e.set_precision(form)
    e.neighbor(SKIN, 10)
    return e


@pytest.mark.parametrize("kind", ["smooth", "plain", "coarse", "kinked"])
@pytest.mark.parametrize("disp", [None, 0.5])
def test_eam_terms_follow_the_fp64_form(kind, disp):
    """disp 0.5: pairs from 1.3 A apart, below the fitted range as well.  The
    bar is the mixed form's: 1e-5 of the largest force (FP32 pair terms, whose
    rounding is 6e-8 of each term)."""
    s = gen.build_slab(4, 2, 2, 9, temperature=300.0, disp=disp, strain=0.02, seed=8)
    a, b = engine(s, "eam", 0, kind), engine(s, "eam", 1, kind)
    for e in (a, b):
        e.compute()
    for x, y in zip(b.forces(), a.forces()):
        assert rel_err(x, y) < 1e-5
    ea, eb = a.energy(), b.energy()
    assert abs(eb["energy"] - ea["energy"]) < 1e-6 * abs(ea["energy"])
    assert np.abs(eb["virial"] - ea["virial"]).max() < 1e-5 * np.abs(ea["virial"]).max()
    assert np.abs(eb["eatom"] - ea["eatom"]).max() < 1e-5 * np.abs(ea["eatom"]).max()
    # a force-only evaluation gives the same forces as one with tallies
    f0 = b.forces()
    b.compute(0, 0)
    for x, y in zip(b.forces(), f0):
        assert np.array_equal(x, y)
    a.close()
    b.close()


@pytest.mark.parametrize("pair", ["lj", "eam"])
@pytest.mark.parametrize("other", [(4, 3, 1, 9), (8, 5, 1, 18), (8, 6, 1, 81)])
def test_forces_do_not_depend_on_lanes_per_site(pair, other):
    """The same replica alone (four lanes a site) and in batches of 19 k, 120 k
    and 630 k sites (four, two and one): equal bit for bit."""
    s = gen.replica(2500, 50, temperature=300.0, strain=0.01, seed=77)
    alone = engine(s, pair, 1)
    batch = engine([gen.build_slab(*other, temperature=300.0, seed=3), s], pair, 1)
    for e in (alone, batch):
        e.setup()
        e.run_nve(11, 0.001)
    f, nf, gf = alone.forces()
    F, NF, GF = batch.forces()
    assert np.array_equal(F[-s.natoms:], f)
    assert np.array_equal(NF[-s.nelements:], nf) and np.array_equal(GF[-s.nelements:], gf)
    alone.close()
    batch.close()
