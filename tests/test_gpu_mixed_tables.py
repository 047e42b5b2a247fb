"""Mixed-form EAM engines with different tables: side by side in one process (the
passes' shared memory grows with the table's cutoff, and one engine's must not
bound another's), and their energies and virials, whose records come beside
those of the forces."""
import threading

import numpy as np
import pytest

from cac_b200 import gen

pytestmark = pytest.mark.gpu


def engine(cut, s, form=1):
    from cac_b200.api import Engine
    p = gen.EamParams(cut=cut)
    frho, rhor, z2r = p.tables()
    e = Engine(0)
    e.upload(s)
    e.pair_eam(dict(nrho=p.nrho, drho=p.drho, nr=p.nr, dr=p.dr, cut=p.cut, mass=p.mass, frho=frho, rhor=rhor, z2r=z2r))
    e.set_precision(form)
    e.neighbor(1.0, 10)
    return e


def test_two_tables_on_two_threads():
    s = gen.build_slab(6, 3, 2, 9, temperature=300.0, seed=3)      # 27,972 sites: resident blocks, records eight times
    engines = [engine(cut, s) for cut in (5.0, 7.0)]
    want = []
    for e in engines:
        e.compute(0, 0)
        want.append([np.array(a, copy=True) for a in e.forces()])
    failures = []

    def work(e, w):
        try:
            for k in range(1500):
                e.compute(0, 0)
                if k % 250 == 0 and not all(np.array_equal(a, b) for a, b in zip(e.forces(), w)):
                    failures.append("forces differ")
        except Exception as ex:
            failures.append(str(ex))

    threads = [threading.Thread(target=work, args=a) for a in zip(engines, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]
    for e in engines:
        e.close()


# four, two and one lanes a site; few and many records
@pytest.mark.parametrize("shape,cut", [((4, 2, 1, 9), 5.5), ((6, 3, 2, 9), 7.0), ((8, 5, 1, 18), 5.5), ((8, 6, 1, 81), 7.0)])
def test_tallies_follow_the_fp64_form(shape, cut):
    """The bar is the mixed form's, 1e-5 of the largest value; forces are the
    same bit for bit with and without tallies."""
    s = gen.build_slab(*shape, temperature=300.0, strain=0.01, seed=9)
    a, b = engine(cut, s, 0), engine(cut, s, 1)
    for e in (a, b):
        e.compute()
    ea, eb = a.energy(), b.energy()
    assert abs(eb["energy"] - ea["energy"]) < 1e-6 * abs(ea["energy"])
    for k in ("eatom", "enode", "virial", "vatom", "vnode"):
        assert np.abs(eb[k] - ea[k]).max() < 1e-5 * np.abs(ea[k]).max(), k
    want = [np.array(f, copy=True) for f in b.forces()]
    b.compute(0, 0)
    assert all(np.array_equal(f, w) for f, w in zip(b.forces(), want))
    a.close()
    b.close()
