"""Mixed-form EAM engines with different tables side by side in one process:
the passes' shared memory grows with the table's cutoff, and one engine's must
not bound another's."""
import threading

import numpy as np
import pytest

from cac_b200 import gen

pytestmark = pytest.mark.gpu


def engine(cut, s):
    from cac_b200.api import MIXED, Engine
    p = gen.EamParams(cut=cut)
    frho, rhor, z2r = p.tables()
    e = Engine(0)
    e.upload(s)
    e.pair_eam(dict(nrho=p.nrho, drho=p.drho, nr=p.nr, dr=p.dr, cut=p.cut, mass=p.mass, frho=frho, rhor=rhor, z2r=z2r))
    e.set_precision(MIXED)
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
