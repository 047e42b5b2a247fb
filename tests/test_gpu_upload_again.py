"""A second system in the same engine: the snapshot and the per-site read-outs of
one of another size are gone (their arrays have that size), as they are in an
engine that never had them."""
import numpy as np
import pytest

from cac_b200 import gen
from helpers import LJ

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("second", [(3, 2, 2, 9), (3, 1, 1, 3)])
@pytest.mark.parametrize("form", [0, 1])
def test_other_sizes_keep_nothing(second, form):
    from cac_b200.api import CacB200Error, Engine
    e = Engine(0)
    e.upload(gen.build_slab(3, 1, 1, 6, temperature=300.0, seed=1))
    e.pair_lj(*LJ)
    e.set_precision(form)
    e.neighbor(1.0, 10)
    e.compute()
    e.snapshot()
    e.upload(gen.build_slab(*second, temperature=300.0, seed=2))
    for call in (e.restore, e.replica_energy, e.energy, lambda: e.device_array("eatom"), lambda: e.device_array("vnode")):
        with pytest.raises(CacB200Error):
            call()
    e.compute()
    e.snapshot()
    want = np.array(e.state()[0], copy=True)
    assert np.isfinite(e.replica_energy()).all()
    e.run_nve(3, 0.001)
    e.restore()
    assert np.array_equal(e.state()[0], want)
    e.close()


def test_same_sizes_keep_the_snapshot():
    from cac_b200.api import Engine
    a, b = (gen.build_slab(3, 1, 1, 6, temperature=300.0, seed=k) for k in (1, 2))
    e = Engine(0)
    e.upload(a)
    e.snapshot()
    e.upload(b)
    e.restore()
    assert np.array_equal(e.state()[0], a.x) and np.array_equal(e.state()[2], a.nodex)
    e.close()
