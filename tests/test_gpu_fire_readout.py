"""The thermo read-out behind a minimisation: the potential energy of the last
evaluation is that of the current step, wherever in its chunk of 25 the
minimisation ended."""
import numpy as np
import pytest

from cac_b200 import gen
from helpers import LJ

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pair,form", [("lj", 0), ("eam", 0), ("eam", 1)])
@pytest.mark.parametrize("maxiter,ftol,every", [(0, 1e-9, 10), (11, 1e-9, 2), (24, 1e-9, 10), (25, 1e-9, 7), (40, 1e-9, 10),
                                                (40, 1e3, 5)])
def test_energy_after_minimisation(pair, form, maxiter, ftol, every, tmp_path):
    from cac_b200.api import Engine
    setfl = str(tmp_path / "cu.setfl")
    gen.write_setfl(gen.EamParams(), setfl)
    e = Engine(0)
    e.upload(gen.build_slab(3, 1, 1, 6, temperature=0.0, disp=0.1, seed=5))
    e.pair_lj(*LJ) if pair == "lj" else e.pair_eam(setfl)
    e.set_precision(form)
    e.neighbor(1.0, every)
    _, _, energy, _ = e.minimize_fire(ftol=ftol, maxiter=maxiter)
    t = e.thermo()
    # the same sum of the same terms, unless a rebuild behind the end has put
    # them in another order
    assert abs(t["pe"] - energy) < (1e-12 if form == 0 else 1e-6) * abs(energy)
    assert np.isfinite(t["etotal"])
    e.close()
