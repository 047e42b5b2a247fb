"""Two atoms at one place: their own pair force is no number, but their densities
and with them the forces and energies of every other site are those of the CPU
restatement."""
import numpy as np
import pytest

from cac_b200 import gen
from helpers import SKIN, rel_err

pytestmark = pytest.mark.gpu


# bars: FP64 parity, and the mixed form's for forces and energies
@pytest.mark.parametrize("form,bar", [(0, 1e-10), (1, 1e-5)])
@pytest.mark.parametrize("shape", [(3, 1, 1, 6), (8, 5, 1, 18)])    # four and two lanes a site
def test_other_sites_of_a_coincident_pair(form, bar, shape, oracle_mod, tmp_path):
    from cac_b200.api import Engine
    path = str(tmp_path / "t.setfl")
    gen.write_setfl(gen.EamParams(rhomax=300.0), path)       # the pair's own density is about 120
    s = gen.build_slab(*shape, temperature=300.0, seed=12)
    a, b = s.natoms // 2, s.natoms // 2 + 1
    s.x[b] = s.x[a]
    st = oracle_mod.OracleState(s)
    ev = oracle_mod.eam_forces(st, oracle_mod.build_list(st, 5.0 + SKIN, True), oracle_mod.Eam(path))
    others = np.ones(s.natoms, bool)
    others[[a, b]] = False
    assert np.isfinite(st.f[others]).all() and not np.isfinite(st.f[~others]).any()
    e = Engine(0)
    e.upload(s)
    e.pair_eam(path)
    e.set_precision(form)
    e.neighbor(SKIN, 10)
    for tallies in (True, False):
        e.compute(*(() if tallies else (0, 0)))
        f, nf, _ = e.forces()
        assert rel_err(f[others], st.f[others]) < bar and rel_err(nf, st.nodef) < bar
        assert not np.isfinite(f[~others]).any()
        if tallies:
            want = ev.eatom[others]
            assert np.abs(e.energy()["eatom"][others] - want).max() < bar * np.abs(want).max()
    e.close()
