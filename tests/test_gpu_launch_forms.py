"""Resident blocks and SM-local runs against one grid launch per pass, bit for
bit, at sizes where both are used: FP64 EAM passes from 100,000 i-sites up
(runs of 64 list slots, the last one short), and mixed passes with more list
slots than the resident blocks take in one stride, alone and in a batch."""
import numpy as np
import pytest

from cac_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,shapes", [(0, [(8, 5, 1, 18)]), (1, [(8, 5, 1, 18)]), (1, [(8, 6, 1, 81)]),
                                         (1, [(6, 4, 2, 15), (3, 1, 1, 3), (7, 4, 1, 18)])])
def test_resident_blocks_equal_grid_launches(form, shapes, tmp_path):
    from cac_b200.api import Engine
    setfl = str(tmp_path / "cu.setfl")
    gen.write_setfl(gen.EamParams(), setfl)
    systems = [gen.build_slab(*shape, temperature=300.0, strain=0.01, seed=31 + i) for i, shape in enumerate(shapes)]
    sites = sum(s.natoms + 8 * s.nelements for s in systems)
    assert sites > 100000 and (form or sites % 64)
    out = []
    for on in (True, False):
        e = Engine(0)
        e.upload_batch(systems) if len(systems) > 1 else e.upload(systems[0])
        e.pair_eam(setfl)
        e.set_precision(form)
        e.neighbor(1.0, 5)
        e.work_queue(on)
        e.setup()
        e.run_nve(12, 0.001)
        out.append([np.array(a, copy=True) for a in (*e.state(), *e.forces())])
        e.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
