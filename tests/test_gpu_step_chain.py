"""Runs whose kernels start before the one ahead of them has ended, against
the same runs with the kernels timed one by one (which puts an event between
any two, so that each waits for the one before), bit for bit: both forms, both
pair styles, a batch, a thermostat, FIRE, and a system above the size from which
launches are plain."""
import numpy as np
import pytest

from cac_b200 import gen

pytestmark = pytest.mark.gpu


def states(shapes, form, pair, what, steps, setfl):
    from cac_b200.api import Engine
    out = []
    for apart in (False, True):
        s = [gen.build_slab(*shape, temperature=300.0, seed=3 + i) for i, shape in enumerate(shapes)]
        e = Engine(0)
        if len(s) > 1:
            e.upload_batch(s)
        else:
            e.upload(s[0])
        if pair == "lj":
            e.pair_lj(0.4093, 2.338, 5.5)
        else:
            e.pair_eam(setfl)
        e.set_precision(form)
        e.neighbor(1.0, 5)
        if what == "langevin":
            e.langevin(300.0, 300.0, 0.1, 777)
        e.profile(apart)
        if what == "fire":
            e.minimize_fire(ftol=1e-9, maxiter=30)
        else:
            e.run_nve(steps, 0.002)
        out.append([np.array(a, copy=True) for a in e.state()] + [np.array(a, copy=True) for a in e.forces()])
        e.close()
    return out


@pytest.mark.parametrize("shapes,form,pair,what", [
    ([(3, 1, 1, 3)], 0, "lj", "nve"), ([(4, 2, 1, 9)], 1, "lj", "nve"), ([(4, 2, 1, 9)], 0, "eam", "nve"),
    ([(4, 2, 3, 9)], 1, "eam", "nve"), ([(3, 1, 1, 3)], 0, "eam", "langevin"), ([(3, 1, 1, 3)], 1, "eam", "langevin"),
    ([(3, 1, 1, 3)], 0, "eam", "fire"), ([(3, 1, 1, 3), (4, 2, 1, 9), (3, 1, 1, 6)], 0, "lj", "nve"),
    ([(3, 1, 1, 3), (4, 2, 1, 9), (3, 1, 1, 6)], 1, "eam", "nve"), ([(12, 8, 2, 102)], 1, "lj", "nve")])
def test_runs_equal_kernels_one_by_one(shapes, form, pair, what, tmp_path):
    setfl = str(tmp_path / "cu.setfl")
    gen.write_setfl(gen.EamParams(), setfl)
    a, b = states(shapes, form, pair, what, 23 if shapes[0][0] < 12 else 7, setfl)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
