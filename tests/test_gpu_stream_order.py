"""Work queued on a context's own stream comes before an ensemble's steps: steps
launched without waiting for them, then a time set, then the ensemble, against the
same calls with a synchronisation after each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hc(harm_lib):
    import harm_cool_b200
    return harm_cool_b200


def test_ensemble_waits_for_its_members(hc):
    shapes = [(96, 96, 1), (24, 20, 4), (40, 200, 1)]
    both = []
    for wait in (True, False):
        ctxs = []
        for s in shapes:
            c = hc.Context(hc.torus_problem(*s))
            c.init_torus()
            c.run(2)
            ctxs.append(c)
        ens = hc.Ensemble(ctxs)
        ens.run(1)
        for rounds in range(3):
            for c in ctxs:
                t, dt = c.time()
                for _ in range(12):
                    c.step_ch()
                c.set_time(t, 0.5 * dt)
                c.set_mass(1.0, 2.0)
                if wait:
                    c.sync()
            ens.run(2)
        both.append([(c.get_prims(), c.time(), c.diag()["mass_in"]) for c in ctxs])
        ens.close()
        for c in ctxs:
            c.close()
    for a, b in zip(*both):
        assert np.array_equal(a[0], b[0]) and a[1:] == b[1:]
