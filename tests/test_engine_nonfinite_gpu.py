"""A position that is not finite in an engine of one replica: the list maintenance reports ACS_FLAG_NONFINITE and nothing
else (every block of its grid takes part in every barrier), and after the status is cleared the engine works on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(cells, tpa):
    """A reduced-unit LJ lattice of 4 cells^3 atoms, one replica, one thread or a warp per atom in the pair kernel (a warp
    per cell or per atom in the list build)."""
    import torch

    from devinproj_b200.engine import Engine, ForceField
    ff = ForceField()
    ff.n_species, ff.lj, ff.lj_cutoff = 1, 1, 2.5
    ff.mass[0], ff.lj_eps[0], ff.lj_sig[0] = 1.0, 1.0, 1.0
    edge = (4 / 0.8442) ** (1 / 3)
    L = cells * edge
    eng = Engine([dict(n=4 * cells ** 3, box=[L] * 3, dt=0.004, rlist=2.8, half_skin=0.15)], ff, maxnb=160, tpa=tpa)
    grid = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    fcc = np.array([[0.25, 0.25, 0.25], [0.75, 0.75, 0.25], [0.75, 0.25, 0.75], [0.25, 0.75, 0.75]])
    rng = np.random.default_rng(cells)
    pos = ((grid + fcc).reshape(-1, 3) * edge + rng.normal(0, 0.03, (4 * cells ** 3, 3))) % L
    vel = rng.normal(0, 0.85, pos.shape)
    return eng, torch.from_numpy(pos).cuda(), torch.from_numpy(vel).cuda(), torch.zeros(len(pos), dtype=torch.int32,
                                                                                        device="cuda")


@pytest.mark.parametrize("cells,tpa", [(6, 32), (10, 32), (20, 1)])
@pytest.mark.parametrize("atom", [0, -1])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("entry", ["set_state", "load_state"])
def test_nonfinite_position_is_reported_alone(cells, tpa, atom, value, entry):
    from devinproj_b200 import _lib
    eng, pos, vel, sp = _engine(cells, tpa)
    eng.set_state(pos, vel, sp)
    eng.run(3, 0, True)
    assert eng.status().flags == 0
    want = eng.records(1)
    bad = pos.clone()
    bad[atom, 1] = value
    if entry == "set_state":
        eng.set_state(bad, vel, sp)
    else:
        eng.load_state(bad, vel)
    eng.run(3, 0, True)
    assert eng.status(clear=True).flags == _lib.FLAG_NONFINITE
    eng.set_state(pos, vel, sp)
    eng.run(3, 0, True)
    assert eng.status().flags == 0
    assert np.array_equal(eng.records(1), want)
