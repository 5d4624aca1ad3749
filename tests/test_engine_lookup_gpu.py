"""The engine's lists where its warps look candidates up in the stencil's occupied cells: gases whose cells are mostly empty,
cells of several chunks, axes of one cell, replicas that are one cell, in both builds, against a k-d tree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RL = 2.8


# replicas as (atoms, box edges in list radii)
@pytest.mark.parametrize("replicas", [
    [(40, (9.3, 8.1, 7.5))],                                   # one atom in 14 cells
    [(1, (3.2, 3.4, 3.1))], [(31, (1.2, 1.1, 1.4))], [(33, (2.9, 2.2, 2.5))], [(700, (2.9, 2.8, 2.6))],
    [(900, (4.1, 1.7, 5.2))], [(900, (2.3, 3.3, 2.9))], [(2500, (3.1, 3.2, 3.3))],
    [(300, (2.5, 2.6, 2.4)), (64, (1.3, 1.3, 1.3)), (500, (5.2, 4.4, 3.6)), (128, (2.9, 3.1, 4.2)), (5, (6.0, 6.0, 6.0))]])
@pytest.mark.parametrize("tpa", [1, 8, 32])
def test_lists_are_the_pairs_within_the_radius(replicas, tpa):
    """FP64 decides in the band, so the sets are equal; pairs within 1e-12 of the radius, which the k-d tree may round
    otherwise, are asked not to occur."""
    import torch
    from scipy.spatial import cKDTree

    from devinproj_b200.engine import Engine, ForceField
    ff = ForceField()
    ff.n_species, ff.lj, ff.lj_cutoff = 1, 1, 2.5
    ff.mass[0], ff.lj_eps[0], ff.lj_sig[0] = 1.0, 1e-9, 1.0   # weak, and at rest: only the first lists count
    boxes = [np.array(b) * RL for _, b in replicas]
    rng = np.random.default_rng(len(replicas) + replicas[0][0])
    pos = [rng.uniform(0, 1, (n, 3)) * b for (n, _), b in zip(replicas, boxes)]
    want = set()
    start = 0
    for p, b in zip(pos, boxes):
        pairs = cKDTree(p, boxsize=b).query_pairs(RL * (1 + 1e-12), output_type="ndarray")
        d = p[pairs[:, 1]] - p[pairs[:, 0]]
        r = np.sqrt(np.sum((d - b * np.round(d / b)) ** 2, axis=1))
        assert np.all(np.abs(r - RL) > 1e-12 * RL)
        for i, j in pairs:
            want |= {(start + int(i), start + int(j)), (start + int(j), start + int(i))}
        start += len(p)
    most = max([1] + list(np.bincount([i for i, _ in want]))) if want else 1
    eng = Engine([dict(n=len(p), box=list(b), dt=1e-6, rlist=RL, half_skin=0.15) for p, b in zip(pos, boxes)], ff,
                 maxnb=int(most + 8) // 8 * 8, tpa=tpa)
    all_pos = torch.from_numpy(np.concatenate(pos)).cuda()
    eng.set_state(all_pos, torch.zeros_like(all_pos), torch.zeros(start, dtype=torch.int32, device="cuda"))
    eng.check("lists")
    keys, _ = eng.list_entries()
    k = keys.cpu().numpy() >> 1
    got = list(zip((k // start).tolist(), (k % start).tolist()))
    assert len(got) == len(set(got)) and set(got) == want
