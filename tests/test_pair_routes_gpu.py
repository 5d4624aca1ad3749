"""The FP64 pair forces on both sides of the rules that choose threads per atom and packed gathers (6000 and 32,768 atoms,
10^6 pairs in all, half the chip's threads), in gases and liquids, with and without a box, against the same sums in torch."""
import numpy as np
import pytest

from tests.test_fp64_kernels_gpu import EPS, _abi, _build_list, _grid

pytestmark = pytest.mark.gpu


def _system(n, rho, seed):
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3) - 1e-9))
    L = (n / rho) ** (1 / 3)
    grid = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return (grid[rng.permutation(len(grid))[:n]] + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) * L / m, np.full(3, L)


def _entries(torch, nbr, nnb, n, maxnb):
    """(i, j) of every list entry."""
    table = nbr.view(-1, maxnb, 32).permute(0, 2, 1).reshape(-1, maxnb)[:n]
    on = torch.arange(maxnb, device="cuda")[None, :] < nnb[:, None]
    i, k = on.nonzero(as_tuple=True)
    return i, table[i, k].long()


# 2369 atoms: 32 and 16 threads an atom meet there; 9473: 16 and 8; 18,945 and 37,889: 8, 4 and 2; 75,777: one
@pytest.mark.parametrize("n", [2368, 2369, 5999, 6000, 9473, 18945, 32767, 32768, 37889, 75776, 75777])
@pytest.mark.parametrize("rho,periodic", [(0.002, True), (0.1, True), (0.9, True), (0.1, False), (0.9, False)])
@pytest.mark.parametrize("species", [1, 2])
def test_pair_routes(n, rho, periodic, species):
    """A pair's term is within 40 roundings of its parts, the exponent's argument takes 4 (alpha r)^2 more; a sum of m terms
    in any order within m roundings of the sum of their sizes (as test_pair_splits has it: 400 and more)."""
    torch, L, st = _abi()
    pos, box = _system(n, rho, n)
    rc, alpha, kc = 2.5, 0.8, 1.3
    rng = np.random.default_rng(1)
    p = torch.from_numpy(pos).cuda()
    sp = torch.from_numpy(rng.integers(0, species, n).astype(np.int32)).cuda()
    q = torch.from_numpy(rng.choice([-1.0, 1.0], n)).cuda()
    eps = np.array([[1.0, 0.8], [0.8, 0.6]])[:species, :species].copy()
    sig = np.array([[1.0, 0.95], [0.95, 0.9]])[:species, :species].copy()
    g = _grid(L, box if periodic else None, 2.8, pos)
    maxnb = 160
    nbr, nnb = _build_list(torch, L, st, p, g, maxnb)
    i, j = _entries(torch, nbr, nnb, n, maxnb)
    d = p[j] - p[i]
    if periodic:
        b = torch.from_numpy(box).cuda()
        d = d - b * torch.round(d / b)
    r2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
    r = r2.sqrt()

    def total(weight, of):
        return torch.zeros((n, 3), dtype=torch.float64, device="cuda").index_add_(0, i, weight[:, None] * of)

    e, s = (torch.from_numpy(x).cuda()[sp[i].long(), sp[j].long()] for x in (eps, sig))
    inside = r2 < (rc * s) ** 2
    s6 = torch.where(inside, (s * s / r2) ** 3, 0.0)
    c6 = (1 / rc ** 2) ** 3
    lj = (total(-24 * e * (2 * s6 ** 2 - s6) / r2, d), total(24 * e * (2 * s6 ** 2 + s6) / r2, d.abs()),
          0.5 * (4 * e * torch.where(inside, s6 ** 2 - s6 - (c6 ** 2 - c6), 0.0)).sum(), 0.5 * (4 * e * (s6 ** 2 + s6 + c6)).sum())
    inside = r < rc
    gauss = 2 * alpha / np.sqrt(np.pi) * torch.exp(-(alpha * r) ** 2) / r
    f = torch.erfc(alpha * r) / r2 + gauss
    erc = float(torch.erfc(torch.tensor(alpha * rc, dtype=torch.float64)))
    sh = erc / rc ** 2 + 2 * alpha / np.sqrt(np.pi) * np.exp(-(alpha * rc) ** 2) / rc
    qq = torch.where(inside, q[i] * q[j], 0.0)
    self_u = float((q ** 2).sum()) * (erc / (2 * rc) + alpha / np.sqrt(np.pi))
    u = torch.erfc(alpha * r) / r
    dsf = (kc * total(-qq * (f - sh) / r, d), kc * total(qq.abs() * (f + sh) / r, d.abs()),
           kc * (0.5 * (qq * (u - erc / rc + sh * (r - rc))).sum() - self_u),
           kc * (0.5 * (qq.abs() * (u + erc / rc + sh * (rc - r))).sum() + self_u))
    near = float(r.min()) if len(r) else 1.0
    tol = (400 + 4 * (alpha * rc) ** 2 + 16 * 2 * 3 ** 0.5 * box.max() / near) * EPS
    for kind, (F, mag, U, Umag) in (("lj", lj), ("dsf", dsf)):
        force = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
        energy = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
        work = torch.empty(L.acs_force_work_bytes(n), dtype=torch.uint8, device="cuda")
        head = (box.ctypes.data if periodic else None, int(periodic), nbr.data_ptr(), nnb.data_ptr(), maxnb)
        tail = (force.data_ptr(), energy.data_ptr(), work.data_ptr(), work.numel(), st)
        if kind == "lj":
            assert L.acs_lj_fp64(p.data_ptr(), sp.data_ptr(), n, *head, species, eps.ctypes.data, sig.ctypes.data, rc, *tail) == 0
        else:
            assert L.acs_dsf_fp64(p.data_ptr(), q.data_ptr(), n, *head, None, None, alpha, rc, kc, *tail) == 0
        assert bool(((force - F).abs() <= tol * mag).all())
        assert abs(float(energy - U)) <= tol * float(Umag) + 1e-300
