"""The FP64 entry points of the C ABI at the sizes where their work splits change: block and warp edges, remainders,
the smallest and largest grids. Each against plain NumPy / torch FP64 of the same quantity."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53

def _abi():
    import torch

    from devinproj_b200 import ewald, learned
    from devinproj_b200.device import stream_handle
    ewald._bind()
    return torch, learned._bind(), stream_handle()


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 65536, 65537, 300001])
def test_conserved_sums(n):
    """KE, P, L: every term passes through fewer than 64 roundings (products, shuffles, 8 warps, blocks / 256 strided
    partials), so each sum is within 64 eps of the sum of its terms' magnitudes."""
    torch, L, st = _abi()
    rng = np.random.default_rng(n)
    pos, vel = rng.uniform(0, 50, (n, 3)), rng.normal(0, 1, (n, 3))
    sp = rng.integers(0, 2, n).astype(np.int32)
    masses = np.array([1.5, 40.0])
    p, v, s = (torch.from_numpy(x).cuda() for x in (pos, vel, sp))
    out = torch.full((7,), float("nan"), dtype=torch.float64, device="cuda")
    work = torch.empty(L.acs_reduce_work_bytes(n), dtype=torch.uint8, device="cuda")
    for _ in range(2):   # the second call finds the ticket as the first left it
        assert L.acs_reduce_conserved(p.data_ptr(), v.data_ptr(), s.data_ptr(), masses.ctypes.data, 2, n, out.data_ptr(),
                                      work.data_ptr(), work.numel(), st) == 0
    mom = masses[sp][:, None] * vel
    ang = np.cross(pos, mom)
    ref = np.concatenate([[0.5 * np.sum(mom * vel)], mom.sum(0), ang.sum(0)])
    mag = np.concatenate([[0.5 * np.sum(np.abs(mom * vel))], np.abs(mom).sum(0),
                          [np.sum(np.abs(pos[:, a] * mom[:, b]) + np.abs(pos[:, b] * mom[:, a]))
                           for a, b in ((1, 2), (2, 0), (0, 1))]])
    assert np.all(np.abs(out.cpu().numpy() - ref) <= 64 * EPS * mag + 64 * EPS * np.abs(ref))


def _grid(L, box, rc, pos=None):
    from devinproj_b200 import _lib
    g = _lib.AcsGrid()
    if box is None:
        lo, hi = (np.ascontiguousarray(x) for x in (np.nanmin(pos, 0), np.nanmax(pos, 0)))
        assert L.acs_grid_setup(C.byref(g), None, 0, lo.ctypes.data, hi.ctypes.data, float(rc)) == 0
    else:
        b = np.ascontiguousarray(box, dtype=float)
        assert L.acs_grid_setup(C.byref(g), b.ctypes.data, 1, None, None, float(rc)) == 0
    g.rc2 = rc ** 2
    return g


def _reference_lists(pos, g):
    """Every atom's neighbours by the reference's binning, stencil and FP64 filter (accusim/forces.py:279-321), in
    stencil order and ascending index within a cell."""
    nc, lo, span = np.array(g.ncell), np.array(g.lo), np.array(g.span)
    with np.errstate(invalid="ignore"):
        t = (pos - lo) / span * nc
        cell = np.where(t >= 1, np.where(t >= nc - 1, nc - 1, np.floor(np.where(np.isfinite(t), t, 0))), 0).astype(int)
    out = []
    for i in range(len(pos)):
        d = cell - cell[i]
        if g.periodic:
            d = np.where(nc >= 3, (d + 1) % nc - 1, d)
        near = np.all(np.abs(d) <= 1, axis=1)
        near[i] = False
        j = np.flatnonzero(near)
        with np.errstate(invalid="ignore", over="ignore"):
            r = pos[j] - pos[i]
            if g.periodic:
                b = np.array(g.box)
                r = r - b * np.round(r / b)
            close = (r[:, 0] * r[:, 0] + r[:, 1] * r[:, 1]) + r[:, 2] * r[:, 2] < g.rc2
        j = j[close]
        rank = (d[j] + 1) @ np.array([9, 3, 1])
        out.append(j[np.lexsort((j, rank))])
    return out


# (cells per axis, atoms, periodic): one cell, the image found per pair (3 cells), stencil images (4 and more), a warp
# per cell (1024 cells and more) with ragged and with crowded cells, open boxes
LIST_FORMS = [((1, 1, 1), 70, True), ((3, 3, 3), 2700, True), ((3, 3, 3), 500, True), ((4, 3, 7), 900, True), ((4, 4, 5), 33, True),
              ((5, 4, 6), 1300, True), ((11, 10, 10), 4500, True), ((4, 16, 17), 4400, True), ((12, 11, 9), 4800, False),
              ((2, 2, 3), 400, False)]


@pytest.mark.parametrize("cells,n,periodic", LIST_FORMS)
@pytest.mark.parametrize("kind", ["inside", "edges", "outside", "clustered"])
@pytest.mark.parametrize("unit", [1.0, 1e-30])
def test_list_is_the_reference_filter_entry_by_entry(cells, n, periodic, kind, unit):
    """Whole lists, in order, for positions inside the box, on cell and box edges, outside it (a caller's unwrapped atoms,
    a NaN, an infinity) and crowded into a few cells; in a unit whose squares underflow FP32 too. Exact."""
    torch, L, st = _abi()
    rng = np.random.default_rng(n)
    rc = 1.1 * unit
    box = (np.array(cells) + rng.uniform(0.02, 0.9, 3) * (np.array(cells) > 1)) * rc
    if cells == (1, 1, 1):
        box = np.array([1.3, 2.2, 2.9]) * rc
    pos = rng.uniform(0, 1, (n, 3)) * box
    if kind == "edges":
        k = rng.integers(0, 3 * n, n)
        edge = rng.integers(0, np.array(cells) + 1, (n, 3)) / np.array(cells) * box
        pos.reshape(-1)[k] = np.nextafter(edge.reshape(-1)[k], rng.choice([-1e9, 1e9], n) * unit)
        pos[:15] = pos[15:30] + rc * np.array([1.0, 0, 0])   # r^2 next to rc^2
        if periodic:
            pos = np.abs(pos)
    elif kind == "outside":
        far = rng.choice(n, n // 4, replace=False)
        pos[far] += rng.integers(-2, 3, (len(far), 3)) * box
        if periodic:
            pos[1], pos[2] = np.nan, [np.inf, 0.1 * rc, 0.2 * rc]
    elif kind == "clustered":
        pos[: n // 2] = box * 0.3 + rng.normal(0, 0.3 * rc, (n // 2, 3))
    g = _grid(L, box if periodic else None, rc, pos)
    ref = _reference_lists(pos, g)
    maxnb = max(max(len(r) for r in ref), 1)
    p = torch.from_numpy(pos).cuda()
    nbr = torch.full(((n + 31) // 32 * 32 * maxnb,), -7, dtype=torch.int32, device="cuda")
    nnb = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    work = torch.empty(L.acs_nlist_work_bytes(n, C.byref(g)) + 4, dtype=torch.uint8, device="cuda")
    assert L.acs_nlist_build(p.data_ptr(), n, C.byref(g), maxnb, nbr.data_ptr(), nnb.data_ptr(), work.data_ptr() + 4,
                             work.numel() - 4, status.data_ptr(), st) == 0
    got_n = nnb.cpu().numpy()
    assert np.array_equal(got_n, [len(r) for r in ref]) and not status.cpu().numpy()[0]
    rows = nbr.cpu().numpy().reshape(-1, maxnb, 32)
    for i, r in enumerate(ref):
        assert np.array_equal(rows[i // 32, :len(r), i % 32], r)
    # one entry too few: every count is still reported, nothing is written past the capacity
    if maxnb > 1:
        nbr.fill_(-7)
        assert L.acs_nlist_build(p.data_ptr(), n, C.byref(g), maxnb - 1, nbr.data_ptr(), nnb.data_ptr(),
                                 work.data_ptr() + 4, work.numel() - 4, status.data_ptr(), st) == 0
        s = status.cpu().numpy()
        assert s[0] == 1 and s[1] == maxnb and np.array_equal(nnb.cpu().numpy(), got_n)
        assert bool((nbr[(n + 31) // 32 * 32 * (maxnb - 1):] == -7).all())


def _build_list(torch, L, st, p, g, maxnb):
    n = len(p)
    nbr = torch.empty((n + 31) // 32 * 32 * maxnb, dtype=torch.int32, device="cuda")
    nnb = torch.empty(n, dtype=torch.int32, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    work = torch.empty(L.acs_nlist_work_bytes(n, C.byref(g)), dtype=torch.uint8, device="cuda")
    assert L.acs_nlist_build(p.data_ptr(), n, C.byref(g), maxnb, nbr.data_ptr(), nnb.data_ptr(), work.data_ptr(),
                             work.numel(), status.data_ptr(), st) == 0
    assert int(status[0].item()) == 0
    return nbr, nnb


def _pairs_within(pos, box, rc):
    """(i, j, d_ij, r^2) of all ordered pairs with r < rc, in the reference's expression; row blocks."""
    out = []
    for a in range(0, len(pos), 400):
        with np.errstate(invalid="ignore"):
            d = pos[None, :, :] - pos[a:a + 400, None, :]
            if box is not None:
                d = d - box * np.round(d / box)
            r2 = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
            i, j = np.nonzero(r2 < rc ** 2)
        keep = i + a != j
        i, j = i[keep], j[keep]
        out.append((i + a, j, d[i, j], r2[i, j]))
    return [np.concatenate(x) for x in zip(*out)]


def _scatter(n, i, x):
    return np.stack([np.bincount(i, x[:, k], minlength=n) for k in range(3)], 1)


# atoms: a block holds 8 (32 phases) or 16 (n = 8193); blocks end ragged
@pytest.mark.parametrize("n", [1, 2, 7, 9, 255, 257, 399, 4095, 4097, 8193])
@pytest.mark.parametrize("species", [1, 3])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("dense", [True, False])
def test_lj_forces(n, species, periodic, dense):
    """Forces and energy against NumPy over the same pairs: a term carries under 25 roundings of the same r^2, amplified
    at most sevenfold by the powers, and an atom's sum under 200 additions, so an atom's force is within 400 eps of the
    sum of its terms' magnitudes. One atom is not finite: it has no pairs."""
    torch, L, st = _abi()
    rng = np.random.default_rng(n + species)
    box = np.array([1.0, 1.2, 0.9]) * (n / 0.8 / 1.08) ** (1 / 3)
    if n > 20:   # a lattice with noise, some atoms left out
        m = np.ceil((n / 1.08) ** (1 / 3) * np.array([1.0, 1.2, 0.9])).astype(int) + 1
        grid = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)
        pos = (grid[rng.permutation(len(grid))[:n]] + 0.5 + rng.normal(0, 0.06, (n, 3))) * box / m
    else:
        pos = rng.uniform(0, 1, (n, 3)) * box
    if n > 8:
        pos[5] = [np.nan, 0.1, 0.2] if periodic else [np.inf, 0.1, 0.2]
    sp = rng.integers(0, species, n).astype(np.int32)
    eps = np.array([[1.0, 0.8, 0.0], [0.8, 1.3, 0.7], [0.0, 0.7, 0.5]])[:species, :species].copy()
    sig = np.array([[1.0, 0.95, 1.0], [0.95, 0.9, 0.85], [1.0, 0.85, 0.8]])[:species, :species].copy()
    cutoff = 2.5
    i, j, d, r2 = _pairs_within(pos, box if periodic else None, cutoff * sig.max())
    e, s = eps[sp[i], sp[j]], sig[sp[i], sp[j]]
    m = (r2 < (cutoff * s) ** 2) & (e > 0)
    i, d, r2, e, s = i[m], d[m], r2[m], e[m], s[m]
    s6 = (s ** 2 / r2) ** 3
    c6 = cutoff ** -6.0
    F = _scatter(n, i, (-24 * e * (2 * s6 ** 2 - s6) / r2)[:, None] * d)
    mag = _scatter(n, i, (24 * e * (2 * s6 ** 2 + s6) / r2)[:, None] * np.abs(d))
    U = 0.5 * np.sum(4 * e * (s6 ** 2 - s6 - (c6 ** 2 - c6)))
    Umag = 0.5 * np.sum(4 * e * (s6 ** 2 + s6 + 1))
    p, spd = torch.from_numpy(pos).cuda(), torch.from_numpy(sp).cuda()
    nbr = nnb = None
    maxnb = 0
    if not dense:
        if n < 2:
            return
        finite = pos[np.isfinite(pos).all(1)]
        g = _grid(L, box if periodic else None, 2.8 * sig.max(), finite)
        maxnb = 400
        nbr, nnb = _build_list(torch, L, st, p, g, maxnb)
    force = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
    energy = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    work = torch.empty(L.acs_force_work_bytes(n) + 8, dtype=torch.uint8, device="cuda")
    b = np.ascontiguousarray(box)
    call = (p.data_ptr(), spd.data_ptr(), n, b.ctypes.data if periodic else None, int(periodic),
            nbr.data_ptr() if nbr is not None else None, nnb.data_ptr() if nnb is not None else None, maxnb, species,
            eps.ctypes.data, sig.ctypes.data, cutoff, force.data_ptr(), energy.data_ptr())
    for extra in ((work.data_ptr() + 8, work.numel() - 8, st), (work.data_ptr() + 8, work.numel() - 8, st), (st,)):
        fn = L.acs_lj_fp64 if len(extra) == 3 else L.acs_lj_fp64_noalloc
        force.fill_(float("nan"))
        assert fn(*call, *extra) == 0
        got = force.cpu().numpy()
        assert np.all(np.abs(got - F) <= 400 * EPS * mag)
        assert abs(energy.item() - U) <= 400 * EPS * (Umag + 1e-300)


# the splits as for LJ; exclusions, an atom that is not finite, uncharged atoms, alpha of zero
@pytest.mark.parametrize("n", [1, 2, 9, 255, 399, 1024, 4097, 8193])
@pytest.mark.parametrize("dense", [True, False])
@pytest.mark.parametrize("alpha", [0.0, 0.8, 9.0])
def test_dsf_forces(n, dense, alpha):
    """Forces and energy against NumPy with SciPy's erfc over the same pairs. A pair's erfc and exponential carry the
    rounding of alpha r, 2 (alpha r)^2 eps of their value, on top of a few eps each: within (60 + 4 (alpha rc)^2) eps of
    the pair's term magnitudes, and an atom's sum adds under 200 roundings of the partial sums."""
    from scipy.special import erfc
    torch, L, st = _abi()
    rng = np.random.default_rng(n)
    rc, kc = 3.0, 1.7
    box = np.array([1.1, 0.9, 1.0]) * max((n / 0.9) ** (1 / 3), 6.2)
    m = np.ceil((n / 0.99) ** (1 / 3) * np.array([1.1, 0.9, 1.0])).astype(int) + 1
    grid = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)
    pos = (grid[rng.permutation(len(grid))[:n]] + 0.5 + rng.normal(0, 0.05, (n, 3))) * box / m
    q = np.where(rng.random(n) < 0.5, 1.0, -1.2)
    q[::7] = 0.0
    if n > 8:
        pos[5] = [np.nan, 0.1, 0.2]
    i, j, d, r2 = _pairs_within(pos, box, rc)
    ex = [] if n < 9 else [(0, int(k)) for k in set(j[i == 0][:3].tolist())] + [(1, n - 1)]
    both = np.array(sorted({p for a, b in ex for p in ((a, b), (b, a))}), dtype=np.int64).reshape(-1, 2)
    start = np.zeros(n + 1, np.int32)
    start[1:] = np.cumsum(np.bincount(both[:, 0], minlength=n))
    keep = ~np.isin(i * n + j, both[:, 0] * n + both[:, 1])
    i, j, d, r = i[keep], j[keep], d[keep], np.sqrt(r2[keep])
    c = 2 * alpha / np.sqrt(np.pi)
    erc = erfc(alpha * rc)
    sh = erc / rc ** 2 + c * np.exp(-(alpha * rc) ** 2) / rc
    er, g = erfc(alpha * r), np.exp(-(alpha * r) ** 2)
    qq = q[i] * q[j]
    F = kc * _scatter(n, i, -(qq * ((er / r ** 2 + c * g / r) - sh) / r)[:, None] * d)
    mag = kc * _scatter(n, i, (np.abs(qq) * ((er / r ** 2 + c * g / r) + sh) / r)[:, None] * np.abs(d))
    self_c = erc / (2 * rc) + alpha / np.sqrt(np.pi)
    U = kc * (0.5 * np.sum(qq * (er / r - erc / rc + sh * (r - rc))) - np.sum(q ** 2) * self_c)
    Umag = kc * (0.5 * np.sum(np.abs(qq) * (er / r + erc / rc + sh * (rc - r))) + np.sum(q ** 2) * self_c)
    p, qd, sd, xd = (torch.from_numpy(x).cuda() for x in (pos, q, start, both[:, 1].astype(np.int32)))
    nbr = nnb = None
    maxnb = 0
    if not dense:
        if n < 2:
            return
        maxnb = 400
        nbr, nnb = _build_list(torch, L, st, p, _grid(L, box, rc + 0.2), maxnb)
    force = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
    energy = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    work = torch.empty(L.acs_force_work_bytes(n), dtype=torch.uint8, device="cuda")
    assert L.acs_dsf_fp64(p.data_ptr(), qd.data_ptr(), n, np.ascontiguousarray(box).ctypes.data, 1,
                          nbr.data_ptr() if nbr is not None else None, nnb.data_ptr() if nnb is not None else None, maxnb,
                          sd.data_ptr() if ex else None, xd.data_ptr() if ex else None, alpha, rc, kc, force.data_ptr(),
                          energy.data_ptr(), work.data_ptr(), work.numel(), st) == 0
    tol = (260 + 4 * (alpha * rc) ** 2) * EPS
    assert np.all(np.abs(force.cpu().numpy() - F) <= tol * mag + 1e-300)
    assert abs(energy.item() - U) <= tol * Umag


# copies of 512 atoms: 13,824 (LJ 8 phases, DSF 32), 32,768 (4, 16), 110,592 (4, 8), 262,144 (4, 2), 626,688 (1, 1)
@pytest.mark.parametrize("copies", [(3, 3, 3), (4, 4, 4), (6, 6, 6), (8, 8, 8), (8, 9, 17)])
def test_pair_splits(copies):
    """Every copy of a periodic system feels the system's own forces. A copy's coordinates are rounded at the whole box's
    size, L eps / 2 each, so a pair's distance is off by at most 2 sqrt(3) L eps and its term by 16 times that over the
    smallest distance (LJ's steepest power 14, DSF's less); to that the bounds of the direct comparisons."""
    from scipy.special import erfc
    torch, L, st = _abi()
    rng = np.random.default_rng(11)
    rc, alpha, kc = 2.5, 0.8, 1.7
    box = np.array([8.6, 8.8, 8.5])
    grid = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (grid + 0.5 + rng.normal(0, 0.06, (512, 3))) * box / 8
    q = np.where(np.arange(512) % 2 == 0, 1.0, -1.2)
    i, j, d, r2 = _pairs_within(pos, box, rc)
    s6, c6, r = r2 ** -3.0, rc ** -6.0, np.sqrt(r2)
    c, erc, qq = 2 * alpha / np.sqrt(np.pi), erfc(alpha * rc), q[i] * q[j]
    sh = erc / rc ** 2 + c * np.exp(-(alpha * rc) ** 2) / rc
    g = erfc(alpha * r) / r ** 2 + c * np.exp(-(alpha * r) ** 2) / r
    er, self_u = erfc(alpha * r) / r, np.sum(q ** 2) * (erc / (2 * rc) + alpha / np.sqrt(np.pi))
    want = [(_scatter(512, i, (-24 * (2 * s6 ** 2 - s6) / r2)[:, None] * d),
             _scatter(512, i, (24 * (2 * s6 ** 2 + s6) / r2)[:, None] * np.abs(d)),
             0.5 * np.sum(4 * (s6 ** 2 - s6 - (c6 ** 2 - c6))), 0.5 * np.sum(4 * (s6 ** 2 + s6 + 1))),
            (kc * _scatter(512, i, -(qq * (g - sh) / r)[:, None] * d),
             kc * _scatter(512, i, (np.abs(qq) * (g + sh) / r)[:, None] * np.abs(d)),
             kc * (0.5 * np.sum(qq * (er - erc / rc + sh * (r - rc))) - self_u),
             kc * (0.5 * np.sum(np.abs(qq) * (er + erc / rc + sh * (rc - r))) + self_u))]
    shift = np.stack(np.meshgrid(*[np.arange(k) for k in copies], indexing="ij"), -1).reshape(-1, 1, 3) * box
    whole = box * copies
    many, times = (pos + shift).reshape(-1, 3), int(np.prod(copies))
    n = len(many)
    p, qd = torch.from_numpy(many).cuda(), torch.from_numpy(np.tile(q, times)).cuda()
    sp = torch.zeros(n, dtype=torch.int32, device="cuda")
    maxnb = 400 if n < 300000 else 128
    nbr, nnb = _build_list(torch, L, st, p, _grid(L, whole, rc + 0.3), maxnb)
    one, b = np.ones((1, 1)), np.ascontiguousarray(whole)
    tol = (400 + 4 * (alpha * rc) ** 2 + 16 * 2 * 3 ** 0.5 * whole.max() / r.min()) * EPS
    for kind, (F, mag, U, Umag) in zip(("lj", "dsf"), want):
        force = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
        energy = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
        work = torch.empty(L.acs_force_work_bytes(n), dtype=torch.uint8, device="cuda")
        tail = (force.data_ptr(), energy.data_ptr(), work.data_ptr(), work.numel(), st)
        if kind == "lj":
            assert L.acs_lj_fp64(p.data_ptr(), sp.data_ptr(), n, b.ctypes.data, 1, nbr.data_ptr(), nnb.data_ptr(), maxnb, 1,
                                 one.ctypes.data, one.ctypes.data, rc, *tail) == 0
        else:
            assert L.acs_dsf_fp64(p.data_ptr(), qd.data_ptr(), n, b.ctypes.data, 1, nbr.data_ptr(), nnb.data_ptr(), maxnb,
                                  None, None, alpha, rc, kc, *tail) == 0
        got = force.cpu().numpy().reshape(times, 512, 3)
        assert np.all(np.abs(got - F) <= tol * mag)
        assert abs(energy.item() / times - U) <= tol * Umag


def _ewald_vectors(kind, box, alpha):
    kmax = {"wide": 17}.get(kind, 4)
    m = np.arange(-kmax, kmax + 1)
    N = np.stack(np.meshgrid(m, m, m, indexing="ij"), -1).reshape(-1, 3)
    N = N[(np.sum(N ** 2, 1) <= kmax ** 2) & np.any(N != 0, 1)]
    rng = np.random.default_rng(5)
    if kind == "wide":          # integers beyond the tables
        N = N[rng.permutation(len(N))[:301]]
    if kind == "order":         # mirrored, but in no order, with unequal weights
        N = N[rng.permutation(len(N))]
    if kind == "half":          # no mirror images
        N = N[(N[:, 0] > 0) | ((N[:, 0] == 0) & (N[:, 1] >= 0))]
    if kind == "twice":         # a vector listed twice
        N = np.concatenate([N, N[:3]])
    if kind == "zero":          # the zero vector among them
        N = np.concatenate([N, [[0, 0, 0]]])
    kv = 2 * np.pi * N / box
    if kind == "free":          # not reciprocal to the box
        kv = kv * rng.uniform(0.9, 1.1, kv.shape)
    k2 = np.maximum(np.sum(kv ** 2, 1), 1e-3)
    w = np.exp(-k2 / (4 * alpha ** 2)) / k2
    return np.ascontiguousarray(kv), w * (rng.uniform(0.5, 2, len(w)) if kind == "order" else 1.0)


# atoms: below, at and above a tile of 32 and a block of 256; above the tiled kernel's range (few partners referenced)
@pytest.mark.parametrize("n,kind", [(n, "lattice") for n in (1, 2, 31, 33, 255, 257, 700, 49153)]
                         + [(300, k) for k in ("order", "half", "twice", "zero", "free", "wide")])
def test_ewald_sum(n, kind):
    """Forces, real-space energy and sum of w |S|^2 against NumPy. Real space as for DSF; a phase k.r carries 8 |k.r| eps
    and a product of three factors a few eps, on S (of at most sum |q|) and on the force's factor."""
    from scipy.special import erfc
    torch, L, st = _abi()
    rng = np.random.default_rng(n)
    box = np.array([9.0, 11.0, 10.0])
    pos = rng.uniform(-0.2, 1.2, (n, 3)) * box        # wrapped or not
    q = rng.choice([-1.0, 1.0, 0.7], n)
    rcut, alpha, kc = 4.4, 0.7, 1.3
    kv, w = _ewald_vectors(kind, box, alpha)
    rows = np.arange(n) if n < 1000 else np.r_[0:40, n - 40:n]
    F, mag = np.zeros((len(rows), 3)), np.zeros((len(rows), 3))
    real = rmag = 0.0
    for a, i in enumerate(rows):
        d = pos - pos[i]
        d = d - box * np.round(d / box)
        r = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
        m = (r < rcut) & (np.arange(n) != i)
        d, r, qq = d[m], r[m], q[i] * q[m]
        e = erfc(alpha * r)
        t = (e / r + 2 * alpha / np.sqrt(np.pi) * np.exp(-(alpha * r) ** 2)) / r ** 2
        F[a] = -np.sum((qq * t)[:, None] * d, 0)
        mag[a] = np.sum((np.abs(qq) * t)[:, None] * np.abs(d), 0)
        real += 0.5 * np.sum(qq * e / r)
        rmag += 0.5 * np.sum(np.abs(qq) * e / r)
    ph = pos @ kv.T
    S = (q[:, None] * np.exp(1j * ph)).sum(0)
    rec = np.sum(w * np.abs(S) ** 2)
    V = float(np.prod(box))
    im = np.imag(np.conj(S)[None, :] * np.exp(1j * ph[rows]))
    F += 4 * np.pi / V * q[rows][:, None] * ((w * im) @ kv)
    wide = (8 * np.abs(ph).max() + 100) * EPS
    Q = np.abs(q).sum()
    tol = (300 + 4 * (alpha * rcut) ** 2) * EPS * mag + 2 * wide * 4 * np.pi / V * np.abs(q[rows])[:, None] * Q * (w @ np.abs(kv))
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (pos, q, kv, w)]
    force = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
    e3 = torch.full((3,), float("nan"), dtype=torch.float64, device="cuda")
    nbytes = L.acs_ewald_work_bytes(n, len(w))
    work = torch.empty(nbytes + 8, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        assert L.acs_ewald_fp64(dev[0].data_ptr(), dev[1].data_ptr(), n, box.ctypes.data, dev[2].data_ptr(),
                                dev[3].data_ptr(), len(w), alpha, rcut, kc, force.data_ptr(), e3.data_ptr(),
                                work.data_ptr() + 8, nbytes, st) == 0
        got = force.cpu().numpy()[rows] / kc
        assert np.all(np.abs(got - F) <= tol)
        e = e3.cpu().numpy()
        if n < 1000:
            assert abs(e[0] - real) <= (300 + 4 * (alpha * rcut) ** 2) * EPS * rmag
        assert abs(e[1] - rec) <= 2 * wide * np.sum(w) * Q ** 2


# boxes whose cells at rmax are one, three (the image found per pair) and four and more per axis; ragged counts
@pytest.mark.parametrize("box,n", [((2.1, 2.3, 2.0), 65), ((3.1, 3.5, 3.3), 700), ((4.2, 6.1, 5.0), 2500), ((9.0, 4.1, 7.7), 5003),
                                   ((2.5, 8.0, 3.9), 33)])
@pytest.mark.parametrize("species", [-1, 1])
@pytest.mark.parametrize("bins", [1, 100, 8192])
def test_pair_histogram(box, n, species, bins):
    """Counts against NumPy's histogram of the reference's distances; distances on bin edges and at rmax, atoms outside the
    box. Exact."""
    torch, L, st = _abi()
    rng = np.random.default_rng(n)
    box, rmax = np.array(box), 1.0
    pos = rng.uniform(0, 1, (n, 3)) * box
    pos[: n // 4] = np.round(pos[: n // 4] * 50) / 50          # distances on edges
    pos[-9:] += rng.integers(-2, 3, (9, 3)) * box
    sp = rng.integers(0, 2, n).astype(np.int32)
    g = _grid(L, box, rmax)
    # pairs the cell grid meets: an atom outside the box sits in an edge cell
    t = pos / np.array(g.span) * np.array(g.ncell)
    nc = np.array(g.ncell)
    cell = np.where(t >= 1, np.where(t >= nc - 1, nc - 1, np.floor(t)), 0).astype(int)
    r = []
    for i in range(n - 1):
        dc = cell[i + 1:] - cell[i]
        dc = np.where(nc >= 3, (dc + 1) % nc - 1, dc)
        m = np.all(np.abs(dc) <= 1, 1)
        if species >= 0:
            m &= (sp[i + 1:] == species) & (sp[i] == species)
        d = pos[i + 1:][m] - pos[i]
        d = d - box * np.round(d / box)
        r.append(np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]))
    r = np.concatenate(r)
    ref = np.histogram(r[r <= rmax], bins=bins, range=(0, rmax))[0]
    p, s = torch.from_numpy(pos).cuda(), torch.from_numpy(sp).cuda()
    hist = torch.full((bins,), -1, dtype=torch.int64, device="cuda")
    work = torch.empty(L.acs_rdf_work_bytes(n, C.byref(g)), dtype=torch.uint8, device="cuda")
    assert L.acs_rdf_hist(p.data_ptr(), s.data_ptr(), n, C.byref(g), species, bins, rmax, hist.data_ptr(), work.data_ptr(),
                          work.numel(), st) == 0
    assert np.array_equal(hist.cpu().numpy(), ref)


# neighbours: none, under a warp's 32, at and over the 128 staged at a time, both species, boxes of one and more cells
@pytest.mark.parametrize("n,edge", [(1, 21.0), (2, 21.0), (9, 24.0), (130, 21.0), (300, 20.5), (1001, 33.0)])
def test_descriptors(n, edge):
    """Invariants and vector features against FP64. FP32 distances (2 ulp) enter the Gaussians with a slope of at most
    0.6 / s and the approximate exponential and cosine are within 4e-7 and 1e-6, so a neighbour's term is off by under
    1e-5 of the cutoff's size; X is rounded to BF16 on top."""
    torch, L, st = _abi()
    rng = np.random.default_rng(n)
    box = np.array([1.0, 1.1, 0.95]) * edge
    rc, r0 = 10.0, 1.8
    dmu = (rc - r0) / 31
    pos = rng.uniform(0, 1, (n, 3)) * box
    if n == 2:
        pos[1] = (pos[0] + [0.0, 0.0, 2.0]) % box
    sp = rng.integers(0, 2, n).astype(np.int32)
    i, j, d, r2 = _pairs_within(pos, box, rc)
    r = np.sqrt(r2)
    mu = r0 + dmu * np.arange(32)
    g = np.exp(-(r[:, None] - mu) ** 2 / (2 * dmu ** 2)) * 0.5 * (np.cos(np.pi * r / rc) + 1)[:, None]
    D, V, count = np.zeros((n, 2, 32)), np.zeros((n, 2, 32, 3)), np.zeros((n, 2, 1))
    np.add.at(D, (i, sp[j]), g)
    np.add.at(V, (i, sp[j]), g[:, :, None] * (d / r[:, None])[:, None, :])
    np.add.at(count, (i, sp[j]), 1.0)
    mean, inv = rng.normal(0, 1, 64).astype(np.float32), rng.uniform(0.5, 2, 64).astype(np.float32)
    p, s = torch.from_numpy(pos).cuda(), torch.from_numpy(sp).cuda()
    nbr, nnb = _build_list(torch, L, st, p, _grid(L, box, rc), 512)
    par = np.array([r0, dmu, 1 / (2 * dmu ** 2), rc, 0, 0], np.float32)
    X = torch.full((n, 80), float("nan"), dtype=torch.bfloat16, device="cuda")
    W = torch.full((n, 64, 3), float("nan"), dtype=torch.float32, device="cuda")
    md, vd = torch.from_numpy(mean).cuda(), torch.from_numpy(inv).cuda()
    assert L.acs_descriptors(p.data_ptr(), s.data_ptr(), n, box.ctypes.data, 1, nbr.data_ptr(), nnb.data_ptr(), 512,
                             par.ctypes.data, md.data_ptr(), vd.data_ptr(), X.data_ptr(), W.data_ptr(), st) == 0
    x = X.float().cpu().numpy()
    tol = 1e-5 * (count + 1)
    assert np.all(np.abs(W.cpu().numpy().reshape(n, 2, 32, 3) - V) <= tol[..., None])
    ref = (D.reshape(n, 64) - mean) * inv
    assert np.all(np.abs(x[:, :64] - ref) <= 2.0 ** -8 * np.abs(ref) + 2 * np.repeat(tol, 32, 2).reshape(n, 64))
    assert np.array_equal(x[:, 64:], np.eye(16, dtype=np.float32)[[15]].repeat(n, 0) + np.eye(16, dtype=np.float32)[sp])


# one row, a tile's last row, a full tile, one row into the next, many tiles
@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
def test_training_step_gradient(n):
    """Loss and gradient against FP64 of the same BF16 weights and inputs (activations and their gradients are rounded to
    BF16, 2^-9 each through three layers: 3e-2 of the gradient's norm, 1e-2 of the loss); buffers that are not
    16-byte aligned give the same bits."""
    torch, L, st = _abi()
    rng = np.random.default_rng(n)
    th = rng.normal(0, 0.12, (3, 64, 80)).astype(np.float32)
    th[1:, :, 65:] = 0
    X = rng.normal(0, 1, (n, 80))
    X[:, 66:79], X[:, 79] = 0, 1
    V, Y = rng.normal(0, 0.7, (n, 64, 3)).astype(np.float32), rng.normal(0, 0.5, (n, 3)).astype(np.float32)
    Xb = torch.from_numpy(X).to(torch.bfloat16)
    q = torch.from_numpy(th).double()
    q[0] = torch.from_numpy(th[0]).to(torch.bfloat16).double()
    q[1:, :, :64] = torch.from_numpy(th[1:, :, :64]).to(torch.bfloat16).double()
    q.requires_grad_(True)
    silu = torch.nn.functional.silu
    h = silu(silu(Xb.double() @ q[0].T) @ q[1][:, :64].T + q[1][:, 64])
    F = torch.einsum("nc,ncd->nd", h @ q[2][:, :64].T + q[2][:, 64], torch.from_numpy(V).double())
    loss = ((F - torch.from_numpy(Y).double()) ** 2).sum() / (3 * n)
    loss.backward()
    ref = q.grad.numpy().reshape(-1)
    out = []
    for shift in (0, 4):
        def device(a):
            b = torch.empty(a.nbytes + 16, dtype=torch.uint8, device="cuda")
            t = b[shift:shift + a.nbytes].view(torch.float32).view(a.shape)
            return t.copy_(torch.from_numpy(a))
        w = torch.from_numpy(th).cuda()
        ws = [x.contiguous().to(torch.bfloat16) for x in (w[0], w[1][:, :64], w[2][:, :64], w[1][:, :64].T, w[2][:, :64].T)]
        w5 = (C.c_void_p * 5)(*[x.data_ptr() for x in ws])
        b2, b3 = w[1][:, 64].contiguous(), w[2][:, 64].contiguous()
        x, v, y, theta = Xb.cuda(), device(V), device(Y), w.reshape(-1).clone()
        m, s, grad = torch.zeros_like(theta), torch.zeros_like(theta), torch.empty_like(theta)
        part = device(np.zeros(L.acs_mlp_grad_bytes(n) // 4, np.float32))
        lp = torch.empty((n + 127) // 128 * 4, device="cuda")
        status = torch.zeros(8, dtype=torch.int32, device="cuda")
        assert L.acs_mlp_train_step(x.data_ptr(), v.data_ptr(), y.data_ptr(), n, w5, b2.data_ptr(), b3.data_ptr(),
                                    theta.data_ptr(), m.data_ptr(), s.data_ptr(), 1e-3, 1, 0.0, part.data_ptr(),
                                    part.numel() * 4, lp.data_ptr(), grad.data_ptr(), status.data_ptr(), st) == 0
        assert int(status[0].item()) == 0
        out.append([t.cpu().numpy() for t in (grad, theta, lp)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert np.linalg.norm(out[0][0] - ref) <= 3e-2 * np.linalg.norm(ref)
    assert abs(out[0][2].sum() - loss.item()) <= 1e-2 * loss.item()


# the one-block binning's limits: 8192 atoms, 8191 cells, one over each
@pytest.mark.parametrize("n,cells", [(8192, (10, 10, 10)), (8193, (10, 10, 10)), (5000, (21, 13, 30)), (5000, (21, 15, 26)),
                                     (5000, (16, 16, 32))])
def test_list_binning_limits(n, cells):
    """Neighbour counts by brute force at the sizes where the binning changes; entries ascend within a cell, so the two
    binnings agree entry by entry with the reference lists of a sample of atoms. Exact."""
    torch, L, st = _abi()
    rng = np.random.default_rng(n)
    rc = 1.0
    box = (np.array(cells) + 0.3) * rc
    pos = rng.uniform(0, 1, (n, 3)) * box
    g = _grid(L, box, rc)
    assert tuple(g.ncell) == cells
    p, b = torch.from_numpy(pos).cuda(), torch.from_numpy(box).cuda()
    nbr, nnb = _build_list(torch, L, st, p, g, 64)
    d = p[None, :, :] - p[:1000, None, :]
    d = d - b * torch.round(d / b)
    close = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2] < rc ** 2
    assert torch.equal(nnb[:1000].long(), close.sum(1) - 1)
    rows = nbr.view(-1, 64, 32)
    for i in range(0, 1000, 37):
        got = rows[i // 32, : int(nnb[i]), i % 32].cpu().numpy()
        cell = np.minimum((pos / box * cells).astype(int), np.array(cells) - 1)
        rank = ((cell[got] - cell[i] + 1) % cells) @ np.array([9, 3, 1])
        assert np.array_equal(got, got[np.lexsort((got, rank))])


@pytest.mark.parametrize("n", [1, 85, 256, 257, 1000, 4096, 4097, 70001])
def test_integrator_kernels(n):
    """Drift and wrap, acceleration and the skin test against NumPy, bit for bit: coordinates inside the box, on its edges,
    one and several boxes away, signed zeros, not finite; the moved atom first, last and absent."""
    torch, L, st = _abi()
    rng = np.random.default_rng(n)
    box = np.array([2.0, 3.7, 1.3])
    pos = rng.uniform(-0.3, 1.3, (n, 3)) * box
    vel = rng.normal(0, 0.2, (n, 3))
    special = np.array([0.0, -0.0, 1.0, -1.0, 2.0, -2.0, 5.5, -7.25, 1e9, np.nan, np.inf, -np.inf, 1e-320, -1e-320])
    k = min(n, 14)
    pos[:k], vel[:k] = (special[:k, None] * box), 0.0
    dt = 0.37
    with np.errstate(invalid="ignore"):
        ref = np.remainder(pos + dt * vel, box)
    p, v = torch.from_numpy(pos).cuda(), torch.from_numpy(vel).cuda()
    assert L.acs_vv_drift_wrap(p.data_ptr(), v.data_ptr(), n, dt, box.ctypes.data, 1, st) == 0
    got = p.cpu().numpy()
    assert np.array_equal(got, ref, equal_nan=True) and np.array_equal(np.signbit(got[~np.isnan(ref)]), np.signbit(ref[~np.isnan(ref)]))
    sp = rng.integers(0, 3, n).astype(np.int32)
    m = np.array([1.7, 22.99, 39.948])
    s, acc = torch.from_numpy(sp).cuda(), torch.empty_like(v)
    assert L.acs_vv_accel(acc.data_ptr(), v.data_ptr(), s.data_ptr(), m.ctypes.data, 3, n, st) == 0
    assert np.array_equal(acc.cpu().numpy(), vel / m[sp][:, None])
    a = rng.uniform(0, 1, (n, 3)) * box
    b = (a + rng.uniform(-0.05, 0.05, (n, 3))) % box
    b[:1] = (a[:1] + [0.2, 0.0, 0.0]) % box
    flag = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    ad = torch.from_numpy(a).cuda()
    for where in (0, n - 1, None):
        c = b.copy()
        if where != 0:
            c[0] = a[0]
        if where:
            c[where] = (a[where] + [0.0, 0.2, 0.0]) % box
        cd = torch.from_numpy(c).cuda()
        assert L.acs_nlist_displacement(cd.data_ptr(), ad.data_ptr(), n, box.ctypes.data, 1, 0.15 ** 2, flag.data_ptr(), st) == 0
        assert int(flag.item()) == (0 if where is None else 1)
    c[n // 2] = np.nan
    cd = torch.from_numpy(c).cuda()
    assert L.acs_nlist_displacement(cd.data_ptr(), ad.data_ptr(), n, box.ctypes.data, 1, 0.15 ** 2, flag.data_ptr(), st) == 0
    assert int(flag.item()) == 1
