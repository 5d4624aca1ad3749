"""Neighbour lists and pair histogram of systems with few atoms per cell (a lane per atom from 20,000 and 50,000 atoms on)
against the reference's binning, stencil and FP64 filter; the candidates come from a k-d tree."""
import ctypes as C

import numpy as np
import pytest

from tests.test_fp64_kernels_gpu import _abi, _grid

pytestmark = pytest.mark.gpu


def _pairs(pos, box, rc):
    """Ordered pairs of finite atoms whose images are no farther than rc and a little, i ascending."""
    from scipy.spatial import cKDTree
    ok = np.flatnonzero(np.isfinite(pos).all(1))
    x = pos[ok]
    if box is not None:
        x = np.mod(x, box)
        x[x >= np.broadcast_to(box, x.shape)] = 0.0
    p = cKDTree(x, boxsize=box).query_pairs(rc * (1 + 1e-9), output_type="ndarray")
    i, j = ok[p[:, 0]], ok[p[:, 1]]
    return np.concatenate([i, j]), np.concatenate([j, i])


def _image(pos, i, j, box):
    d = pos[j] - pos[i]
    if box is not None:
        d = d - box * np.round(d / box)
    return d, (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]


def _positions(kind, n, cells, box, rc, periodic, unit):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, 1, (n, 3)) * box
    if kind == "edges":   # on cell edges and next to them, and pairs next to the radius
        k = rng.integers(0, 3 * n, n)
        edge = rng.integers(0, np.array(cells) + 1, (n, 3)) / np.array(cells) * box
        pos.reshape(-1)[k] = np.nextafter(edge.reshape(-1)[k], rng.choice([-1e9, 1e9], n) * unit)
        pos[:15] = pos[15:30] + rc * np.array([1.0, 0, 0])
        if periodic:
            pos = np.abs(pos)
    elif kind == "outside":   # a caller's unwrapped atoms, a NaN, an infinity
        far = rng.choice(n, n // 4, replace=False)
        pos[far] += rng.integers(-2, 3, (len(far), 3)) * box
        if periodic:
            pos[1], pos[2] = np.nan, [np.inf, 0.1 * rc, 0.2 * rc]
    elif kind == "clustered":
        pos[:3000] = box * 0.3 + rng.normal(0, 2 * rc, (3000, 3))
        if periodic:
            pos[:3000] %= box
    return pos


# one axis of one cell and of three (the image found per pair), stencil images, open boxes; at the first size and above
@pytest.mark.parametrize("cells,n,periodic", [((1, 90, 91), 20000, True), ((3, 50, 51), 20001, True), ((30, 16, 15), 20500, True),
                                              ((40, 33, 35), 20223, True), ((28, 29, 27), 20031, False)])
@pytest.mark.parametrize("kind", ["inside", "edges", "outside", "clustered"])
@pytest.mark.parametrize("unit", [1.0, 1e-30])
def test_sparse_list(cells, n, periodic, kind, unit):
    torch, L, st = _abi()
    rc = 1.1 * unit
    box = (np.array(cells) + np.array([0.3, 0.6, 0.8])) * rc
    pos = _positions(kind, n, cells, box, rc, periodic, unit)
    g = _grid(L, box if periodic else None, rc, pos)
    nc = np.array(g.ncell)
    assert n < 4 * np.prod(nc)
    with np.errstate(invalid="ignore"):
        t = (pos - np.array(g.lo)) / np.array(g.span) * nc
        cell = np.where(t >= 1, np.where(t >= nc - 1, nc - 1, np.floor(np.where(np.isfinite(t), t, 0))), 0).astype(int)
    i, j = _pairs(pos / unit, box / unit if periodic else None, rc / unit)
    _, r2 = _image(pos, i, j, box if periodic else None)
    d = cell[j] - cell[i]
    if periodic:
        d = np.where(nc >= 3, (d + 1) % nc - 1, d)
    keep = (r2 < g.rc2) & np.all(np.abs(d) <= 1, axis=1)
    i, j, d = i[keep], j[keep], d[keep]
    order = np.lexsort((j, (d + 1) @ np.array([9, 3, 1]), i))
    i, j = i[order], j[order]
    count = np.bincount(i, minlength=n)
    place = np.arange(len(i)) - (np.cumsum(count) - count)[i]
    maxnb = int(count.max())
    p = torch.from_numpy(pos).cuda()
    nbr = torch.full(((n + 31) // 32 * 32 * maxnb,), -7, dtype=torch.int32, device="cuda")
    nnb = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    work = torch.empty(L.acs_nlist_work_bytes(n, C.byref(g)), dtype=torch.uint8, device="cuda")
    assert L.acs_nlist_build(p.data_ptr(), n, C.byref(g), maxnb, nbr.data_ptr(), nnb.data_ptr(), work.data_ptr(),
                             work.numel(), status.data_ptr(), st) == 0
    want = np.full((n + 31) // 32 * 32 * maxnb, -7, np.int32)
    want[i // 32 * maxnb * 32 + place * 32 + i % 32] = j
    assert np.array_equal(nnb.cpu().numpy(), count) and np.array_equal(nbr.cpu().numpy(), want)
    assert not status.cpu().numpy()[0]
    # one entry too few: every count is reported, nothing is written past the capacity
    nbr.fill_(-7)
    assert L.acs_nlist_build(p.data_ptr(), n, C.byref(g), maxnb - 1, nbr.data_ptr(), nnb.data_ptr(), work.data_ptr(),
                             work.numel(), status.data_ptr(), st) == 0
    s = status.cpu().numpy()
    assert s[0] == 1 and s[1] == maxnb and np.array_equal(nnb.cpu().numpy(), count)
    assert bool((nbr[(n + 31) // 32 * 32 * (maxnb - 1):] == -7).all())


@pytest.mark.parametrize("cells,n", [((1, 140, 141), 50000), ((3, 80, 81), 50001), ((50, 36, 37), 50033)])
@pytest.mark.parametrize("kind", ["inside", "edges", "outside"])
@pytest.mark.parametrize("species", [-1, 1])
def test_sparse_histogram(cells, n, kind, species):
    """Counts equal to the reference's rdf on the pairs its cells hold (positions outside the box are binned into the edge
    cells, as the list's)."""
    torch, L, st = _abi()
    rmax, bins = 1.1, 37
    box = (np.array(cells) + np.array([0.3, 0.6, 0.8])) * rmax
    pos = _positions(kind, n, cells, box, rmax, True, 1.0)
    sp = np.random.default_rng(1).integers(0, 2, n).astype(np.int32)
    g = _grid(L, box, rmax)
    nc = np.array(g.ncell)
    assert n < 4 * np.prod(nc)
    with np.errstate(invalid="ignore"):
        t = pos / box * nc
        cell = np.where(t >= 1, np.where(t >= nc - 1, nc - 1, np.floor(np.where(np.isfinite(t), t, 0))), 0).astype(int)
    i, j = _pairs(pos, box, rmax)
    i, j = i[i < j], j[i < j]
    d = cell[j] - cell[i]
    d = np.where(nc >= 3, (d + 1) % nc - 1, d)
    keep = np.all(np.abs(d) <= 1, axis=1)
    if species >= 0:
        keep &= (sp[i] == species) & (sp[j] == species)
    r = np.sqrt(_image(pos, i[keep], j[keep], box)[1])
    want = np.histogram(r[r <= rmax], bins=bins, range=(0.0, rmax))[0]
    p, s = torch.from_numpy(pos).cuda(), torch.from_numpy(sp).cuda()
    hist = torch.full((bins,), -1, dtype=torch.int64, device="cuda")
    work = torch.empty(L.acs_rdf_work_bytes(n, C.addressof(g)), dtype=torch.uint8, device="cuda")
    assert L.acs_rdf_hist(p.data_ptr(), s.data_ptr(), n, C.addressof(g), species, bins, rmax, hist.data_ptr(),
                          work.data_ptr(), work.numel(), st) == 0
    assert np.array_equal(hist.cpu().numpy(), want)
