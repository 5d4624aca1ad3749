"""Single pair terms of the FP64 kernels against 40 digits: the force of one pair (a dimer, two ions far from the others)
is its term, so no sum averages the term's error.

The tolerance is the root mean square error of the plain FP64 expression (IEEE square root and division, libm's erfc and
exp) on the same distances, per range of distance, and on top of it, where the term holds them, that of an erfc and an
exponential that are 1.5 units of 2^-53 off: the root mean square bound stated at `erfc_exp`."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -53
EDGES = np.array([1e-3, 0.1, 0.3, 0.6, 1.0])   # of the cutoff


def _rms(error, r, rc):
    return np.array([np.sqrt(np.mean(error[(r >= a * rc) & (r < b * rc)] ** 2)) for a, b in zip(EDGES, EDGES[1:])]) / UNIT


def _dimers(torch, r):
    """2 m atoms: the pair (2 k, 2 k + 1) at distance r[k] on the x axis, each listing the other only."""
    n = 2 * len(r)
    pos = np.zeros((n, 3))
    pos[1::2, 0] = r
    nbr = torch.zeros((n + 31) // 32 * 32, dtype=torch.int32)
    nbr[:n] = torch.arange(n, dtype=torch.int32) ^ 1
    return torch.from_numpy(pos).cuda(), nbr.cuda(), torch.ones(n, dtype=torch.int32, device="cuda")


def _exact(r, alpha, rc):
    """erfc(alpha r) / r, the force of it, and the shift at rc, to 40 digits."""
    import mpmath as mp
    with mp.workdps(40):
        a, c = mp.mpf(alpha), 2 * mp.mpf(alpha) / mp.sqrt(mp.pi)
        u = [mp.erfc(a * mp.mpf(x)) / mp.mpf(x) for x in r]
        f = [y / mp.mpf(x) + c * mp.exp(-(a * mp.mpf(x)) ** 2) / mp.mpf(x) for x, y in zip(r, u)]
        shift = mp.erfc(a * rc) / mp.mpf(rc) ** 2 + c * mp.exp(-(a * rc) ** 2) / rc
    return u, f, shift


def _relative(got, exact, scale):
    import mpmath as mp
    with mp.workdps(40):
        return np.array([float((mp.mpf(float(g)) - e) / s) for g, e, s in zip(got, exact, scale)])


@pytest.mark.parametrize("alpha,rc", [(0.0, 3.0), (0.2, 12.0), (0.8, 3.0), (1.9, 3.0)])
def test_dsf_pair(alpha, rc):
    from scipy.special import erfc
    import torch

    from devinproj_b200 import _lib
    from devinproj_b200.device import stream_handle
    L = _lib.lib()
    rng = np.random.default_rng(5)
    r = np.concatenate([rng.uniform(a * rc, b * rc, 1500) for a, b in zip(EDGES, EDGES[1:])])
    pos, nbr, nnb = _dimers(torch, r)
    n = len(pos)
    q = torch.ones(n, dtype=torch.float64, device="cuda")
    force, energy = torch.empty_like(pos), torch.empty(1, dtype=torch.float64, device="cuda")
    work = torch.empty(L.acs_force_work_bytes(n), dtype=torch.uint8, device="cuda")
    assert L.acs_dsf_fp64(pos.data_ptr(), q.data_ptr(), n, None, 0, nbr.data_ptr(), nnb.data_ptr(), 1, None, None, alpha, rc,
                          1.0, force.data_ptr(), energy.data_ptr(), work.data_ptr(), work.numel(), stream_handle()) == 0
    _, f, shift = _exact(r, alpha, rc)
    c, erc = 2 * alpha / np.sqrt(np.pi), erfc(alpha * rc)
    root = np.sqrt(r * r)
    ir, ar = 1.0 / root, alpha * root
    plain = ((erfc(ar) * (ir * ir) + c * np.exp(-(ar * ar)) * ir) - (erc / (rc * rc) + c * np.exp(-(alpha * rc) ** 2) / rc)) * ir * r
    exact, scale = [x - shift for x in f], [x + shift for x in f]
    want = _rms(_relative(plain, exact, scale), r, rc)
    got = _rms(_relative(force[1::2, 0].cpu().numpy(), exact, scale), r, rc)
    print(got, want)
    assert np.all(got <= 1.05 * np.sqrt(want ** 2 + (1.5 if alpha else 0.0) ** 2))


def test_lj_pair():
    """Against the plain expression with the product-difference 2 s^2 - s in one FMA (here in extended precision), which is
    the same number of roundings: 2% for the sampling of rare differences."""
    import torch

    from devinproj_b200 import _lib
    from devinproj_b200.device import stream_handle
    L = _lib.lib()
    rng = np.random.default_rng(7)
    bins = np.array([0.8, 1.0, 1.2, 1.5, 2.0, 2.5])
    r = np.concatenate([rng.uniform(a, b, 40000) for a, b in zip(bins, bins[1:])])
    pos, nbr, nnb = _dimers(torch, r)
    n = len(pos)
    sp, one = torch.zeros(n, dtype=torch.int32, device="cuda"), np.ones(1)
    force, energy = torch.empty_like(pos), torch.empty(1, dtype=torch.float64, device="cuda")
    work = torch.empty(L.acs_force_work_bytes(n), dtype=torch.uint8, device="cuda")
    assert L.acs_lj_fp64(pos.data_ptr(), sp.data_ptr(), n, None, 0, nbr.data_ptr(), nnb.data_ptr(), 1, 1, one.ctypes.data,
                         one.ctypes.data, 2.5, force.data_ptr(), energy.data_ptr(), work.data_ptr(), work.numel(),
                         stream_handle()) == 0
    ext = r.astype(np.longdouble)
    exact, terms = 24 * (2 * ext ** -12 - ext ** -6) / ext, 24 * (2 * ext ** -12 + ext ** -6) / ext
    ir2 = 1.0 / (r * r)
    s6 = ir2 * ir2 * ir2
    plain = 24 * ((2 * s6).astype(np.longdouble) * s6 - s6).astype(float) * ir2 * r
    for a, b in zip(bins, bins[1:]):
        k = (r >= a) & (r < b)
        got, want = (np.sqrt(np.mean(((x - exact) / terms)[k].astype(float) ** 2)) / UNIT
                     for x in (force[1::2, 0].cpu().numpy(), plain))
        print(a, b, got, want)
        assert got <= 1.02 * want


def test_ewald_pair():
    """Two ions, the reciprocal weights zero: the force and the energy are one real-space term."""
    from scipy.special import erfc
    import torch

    from devinproj_b200 import ewald
    from devinproj_b200.device import stream_handle
    L = ewald._bind()
    rng = np.random.default_rng(6)
    rc = 20.0
    alpha = 4 / rc
    r = np.concatenate([rng.uniform(a * rc, b * rc, 500) for a, b in zip(EDGES, EDGES[1:])])
    pos = _dimers(torch, r)[0].reshape(-1, 2, 3).contiguous()
    box = np.array([50.0, 60.0, 70.0])
    q, kw = torch.ones(2, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    kv = torch.tensor([[0.1, 0.2, 0.3]], dtype=torch.float64, device="cuda")
    force = torch.empty_like(pos)
    energy = torch.empty((len(r), 3), dtype=torch.float64, device="cuda")
    work = torch.empty(L.acs_ewald_work_bytes(2, 1), dtype=torch.uint8, device="cuda")
    for k in range(len(r)):
        assert L.acs_ewald_fp64(pos[k].data_ptr(), q.data_ptr(), 2, box.ctypes.data, kv.data_ptr(), kw.data_ptr(), 1, alpha, rc,
                                1.0, force[k].data_ptr(), energy[k].data_ptr(), work.data_ptr(), work.numel(),
                                stream_handle()) == 0
    u, f, _ = _exact(r, alpha, rc)
    root = np.sqrt(r * r)
    er = erfc(alpha * root) / root
    plain = (er + 2 * alpha / np.sqrt(np.pi) * np.exp(-(alpha * root) ** 2)) / (r * r) * r
    for got, expr, exact in ((force[:, 1, 0], plain, f), (energy[:, 0], er, u)):
        want = _rms(_relative(expr, exact, exact), r, rc)
        have = _rms(_relative(got.cpu().numpy(), exact, exact), r, rc)
        print(have, want)
        assert np.all(have <= 1.05 * np.sqrt(want ** 2 + 1.5 ** 2))


def test_descriptor_pair():
    """One neighbour: a vector feature is g fc(r) / r, the same number for the three axes, times the FP32 component of d,
    rounded once. So V_x / d_x and V_y / d_y differ by at most two roundings, 2^-23."""
    import torch

    from devinproj_b200 import learned
    from devinproj_b200.device import stream_handle
    L = learned._bind()
    rng = np.random.default_rng(8)
    m = 2000
    pos = np.zeros((2 * m, 3))
    u = rng.normal(0, 1, (m, 3))
    pos[1::2] = u / np.linalg.norm(u, axis=1)[:, None] * rng.uniform(1.5, 9.5, m)[:, None]
    p, nbr, nnb = _dimers(torch, np.zeros(m))
    p = torch.from_numpy(pos).cuda()
    sp = torch.zeros(2 * m, dtype=torch.int32, device="cuda")
    rbf = learned.rbf_params()
    params = np.array([rbf["r0"], rbf["dmu"], 1 / (2 * rbf["s"] ** 2), rbf["rc"], 0, 0], dtype=np.float32)
    mean, inv_std = torch.zeros(64, device="cuda"), torch.ones(64, device="cuda")
    X = torch.empty((2 * m, 80), dtype=torch.bfloat16, device="cuda")
    V = torch.empty((2 * m, 64, 3), device="cuda")
    assert L.acs_descriptors(p.data_ptr(), sp.data_ptr(), 2 * m, None, 0, nbr.data_ptr(), nnb.data_ptr(), 1,
                             params.ctypes.data, mean.data_ptr(), inv_std.data_ptr(), X.data_ptr(), V.data_ptr(),
                             stream_handle()) == 0
    d = pos[1::2].astype(np.float32).astype(np.float64)
    q = V.cpu().numpy()[::2, :32].astype(np.float64) / d[:, None, :]
    big = np.abs(V.cpu().numpy()[::2, :32]).min(2) > 1e-30   # no subnormal numbers among them
    q = q[big]
    spread = (q.max(1) - q.min(1)) / np.abs(q).mean(1)
    print(len(spread), spread.max() * 2 ** 23)
    assert len(spread) > m and spread.max() <= 2.0 ** -23 * (1 + 1e-6)


# 110,592 atoms with 250 pairs each (several threads per atom there, by the rule's second part) and 13,824 with 55
@pytest.mark.parametrize("n_side,rc", [(48, 4.1), (24, 2.5)])
def test_lj_bits_do_not_depend_on_the_list_capacity(n_side, rc):
    """The same list in buffers of three capacities: the same force and energy, bit for bit, as after a regrow on overflow."""
    import torch

    from tests.test_fp64_kernels_gpu import _abi, _build_list, _grid
    _, L, st = _abi()
    rng = np.random.default_rng(n_side)
    n = n_side ** 3
    box = np.array([1.0, 1.0, 1.0]) * (n / 0.8442) ** (1 / 3)
    grid = np.stack(np.meshgrid(*[np.arange(n_side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = torch.from_numpy((grid + 0.5 + rng.normal(0, 0.05, (n, 3))) * box / n_side % box).cuda()
    sp, one = torch.zeros(n, dtype=torch.int32, device="cuda"), np.ones(1)
    g = _grid(L, box, 1.12 * rc)
    work = torch.empty(L.acs_force_work_bytes(n), dtype=torch.uint8, device="cuda")
    expected = int(4 / 3 * np.pi * (1.12 * rc) ** 3 * 0.8442)
    out = []
    for maxnb in (expected + 40, 2 * expected + 40, 4 * expected):
        nbr, nnb = _build_list(torch, L, st, pos, g, maxnb)
        force, energy = torch.empty_like(pos), torch.empty(1, dtype=torch.float64, device="cuda")
        assert L.acs_lj_fp64(pos.data_ptr(), sp.data_ptr(), n, box.ctypes.data, 1, nbr.data_ptr(), nnb.data_ptr(), maxnb, 1,
                             one.ctypes.data, one.ctypes.data, rc, force.data_ptr(), energy.data_ptr(), work.data_ptr(),
                             work.numel(), st) == 0
        out.append(torch.cat([force.reshape(-1), energy]).cpu())
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
