"""The rotation at the edges of its column groups (64, 256 and 1024 columns, one to four per thread)
and for one to nine maps, against the oracle's Wigner d(pi/2).  Tolerance 1e-12 x max|alm|, the FP64
level's bound (the recursion's rounding grows like a few l 2^-53)."""
import numpy as np
import pytest

from oracle import dsht_oracle as O

pytestmark = pytest.mark.gpu


def _random_alm(rng, Nl):
    n = Nl * (Nl + 1) // 2
    a = rng.normal(size=n) + 1j * rng.normal(size=n)
    a[:Nl] = a[:Nl].real
    return a


@pytest.mark.parametrize("Nl", [1, 2, 3, 4, 5, 63, 64, 65, 128, 255, 257, 320, 513, 770, 1030])
def test_rotate_back_edges(Nl):
    import torch
    from directsht_b200 import DirectSHT
    from directsht_b200 import _lib as L
    rng = np.random.default_rng(Nl)
    a = _random_alm(rng, Nl)
    d = DirectSHT(Nl, 2)
    rot, out = torch.from_numpy(a).cuda(), torch.empty(len(a), dtype=torch.complex128, device="cuda")
    L.check(d._lib.dsht_rotate_back(d._plan, L.ptr(rot), None, L.ptr(out), None))
    add = torch.from_numpy(_random_alm(rng, Nl)).cuda()
    both = torch.empty_like(out)
    L.check(d._lib.dsht_rotate_back(d._plan, L.ptr(rot), L.ptr(add), L.ptr(both), None))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    # degrees at the column edges and the largest
    index = lambda l, m: m * (2 * Nl - 1 - m) // 2 + l
    for l in sorted({0, min(2, Nl - 1), Nl // 2, Nl - 1}):
        D = O.wigner_d_halfpi_column(l)  # [m', m] for m', m >= 0
        al = np.array([a[index(l, m)] for m in range(l + 1)])
        k = np.arange(l + 1)
        for m in range(l + 1):
            even = (l + m + k) % 2 == 0
            wt = np.where(k > 0, 2.0, 1.0)
            re = (D[:, m] * wt * al.real)[even].sum()
            im = (D[:, m] * 2.0 * al.imag)[~even & (k > 0)].sum()
            assert abs(got[index(l, m)] - (re + 1j * im)) <= 1e-12 * np.abs(al).max() * max(1, l) ** 0.5, (l, m)
    np.testing.assert_array_equal(both.cpu().numpy(), add.cpu().numpy() + got)


@pytest.mark.parametrize("nmaps", [2, 3, 4, 5, 7, 9])
def test_maps_equal_single_rotations(nmaps):
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(nmaps)
    Nl, N = 300, 500
    th, ph = np.arccos(rng.uniform(0.6, 1.0, N)), rng.uniform(0, 2 * np.pi, N)
    w = rng.normal(size=(nmaps, N))
    d = DirectSHT(Nl, 40)
    got = d.call_maps(th, ph, w)
    for k in range(nmaps):
        ref = d(th, ph, w[k])
        assert np.abs(got[k] - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("Nl", [1, 64, 65, 300, 1030])
def test_rotate_back_in_place(Nl):
    """alm_out may be any of the inputs: the result is that of separate arrays, bit for bit."""
    import torch
    from directsht_b200 import DirectSHT
    from directsht_b200 import _lib as L
    rng = np.random.default_rng(Nl)
    d = DirectSHT(Nl, 2)
    a, b = (torch.from_numpy(_random_alm(rng, Nl)).cuda() for _ in range(2))

    def rotate(rot, add, out):
        L.check(d._lib.dsht_rotate_back(d._plan, L.ptr(rot), None if add is None else L.ptr(add), L.ptr(out), None))
        torch.cuda.synchronize()
        return out

    new = lambda: torch.full_like(a, float("nan"))
    sum_ab, rot_a, sum_aa = rotate(a, b, new()), rotate(a, None, new()), rotate(a, a, new())
    x, y = a.clone(), b.clone()
    assert torch.equal(rotate(x, y, x), sum_ab) and torch.equal(y, b)
    y = b.clone()
    assert torch.equal(rotate(a, y, y), sum_ab)
    x = a.clone()
    assert torch.equal(rotate(x, None, x), rot_a)
    x = a.clone()
    assert torch.equal(rotate(x, x, x), sum_aa)
