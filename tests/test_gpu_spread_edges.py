"""The fused spread's edges: candidate counts around a warp's 32 and a CTA's 256, atoms that all share
one bin (so that it overflows), row blocks of every shape the block rule picks, and charges and atom
counts that force the carry form of the accumulation on every tile.  The fused evaluation must give the staged calls' forces, energy and
virial bit for bit (the staged spread adds every contribution to the int64 grid by itself)."""
import numpy as np
import pytest

from gpu_recip_b200 import systems as S

pytestmark = pytest.mark.gpu


def _both(torch, s):
    from gpu_recip_b200 import CudaPMERecip, recip_from_box
    n = s.natom
    x = torch.from_numpy(s.xyzq).cuda()
    out = []
    for staged in (False, True):
        p = CudaPMERecip(*s.nfft, s.order)
        f = torch.zeros((n, 3), device="cuda")
        r = recip_from_box(s.box)
        for _ in range(2):          # the second evaluation takes the atoms in the bins' order
            p.energy_virial.clear()
            if staged:
                p.spread_charge(x, n, r)
                p.r2c_fft()
                p.scalar_sum(r, s.kappa, True, True)
                p.c2r_fft()
                p.gather_force(x, n, r, 1, f)
            else:
                p.eval(r, x, n, s.kappa, True, True, f, 1)
        p.energy_virial.copyToHost()
        out.append((f.cpu().numpy(), p.energy_virial.getEnergy("recip"), p.energy_virial.getVirial()))
        p.close()
    return out


@pytest.mark.parametrize("order", [4, 6, 8])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 700])
def test_candidate_counts_in_one_place(cuda, order, n):
    """All atoms within half a grid spacing: one bin holds them, and overflows beyond its capacity."""
    rng = np.random.default_rng(10 * n + order)
    x = np.empty((n, 4), np.float32)
    x[:, :3] = np.array([31.7, 0.2, 15.1]) + rng.random((n, 3)) * 0.5
    x[:, 3] = rng.normal(0.0, 0.5, n)
    a, b = _both(cuda, S.PmeSystem("one place", x, (32.0, 32.0, 32.0), (32, 32, 32), order, 0.34))
    assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("nfft,waters,q", [
    ((16, 16, 16), 100, 1.0), ((24, 25, 27), 400, 1.0), ((32, 32, 32), 1000, 1.0), ((45, 40, 50), 2000, 1.0),
    ((64, 54, 60), 6000, 1.0), ((120, 75, 81), 20000, 1.0), ((512, 16, 18), 1500, 1.0),
    ((32, 32, 32), 1000, 60.0), ((64, 54, 60), 6000, 200.0),      # some tiles near the split form's bound
])
@pytest.mark.parametrize("order", [4, 6, 8])
def test_block_shapes(cuda, order, nfft, waters, q):
    box = tuple(float(n) * 0.98 for n in nfft)
    x = S.water_box(waters, box, 77 + order)
    x[:, 3] *= q
    a, b = _both(cuda, S.PmeSystem("blocks", x, box, nfft, order, 0.33))
    assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2])


# cube of the largest weight of the order-P spline
PEAK3 = {4: (2.0 / 3.0) ** 3, 6: 0.55 ** 3, 8: (151.0 / 315.0) ** 3}


def _fewest_candidates(s, order):
    """The fewest atoms whose stencils reach a block of rows, over all places: what any tile of any block
    shape has as candidates at least (one row; larger blocks reach more)."""
    ny, nz = s.nfft[1], s.nfft[2]
    iy = np.floor(s.xyzq[:, 1] / s.box[1] * ny).astype(int) % ny
    iz = np.floor(s.xyzq[:, 2] / s.box[2] * nz).astype(int) % nz
    h = np.zeros((ny, nz))
    np.add.at(h, (iy, iz), 1)
    reach = sum(np.roll(h, (a, b), (0, 1)) for a in range(order) for b in range(order))
    return int(reach.min())


def _assert_carry(s, order, fewest):
    """The split form's bound on its upper sums, 256 n^2 |q|max M^3 at least (its exponent is the largest k
    with n 2^k < 2^32), is beyond 2^31 for n = fewest candidates, so every tile takes the carry form."""
    q = float(np.abs(s.xyzq[:, 3]).max())
    assert 256.0 * fewest ** 2 * q * PEAK3[order] > 1.2 * 2.0 ** 31


@pytest.mark.parametrize("nfft,waters", [((32, 32, 32), 1000), ((64, 54, 60), 6000), ((45, 40, 50), 2000)])
@pytest.mark.parametrize("order", [4, 6, 8])
def test_carry_form_by_charge(cuda, order, nfft, waters):
    """Charges that no tile's split form holds.  Energy and virial (fixed point at 2^32) are beyond their
    range at such charges; the forces are not."""
    box = tuple(float(n) * 0.98 for n in nfft)
    x = S.water_box(waters, box, 90 + order)
    s = S.PmeSystem("carry", x, box, nfft, order, 0.33)
    fewest = _fewest_candidates(s, order)
    x[:, 3] *= np.float32(2.0 ** 23 * 2.0 / (fewest ** 2 * PEAK3[order] * np.abs(x[:, 3]).max()))
    _assert_carry(s, order, fewest)
    a, b = _both(cuda, s)
    assert np.abs(b[0]).max() > 0 and np.isfinite(b[0]).all() and np.array_equal(a[0], b[0])


@pytest.mark.parametrize("order", [4, 6, 8])
def test_carry_form_by_count(cuda, order):
    """14,000 ions in one place: every tile has the atoms beyond that bin's capacity as candidates."""
    rng = np.random.default_rng(order)
    x = np.empty((14000, 4), np.float32)
    x[:, :3] = np.array([15.3, 0.1, 31.8]) + rng.random((14000, 3)) * 0.6
    x[:, 3] = np.where(np.arange(14000) % 2, 1.0, -1.0)
    s = S.PmeSystem("one place", x, (32.0, 32.0, 32.0), (32, 32, 32), order, 0.34)
    _assert_carry(s, order, 14000 - 2000)   # a bin holds some hundreds of them
    a, b = _both(cuda, s)
    assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2])
