"""The fused spread's edges: candidate counts around a warp's 32 and a CTA's 256, atoms that all share
one bin (so that it overflows), row blocks of every shape the block rule picks, and charges that force
the carry form of the accumulation.  The fused evaluation must give the staged calls' forces, energy and
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
    ((32, 32, 32), 1000, 60.0), ((64, 54, 60), 6000, 200.0),      # the carry form
])
@pytest.mark.parametrize("order", [4, 6, 8])
def test_block_shapes(cuda, order, nfft, waters, q):
    box = tuple(float(n) * 0.98 for n in nfft)
    x = S.water_box(waters, box, 77 + order)
    x[:, 3] *= q
    a, b = _both(cuda, S.PmeSystem("blocks", x, box, nfft, order, 0.33))
    assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2])
