"""Single systems that fill a part of their box only (slabs, a droplet): forces, energy and virial are the
staged calls', bit for bit, and the atoms' bins hold them (the list of surplus atoms, which every tile reads,
made such evaluations ten times as long)."""
import numpy as np
import pytest

from gpu_recip_b200 import systems as S

pytestmark = pytest.mark.gpu


def _system(nfft, order, shape):
    box = np.array(nfft, float)
    part = box.copy()
    if shape == "droplet":
        part *= 0.55
    else:
        part["xyz".index(shape[0])] /= int(shape[1])
    x = S.water_box(int(part.prod() * 8000 / 62.1 ** 3), part, 17)
    if shape == "droplet":
        x = x[((x[:, :3] - part / 2) ** 2).sum(1) < (part.min() / 2) ** 2]
        x[:, :3] += np.float32(0.2) * box.astype(np.float32)
    return S.PmeSystem(shape, np.ascontiguousarray(x), tuple(box), nfft, order, 0.33)


def _eval(torch, p, s, x, staged):
    from gpu_recip_b200 import recip_from_box
    n = s.natom
    f = torch.zeros((n, 3), device="cuda")
    r = recip_from_box(s.box)
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
    return f.cpu().numpy(), p.energy_virial.getEnergy("recip"), p.energy_virial.getVirial()


@pytest.mark.parametrize("shape", ["z4", "y2", "x3", "z20", "droplet"])
@pytest.mark.parametrize("nfft,order", [((48, 40, 96), 4), ((64, 64, 64), 6), ((60, 54, 72), 8)])
def test_part_of_the_box(cuda, nfft, order, shape):
    from gpu_recip_b200 import CudaPMERecip
    s = _system(nfft, order, shape)
    x = cuda.from_numpy(s.xyzq).cuda()
    p = CudaPMERecip(*nfft, order)
    want = _eval(cuda, CudaPMERecip(*nfft, order), s, x, True)
    for _ in range(2):
        got = _eval(cuda, p, s, x, False)
        assert np.array_equal(got[0], want[0]) and got[1] == want[1] and np.array_equal(got[2], want[2])


def test_slab_takes_about_as_long_as_a_full_box(cuda):
    """75,000 atoms on 144^3, in a quarter of the box and in all of it: 1.1 times as long here, 10 where the
    bins held 1.5 times their mean only."""
    from gpu_recip_b200 import CudaPMERecip, recip_from_box
    n = (144, 144, 144)
    slab = _system(n, 4, "z4")
    full = S.PmeSystem("full", S.water_box(slab.natom // 3, (144.0,) * 3, 3), (144.0,) * 3, n, 4, 0.33)
    us = []
    for s in (slab, full):
        p = CudaPMERecip(*n, 4)
        x = cuda.from_numpy(s.xyzq).cuda()
        f = cuda.zeros((s.natom, 3), device="cuda")
        r = recip_from_box(s.box)
        times = []
        for k in range(25):
            a, b = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            a.record()
            p.eval(r, x, s.natom, s.kappa, False, False, f, 1)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        us.append(sorted(times)[8] * 1e3)
    assert us[0] < 3.0 * us[1], us
