"""The launch of a single system's evaluation: the build of the kernel is the one that the row blocks were
chosen for, and the inverse x pass runs inside the gather only where the gather is one wave.  The shapes
change the time alone: forces, energy and virial are the staged calls', bit for bit."""
import functools

import numpy as np
import pytest

from gpu_recip_b200 import systems as S

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _system(nfft, order):
    box = tuple(float(n) for n in nfft)
    waters = int(np.prod(box) * 8000 / 62.1 ** 3)
    return S.PmeSystem("launch", S.water_box(waters, box, 5), box, nfft, order, 0.33)


def _eval(torch, p, s, x, staged=False):
    from gpu_recip_b200 import recip_from_box
    f = torch.zeros((s.natom, 3), device="cuda")
    r = recip_from_box(s.box)
    p.energy_virial.clear()
    if staged:
        p.spread_charge(x, s.natom, r)
        p.r2c_fft()
        p.scalar_sum(r, s.kappa, True, True)
        p.c2r_fft()
        p.gather_force(x, s.natom, r, 1, f)
    else:
        p.eval(r, x, s.natom, s.kappa, True, True, f, 1)
    p.energy_virial.copyToHost()
    return f.cpu().numpy(), p.energy_virial.getEnergy("recip"), p.energy_virial.getVirial()


@pytest.mark.parametrize("nfft,order,three,fused_x", [
    ((64, 64, 64), 4, False, True),       # 256 tiles of 4 x 4 rows: one wave of 2 CTAs per SM
    ((40, 128, 64), 4, False, False),     # 512: more than one wave
    ((72, 72, 72), 4, True, False),       # 432 of 4 x 3 rows: one wave of 3 CTAs per SM
    ((81, 81, 81), 6, True, False),       # 441 of 4 x 4 rows
    ((90, 75, 80), 8, True, False),       # 380 of 4 x 4 rows
    ((128, 125, 128), 8, False, False),   # 1024 of 4 x 4 rows: faster in four waves of 2 than in three of 3
])
def test_build_follows_the_row_blocks(cuda, nfft, order, three, fused_x):
    from gpu_recip_b200 import CudaPMERecip
    from gpu_recip_b200.pme import TRACE_STEP_STAMPS
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    if sms != 148:
        pytest.skip("the tile counts are for 148 SMs")
    s = _system(nfft, order)
    x = cuda.from_numpy(s.xyzq).cuda()
    p = CudaPMERecip(*nfft, order)
    buf = cuda.zeros(1024 * 14 + TRACE_STEP_STAMPS, dtype=cuda.int64, device="cuda")
    p.set_trace(buf, 1024)
    got = _eval(cuda, p, s, x)
    p.set_trace(None)
    ran = buf[:1024 * 14].view(1024, 7, 2)[:, :, 0].cpu().numpy() > 0
    assert (ran[:, 1].sum() > 2 * sms) == three
    assert ran[:, 5].any() != fused_x
    want = _eval(cuda, CudaPMERecip(*nfft, order), s, x, staged=True)
    assert np.array_equal(got[0], want[0]) and got[1] == want[1] and np.array_equal(got[2], want[2])
    p.close()


@pytest.mark.parametrize("schedule,z_passes", [(0, True), (3, False)])
def test_cluster_planes_asked_for_are_run(cuda, schedule, z_passes):
    """72^3 order 4 runs the throughput build by itself, with y and z passes; the cluster planes, which only
    the latency build has, where the caller asks for them."""
    from gpu_recip_b200 import CudaPMERecip
    from gpu_recip_b200.pme import TRACE_STEP_STAMPS
    s = _system((72, 72, 72), 4)
    x = cuda.from_numpy(s.xyzq).cuda()
    p = CudaPMERecip(72, 72, 72, 4)
    p.set_fft_schedule(schedule)
    buf = cuda.zeros(1024 * 14 + TRACE_STEP_STAMPS, dtype=cuda.int64, device="cuda")
    p.set_trace(buf, 1024)
    got = _eval(cuda, p, s, x)
    p.set_trace(None)
    assert bool((buf[:1024 * 14].view(1024, 7, 2)[:, 3, 0] > 0).any()) == z_passes
    want = _eval(cuda, CudaPMERecip(72, 72, 72, 4), s, x, staged=True)
    assert np.array_equal(got[0], want[0]) and got[1] == want[1] and np.array_equal(got[2], want[2])


def test_changed_order_takes_its_own_row_block(cuda):
    """Order 8 on 32^3 has blocks of 4 x 1 rows (256 tiles), order 4 of 3 x 3 (121): a handle whose order
    changes before its first evaluation is launched as one made with that order."""
    from gpu_recip_b200 import CudaPMERecip
    from gpu_recip_b200.pme import TRACE_STEP_STAMPS
    s = _system((32, 32, 32), 4)
    x = cuda.from_numpy(s.xyzq).cuda()
    tiles = []
    for first in (4, 8):
        p = CudaPMERecip(32, 32, 32, first)
        p.set_order(4)
        buf = cuda.zeros(1024 * 14 + TRACE_STEP_STAMPS, dtype=cuda.int64, device="cuda")
        p.set_trace(buf, 1024)
        _eval(cuda, p, s, x)
        p.set_trace(None)
        tiles.append(int((buf[:1024 * 14].view(1024, 7, 2)[:, 1, 0] > 0).sum()))
        p.close()
    assert tiles[0] == tiles[1]


@pytest.mark.parametrize("evaluated", [False, True])
@pytest.mark.parametrize("nfft", [(32, 32, 32), (72, 72, 72)])
@pytest.mark.parametrize("first,order", [(4, 8), (8, 4), (6, 4), (4, 6)])
def test_changed_order_gives_a_new_handles_bits(cuda, nfft, first, order, evaluated):
    """Whether or not the handle has evaluated at its first order: order 4 to 8 and back."""
    from gpu_recip_b200 import CudaPMERecip
    s = _system(nfft, order)
    x = cuda.from_numpy(s.xyzq).cuda()
    p = CudaPMERecip(*nfft, first)
    if evaluated:
        _eval(cuda, p, s, x)
    p.set_order(order)
    want = _eval(cuda, CudaPMERecip(*nfft, order), s, x)
    for _ in range(2):
        got = _eval(cuda, p, s, x)
        assert np.array_equal(got[0], want[0]) and got[1] == want[1] and np.array_equal(got[2], want[2])
    p.close()


def test_row_block_follows_the_number_of_atoms(cuda):
    """48^3 order 4: blocks of 4 x 4 rows (144 tiles) at 0.1 atoms per grid point, 3 x 3 (256) at 0.2; a
    handle that grows from the one to the other takes the new block and keeps its results."""
    from gpu_recip_b200 import CudaPMERecip
    from gpu_recip_b200.pme import TRACE_STEP_STAMPS
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    if sms != 148:
        pytest.skip("the tile counts are for 148 SMs")
    p = CudaPMERecip(48, 48, 48, 4)
    for waters, tiles in ((3700, 144), (7400, 256), (3700, 256)):
        box = (48.0,) * 3
        s = S.PmeSystem("atoms", S.water_box(waters, box, 6), box, (48, 48, 48), 4, 0.33)
        x = cuda.from_numpy(s.xyzq).cuda()
        buf = cuda.zeros(1024 * 14 + TRACE_STEP_STAMPS, dtype=cuda.int64, device="cuda")
        p.set_trace(buf, 1024)
        got = _eval(cuda, p, s, x)
        p.set_trace(None)
        # a CTA per tile (and one for the record)
        assert int((buf[:1024 * 14].view(1024, 7, 2)[:, 1, 0] > 0).sum()) in (tiles, tiles + 1)
        want = _eval(cuda, CudaPMERecip(48, 48, 48, 4), s, x, staged=True)
        assert np.array_equal(got[0], want[0]) and got[1] == want[1] and np.array_equal(got[2], want[2])
    p.close()


@pytest.mark.parametrize("nfft,order", [((16, 512, 512), 4), ((24, 400, 360), 8)])
def test_grids_whose_tiles_leave_one_cta_per_sm(cuda, nfft, order):
    """The z tiles of long y and z axes take more than half an SM's shared memory: the row block is still
    one of many rows (an evaluation with blocks of one row took 20 to 40 times the staged calls), and the
    bits are theirs."""
    from gpu_recip_b200 import CudaPMERecip
    s = _system(nfft, order)
    x = cuda.from_numpy(s.xyzq).cuda()
    p = CudaPMERecip(*nfft, order)
    ms, out = [], []
    for staged in (False, True):
        for k in range(4):
            a, b = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            a.record()
            got = _eval(cuda, p, s, x, staged)
            b.record()
            b.synchronize()
        ms.append(a.elapsed_time(b))
        out.append(got)
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1] and np.array_equal(out[0][2], out[1][2])
    assert ms[0] < 4.0 * ms[1], ms
