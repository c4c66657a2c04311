"""Direct-space PME on the GPU (include/pme_direct.h) against the reference's direct test and
the FP64 oracle.  Bars: the reference driver's own tolerances on its 23,558-atom fixture
(gpu_direct.cu:158-222: forces 7.72e-4 / 7.73e-4, energies 0.007, virial 3.13); against the
oracle a force relative RMS of 1e-5 and energies within 1e-6 relative; identical int64 forces
and energies from run to run."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORCE_SCALE = 2.0 ** 40


@pytest.fixture(scope="module")
def fx():
    from tests.conftest import GOLDEN
    return dict(np.load(os.path.join(GOLDEN, "ref_direct_23558.npz")))


def _make(torch, d, with14=False):
    from gpu_recip_b200.direct import CudaPMEDirectForce
    n = d["xyzq"].shape[0]
    dr = CudaPMEDirectForce()
    dr.setup(*d["box"], float(d["kappa"]), float(d["roff"]), float(d.get("ron", 0.0)), float(d.get("e14fac", 1.0)))
    dr.set_vdwparam(d["vdwparam"])
    dr.set_vdwtype(d["vdwtype"])
    if "iblo14" in d:
        dr.set_exclusions(d["iblo14"], d["inb14"], d.get("loc2glo"))
    if with14:
        dr.set_vdwparam14(d["vdwparam14"])
        dr.set_14_list(d["in14"], d["ex14"])
    x = torch.from_numpy(np.ascontiguousarray(d["xyzq"], dtype=np.float32)).cuda()
    stride = ((n + 63) // 64) * 64
    return dr, x, n, stride


def _run(torch, dr, x, n, stride, with14=False):
    f = torch.zeros(3 * stride, dtype=torch.int64, device="cuda")
    dr.energy_virial.clear()
    dr.calc_force(x, n, True, True, stride, f)
    if with14:
        dr.calc_14_force(x, True, True, stride, f)
    torch.cuda.synchronize()
    ev = dr.energy_virial
    ev.copyToHost()
    fi = f.view(3, stride)[:, :n].T.cpu().numpy()
    return fi, dict(vdw=ev.getEnergy("vdw"), elec=ev.getEnergy("elec"), excl=ev.getEnergy("excl")), ev.getVirial()


def test_direct_reference_fixture_main_list(cuda, fx):
    dr, x, n, stride = _make(cuda, fx)
    fi, e, vir = _run(cuda, dr, x, n, stride)
    f = fi.astype(np.float64) / FORCE_SCALE
    assert np.abs(f - fx["force_main"]).max() <= fx["tol_force_main"]
    assert abs(e["vdw"] - fx["energy_vdw"]) < fx["tol_energy"]
    assert abs(e["elec"] - fx["energy_elec"]) < fx["tol_energy"]
    assert np.abs(vir - fx["virial"]).max() < fx["tol_virial"]
    # run to run: the same int64 forces and energies
    fi2, e2, vir2 = _run(cuda, dr, x, n, stride)
    assert np.array_equal(fi, fi2) and e == e2 and np.array_equal(vir, vir2)
    dr.close()


def test_direct_reference_fixture_total_with_14_lists(cuda, fx, oracle):
    dr, x, n, stride = _make(cuda, fx, with14=True)
    fi, e, _ = _run(cuda, dr, x, n, stride, with14=True)
    f = fi.astype(np.float64) / FORCE_SCALE
    assert np.abs(f - fx["force_total"]).max() <= fx["tol_force_total"]
    _, ev14, ee14, ex14, _ = oracle.direct_14(fx["xyzq"].astype(np.float64), fx["box"], float(fx["kappa"]),
                                              float(fx["roff"]), float(fx["e14fac"]), fx["vdwparam14"],
                                              fx["vdwtype"], fx["in14"], fx["ex14"])
    assert abs(e["excl"] - ex14) < 1e-6 * abs(ex14)
    assert abs(e["vdw"] - (fx["energy_vdw"] + ev14)) < fx["tol_energy"]
    assert abs(e["elec"] - (fx["energy_elec"] + ee14)) < fx["tol_energy"]
    dr.close()


def test_direct_matches_fp64_oracle_on_fixture(cuda, fx, oracle):
    dr, x, n, stride = _make(cuda, fx)
    fi, e, vir = _run(cuda, dr, x, n, stride)
    ptr, idx = oracle.exclusions_csr(fx["iblo14"], fx["inb14"], n, fx["loc2glo"])
    vp32 = fx["vdwparam"].astype(np.float32).astype(np.float64)   # the library holds FP32 parameters
    fo, ev, ee, vo = oracle.direct_force(fx["xyzq"].astype(np.float32).astype(np.float64), fx["box"],
                                         float(fx["kappa"]), float(fx["roff"]), vp32, fx["vdwtype"], ptr, idx)
    f = fi.astype(np.float64) / FORCE_SCALE
    rms = np.sqrt(((f - fo) ** 2).sum() / (fo ** 2).sum())
    assert rms <= 1e-5, rms
    assert abs(e["vdw"] - ev) <= 1e-6 * abs(ev)
    assert abs(e["elec"] - ee) <= 1e-6 * abs(ee)
    assert np.abs(vir - vo).max() <= 1e-5 * np.abs(vo).max()
    dr.close()


def _lattice(box=24.0, per=6, seed=3):
    """Charges on a jittered lattice with exclusions to the +x lattice neighbour (wrapping pairs sit
    180 indices apart: the explicit far-list path), two vdW types."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(per)] * 3, indexing="ij"), -1).reshape(-1, 3)
    n = per ** 3
    sp = box / per
    x = np.empty((n, 4))
    x[:, :3] = g * sp + rng.uniform(-0.3, 0.3, (n, 3))
    x[:, 3] = rng.choice([-0.8, 0.4], n)
    iblo, inb = [], []
    for i in range(n):
        gx, gy, gz = g[i]
        j = int(((gx + 1) % per) * per * per + gy * per + gz)
        inb.append(j + 1)
        iblo.append(len(inb))
    return dict(xyzq=x.astype(np.float32), box=np.array([box, box, box]), kappa=np.array(0.35),
                roff=np.array(9.0), vdwparam=np.array([1.0e2, 1.2e5, 6.0e1, 1.6e5, 2.9e2, 5.0e5]),
                vdwtype=(np.arange(n) % 2).astype(np.int32), iblo14=np.array(iblo, np.int32),
                inb14=np.array(inb, np.int32))


@pytest.mark.parametrize("box", [24.0, 40.0])   # 24 A: fewer cells than offsets on every axis
def test_direct_lattice_with_far_exclusions_matches_oracle(cuda, oracle, box):
    d = _lattice(box=box, per=6 if box == 24.0 else 10)
    dr, x, n, stride = _make(cuda, d)
    fi, e, vir = _run(cuda, dr, x, n, stride)
    ptr, idx = oracle.exclusions_csr(d["iblo14"], d["inb14"], n)
    vp32 = d["vdwparam"].astype(np.float32).astype(np.float64)
    fo, ev, ee, vo = oracle.direct_force(d["xyzq"].astype(np.float64), d["box"], float(d["kappa"]),
                                         float(d["roff"]), vp32, d["vdwtype"], ptr, idx)
    f = fi.astype(np.float64) / FORCE_SCALE
    assert np.sqrt(((f - fo) ** 2).sum() / (fo ** 2).sum()) <= 1e-5
    assert abs(e["vdw"] - ev) <= 1e-6 * abs(ev) + 1e-6 and abs(e["elec"] - ee) <= 1e-6 * abs(ee)
    assert np.abs(vir - vo).max() <= 1e-5 * np.abs(vo).max()
    dr.close()


def test_direct_electrostatics_only_and_no_exclusions(cuda, oracle):
    from gpu_recip_b200.direct import CudaPMEDirectForce, ELEC_NONE, EWALD, VDW_NONE
    d = _lattice()
    n = d["xyzq"].shape[0]
    dr = CudaPMEDirectForce()
    dr.setup(24.0, 24.0, 24.0, 0.35, 9.0, 7.5, 1.0, VDW_NONE, EWALD)
    x = cuda.from_numpy(d["xyzq"]).cuda()
    fi, e, _ = _run(cuda, dr, x, n, n)
    ptr = np.zeros(n + 1, np.int32)
    fo, ev, ee, _ = oracle.direct_force(d["xyzq"].astype(np.float64), d["box"], 0.35, 9.0, np.zeros(2),
                                        np.zeros(n, np.int32), ptr, np.zeros(0, np.int32))
    f = fi.astype(np.float64) / FORCE_SCALE
    assert np.sqrt(((f - fo) ** 2).sum() / (fo ** 2).sum()) <= 1e-5
    assert e["vdw"] == 0.0 and abs(e["elec"] - ee) <= 1e-6 * abs(ee)
    dr.close()


def test_direct_argument_checks(cuda):
    from gpu_recip_b200 import _capi
    from gpu_recip_b200.direct import CudaPMEDirectForce
    dr = CudaPMEDirectForce()
    x = cuda.zeros((4, 4), device="cuda")
    f = cuda.zeros(12, dtype=cuda.int64, device="cuda")
    with pytest.raises(_capi.PMEError) as e:       # before setup
        dr.calc_force(x, 4, True, True, 4, f)
    assert e.value.status == _capi.PME_ESTATE
    with pytest.raises(_capi.PMEError) as e:       # roff beyond half the box
        dr.setup(10.0, 10.0, 10.0, 0.3, 9.0, 7.5, 1.0)
    assert e.value.status == _capi.PME_EINVAL
    with pytest.raises(_capi.PMEError) as e:       # a model that is not built
        dr.setup(30.0, 30.0, 30.0, 0.3, 9.0, 7.5, 1.0, 2, 101)
    assert e.value.status == _capi.PME_EUNSUPPORTED
    dr.setup(30.0, 30.0, 30.0, 0.3, 9.0, 7.5, 1.0)
    dr.set_vdwparam([1.0, 2.0, 3.0, 4.0, 5.0, 6.0])          # 2 types
    dr.set_vdwtype([0, 1, 2, 0])                             # type 2 is beyond the table
    with pytest.raises(_capi.PMEError) as e:
        dr.calc_force(x, 4, True, True, 4, f)
    assert e.value.status == _capi.PME_EINVAL
    dr.set_vdwtype([0, 1, 1, 0])
    dr.set_vdwparam14([1.0, 2.0, 3.0, 4.0, 5.0, 6.0])
    dr.set_14_list([[0, 9, 13]], [])                         # atom 9 of 4
    with pytest.raises(_capi.PMEError) as e:
        dr.calc_14_force(x, True, True, 4, f)
    assert e.value.status == _capi.PME_EINVAL
    with pytest.raises(_capi.PMEError) as e:                 # loc2glo not a permutation
        dr.set_exclusions([1, 1, 1, 1], [2], [0, 0, 1, 2])
    assert e.value.status == _capi.PME_EINVAL
    dr.close()


@pytest.mark.parametrize("box,n", [(20.0, 3000), (40.0, 24000)])   # every axis with too few cells; shifts
def test_direct_dense_cells_many_chunks(cuda, oracle, box, n):
    """About 90 atoms per cell (three 32-atom chunks each): electrostatics only (random charges
    closer than any vdW model would allow), against the FP64 oracle."""
    from gpu_recip_b200.direct import CudaPMEDirectForce, EWALD, VDW_NONE
    rng = np.random.default_rng(n)
    x = np.empty((n, 4), np.float32)
    x[:, :3] = rng.random((n, 3)) * box
    x[:, 3] = rng.normal(0.0, 0.3, n)
    dr = CudaPMEDirectForce()
    dr.setup(box, box, box, 0.35, 9.0, 7.5, 1.0, VDW_NONE, EWALD)
    xd = cuda.from_numpy(x).cuda()
    fi, e, vir = _run(cuda, dr, xd, n, n)
    fo, _, ee, vo = oracle.direct_force(x.astype(np.float64), np.array([box] * 3), 0.35, 9.0, np.zeros(2),
                                        np.zeros(n, np.int32), np.zeros(n + 1, np.int32), np.zeros(0, np.int32))
    f = fi.astype(np.float64) / FORCE_SCALE
    assert np.sqrt(((f - fo) ** 2).sum() / (fo ** 2).sum()) <= 1e-6
    assert abs(e["elec"] - ee) <= 1e-7 * abs(ee) + 1e-6
    assert np.abs(vir - vo).max() <= 1e-6 * np.abs(vo).max()
    dr.close()


def test_direct_vdw_only(cuda, oracle):
    """ELEC_NONE: only the shifted Lennard-Jones terms (the oracle with the charges set to 0)."""
    from gpu_recip_b200.direct import CudaPMEDirectForce, ELEC_NONE, VDW_VSH
    d = _lattice()
    n = d["xyzq"].shape[0]
    dr = CudaPMEDirectForce()
    dr.setup(24.0, 24.0, 24.0, 0.35, 9.0, 7.5, 1.0, VDW_VSH, ELEC_NONE)
    dr.set_vdwparam(d["vdwparam"])
    dr.set_vdwtype(d["vdwtype"])
    dr.set_exclusions(d["iblo14"], d["inb14"])
    x = cuda.from_numpy(d["xyzq"]).cuda()
    fi, e, vir = _run(cuda, dr, x, n, n)
    xq0 = d["xyzq"].astype(np.float64).copy()
    xq0[:, 3] = 0.0
    ptr, idx = oracle.exclusions_csr(d["iblo14"], d["inb14"], n)
    fo, ev, ee, vo = oracle.direct_force(xq0, d["box"], 0.35, 9.0, d["vdwparam"].astype(np.float32).astype(np.float64),
                                         d["vdwtype"], ptr, idx)
    f = fi.astype(np.float64) / FORCE_SCALE
    assert e["elec"] == 0.0 and ee == 0.0
    assert np.sqrt(((f - fo) ** 2).sum() / (fo ** 2).sum()) <= 1e-6
    assert abs(e["vdw"] - ev) <= 1e-6 * abs(ev)
    dr.close()


@pytest.mark.parametrize("box,n,roff,ntype,kappa", [
    ((18.0, 18.0, 18.0), 1, 9.0, 0, 0.35),          # one atom; a cutoff of half the box
    ((18.0, 18.0, 18.0), 9, 9.0, 0, 0.35),          # partial clusters, columns visited at several images
    ((18.0, 18.0, 18.0), 1500, 9.0, 0, 0.35),
    ((20.0, 22.0, 19.0), 12000, 9.0, 0, 0.35),      # dense: narrow columns, queues that fill
    ((200.0, 150.0, 180.0), 500, 9.0, 0, 0.35),     # sparse: wide columns, long clusters
    ((18.1, 40.0, 90.0), 3000, 7.0, 0, 0.0),        # uneven box, plain Coulomb
    ((60.0, 40.0, 45.0), 1000, 20.0, 0, 0.25),      # a long cutoff
    ((24.0, 24.0, 24.0), 216, 9.0, 3, 0.35),        # vdW types in the square table
    ((24.0, 24.0, 24.0), 216, 9.0, 70, 0.35),       # more types than the square table holds
])
def test_direct_cluster_edges_match_oracle(cuda, oracle, box, n, roff, ntype, kappa):
    """Cluster and column edges of the pair kernel.  Forces, energies and virial are sums of FP64 terms
    rounded once to 2^-40 and 2^-32; the parameters are exact in FP32, so 1e-8 leaves room for the
    Ewald table (3e-10 per pair) and the rounding of sums that cancel."""
    from gpu_recip_b200.direct import CudaPMEDirectForce, EWALD, VDW_NONE, VDW_VSH
    rng = np.random.default_rng(n + ntype)
    x = np.empty((n, 4), np.float32)
    if ntype:   # in the box: wrapping a coordinate in FP32 would move it by up to its last bit (1e-6 A)
        x[:, :3] = np.mod(_lattice()["xyzq"][:, :3], np.float32(24.0))
    else:
        x[:, :3] = rng.random((n, 3)) * np.array(box) * 0.999999
    x[:, 3] = rng.integers(-8, 9, n) / 16.0
    dr = CudaPMEDirectForce()
    dr.setup(*box, kappa, roff, roff - 1.5, 1.0, VDW_VSH if ntype else VDW_NONE, EWALD)
    vp, vt = np.zeros(2), np.zeros(n, np.int32)
    if ntype:
        vp = np.float32(rng.random(ntype * (ntype + 1))).astype(np.float64) * np.tile([1.0e2, 1.0e5], ntype * (ntype + 1) // 2)
        vp = vp.astype(np.float32).astype(np.float64)
        vt = rng.integers(0, ntype, n).astype(np.int32)
        dr.set_vdwparam(vp)
        dr.set_vdwtype(vt)
        vp = np.stack([(6 * vp[0::2].astype(np.float32)).astype(np.float64) / 6,
                       (12 * vp[1::2].astype(np.float32)).astype(np.float64) / 12], 1).reshape(-1)
    xd = cuda.from_numpy(x).cuda()
    stride = ((n + 63) // 64) * 64
    fi, e, vir = _run(cuda, dr, xd, n, stride)
    fo, ev, ee, vo = oracle.direct_force(x.astype(np.float64), np.array(box), kappa, roff, vp, vt,
                                         np.zeros(n + 1, np.int32), np.zeros(0, np.int32))
    f = fi.astype(np.float64) / FORCE_SCALE
    assert np.sqrt(((f - fo) ** 2).sum()) <= 1e-8 * np.sqrt((fo ** 2).sum()) + 1e-9
    assert abs(e["vdw"] - ev) <= 1e-8 * abs(ev) + 1e-6 and abs(e["elec"] - ee) <= 1e-8 * abs(ee) + 1e-6
    assert np.abs(vir - vo).max() <= 1e-7 * np.abs(vo).max() + 1e-6
    fi2, e2, vir2 = _run(cuda, dr, xd, n, stride)      # the forces-only kernel and the same sums again
    fz = cuda.zeros(3 * stride, dtype=cuda.int64, device="cuda")
    dr.calc_force(xd, n, False, False, stride, fz)
    assert np.array_equal(fi, fi2) and e == e2 and np.array_equal(vir, vir2)
    assert np.array_equal(fi, fz.view(3, stride)[:, :n].T.cpu().numpy())
    dr.close()


@pytest.mark.parametrize("ntype", [30, 37, 38, 45, 46, 47, 48, 64, 65, 200])
def test_types_that_no_atom_has_change_nothing(cuda, ntype):
    """The same parameters in a table of 3 types (held as a square in shared memory) and in a larger one, on
    both sides of where the square gives way to the packed triangle: the same forces, energies and virial."""
    from gpu_recip_b200.direct import CudaPMEDirectForce
    d = _lattice()
    n = d["xyzq"].shape[0]
    x = cuda.from_numpy(np.ascontiguousarray(d["xyzq"], dtype=np.float32)).cuda()
    vp = np.zeros(ntype * (ntype + 1), np.float32)
    vp[:12] = np.random.default_rng(4).random(12) * np.tile([1.0e2, 1.0e5], 6)
    out = []
    for m in (3, ntype):
        dr = CudaPMEDirectForce()
        dr.setup(24.0, 24.0, 24.0, 0.35, 9.0, 7.5, 1.0)
        dr.set_vdwparam(vp[:m * (m + 1)])
        dr.set_vdwtype(np.arange(n, dtype=np.int32) % 3)
        f, e, v = _run(cuda, dr, x, n, n)
        g = cuda.zeros(3 * n, dtype=cuda.int64, device="cuda")
        dr.calc_force(x, n, False, False, n, g)
        assert np.array_equal(f, g.view(3, n).T.cpu().numpy())
        out.append((f, e, v))
        dr.close()
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1] and np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("box", [(40.0, 40.0, 40.0), (62.0, 70.0, 55.0)])
def test_breathing_box_needs_no_new_work_space(cuda, box):
    """Edges up to 4% longer than at the first call: calc_force allocates nothing (an allocation ends a
    stream capture) and gives what a new handle gives for that box."""
    from gpu_recip_b200.direct import CudaPMEDirectForce, EWALD, VDW_NONE
    n = int(0.1 * np.prod(box))
    rng = np.random.default_rng(11)
    stream = cuda.cuda.Stream()
    with cuda.cuda.stream(stream):
        x = cuda.from_numpy(np.concatenate([rng.random((n, 3)) * box, rng.normal(0.0, 0.4, (n, 1))], 1).astype(np.float32)).cuda()
        f, g = (cuda.zeros(3 * n, dtype=cuda.int64, device="cuda") for _ in range(2))
        dr = CudaPMEDirectForce(stream)
        dr.setup(*box, 0.33, 9.0, 7.5, 1.0, VDW_NONE, EWALD)
        dr.calc_force(x, n, False, False, n, f)
    stream.synchronize()
    for scale in (1.01, 1.025, 1.04):
        dr.set_box_size(*(scale * b for b in box))
        graph = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(graph, stream=stream):
            dr.calc_force(x, n, False, False, n, f)
        f.zero_()
        g.zero_()
        graph.replay()
        new = CudaPMEDirectForce()
        new.setup(*(scale * b for b in box), 0.33, 9.0, 7.5, 1.0, VDW_NONE, EWALD)
        new.calc_force(x, n, False, False, n, g)
        cuda.cuda.synchronize()
        assert cuda.equal(f, g) and f.abs().max() > 0
        del graph
        new.close()
    dr.close()


def test_handles_of_unlike_tables_in_two_threads(cuda):
    """A handle with 64 vdW types and one with two, each in a thread with its own stream: neither's
    launches depend on the shared memory that the other's tables take."""
    import threading
    from gpu_recip_b200.direct import CudaPMEDirectForce
    d = _lattice()
    n = d["xyzq"].shape[0]
    failed, out = [], {}

    def work(ntype):
        try:
            stream = cuda.cuda.Stream()
            dr = CudaPMEDirectForce(stream)
            dr.setup(24.0, 24.0, 24.0, 0.35, 12.0, 10.0, 1.0)
            dr.set_vdwparam(np.ones(ntype * (ntype + 1), np.float32))
            dr.set_vdwtype(np.arange(n, dtype=np.int32) % ntype)
            with cuda.cuda.stream(stream):
                x = cuda.from_numpy(np.ascontiguousarray(d["xyzq"], dtype=np.float32)).cuda()
                f = cuda.zeros(3 * n, dtype=cuda.int64, device="cuda")
                for _ in range(1500):
                    f.zero_()
                    dr.calc_force(x, n, True, True, n, f)
                stream.synchronize()
                out[ntype] = f.cpu().numpy(), dr
        except Exception as e:   # raised again by the assertion below
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(t,)) for t in (64, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for ntype, (f, dr) in out.items():
        g = cuda.zeros(3 * n, dtype=cuda.int64, device="cuda")
        cuda.cuda.synchronize()
        dr.calc_force(cuda.from_numpy(np.ascontiguousarray(d["xyzq"], dtype=np.float32)).cuda(), n, True, True, n, g)
        cuda.cuda.synchronize()
        assert np.array_equal(f, g.cpu().numpy())
        dr.close()
