"""The direct-space engine's host-side choices (csrc/pme_direct_plan.h) and exact sums
(csrc/pme_direct_math.h), compiled with the undefined behaviour sanitizer and checked without a GPU."""
import itertools
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "direct_plan")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined,float-cast-overflow", "-fno-sanitize-recover=all",
                    "-I", os.path.join(ROOT, "gpu_recip_b200", "csrc"), os.path.join(ROOT, "tests", "cpp", "direct_plan.cpp"),
                    "-o", exe], check=True)

    def run(what, lines):
        text = "".join(" ".join(repr(v) for v in line) + "\n" for line in lines)
        r = subprocess.run([exe, what], input=text, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        return [line.split() for line in r.stdout.splitlines()]
    return run


def test_columns_stay_within_their_tables(plan):
    """Any accepted box and cutoff (at most half the shortest edge): indices that fit, no offset that
    wraps twice, no pair within the cutoff beyond the columns in reach."""
    edges = [0.5, 18.0, 62.1, 500.0, 1.0e4, 1.0e6]
    cases = [(*b, f * min(b), n) for b in itertools.product(edges, repeat=3)
             for f in (0.5, 0.49999, 0.145, 0.02, 2e-5, 1e-9, 1e-30) for n in (1, 24000, 10 ** 6, 10 ** 9)]
    out = np.array(plan("columns", cases), float)
    box, roff = np.array([c[:3] for c in cases]), np.array([c[3] for c in cases])
    nx, ncol, reach, cells = out[:, 0], out[:, 1:3], out[:, 3:4], out[:, 4]
    assert (nx >= 1).all() and (nx <= 1024).all() and (ncol.prod(1) <= 2 ** 22).all()
    assert (cells == ncol.prod(1) * (nx + 1)).all() and (cells <= 16.0e6 + 2 ** 22).all()
    assert (reach >= 1).all() and (reach <= 4).all() and (ncol >= reach).all()
    assert (reach * box[:, 1:] / ncol >= roff[:, None] * 1.00001 * (1 - 1e-12)).all()


def test_columns_of_usual_systems(plan):
    """24,000 and 192,000 atoms of water at 9 A, and a cutoff of half the box."""
    out = plan("columns", [(62.1, 62.1, 62.1, 9.0, 24000), (124.2, 124.2, 124.2, 9.0, 192000), (18.0, 18.0, 18.0, 9.0, 600)])
    assert [[int(v) for v in row[:4]] for row in out] == [[62, 13, 13, 2], [124, 27, 27, 2], [18, 3, 3, 2]]


def test_square_of_types_keeps_the_ctas(plan):
    """228 KB per SM, cutoffs of 9 and 12 A, forces only and with energies: the square of types takes what
    five CTAs leave, and no more."""
    tables = [171 * 48, 171 * 96, 199 * 48, 199 * 96]
    most = [int(row[0]) for row in plan("types", [(t, 228 * 1024) for t in tables])]
    assert most == [int(((228 * 1024) // 5 - 1024 - 19072 - t) // 8) ** 0.5 // 1 for t in tables]
    assert most[0] > 40 and most[0] < 48 and most[1] > 32 and most[1] < 40
    # a long cutoff (60 A, with energies: 345 intervals) leaves fewer CTAs anyway: a few types cost none of them
    assert 5 * (19072 + 1024 + 345 * 96) > 228 * 1024
    assert int(plan("types", [(345 * 96, 228 * 1024)])[0][0]) >= 25


@pytest.mark.parametrize("roff", [9.0, 12.0, 20.0])
@pytest.mark.parametrize("kappa", [0.0, 0.25, 0.32, 0.45, 1.0])
def test_ewald_table_errors(plan, kappa, roff):
    """The table against erfc and exp in FP64, over pairs uniform in volume from 1.5 A to the cutoff: a
    hundredth of the largest errors of a cubic Hermite table of 4,096 even intervals (3.5e-10 of F r and
    6e-11 of E at 9 A), and of its rms errors (6e-12 and 1e-12)."""
    from scipy.special import erfc
    c = np.array(plan("ewald", [(kappa, roff)]), float)
    assert c.shape == (np.searchsorted([(32 + i % 32) * 2.0 ** (i // 32) / 16 for i in range(512)], roff ** 2, side="right"), 12)
    rng = np.random.default_rng(9)
    r = np.sort(np.cbrt(rng.uniform(1.5 ** 3, roff ** 3, 200000)))
    s = r * r
    m, e = np.frexp(s)                                  # s = 2 m 2^(e-1), 2 m in [1, 2)
    i = 32 * (e - 2) + np.floor((2 * m - 1) * 32).astype(int)
    t = s - (2.0 ** (e - 1) * (1 + (np.floor((2 * m - 1) * 32) + 0.5) / 32))
    p = c[i]
    F, E = (sum(p[:, o + k] * t ** k for k in range(6)) for o in (0, 6))
    E0 = erfc(kappa * r) / r
    F0 = (-2 / np.sqrt(np.pi) * kappa * np.exp(-kappa ** 2 * s) - E0) / s
    dF, dE = np.abs(F - F0) * r, np.abs(E - E0)
    assert dF.max() <= 3.5e-12 and dE.max() <= 6e-13
    assert np.sqrt((dF ** 2).mean()) <= 6e-14 and np.sqrt((dE ** 2).mean()) <= 1e-14


def test_room_for_a_longer_box(plan):
    """Edges up to 5% longer take no more cells than were made room for, whatever the box and density."""
    rng = np.random.default_rng(5)
    cases = []
    for _ in range(300):
        box = np.exp(rng.uniform(np.log(19.0), np.log(300.0), 3))
        n = int(np.exp(rng.uniform(np.log(1e-5), np.log(0.2))) * box.prod()) + 1
        cases += [(*(s * box).tolist(), 9.0, n) for s in (1.0, 1.003, 1.01, 1.02, 1.03, 1.04, 1.0499)]
    out = np.array(plan("columns", cases), float).reshape(-1, 7, 7)
    room, cells, columns = out[:, 0, 5], out[:, :, 4], out[:, :, 1] * out[:, :, 2]
    assert (cells <= room[:, None]).all() and (columns <= out[:, 0, 6][:, None]).all()


def test_force_sums_are_exact(plan):
    """Sums of terms rounded to 2^-40: exact at every step, in defined arithmetic, small and large terms."""
    rng = np.random.default_rng(3)
    v = np.concatenate([rng.normal(0.0, 300.0, 400).clip(-1023.9, 1023.9), [1023.999, -1023.999, 0.0, -0.0, 0.5 ** 41, -0.5 ** 41],
                        rng.normal(0.0, 4000.0, 200)])
    rng.shuffle(v)
    got = [int(row[0]) for row in plan("sums", [(float(x),) for x in v])]
    want = np.cumsum([int(np.rint(x * 2.0 ** 40)) for x in v], dtype=object)
    assert got == list(want)
