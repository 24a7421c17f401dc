"""The arithmetic that the kernels' fast forms rest on, and those forms themselves, on the device
(tests/cpp/device_forms_check.cu, compiled here against the engine's library): quotients, reciprocals and roots
correctly rounded as / and sqrt are (Markstein 1990), the force, value and expansions of the orbits, angles
and searches against the node form and evalPowerLaw."""
import os
import subprocess

import pytest

from conftest import ROOT, GOLDEN

pytestmark = pytest.mark.gpu

LIBDIR = os.path.join(ROOT, "agama_b200", "_lib")
COEFS = ["cfg1", "cfg2", "cfg3", "cfg4", "cfg5"]


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    from agama_b200 import build
    exe = str(tmp_path_factory.mktemp("forms") / "device_forms_check")
    r = subprocess.run([build.NVCC, os.path.join(ROOT, "tests", "cpp", "device_forms_check.cu"), "-o", exe, "-L" + LIBDIR,
                        "-lagama_b200", "-lcudart", "-Xlinker", "-rpath=" + LIBDIR] + build.COMMON + build.CUDA_FLAGS,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe] + [os.path.join(GOLDEN, c + ".coef") for c in COEFS], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    out = {}
    for line in r.stdout.splitlines():
        what, name, differ, most = line.split()
        out[what, name] = int(differ), float(most)
    return out


@pytest.mark.parametrize("exponents", [0, 2, 60, 300])
def test_arithmetic(results, exponents):
    of = {name: v for (what, name), v in results.items() if what == "arithmetic%d" % exponents}
    # correctly rounded, also the quotient by the one kind of divisor (a fraction of ones alone) whose
    # reciprocal the step may leave one unit off
    for name in ("reciprocal", "quotient", "quotient_ones", "root"):
        assert of[name][0] == 0, name
    # within one unit; the root's factors are both rounded, and so is the value 1 / sqrt it is compared with
    for name, units in (("reciprocal_ones", 1), ("rcp", 1), ("normal_quotient", 1), ("rsqrt", 2), ("normal_root", 2)):
        assert of[name][1] <= units, name


@pytest.mark.parametrize("k", range(len(COEFS)))
def test_forms(results, k):
    of = {name: v for (what, name), v in results.items() if what == "forms%d" % (k + 1)}
    # the same operations with other contractions: some tens of roundings of terms of the scale of the sum
    for name in ("force", "value", "axis", "axis_slope"):
        assert of[name][1] <= 64, name
    # the two forms of a Cartesian point round r^2 by themselves: config 2's outer expansion has the
    # conditioning that test_potential_gpu allows for beyond the grid (1e-11)
    assert of["terms"][1] <= (1e-11 * 2 ** 52 if COEFS[k] == "cfg2" else 64)
    # other recurrences of the Legendre functions (their rounding errors grow as l^2)
    for name in ("branch", "branch_slope"):
        assert of[name][1] <= 1000, name
