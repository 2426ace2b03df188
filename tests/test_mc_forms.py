"""The MohrCoulomb update's two forms (mpm_math.cuh, mpm_return.cuh) on the host, linked into one
program (mc_forms.cpp): the form of the mixed path against 80-bit arithmetic and, over whole
updates, against the form that the FP64 path takes.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mpm_b200", "csrc")


@pytest.fixture(scope="module")
def forms(tmp_path_factory):
    d = tmp_path_factory.mktemp("forms")
    objs = []
    for name, flags in (("written", []), ("reciprocal", ["-DMPM_MC_RECIPROCALS"])):
        objs.append(str(d / (name + ".o")))
        subprocess.check_call(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", CSRC] + flags +
                              ["-c", os.path.join(HERE, "mc_forms.cpp"), "-o", objs[-1]])
    exe = str(d / "forms")
    subprocess.check_call(["g++"] + objs + ["-o", exe])
    return {r[0]: [float(x) for x in r[1:]] for r in map(str.split, subprocess.check_output([exe], text=True).splitlines())}


def test_each_form_keeps_its_own_definitions(forms):
    """The forms round differently, so equal bits everywhere would mean that the linker merged them."""
    assert forms["same_bits"][0] < 2000


def test_lode_angle_from_the_triple_angle_equation(forms):
    """sin, cos and the angle for cos 3 theta in [-1, 1] and up to both ends of it: the last correction
    and what follows are at most eight roundings each, and eight more for the angle."""
    sn, cs, th = forms["lode"]
    assert sn < 8 * 2.0 ** -53 and cs < 8 * 2.0 ** -53 and th < 16 * 2.0 ** -53


def test_single_evaluations(forms):
    """Yield functions, dF/dsigma, dP/dsigma, dP/dq, softening and Lode angle within 16 roundings of 80
    bits, each of the size that the invariants carry (mc_forms.cpp); shear, tensile and softening points."""
    assert all(n > 1000 for n in forms["evals"])
    assert max(forms["eval_errors"]) < 16, forms["eval_errors"]


def test_whole_updates(forms):
    """Random updates, one in seventeen from an exact triaxial corner: the same yield states and numbers
    of corrections, stresses on or inside the yield surface (to the update's tolerance of 0.1), and 99 %
    of the stresses within 1e-13: an update is a few corrections of some hundred roundings each."""
    n, finite, counts, yields, corrections, shear, tensile, off_surface = forms["returns"]
    assert shear > 1000 and tensile > 1000 and corrections > 5000
    assert finite == yields == n and off_surface == 0
    assert counts >= 0.999 * n  # a correction more where the tolerance is met within a rounding
    assert forms["stress"][1] < 1e-13
