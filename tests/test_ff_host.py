"""The solver's sums of float-float products lose no more than float-float additions do."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ff") / "ff_host")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", os.path.join(HERE, "ff_host.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("terms", [7, 32])
@pytest.mark.parametrize("kind", ["laplacian", "positive", "binades"])
def test_sums_of_products_keep_the_precision_of_float_float_additions(exe, terms, kind):
    k = ["laplacian", "positive", "binades"].index(kind)
    rms, worst, ref_rms, ref_worst = map(float, subprocess.run([exe, str(terms), str(k)], check=True, capture_output=True,
                                                               text=True).stdout.split())
    print("rms %.3f largest %.3f, additions %.3f %.3f (2^-48)" % (rms, worst, ref_rms, ref_worst))
    assert rms <= ref_rms and worst <= ref_worst
