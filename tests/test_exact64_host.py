"""The FP64 kernels' short forms (falcon_gb300/csrc/exact64.cuh) compiled for the CPU:
each gives the bits of the reference's expression."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _compile(tmp, *flags):
    exe = str(tmp / "exact64_host")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", *flags, os.path.join(HERE, "exact64_host.cpp"), "-o", exe],
                   check=True)
    return exe


def _run(*cmd):
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return _compile(tmp_path_factory.mktemp("exact64"))


@pytest.mark.parametrize("form", ["slopes", "fluxes", "quotients", "limiters", "ghosts"])
def test_short_form_is_the_expression(exe, form):
    _run(exe, form, "2000000", "7")


@pytest.mark.parametrize("form,count", [("far_ghost_case", 1), ("far_ghosts", 5000000)])
def test_ghost_with_large_corners_off_along_several_axes(exe, form, count):
    """Corners off along several axes weigh up to 2^-80, and those that the reference adds
    before the large corner take part in its rounding."""
    _run(exe, form, str(count), "11")


@pytest.mark.parametrize("form", ["slopes", "fluxes", "quotients", "limiters", "ghosts"])
def test_short_forms_have_no_undefined_arithmetic(tmp_path, form):
    """Signed overflow and shifts of negative values end the program."""
    exe = _compile(tmp_path, "-fsanitize=undefined", "-fsanitize-undefined-trap-on-error")
    _run(exe, form, "200000", "3")
