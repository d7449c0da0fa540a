"""The loading and the issuing role of k_comb256's blocks (csrc/comb_roles.cuh),
compiled for the host, with every one of their waits running out in turn: the
role says so, and leaves nothing in flight that would touch the shared or the
tensor memory of the next block."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
OK, WRONG, IN_FLIGHT = 1, 2, 4


@pytest.fixture(scope="module")
def roles(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("roles") / "comb_roles_host.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared",
                           '-DFT_HOST_EMULATION="../../tests/host/ptx_emul.h"', "-o", so,
                           os.path.join(HERE, "host", "comb_roles_host.cpp")])
    return ctypes.CDLL(so)


@pytest.mark.parametrize("steps", [0, 1, 2, 3, 4, 5, 6, 7, 32, 66])
def test_loads(roles, steps):
    assert roles.hr_load(steps, 0) == OK
    before = max(0, steps - 3)  # waits for a free buffer; those at the end cannot be made good
    last = 2 * min(3, steps)
    for fail in range(1, before + 1):
        assert roles.hr_load(steps, fail) == 0, fail
    for fail in range(before + 1, before + last + 1):
        assert roles.hr_load(steps, fail) in (0, IN_FLIGHT), fail
    assert roles.hr_load(steps, before + last + 1) == OK


@pytest.mark.parametrize("steps", [0, 1, 2, 3, 4, 5, 6, 7, 32, 66])
def test_products(roles, steps):
    assert roles.hr_issue(steps, 0) == OK
    for fail in range(1, 2 * steps + 1):
        assert roles.hr_issue(steps, fail) == 0, fail
    if steps:
        assert roles.hr_issue(steps, 2 * steps + 1) == IN_FLIGHT  # the wait for the last product itself
    assert roles.hr_issue(steps, 2 * steps + 2) == OK
