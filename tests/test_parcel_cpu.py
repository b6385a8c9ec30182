"""The depth-first kernel's parcel protocol (csrc/cp_parcel.cuh), built for the host."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "circlepacking_b200", "csrc")
SLOTS, TAKEN = 1 << 12, 0xFF


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("parcel") / "libparcel.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-shared", "-fPIC", "-I" + CSRC,
                    os.path.join(HERE, "parcel_host.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.p_claim.argtypes = [ctypes.c_void_p, ctypes.c_ulonglong, ctypes.c_uint, ctypes.c_uint]
    L.p_ready.argtypes = [ctypes.c_ulonglong, ctypes.c_ulonglong, ctypes.c_uint]
    L.p_left.argtypes = [ctypes.c_ulonglong, ctypes.c_ulonglong]
    L.p_epochs.argtypes = [ctypes.c_long, ctypes.c_int]
    L.p_epochs.restype = ctypes.c_long
    L.p_stress.restype = L.p_hand_over.restype = ctypes.c_long
    return L


@pytest.mark.parametrize("epoch", [1, 5, (1 << 24) - 1])
def test_one_giver_per_slot(host, epoch):
    """Parcels d, d + slots and d + 2 slots want one slot: a giver is refused from the moment another one
    may write, before anything is published, until the parcel has been taken."""
    old = (epoch - 1) << 40 | 3 << 8 | TAKEN  # another launch's flag
    flag = ctypes.c_ulonglong(old)
    claim = lambda d: bool(host.p_claim(ctypes.byref(flag), epoch, d, SLOTS))
    assert claim(3)
    assert not claim(3 + SLOTS)  # the first one has published nothing yet
    flag.value = epoch << 40 | 3 << 8 | 32
    assert not claim(3 + SLOTS)  # ready
    flag.value |= TAKEN
    assert claim(3 + 2 * SLOTS)
    assert flag.value == epoch << 40 | (3 + 2 * SLOTS) << 8
    assert not claim(3 + SLOTS)  # claimed
    flag.value |= TAKEN
    assert claim(3 + SLOTS)


def test_claims_exclude_each_other(host):
    assert host.p_stress(8, 3, 20000) == 0


def test_slot_is_passed_on_by_the_whole_warp(host):
    """The flag moves when every lane has read or written, not when the first one has."""
    assert host.p_hand_over(200) == 0


@pytest.mark.parametrize("n", [0, 1, 32, TAKEN])
def test_only_parents_that_are_there_are_read(host, n):
    """A taken parcel is none, neither for the ticket that once waited for it (epochs come back) nor as a left-over."""
    e, d = 9, 70000
    there = n if n != TAKEN else 0
    for epoch in (e, e + (1 << 24)):
        assert host.p_ready(e << 40 | d << 8 | n, epoch, d) == there
        assert host.p_left(e << 40 | d << 8 | n, epoch) == there
    assert host.p_ready(e << 40 | d << 8 | n, e, d + SLOTS) == host.p_ready(e << 40 | d << 8 | n, e + 1, d) == 0
    assert host.p_left(e << 40 | d << 8 | n, e + 1) == 0


@pytest.mark.parametrize("launches", [1, 3, 1 << 20])
def test_epochs_do_not_come_back_over_uncleared_flags(host, launches):
    assert host.p_epochs((1 << 25) // launches + 3, launches) == 0
