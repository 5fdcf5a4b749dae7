"""The engine's host side when an allocation fails, on the CPU.

host_check.cpp compiles engine.cu and batch_host.cu against a fake CUDA runtime in which the k-th
allocation of a call fails. Whatever k is, that call returns an error and the
next one runs on arrays, tables and fluxes of its own. And what a context costs
before it has done much.
"""
import os
import shutil
import subprocess

import pytest

from lcurve_re_b200 import workloads as W

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "host", "host_check.cpp")
EXE = os.path.join(HERE, "host", "_build", "host_check")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def host_check():
    if shutil.which("g++") is None or not os.path.isdir(os.path.join(CUDA, "include")):
        pytest.skip("g++ or the CUDA headers are not available")
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    subprocess.check_call(["g++", "-x", "c++", "-std=c++17", "-O1", "-pthread",
                           "-I" + os.path.join(CUDA, "include"),
                           "-I" + os.path.join(ROOT, "include"), "-o", EXE, SRC])
    return EXE


def _run(exe, mode, a, b):
    blob = bytes(W.model(**dict(dict(nlat1f=20, nlat2f=24), **a)).to_c()) + bytes(W.model(**b).to_c())
    out = subprocess.run([exe, mode], input=blob, capture_output=True, timeout=300)
    assert out.returncode == 0, out.stderr.decode()[-2000:]
    return int(out.stdout.split()[0])


@pytest.mark.parametrize("nlat1,nlat2", [(60, 70), (20, 70), (90, 24)])
def test_ring_tables_after_a_failed_allocation(host_check, nlat1, nlat2):
    """A grid's ring table is kept for its strip count: not past another one's failure."""
    assert _run(host_check, "rings", {}, dict(nlat1f=nlat1, nlat2f=nlat2)) >= 8


@pytest.mark.parametrize("over", [dict(t1=15000.0, t2=3000.0, beam_factor1=1.3),
                                  dict(t1=15000.0, mucrit1=0.2), dict(t2=3500.0, limb2="Poly")])
def test_fluxes_after_a_failed_allocation(host_check, over):
    """The reuse of a model's fluxes ends when another model's call has overwritten them."""
    _run(host_check, "cache", {}, dict(nlat1f=20, nlat2f=24, **over))


def test_points_after_a_failed_allocation(host_check):
    """Points that did not fit are refused, and no call takes the freed ones for them."""
    assert _run(host_check, "data", {}, dict(nlat1f=20, nlat2f=24)) >= 2


def test_pinned_memory_waits_until_it_pays(host_check):
    """Contexts share one pinned block; past it a context of few calls pins nothing, and one of
    many does so once, and undoes it."""
    _run(host_check, "pin", {}, {})


def test_first_calls_make_few_large_allocations(host_check):
    """Each takes a third of a millisecond: per grid of 326,000 faces its points, the state of
    its eclipse candidates, its records and their ranges."""
    assert _run(host_check, "first", dict(nlat1f=506, nlat2f=506), {}) <= 8


@pytest.mark.parametrize("nlat1,nlat2", [(60, 70), (20, 70), (90, 24)])
def test_batches_after_a_failed_allocation(host_check, nlat1, nlat2):
    """Ring tables that a failed layout added to the pool reach the device with the next one."""
    assert _run(host_check, "batch", {}, dict(nlat1f=nlat1, nlat2f=nlat2)) >= 8


def test_batches_after_their_points_moved(host_check):
    """Points that grew and shrank back lie in the same block, their offsets in another: the
    captured graph goes with both."""
    _run(host_check, "moved", {}, {})
