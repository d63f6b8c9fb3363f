"""The GPU.cuh drop-in's host side against a stand-in for the library (dropin_stub.cpp): no GPU needed."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DROPIN = os.path.join(ROOT, "bacterial-classification_gb300", "dropin")


@pytest.fixture(scope="module")
def stub(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("dropin") / "stub")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-DHV_DIM=64", "-I" + DROPIN, "-I" + os.path.join(ROOT, "include"),
                           os.path.join(ROOT, "tests", "dropin_stub.cpp"), os.path.join(DROPIN, "gpu_dropin.cpp"), "-o", exe])
    return lambda limit, status=0: subprocess.run([exe, str(limit), str(status)], capture_output=True, text=True,
                                                  check=True).stdout.split("\n")[:-1]


def test_a_full_card_searches_with_the_least_workspace(stub):
    assert stub(2 << 30) == ["work %d" % (1 << 30), "found 1"]
    assert stub(1 << 20) == ["work 4096", "found 1"]
    assert stub(1 << 10) == ["threw hdc_device_alloc: stub"]


def test_a_search_that_gave_up_is_an_error(stub):
    """The tensor-core search reports a bounded wait that ran out in the status word only, with partial results."""
    assert stub(2 << 30, 103)[-1].startswith("threw ") and "103" in stub(2 << 30, 103)[-1]
