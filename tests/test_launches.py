"""Which kernels a call launches, and what is left of a call whose launch is refused: on the CPU, with a stand-in for the CUDA runtime."""
import pytest

from tests import launches


def test_prefill_in_two_parts_covers_every_slice():
    rc, got = launches.prefill(16, 32, 8192)
    assert rc == 0 and [g[1:] for g in got] == [(888, 64, False), (136, 128, True)]
    rc, got = launches.prefill(16, 32, 255)
    assert rc == 0 and [g[1:] for g in got] == [(1024, 64, False)]


@pytest.mark.parametrize("bits", [4, 2])
def test_second_part_refused_beside_the_first_follows_it(bits):
    """A refused launch leaves no prefill half written."""
    rc, got = launches.prefill(16, 32, 8192, bits, fail=[("cudaLaunchKernelExC", 1)])
    assert rc == 0 and [g[1:] for g in got] == [(888, 64, False), (136, 128, False)]
    rc, got = launches.prefill(16, 32, 8192, bits)      # and no error stays behind for the next call
    assert rc == 0 and len(got) == 2


@pytest.mark.parametrize("function", ["cudaFuncGetAttributes", "cudaLaunchKernel"])
def test_refused_before_the_first_part(function):
    rc, got = launches.prefill(16, 32, 8192, fail=[(function, 1)])
    assert rc != 0 and got == []
    rc, got = launches.prefill(16, 32, 8192)
    assert rc == 0 and len(got) == 2
