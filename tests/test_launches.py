"""Which kernels a call launches, and what is left of a call whose launch is refused: on the CPU, with a stand-in for the CUDA runtime."""
import pytest

from adkv_b200 import _lib
from tests import launches, test_gpu_prefill_parts, test_gpu_segments, test_gpu_tensor_step, test_gpu_tile_edges
from tests.util import SMAX, SMIN, WIDE

USUAL = (SMIN, SMAX)


def test_prefill_in_two_parts_covers_every_slice():
    rc, got = launches.prefill(16, 32, 8192)
    assert rc == 0 and [g[1:] for g in got] == [(888, 64, False), (136, 128, True)]
    rc, got = launches.prefill(16, 32, 255)
    assert rc == 0 and [g[1:] for g in got] == [(1024, 64, False)]


@pytest.mark.parametrize("slices,T,bits,split", [(592, 4000, 4, 0), (594, 256, 4, 592), (594, 255, 4, 0), (740, 256, 4, 592), (742, 4000, 4, 0),
                                                 (740, 2047, 2, 0), (740, 2048, 2, 592), (890, 383, 2, 0), (890, 384, 2, 888), (1186, 255, 2, 0),
                                                 (1186, 256, 2, 1184), (1628, 256, 4, 1480), (1778, 4000, 4, 0), (446, 4000, 4, 0)])
def test_lines_of_the_second_part(slices, T, bits, split):
    rc, got = launches.prefill(slices // 2, 1, T, bits)
    assert rc == 0 and [g[1] for g in got] == ([split, slices - split] if split else [slices])


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


# query heads per KV head, bits, streams: fewest tokens of the tensor cores' kernel (None: never)
LINES = [(1, 4, 1, 32), (1, 4, 148, 32), (1, 4, 149, 64), (1, 4, 296, 64), (1, 4, 297, 256), (1, 2, 297, 128), (1, 4, 444, 256), (1, 4, 445, None),
         (2, 4, 148, 32), (2, 2, 296, 64), (2, 4, 297, 100), (2, 4, 445, 256), (2, 2, 740, 256), (2, 4, 741, None),
         (4, 4, 148, 32), (4, 2, 297, 100), (4, 4, 445, 128), (4, 2, 740, 128), (4, 4, 741, 256), (4, 4, 1184, 256), (4, 4, 1185, 512),
         (4, 4, 2368, 512), (4, 4, 2369, None), (8, 4, 64, None)]


@pytest.mark.parametrize("G,bits,streams,fewest", LINES)
def test_lines_of_the_tensor_cores(G, bits, streams, fewest):
    for T in (31, 32, 63, 64, 99, 100, 127, 128, 255, 256, 511, 512, 600):
        kernel, ctas = launches.decode(bits, G, streams, 1, T, USUAL)
        assert ctas == streams and (kernel == "tensor") == (fewest is not None and T >= fewest), (T, kernel)


# the same for device-side lengths, by what the cache can hold
@pytest.mark.parametrize("G,streams,fewest", [(1, 148, 128), (1, 149, None), (2, 149, 128), (2, 296, 128), (2, 297, 512), (2, 592, 512), (2, 593, None),
                                              (4, 296, 128), (4, 297, 512), (4, 740, 512), (4, 741, None)])
def test_lines_with_device_side_lengths(G, streams, fewest):
    for words in (15, 16, 17, 63, 64, 65, 80):      # one token less than the words hold
        kernel, _ = launches.decode_varlen(4, G, streams, 1, 8 * words, USUAL)
        assert (kernel == "tensor") == (fewest is not None and 8 * words - 1 >= fewest), (words, kernel)


def test_line_to_token_segments():
    for T, kernel in ((127, "tensor"), (700, "tensor"), (701, "segments"), (4000, "segments")):
        assert launches.decode(2, 1, 148, 1, T, USUAL)[0] == kernel
        assert launches.decode_ckpt(2, 1, 8, 1, T, 1024, USUAL)[0] == "tensor"
    assert launches.decode(2, 1, 149, 1, 4000, USUAL)[0] == "tensor"
    assert launches.decode(4, 1, 148, 1, 4000, USUAL)[0] == launches.decode(2, 2, 148, 1, 4000, USUAL)[0] == "tensor"


@pytest.mark.parametrize("bounds,takes", [((SMIN, SMAX), True), (WIDE, False), ((2.0 ** -7, 64.0), True), ((2.0 ** -7, 64.01), False), ((4.0, 32768.0), True),
                                          ((4.0, 32769.0), False), ((1.0, float("inf")), False), ((1.0, float("nan")), False),
                                          ((float("nan"), 1.0), False), ((0.0, 1.0), False), ((1e-9, 8e-5), True), ((1e-9, 9e-9), False),
                                          ((0.0, 0.0), False), ((1.0, 0.5), True)])
def test_scale_bounds_of_the_tensor_cores(bounds, takes):
    """Up to 2 ** 13 apart, counted from the quantiser's eps on, scale_max from there to 32768."""
    for G, bits in ((1, 4), (4, 2)):
        assert (launches.decode(bits, G, 8, 8, 500, bounds)[0] == "tensor") == takes
        assert (launches.decode_ckpt(bits, G, 2, 8, 500, 256, bounds)[0] == "tensor") == takes
        assert (launches.decode_varlen(bits, G, 8, 8, 500, bounds)[0] == "tensor") == takes


def test_flags_and_states_of_the_tensor_cores():
    split, no_split = _lib.FLAG_SPLIT_CHANNELS, _lib.FLAG_NO_SPLIT_CHANNELS
    assert launches.decode(4, 1, 8, 8, 500, USUAL, flags=launches.FAST | split)[0] == "narrow"
    assert launches.decode(4, 1, 8, 8, 500, USUAL, flags=launches.FAST | no_split)[0] == "whole"
    assert launches.decode(4, 1, 8, 8, 500, USUAL, flags=0)[0] == "narrow"
    assert launches.decode(4, 1, 8, 8, 500, USUAL, tails=False)[0] == "narrow"
    assert launches.decode_ckpt(4, 1, 8, 8, 500, 256, USUAL, flags=0)[0] == "split"
    assert launches.decode_ckpt(4, 1, 8, 8, 500, 256, USUAL, flags=launches.FAST | _lib.FLAG_SELFTEST_MUTE_K)[0] == "tensor"


def test_gpu_tests_reach_the_kernels_they_name():
    for B, Hq, Hkv, T, bits in test_gpu_segments.SHAPES:
        kernel, _ = launches.decode(bits, Hq // Hkv, B, Hkv, T, WIDE)
        assert kernel == ("segments" if T >= 128 else "narrow")
        kernel, _ = launches.decode(bits, Hq // Hkv, B, Hkv, T, USUAL)
        assert kernel == ("narrow" if T < 32 else "segments" if T == 777 else "tensor")
    for bits, G, T in test_gpu_tile_edges.SEGMENTS:
        assert launches.decode(bits, G, 2, 2, T, WIDE)[0] == "segments"
    for bounds, kernel in ((USUAL, "tensor"), (WIDE, "segments")):
        assert launches.decode_varlen(4, 2, 3, 2, 641, bounds)[0] == launches.decode_varlen(2, 4, 11, 2, 700, bounds)[0] == kernel
    assert launches.decode(4, 1, 1, 2, 700, (0.0, 4.0))[0] == "segments"
    for B, Hkv, G, bits, room in test_gpu_tensor_step.RAGGED:
        assert launches.decode_varlen(bits, G, B, Hkv, room, USUAL) == ("tensor", B * Hkv)
    two = [len(launches.prefill(B, H, T - start, bits)[1]) == 2 for B, H, T, bits, interval, start in test_gpu_prefill_parts.SHAPES]
    assert two == [True, False, True, True, False, True, False, True, True]


def test_smoke_run_reaches_the_default_kernels():
    assert launches.decode(4, 2, 2, 2, 260, USUAL)[0] == "tensor"
    assert len(launches.prefill(298, 2, 260)[1]) == 2


@pytest.mark.parametrize("step", [lambda **kw: launches.decode(4, 1, 8, 8, 500, USUAL, **kw), lambda **kw: launches.decode(4, 1, 8, 8, 500, WIDE, **kw),
                                  lambda **kw: launches.decode_ckpt(4, 1, 8, 8, 500, 256, USUAL, **kw)], ids=["tensor", "segments", "ckpt"])
@pytest.mark.parametrize("function", ["cudaFuncSetAttribute", "cudaLaunchKernel"])
def test_error_of_a_refused_step_is_its_own(step, function):
    """The call reports it, launches nothing, and the next call does not find it."""
    rc, got = step(fail=[(function, 1)])
    assert rc == 701 and got == []
    assert launches.library().fake_last_error() == 0


def test_error_before_a_static_step_is_its_own():
    rc, got = launches.decode_static(4, 1, 8, 8, 500, 256, USUAL, fail=[("cudaGetDevice", 1)])
    assert rc == 701 and got == [] and launches.library().fake_last_error() == 0
    assert launches.decode_static(4, 1, 8, 8, 500, 256, USUAL)[0] == "tensor"


@pytest.mark.parametrize("T", [500, 4000])      # the merge of few segments, and the other
def test_merge_refused_beside_the_segments_follows_them(T):
    rc, got = launches.decode_ckpt(4, 1, 8, 8, T, 256, USUAL, fail=[("cudaLaunchKernelExC", 1)])
    assert rc == 0 and "merge" in got[1][0] and not got[1][3]
    assert launches.library().fake_last_error() == 0


def test_error_of_a_refused_merge_is_its_own():
    rc, got = launches.decode_ckpt(4, 1, 8, 8, 500, 256, USUAL, fail=[("cudaLaunchKernelExC", 1), ("cudaLaunchKernel", 2)])
    assert rc == 701 and len(got) == 1
    assert launches.library().fake_last_error() == 0
