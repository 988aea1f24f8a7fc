"""The choice between the streaming and the tensor-core decode attention, and between key splits, from the measured times that it rests on (no GPU)."""
import pytest

from mary_b200.ops.cuda import stream_split


@pytest.mark.parametrize("units,span,measured", [(256, 1024, 56), (64, 2000, 30), (8, 777, 8), (16, 4000, 30), (16, 8000, 52), (8, 4000, 19), (1, 16000, 52), (4, 8000, 30)])
def test_estimates_are_near_what_was_measured(units, span, measured):
    assert 0.6 * measured < stream_split(units, span)[2] < 1.3 * measured


def test_clusters_of_eight_that_do_not_fit_side_by_side():
    """16 units of 4000 keys of 256 in bf16: 128 CTAs on the 112 SMs that clusters of 8 reach.  The tensor-core kernel takes 15 us + the bytes at 5.3 TB/s."""
    assert stream_split(16, 4000)[2] > 15.0 + 2 * 4000 * 8 * 1024 / 5.3e6


def test_few_long_sequences_and_short_ones():
    """One sequence of 4000 keys: 19 us streamed, 23 on the tensor cores; two of 8000: 52 and 37."""
    assert stream_split(8, 4000)[2] < 15.0 + 4000 * 8 * 1024 / 5.3e6
    assert stream_split(16, 8000)[2] > 15.0 + 2 * 8000 * 8 * 1024 / 5.3e6


def test_splits_are_what_the_kernel_takes():
    for units in (1, 3, 16, 100, 148, 149, 5000):
        for span in (1, 31, 64, 777, 4000, 64000):
            nsplit, warps, t = stream_split(units, span)
            assert nsplit in (1, 2, 4, 8) and warps in (4, 8) and t > 0 and (nsplit == 1 or span >= 32 * nsplit)
