"""Which kernels a call launched is read from the profiler's activity records, which may miss some
(a region of microseconds at the window's edge): an incomplete list must not decide anything."""
import pytest

from tests.helpers import launched_back_projectors, require_records

A, B = "void etcu::bp_block_kernel<256, false, 0>(etcu::BpBlockArgs)", "void etcu::bp_parallel_kernel<false, 0, 0>()"
FP = "void etcu::forward_project_kernel<float, false, 1>(etcu::FpArgs)"


def _records(*lists):
    seen, it = [], iter(lists)

    def record(run, pad):
        seen.append(pad)
        run()
        return next(it)
    return seen, record


def test_incomplete_records_are_taken_again():
    runs = []
    pads, record = _records([], [FP], [FP, A, "Memcpy HtoD"])
    assert launched_back_projectors(lambda: runs.append(1), 1, record) == {A}
    assert len(runs) == 3 and pads == sorted(pads) and pads[0] > 0
    _, record = _records([FP, A], [FP, FP, A, B])
    assert launched_back_projectors(lambda: None, 2, record) == {A, B}


def test_records_that_stay_incomplete_decide_nothing():
    _, record = _records([FP], [FP, A], [A], [])
    names = launched_back_projectors(lambda: None, 2, record)
    assert names is None
    require_records({A}, {B})
    with pytest.raises(pytest.skip.Exception):
        require_records({A}, names)
