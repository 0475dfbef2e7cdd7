"""Which product runs, asked where there is no device to answer."""
import pytest
import torch


@pytest.mark.skipif(torch.cuda.is_available(), reason="the question has an answer here")
def test_an_answer_that_does_not_come_is_an_error_each_time():
    """How many clusters fit is asked of the device; without one the choice is not made, and nothing is remembered."""
    from dispec_b200.ops import library, tuning
    for _ in range(2):
        with pytest.raises(library.KernelError, match="how many clusters"):
            tuning._few_rows_faster(300, 1536, 8960, 148)
