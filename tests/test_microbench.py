"""The matvec microbenchmark times the kernel that it names."""
import pytest

from camelid_b200 import microbench


@pytest.mark.parametrize("kernel, batch, choice", [("staged", 1, 16), ("staged", 32, 16), ("rows", 3, 0), ("rows", 32, 0), ("tcgen05", 9, 32), ("direct", 4, 1),
                                                   ("mma", 32, 4)])
def test_choice_of_a_kernel(kernel, batch, choice):
    assert microbench.kernel_choice(kernel, batch) == choice


@pytest.mark.parametrize("kernel, batch", [("rows", 1), ("rows", 2), ("rows", 33), ("mma", 33)])
def test_a_batch_that_another_kernel_would_serve_is_refused(kernel, batch):
    with pytest.raises(ValueError):
        microbench.kernel_choice(kernel, batch)
