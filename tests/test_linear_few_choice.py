"""Which bfloat16 products of few rows the framework's own kernel takes: the matrix decides, not the number of rows."""
from __future__ import annotations

from quanta_b200 import kernels

SIZES = [(k, n) for k in (16, 48, 64, 72, 768, 2048, 3072, 5632, 6144, 8192, 8208, 12288, 12304, 16384) for n in (1, 16, 2048, 2368, 2369, 8192, 200064)]


def test_every_number_of_rows_has_the_same_kernel():
    most = kernels.LINEAR_FEW_MAX
    for k, n in SIZES:
        assert {kernels.linear_few_takes(rows, k, n) for rows in range(1, most + 1)} == {kernels.linear_few_takes(1, k, n)}, (k, n)
        assert not kernels.linear_few_takes(0, k, n) and not kernels.linear_few_takes(most + 1, k, n)


def test_the_sizes_that_it_takes():
    taken = {(k, n) for k, n in SIZES if kernels.linear_few_takes(8, k, n)}
    assert {(3072, 8192), (2048, 200064), (8192, 200064), (12288, 2368), (64, 1)} <= taken
    assert not {(48, 16), (72, 2048), (8208, 2369), (12288, 8192), (12304, 2048)} & taken
