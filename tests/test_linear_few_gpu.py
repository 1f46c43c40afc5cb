"""The bfloat16 product of few rows against float64.  Tolerance: the operands are exact, a float32 sum of K products in any order is within
2 K 2^-24 sum |x_i w_i| of the exact one (Higham, Accuracy and Stability of Numerical Algorithms, section 3.1; twice gamma_K, since the
tensor cores may truncate where an addition would round), and a bfloat16 result (eight significant bits) is rounded once more, by at most 2^-8 of itself."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24


def _operands(n, k, m, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(n, k, device=DEV, generator=g).to(torch.bfloat16)
    return x, torch.randn(m, k, device=DEV, generator=g).to(torch.bfloat16)


def _within(out, x, w):
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bound = 2 * x.shape[1] * U * size + (2.0 ** -8 * want.abs() if out.dtype == torch.bfloat16 else 0.0)
    return torch.all((out.double() - want).abs() <= bound)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("n,k,m", [(1, 16, 1), (1, 64, 15), (2, 528, 17), (7, 1024, 16), (8, 2048, 33), (8, 4624, 40), (9, 64, 31), (12, 2064, 100),
                                   (16, 3072, 2400), (17, 80, 16), (24, 2048, 2368), (32, 5632, 48), (32, 1040, 2400)])
def test_linear_few(n, k, m, early, dtype):
    from quanta_b200 import kernels
    x, w = _operands(n, k, m, n * 100 + m)
    out = torch.full((n, m), float("nan"), device=DEV, dtype=dtype)
    torch.cuda.synchronize()                    # the weights are settled
    kernels.linear_few(x, w, out, early=early)
    assert _within(out, x, w)
    for rows in {1, min(n, 8), min(n, 16), n}:  # a row's sums depend neither on the others nor on how many there are
        some = torch.empty((rows, m), device=DEV, dtype=dtype)
        kernels.linear_few(x[:rows].contiguous(), w, some, early=early)
        assert torch.equal(some, out[:rows])


@pytest.mark.parametrize("dtype", [None, torch.float32])
def test_linear_takes_few_rows_and_leaves_the_rest(dtype):
    """Through ``matmul.linear``: rows with and without spare ones, widths and places the kernel does not take, and more rows."""
    from quanta_b200.matmul import empty_rows, linear
    flat = torch.randn(4 * 128 + 8, device=DEV).to(torch.bfloat16)
    pairs = [_operands(n, k, m, n + k) for n, k, m in ((1, 16, 40), (3, 72, 40), (5, 64, 24), (16, 256, 4000), (17, 2048, 4000), (33, 128, 50))]
    pairs.append((flat[8:].view(4, 128), _operands(1, 128, 9, 3)[1]))            # 16 bytes past a 32-byte boundary
    spare = empty_rows(5, 128, dtype=torch.bfloat16, device=DEV)
    spare.copy_(torch.randn(5, 128, device=DEV))
    pairs.append((spare, _operands(1, 128, 70, 4)[1]))
    for x, w in pairs:
        out = linear(x, w, out_dtype=dtype)
        assert out.shape == (x.shape[0], w.shape[0]) and out.dtype == (dtype or torch.bfloat16) and _within(out, x, w)


@pytest.mark.parametrize("k,m", [(3072, 8192), (2048, 11264), (2048, 2048), (768, 3072), (5632, 2048), (72, 300), (16384, 2048)])
def test_a_rows_numbers_do_not_depend_on_the_step(k, m):
    """Large and small matrices, of this kernel and of the library (rows that are no multiple of 16, long ones): a row has the same bits in every
    step of up to 32 rows, and in a larger one it is within the same bound."""
    from quanta_b200.matmul import empty_rows, linear, linear_silu
    x, w = _operands(33, k, m, k + m)
    rows = []
    for n in (1, 7, 8, 9, 16, 17, 31, 32, 33):
        some = empty_rows(n, k, dtype=torch.bfloat16, device=DEV)
        some.copy_(x[:n])
        rows.append((n, linear(some, w, out_dtype=torch.float32), linear_silu(some, w)))
    for n, out, act in rows:
        assert _within(out, x[:n], w)
        if n <= 32:
            assert torch.equal(out, rows[-2][1][:n]), n
            assert (act is None) == (rows[0][2] is None) and (act is None or torch.equal(act, rows[-2][2][:n])), n


def test_what_hangs_on_the_product_stays_with_torch():
    from quanta_b200.matmul import linear
    x, w = _operands(3, 64, 32, 5)
    xg, wg = x.clone().requires_grad_(), torch.nn.Parameter(w.clone())
    linear(xg, wg).float().sum().backward()
    assert xg.grad is not None and wg.grad is not None
    with pytest.raises(RuntimeError):
        linear(x, w[:, :48])
    with pytest.raises(RuntimeError):
        linear(x, w, out_dtype=torch.float16)


def test_infinities_and_nan_stay_in_their_rows():
    from quanta_b200 import kernels
    x, w = _operands(9, 2048, 48, 6)
    x[3, 5], x[4, 7], w[20, 9] = float("inf"), float("nan"), float("inf")
    out = torch.empty((9, 48), device=DEV)
    kernels.linear_few(x, w, out)
    want = x.float() @ w.float().T
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isinf(out), torch.isinf(want))
