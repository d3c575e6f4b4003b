"""The forms of the 32-bit product: tiles with two chains an instruction and whole stages of few tokens give every output the one
chain of multiply-adds in order of k that the other forms give it, at the edges of tiles and stages."""

import pytest
import torch

from tests.test_gpu_kernels import DEV, F, rand

pytestmark = pytest.mark.gpu


def check(x, w, out_dtype):
    got = F().linear_f32(x, w, out_dtype)
    K = x.shape[1]
    want = x.double() @ w.double().T
    bound = K * 2.0**-24 * (x.double().abs() @ w.double().abs().T) + (0 if out_dtype == torch.float32 else 2.0**-8) * want.abs()
    assert ((got.double() - want).abs() <= bound).all()
    # the same rows one at a time, over rows of W that neither whole groups of eight nor whole tiles hold
    some = sorted({0, x.shape[0] // 2, x.shape[0] - 1})
    n = min(w.shape[0], 1003)
    for m in some:
        assert torch.equal(F().linear_f32(x[m:m + 1], w[-n:].contiguous(), out_dtype)[0], got[m, -n:]), f"row {m}"


@pytest.mark.parametrize("a_dtype,out_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("M,N,K", [(65, 17024, 16), (64, 33280, 17), (127, 17024, 40), (130, 16640, 100), (200, 8448, 129)])
def test_tiles_of_pairs(M, N, K, a_dtype, out_dtype):
    check(rand(M, K, seed=M).to(a_dtype).to(DEV), rand(N, K, seed=N).float().to(DEV), out_dtype)


@pytest.mark.parametrize("a_dtype,out_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("M", [1, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(8, 128), (1024, 640), (2368, 768), (1032, 1152)])
def test_whole_stages_of_few_tokens(M, N, K, a_dtype, out_dtype):
    check(rand(M, K, seed=M + 7).to(a_dtype).to(DEV), rand(N, K, seed=N).float().to(DEV), out_dtype)
