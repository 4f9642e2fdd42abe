"""The held-out perplexity of more pairs than every block takes in one chunk
(1,048,576 for rows of a warp, 4,194,304 for shorter ones is the limit), through
ammsb_perplexity_noalloc: each average and the result against the plain
expression in FP64, within the 1e-5 of test_gpu_parity."""
import ctypes

import pytest

from mcmc_for_ammsb_gb300 import _native

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,bf16,pairs", [(256, True, 1048577), (128, False, 2200001), (40, False, 4194304),
                                          (1024, True, 1100000)])
def test_perplexity_of_several_chunks_a_block(native_lib, K, bf16, pairs):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    gen = torch.Generator(device="cuda").manual_seed(pairs)
    n, eps = 300, 1e-7
    pi = torch.rand(n, K, device="cuda", generator=gen) + 0.01
    pi = (pi / pi.sum(1, keepdim=True)).to(torch.bfloat16 if bf16 else torch.float32)
    beta = torch.rand(K, device="cuda", generator=gen)
    a, b = (torch.randint(n, (pairs,), device="cuda", generator=gen, dtype=torch.int32) for _ in range(2))
    y = (torch.rand(pairs, device="cuda", generator=gen) < 0.5).to(torch.uint8)
    # both kinds of every pair of rows, as matrix products
    x, w = pi.double(), beta.double()
    f, link = x @ x.T, (x * w) @ x.T
    p = torch.where(y.bool(), link[a.long(), b.long()],
                    ((f - link) + (1 - f) * (1 - eps))[a.long(), b.long()]).clamp_min(1e-30)
    ppx = torch.zeros(pairs, device="cuda")
    for count in (1, 2):  # the average of equal values is the value
        out = ctypes.c_double()
        assert native_lib.ammsb_perplexity_noalloc(
            pi.data_ptr(), _native.PI_BF16 if bf16 else _native.PI_F32, K, K, n, beta.data_ptr(), eps, a.data_ptr(),
            b.data_ptr(), y.data_ptr(), pairs, ppx.data_ptr(), count, torch.cuda.current_stream().cuda_stream,
            ctypes.byref(out)) == 0
        assert float(((ppx.double() - p) / p).abs().max()) < 1e-5
        assert out.value == pytest.approx(float(-p.log().mean()), rel=1e-5)
