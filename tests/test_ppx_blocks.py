"""The held-out perplexity where its blocks, lane groups and chunks have
remainders, through ammsb_perplexity_noalloc on the caller's memory: each
running average and the result against the plain expression in FP64, within
the 1e-5 of test_gpu_parity."""
import ctypes
import math

import pytest

from mcmc_for_ammsb_gb300 import _native

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# lanes per pair from one to a warp; 32 to 256 pairs per block, one block and
# several, one pair past a block, more blocks than the last one's threads
@pytest.mark.parametrize("K,bf16", [(1, False), (4, False), (30, False), (100, True), (256, True), (1000, False),
                                    (1024, True)])
@pytest.mark.parametrize("pairs", [1, 31, 33, 255, 257, 9000])
def test_perplexity_at_block_remainders(native_lib, K, bf16, pairs):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    gen = torch.Generator(device="cuda").manual_seed(pairs)
    n, per, eps = 400, 8 if bf16 else 4, 1e-7
    pi = torch.full((n, -(-K // per) * per), float("nan"), device="cuda")
    rows = torch.rand(n, K, device="cuda", generator=gen) + 0.01
    pi[:, :K] = rows / rows.sum(1, keepdim=True)
    pi = pi.to(torch.bfloat16 if bf16 else torch.float32)
    beta = torch.rand(K, device="cuda", generator=gen)
    a, b = (torch.randint(n, (pairs,), device="cuda", generator=gen, dtype=torch.int32) for _ in range(2))
    y = (torch.rand(pairs, device="cuda", generator=gen) < 0.5).to(torch.uint8)
    f = pi[a.long(), :K].double() * pi[b.long(), :K].double()
    p = torch.where(y.bool(), (f * beta).sum(1),
                    (f * (1 - beta)).sum(1) + (1 - f.sum(1)) * (1 - eps)).clamp_min(1e-30)
    ppx = torch.zeros(pairs, device="cuda")
    for count in (1, 2, 3):  # the average of equal values is the value
        out = ctypes.c_double()
        rc = native_lib.ammsb_perplexity_noalloc(
            pi.data_ptr(), _native.PI_BF16 if bf16 else _native.PI_F32, K, pi.shape[1], n, beta.data_ptr(), eps,
            a.data_ptr(), b.data_ptr(), y.data_ptr(), pairs, ppx.data_ptr(), count,
            torch.cuda.current_stream().cuda_stream, ctypes.byref(out))
        assert rc == 0
        assert float(((ppx.double() - p) / p).abs().max()) < 1e-5
        assert out.value == pytest.approx(float(-p.log().mean()), rel=1e-5, abs=1e-5)


# the logarithms are taken of products of four averages: of the smallest ones
# (a link between disjoint rows has p = 1e-30), and with a negative average in
# the caller's array, whose logarithm is NaN
@pytest.mark.parametrize("K", [2, 32, 128])
def test_perplexity_of_the_smallest_averages(native_lib, K):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    pairs = 100
    pi = torch.zeros(2, -(-K // 4) * 4, device="cuda")
    pi[0, 0], pi[1, 1] = 1.0, 1.0
    beta = torch.full((K,), 0.5, device="cuda")
    a = torch.zeros(pairs, dtype=torch.int32, device="cuda")
    b, y = torch.ones_like(a), torch.ones(pairs, dtype=torch.uint8, device="cuda")
    ppx = torch.zeros(pairs, device="cuda")

    def call(count):
        out = ctypes.c_double()
        assert native_lib.ammsb_perplexity_noalloc(
            pi.data_ptr(), _native.PI_F32, K, pi.shape[1], 2, beta.data_ptr(), 1e-7, a.data_ptr(), b.data_ptr(),
            y.data_ptr(), pairs, ppx.data_ptr(), count, 0, ctypes.byref(out)) == 0
        return out.value

    tiny = float(torch.tensor(1e-30))
    assert call(1) == pytest.approx(-math.log(tiny), rel=1e-12)
    ppx[7] = ppx[10] = -1.0
    assert math.isnan(call(2))
