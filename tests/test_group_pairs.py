"""Pair grouping and the edge log-likelihood where their tiles and rows have
remainders.  Grouping: the CUDA sort against the stable torch sort of the same
lists on the CPU, exactly.  Gradients: against torch's own autograd of the
plain expression in FP64, within the tolerances of test_adjoint (FP64 1e-11,
FP32 1e-4 of the largest gradient)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu(native_lib):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")


# one warp, a tile of 2,048 and its neighbours, many tiles, no pairs; keys of
# one to three digits, all equal, more keys than one block's pointers
@pytest.mark.parametrize("pairs", [0, 1, 33, 2047, 2048, 2049, 50001])
@pytest.mark.parametrize("n_src,n_nbr", [(1, 1), (50, 2000), (513, 20000), (5000, 300001)])
@pytest.mark.parametrize("order", ["sorted", "random", "one"])
def test_groups_equal_a_stable_sort(pairs, n_src, n_nbr, order):
    from mcmc_for_ammsb_gb300.autograd import group_pairs
    rng = np.random.default_rng([pairs, n_src, len(order)])
    src = rng.integers(0, n_src, pairs)
    nbr = rng.integers(0, n_nbr, pairs)
    if order == "sorted":
        src = np.sort(src)
    if order == "one":
        src[:], nbr[:] = n_src - 1, n_nbr // 2
    lists = [torch.from_numpy(src), torch.from_numpy(nbr),
             torch.from_numpy(rng.integers(0, 2, pairs).astype(np.uint8))]
    want = group_pairs(*lists, n_src, n_nbr)
    got = group_pairs(*(t.cuda() for t in lists), n_src, n_nbr)
    for g, w in zip(got, want):
        assert g.dtype == w.dtype and torch.equal(g.cpu(), w)


def test_pairs_past_the_rows_come_last():
    from mcmc_for_ammsb_gb300.autograd import group_pairs
    src = torch.tensor([7, 1, 9, 0, 1], dtype=torch.int32)
    nbr = torch.tensor([0, 5, 2, 5, 40])
    y = torch.tensor([True, False, True, False, True])
    for g, w in zip(group_pairs(src.cuda(), nbr.cuda(), y.cuda(), 2, 6), group_pairs(src, nbr, y, 2, 6)):
        assert torch.equal(g.cpu(), w)
    with pytest.raises(RuntimeError):
        group_pairs((src - 1).cuda(), nbr.cuda(), y.cuda(), 2, 6)


# 16-byte vectors and single elements; rows of less than a vector to the widest
@pytest.mark.parametrize("K", [2, 4, 6, 17, 66, 130, 516, 1001, 1024])
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-11), (torch.float32, 1e-4)])
def test_gradients_at_row_remainders(K, dtype, tol):
    from mcmc_for_ammsb_gb300.autograd import edge_log_likelihood
    from test_adjoint import torch_reference
    gen = torch.Generator(device="cuda").manual_seed(K)
    n_src, n_nbr, eps = 37, 90, 1e-7
    # sources with no pair, with one, and with more than a block's groups take
    counts = torch.tensor([0, 1, 200] + [5] * (n_src - 3), device="cuda")
    src = torch.arange(n_src, device="cuda").repeat_interleave(counts)
    nbr = torch.randint(n_nbr - 1, src.shape, device="cuda", generator=gen)  # the last row has none
    nbr[:100] = 3  # a neighbour row with more pairs than a warp's lanes
    y = (torch.rand(src.shape, device="cuda", generator=gen) < 0.3).to(torch.uint8)
    perm = torch.randperm(len(src), device="cuda", generator=gen)
    src, nbr, y = src[perm], nbr[perm], y[perm]
    phi = 0.1 + torch.rand(n_src, K, device="cuda", generator=gen, dtype=torch.float64)
    pi = 0.1 + torch.rand(n_nbr, K, device="cuda", generator=gen, dtype=torch.float64)
    pi /= pi.sum(1, keepdim=True)
    theta = 0.5 + torch.rand(K, 2, device="cuda", generator=gen, dtype=torch.float64)
    ref = [t.clone().requires_grad_() for t in (phi, pi, theta)]
    want = torch_reference(*ref, src, nbr, y, eps)
    mine = [t.to(dtype).requires_grad_() for t in (phi, pi, theta)]
    got = edge_log_likelihood(*mine, src, nbr, y, eps)
    assert float(got.detach()) == pytest.approx(float(want.detach()), rel=max(tol, 1e-12))
    for rerun in range(2):  # the backward leaves what it reads
        grads = torch.autograd.grad(got, mine, retain_graph=True)
        for g, w in zip(grads, torch.autograd.grad(want, ref, retain_graph=True)):
            assert float((g.double() - w).abs().max()) <= tol * float(w.abs().max()), rerun


@pytest.mark.parametrize("pairs", [100, 5000])
@pytest.mark.parametrize("which,bad", [("src", -1), ("src", 50), ("nbr", -3), ("nbr", 2000), ("nbr", 1 << 40)])
def test_out_of_range_indices_are_refused(pairs, which, bad):
    from mcmc_for_ammsb_gb300.autograd import edge_log_likelihood
    phi = torch.rand(50, 16, device="cuda", dtype=torch.float64) + 0.1
    pi = torch.full((2000, 16), 1 / 16, device="cuda", dtype=torch.float64)
    theta = torch.ones(16, 2, device="cuda", dtype=torch.float64)
    lists = dict(src=torch.randint(50, (pairs,), device="cuda"),
                 nbr=torch.randint(2000, (pairs,), device="cuda"))
    y = torch.zeros(pairs, dtype=torch.uint8, device="cuda")
    edge_log_likelihood(phi, pi, theta, lists["src"], lists["nbr"], y, 1e-7)
    lists[which][pairs // 2] = bad
    with pytest.raises(IndexError):
        edge_log_likelihood(phi, pi, theta, lists["src"], lists["nbr"], y, 1e-7)
