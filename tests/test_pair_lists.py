"""Pair lists as callers may pass them to the edge log-likelihood."""
import ctypes

import pytest

from mcmc_for_ammsb_gb300 import _native

torch = pytest.importorskip("torch")


@pytest.fixture
def gpu(native_lib):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")


def lists(device="cpu"):
    return [torch.tensor(x, device=device) for x in ([0, 1, 1], [2, 0, 1], [1, 0, 0])]


# no pointer of another device, and no list of other than one dimension, gets
# as far as a kernel (the meta device stands for any other one)
@pytest.mark.parametrize("which", [0, 1, 2])
def test_lists_of_another_device_are_refused(which):
    from mcmc_for_ammsb_gb300.autograd import _as_lists
    mixed = lists()
    mixed[which] = mixed[which].to("meta")
    with pytest.raises(RuntimeError):
        _as_lists(*mixed)


@pytest.mark.gpu
@pytest.mark.parametrize("which", [0, 1, 2])
def test_mixed_lists_are_refused(gpu, which):
    from mcmc_for_ammsb_gb300.autograd import edge_log_likelihood, group_pairs
    phi, theta = torch.ones(3, 4, device="cuda"), torch.ones(4, 2, device="cuda")
    mixed = lists("cuda")
    mixed[which] = mixed[which].cpu()
    with pytest.raises(RuntimeError):
        edge_log_likelihood(phi, phi / 4, theta, *mixed, 1e-7)
    if which:  # lists led by a CPU one are grouped by torch
        with pytest.raises(RuntimeError):
            group_pairs(*mixed, 3, 3)
    flat = lists("cuda")
    if which < 2:
        flat[which] = flat[which][:, None]
        with pytest.raises(RuntimeError):
            group_pairs(*flat, 3, 3)
        with pytest.raises(RuntimeError):
            edge_log_likelihood(phi, phi / 4, theta, *flat, 1e-7)


# every index outside the rows is skipped and flagged, whatever its value: the
# loss is that of the other pairs (their sum in another order, hence the
# tolerances of test_adjoint), and no word of the workspace is read unwritten
@pytest.mark.gpu
@pytest.mark.parametrize("bad", [-1, -2, -3, -2**31, 90, 2**31 - 1])
@pytest.mark.parametrize("K,dtype,tol", [(16, torch.float64, 1e-11), (17, torch.float32, 1e-4),
                                         (256, torch.float32, 1e-4)])
def test_any_index_out_of_range_is_flagged(gpu, native_lib, bad, K, dtype, tol):
    n_src, n_nbr, per = 5, 90, 40
    gen = torch.Generator(device="cuda").manual_seed(K)
    phi, pi = (torch.rand(n, K, device="cuda", generator=gen, dtype=dtype) + 0.1 for n in (n_src, n_nbr))
    pi /= pi.sum(1, keepdim=True)
    theta = torch.rand(K, 2, device="cuda", generator=gen, dtype=dtype) + 0.5
    nbr = torch.randint(n_nbr, (n_src * per,), device="cuda", generator=gen, dtype=torch.int32)
    y = (torch.rand(n_src * per, device="cuda", generator=gen) < 0.3).to(torch.uint8)
    code = _native.REAL_F64 if dtype == torch.float64 else _native.REAL_F32

    def forward(nbr, y, per):
        ptr = torch.arange(n_src + 1, device="cuda") * per
        size = native_lib.ammsb_edge_loglik_workspace_size(code, K, n_src, len(nbr))
        ws = torch.full((size // phi.element_size(),), float("nan"), device="cuda", dtype=dtype)
        loss, flags = torch.zeros((), device="cuda", dtype=dtype), ctypes.c_int32()
        p = [ctypes.c_void_p(t.data_ptr()) for t in (phi, pi, theta, ptr, nbr, y, loss, ws)]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert native_lib.ammsb_edge_loglik_forward(code, K, p[0], K, p[1], K, n_nbr, p[2], 1e-7, p[3], n_src,
                                                    p[4], p[5], len(nbr), p[6], p[7], stream) == 0
        assert native_lib.ammsb_edge_loglik_status(p[7], stream, ctypes.byref(flags)) == 0
        return float(loss), flags.value

    marked = nbr.clone().view(n_src, per)
    marked[:, [0, 7, per - 1]] = bad
    keep = torch.ones(per, dtype=torch.bool, device="cuda")
    keep[[0, 7, per - 1]] = False
    want, clean = forward(nbr.view(n_src, per)[:, keep].reshape(-1), y.view(n_src, per)[:, keep].reshape(-1), per - 3)
    got, flags = forward(marked.reshape(-1), y, per)
    assert clean == 0 and flags == 1
    assert got == pytest.approx(want, rel=tol)


# a neighbour list longer than the source list: its tail takes no part, but
# has to be in range
@pytest.mark.gpu
def test_a_longer_neighbour_list_is_checked_to_its_end(gpu):
    from mcmc_for_ammsb_gb300.autograd import edge_log_likelihood
    phi, theta = torch.ones(3, 4, device="cuda"), torch.ones(4, 2, device="cuda")
    src, nbr, y = lists("cuda")
    want = edge_log_likelihood(phi, phi / 4, theta, src, nbr, y, 1e-7)
    longer = torch.cat([nbr, nbr])
    assert torch.equal(edge_log_likelihood(phi, phi / 4, theta, src, longer, y, 1e-7), want)
    for bad in (-1, 3):
        longer[-1] = bad
        with pytest.raises(IndexError):
            edge_log_likelihood(phi, phi / 4, theta, src, longer, y, 1e-7)


# more rows than an int32 can name, of which the pairs name the first and the
# last that it can: the pointers are those of the sorted list (exact)
@pytest.mark.gpu
def test_more_rows_than_an_int32_names(gpu):
    from mcmc_for_ammsb_gb300.autograd import group_pairs
    n_src, last = 2**31 + 5, 2**31 - 1
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    src = torch.tensor([last, 0, last, 7], device="cuda")
    src_ptr, pair_nbr, _, pair_src, _, _ = group_pairs(src, torch.tensor([2, 0, 1, 1], device="cuda"),
                                                       torch.zeros_like(src), n_src, 3)
    assert pair_src.tolist() == [0, 7, last, last] and pair_nbr.tolist() == [0, 1, 2, 1]
    assert src_ptr.shape[0] == n_src + 1
    for at, want in ((0, 0), (1, 1), (7, 1), (8, 2), (last, 2), (last + 1, 4), (n_src, 4)):
        assert int(src_ptr[at]) == want, at


# so many source rows that the forward's blocks do not fit one grid dimension:
# K = 1, phi = 1 and theta = (1, 1) give every pair p = eps + (1/2 - eps) pi for
# a link and dL/dphi = 0 of every row (a row's pi is 1 whatever phi); FP32's
# roundings of p and its logarithm allow 1e-6
@pytest.mark.gpu
def test_more_sources_than_a_grid_dimension(gpu):
    import math
    from mcmc_for_ammsb_gb300.autograd import edge_log_likelihood
    n_src, last = 2**31 + 5, 2**31 - 1
    if torch.cuda.mem_get_info()[0] < 120 << 30:
        pytest.skip("needs 120 GB of device memory")
    phi = torch.ones(n_src, 1, device="cuda").requires_grad_()
    pi = torch.tensor([[0.25], [0.5]], device="cuda").requires_grad_()
    theta = torch.ones(1, 2, device="cuda").requires_grad_()
    src = torch.tensor([0, last, last], device="cuda")
    loss = edge_log_likelihood(phi, pi, theta, src, torch.tensor([0, 1, 0], device="cuda"),
                               torch.ones(3, dtype=torch.uint8, device="cuda"), 1e-3)
    p = [1e-3 + (0.5 - 1e-3) * x for x in (0.25, 0.5)]
    assert float(loss.detach()) == pytest.approx(2 * math.log(p[0]) + math.log(p[1]), rel=1e-6)
    dphi, dpi, _ = torch.autograd.grad(loss, [phi, pi, theta])
    assert float(dphi[1:8].abs().max()) == 0.0 and float(dphi[last + 1:].abs().max()) == 0.0
    assert float(dphi[[0, last]].abs().max()) <= 1e-6
    assert dpi[:, 0].tolist() == pytest.approx([2 * 0.499 / p[0], 0.499 / p[1]], rel=1e-6)
