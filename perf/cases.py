"""The work that users of the sampler have it do, as timed cases.

Five kinds, each through the package's public entry points:

  chain     iterations of one Markov chain (MCMCSamplerStochastic.step) with
            what a training loop reads between its intervals: the held-out
            perplexity with its running averages, beta and, where N x K is
            small enough to look at during training, pi
  batch     many independent chains advanced together (ChainBatch.step)
  init      a chain's initial state, phi ~ Gamma(1, 1) (init())
  heldout   the held-out perplexity of a state in the caller's own device
            memory (ammsb_perplexity_noalloc)
  gradient  the minibatch edge log-likelihood and its gradients through
            torch.autograd (edge_log_likelihood)

Sizes are those of the package's workloads (workloads.py), of its tests and
of the options' derived defaults (K = 300, num-node-sample N / 50, minibatch
N / 10).  The graphs are planted communities, drawn here with numpy so that
exact() can restate a case without the package: overlapping communities of
log-uniform sizes, a tenth as many background edges, held-out and test sets
of links and as many non-links.

exact() restates the same draws (Philox4x32-10 streams) and the model's
update in 64 bits.
"""
import ctypes
import math

import numpy as np
import torch

from mcmc_for_ammsb_gb300 import ChainBatch, MCMCSamplerStochastic, Network, Options, _native
from mcmc_for_ammsb_gb300.autograd import edge_log_likelihood

EPSILON = 1e-7  # mcmc.epsilon's default, the sampler's and the gradients'
SCHEDULE = (0.01, 1024.0, 0.55)  # a, b, c of the step size, as in workloads.py


def listed():
    return [
        # a script that tries things on a small graph, one iteration at a
        # time, looking at the communities after each: latency alone
        dict(name="chain-single", kind="chain", n=2000, K=16, bf16=False, m=32, nns=32,
             degree=4, held=0.02, iters=1, ppx=False, read_pi=True),
        # the small workload's interval: 100 iterations, then the perplexity
        dict(name="chain-small", kind="chain", n=5000, K=32, bf16=False, m=500, nns=32,
             degree=4, held=0.02, iters=100, ppx=True, read_pi=True),
        # the options' derived defaults on 10k nodes (K = 300, N / 50, N / 10,
        # interval 50): a row length that is no power of two
        dict(name="chain-defaults", kind="chain", n=10000, K=300, bf16=False, m=1000, nns=200,
             degree=8, held=0.1, iters=50, ppx=True, read_pi=True),
        # the mid workload's shapes (100,000 nodes, K = 256), an interval of 500
        dict(name="chain-mid", kind="chain", n=100000, K=256, bf16=True, m=512, nns=64,
             degree=8, held=0.02, iters=500, ppx=True, read_pi=False),
        # the large workload's kernel shapes on 400,000 nodes (pi far larger
        # than the L2 cache): the headline configuration
        dict(name="chain-large", kind="chain", n=400000, K=1024, bf16=True, m=4096, nns=128,
             degree=16, held=0.002, iters=100, ppx=True, read_pi=False),
        # wide single-precision rows of a ragged length
        dict(name="chain-wide-f32", kind="chain", n=150000, K=1000, bf16=False, m=2000, nns=100,
             degree=16, held=0.002, iters=50, ppx=True, read_pi=False),
        # the batching workload: a parameter sweep of chains, own graphs and sizes
        dict(name="batch-32", kind="batch", chains=32, n_lo=1000, n_hi=50000, m_lo=32, m_hi=1024,
             nns=32, degree=6, held=0.02, iters=100),
        # the start of a chain of 30,000 nodes: its initial state
        dict(name="init", kind="init", n=30000, K=256, bf16=False),
        # the evaluation of a large model's held-out pairs in a host program
        # that owns the device memory
        dict(name="heldout-large", kind="heldout", n=500000, K=1024, bf16=True, pairs=86246),
        # the differentiation workload: 50 nodes x 32 neighbours, FP64
        dict(name="gradient-small", kind="gradient", n_src=50, per=32, n_nbr=2000, K=16, f64=True),
        # a minibatch of the mid workload's shapes in single precision
        dict(name="gradient-mid", kind="gradient", n_src=513, per=65, n_nbr=20000, K=256,
             f64=False),
        # a minibatch of the large workload's shapes, ragged rows
        dict(name="gradient-large", kind="gradient", n_src=4097, per=129, n_nbr=200000, K=1000,
             f64=False),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["chain", "chain", "chain", "batch", "init", "heldout", "gradient",
                       "gradient"])
    if kind == "chain":
        # nodes x row length within the largest listed state
        K = log_int(8, 1024)
        n = log_int(2000, min(400000, 400000 * 1024 // K))
        nns = log_int(16, min(200, n // 10))
        m = log_int(32, min(4096, n // 4))
        bf16 = rng.random() < 0.5
        # a pass of at most the listed ones' work: an iteration is a fixed cost
        # of some tens of microseconds and, half the time, m x nns row reads
        iters = int(8e-3 / (25e-6 + m * nns * K * (1 if bf16 else 2) / 4e12))
        iters = max(1, min(300, iters))
        return dict(kind=kind, n=n, K=K, bf16=bf16, m=m, nns=nns,
                    degree=rng.choice([4, 8, 16]), held=0.02 if n < 100000 else 0.002,
                    iters=iters, ppx=True, read_pi=n * K <= 5000000)
    if kind == "batch":
        return dict(kind=kind, chains=rng.randint(2, 32), n_lo=1000, n_hi=log_int(2000, 50000),
                    m_lo=32, m_hi=log_int(64, 1024), nns=log_int(16, 64), degree=6, held=0.02,
                    iters=rng.randint(8, 100))
    if kind == "init":
        K = log_int(8, 1024)
        return dict(kind=kind, n=log_int(2000, max(2001, 7680000 // K)), K=K,
                    bf16=rng.random() < 0.3)
    if kind == "heldout":
        K = log_int(8, 1024)
        return dict(kind=kind, n=log_int(5000, 500000), K=K, bf16=rng.random() < 0.5,
                    pairs=log_int(300, 86246))
    f64 = rng.random() < 0.4
    K = log_int(8, 512 if f64 else 1024)
    n_src = log_int(16, 4097)
    per = log_int(8, 129)
    return dict(kind=kind, n_src=n_src, per=per, n_nbr=log_int(1000, 100000 if f64 else 200000),
                K=K, f64=f64)


# -- inputs -------------------------------------------------------------------

def planted_edges(rng, n, degree):
    """Undirected pairs of a graph of overlapping communities (duplicates and
    self-pairs included, as a text file of edges may have them): every node
    belongs to one community, three in ten to a second one."""
    pairs = []
    for nodes, deg in ((rng.permutation(n), degree), (rng.permutation(n)[:3 * n // 10], degree)):
        sizes = np.exp(rng.uniform(math.log(10), math.log(min(500, len(nodes) // 2)),
                                   size=len(nodes) // 10 + 1)).astype(np.int64)
        ends = np.minimum(np.cumsum(sizes), len(nodes))
        ends = ends[:np.searchsorted(ends, len(nodes)) + 1]
        starts = np.concatenate([[0], ends[:-1]])
        which = np.repeat(np.arange(len(ends)), ends - starts)
        count = len(nodes) * deg // 2
        at = rng.integers(0, len(nodes), count)
        c = which[at]
        to = starts[c] + (rng.random(count) * (ends[c] - starts[c])).astype(np.int64)
        pairs.append(np.stack([nodes[at], nodes[to]]))
    count = n * degree // 20
    pairs.append(rng.integers(0, n, (2, count)))
    return np.concatenate(pairs, axis=1)


def unique_keys(a, b, n):
    """Sorted keys min * n + max of the pairs, without self-pairs."""
    lo, hi = np.minimum(a, b), np.maximum(a, b)
    keys = (lo * n + hi)[lo != hi]
    keys.sort()
    return keys[np.concatenate([[True], keys[1:] != keys[:-1]])] if len(keys) else keys


def is_in(sorted_keys, keys):
    at = np.minimum(np.searchsorted(sorted_keys, keys), max(len(sorted_keys) - 1, 0))
    return sorted_keys[at] == keys if len(sorted_keys) else np.zeros(keys.shape, bool)


def make_graph(seed, n, degree, held):
    """(sorted edge keys, held-out and test sets as (a, b, y)) of a seed."""
    rng = np.random.default_rng([seed, n, degree])
    pairs = planted_edges(rng, n, degree)
    edges = unique_keys(pairs[0], pairs[1], n)
    # links, and as many non-links, of each set: a share of the links drawn
    # (the package's split takes it of the distinct ones), the same for every seed
    count = max(4, int(held * n * degree * 0.6) // 2)
    links = edges[rng.permutation(len(edges))[:2 * count]]
    pairs = rng.integers(0, n, (2, 4 * count + 64))
    others = unique_keys(pairs[0], pairs[1], n)
    others = rng.permutation(others[~is_in(edges, others)])[:2 * count]
    sets = []
    for s in range(2):
        keys = np.concatenate([links[s * count:(s + 1) * count], others[s * count:(s + 1) * count]])
        y = np.concatenate([np.ones(count, np.uint8), np.zeros(len(keys) - count, np.uint8)])
        sets.append(((keys // n).astype(np.int32), (keys % n).astype(np.int32), y))
    return edges, sets[0], sets[1]


def make_sampler(seed, n, K, bf16, m, nns, degree, held, chain=0):
    edges, held_out, test = make_graph(seed, n, degree, held)
    net = Network.from_edges(n, edges // n, edges % n)
    net.held_out, net.test = held_out, test
    a, b, c = SCHEDULE
    opt = Options(K=K, mini_batch_size=m, num_node_sample=nns, pi_dtype=int(bf16), chain=chain,
                  held_out_ratio=held, epsilon=EPSILON, a=a, b=b, c=c,
                  random_seed=seed & 0x7fffffff)
    return MCMCSamplerStochastic(opt, net)


def batch_members(case):
    """The arguments of each chain of a batch: N, K and the minibatch size drawn
    as the batching workload draws them, the same for every seed."""
    rng = np.random.default_rng(case["chains"])
    for i in range(case["chains"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        K = int(rng.choice([16, 32, 64, 128]))
        m = int(round(math.exp(rng.uniform(math.log(case["m_lo"]), math.log(case["m_hi"])))))
        yield dict(n=n, K=K, bf16=True, m=min(m, n // 2), nns=case["nns"], degree=case["degree"],
                   held=case["held"], chain=i)


def make_rows(gen, n, K, device, dtype):
    """phi rows as the sampler draws them: iid Gamma(1, 1)."""
    return torch.empty(n, K, device=device, dtype=dtype).exponential_(generator=gen)


def make_gradient(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.float64 if case["f64"] else torch.float32
    K = case["K"]
    phi = make_rows(gen, case["n_src"], K, "cuda", dtype)
    pi = make_rows(gen, case["n_nbr"], K, "cuda", dtype)
    pi /= pi.sum(1, keepdim=True)
    theta = 0.5 + make_rows(gen, K, 2, "cuda", dtype)
    pairs = case["n_src"] * case["per"]
    src = torch.arange(case["n_src"], device="cuda").repeat_interleave(case["per"])
    nbr = torch.randint(case["n_nbr"], (pairs,), device="cuda", generator=gen)
    y = (torch.rand(pairs, device="cuda", generator=gen) < 0.1).to(torch.uint8)
    return phi, pi, theta, src, nbr, y


def make_heldout(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, K, per = case["n"], case["K"], 8 if case["bf16"] else 4
    stride = -(-K // per) * per
    pi = torch.zeros(n, stride, device="cuda",
                     dtype=torch.bfloat16 if case["bf16"] else torch.float32)
    for r in range(0, n, 65536):
        x = make_rows(gen, min(65536, n - r), K, "cuda", torch.float32)
        pi[r:r + 65536, :K] = (x / x.sum(1, keepdim=True)).to(pi.dtype)
    beta = torch.rand(K, device="cuda", generator=gen)
    a = torch.randint(n, (case["pairs"],), device="cuda", generator=gen, dtype=torch.int32)
    b = torch.randint(n, (case["pairs"],), device="cuda", generator=gen, dtype=torch.int32)
    y = (torch.arange(case["pairs"], device="cuda") < case["pairs"] // 2).to(torch.uint8)
    return pi, beta, a, b, y


# -- the cases ----------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "chain":
        state["s"] = make_sampler(seed, *(case[k] for k in ("n", "K", "bf16", "m", "nns", "degree",
                                                            "held"))).init()
    elif kind == "batch":
        state["s"] = [make_sampler(seed + i, **a).init()
                      for i, a in enumerate(batch_members(case))]
        state["batch"] = ChainBatch(state["s"])
    elif kind == "init":
        state["s"] = make_sampler(seed, case["n"], case["K"], case["bf16"], 64, 32, 2,
                                  0.02).create()
    elif kind == "heldout":
        state["tensors"] = make_heldout(case, seed)
        state["ppx"] = torch.zeros(case["pairs"], device="cuda")
        state["count"] = 0
    else:
        phi, pi, theta, src, nbr, y = make_gradient(case, seed)
        state["leaves"] = [t.requires_grad_() for t in (phi, pi, theta)]
        state["pairs"] = (src, nbr, y)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "chain":
        s = state["s"]
        s.step(case["iters"])
        out = {}
        if case["ppx"]:
            out["perplexity"] = s.cal_perplexity_held_out()
            out["held_out"] = s.ppx_per_heldout_edge
        out["beta"] = s.beta
        if case["read_pi"]:
            out["pi"] = s.pi
        return out
    if kind == "batch":
        state["batch"].step(case["iters"])
        ppx = [s.cal_perplexity_held_out() for s in state["s"]]
        return {"perplexity": np.array(ppx, np.float32),
                "held_out": np.concatenate([s.ppx_per_heldout_edge for s in state["s"]]),
                "beta": np.concatenate([s.beta for s in state["s"]])}
    if kind == "init":
        s = state["s"]
        s.init()
        return {"pi": s.pi, "beta": s.beta}
    if kind == "heldout":
        pi, beta, a, b, y = state["tensors"]
        state["count"] += 1
        value = ctypes.c_double()
        code = _native.lib().ammsb_perplexity_noalloc(
            pi.data_ptr(), _native.PI_BF16 if case["bf16"] else _native.PI_F32, case["K"],
            pi.shape[1], pi.shape[0], beta.data_ptr(), EPSILON, a.data_ptr(), b.data_ptr(),
            y.data_ptr(), case["pairs"], state["ppx"].data_ptr(), state["count"],
            torch.cuda.current_stream().cuda_stream, ctypes.byref(value))
        if code != _native.AMMSB_OK:
            raise _native.AmmsbError(code, "ammsb_perplexity_noalloc")
        return {"perplexity": value.value, "held_out": state["ppx"]}
    loss = edge_log_likelihood(*state["leaves"], *state["pairs"], EPSILON)
    grads = torch.autograd.grad(loss, state["leaves"])
    return {"loss": loss.detach(), "phi": grads[0], "pi": grads[1], "theta": grads[2]}


def chain_work(n, K, bf16, m, nns, degree, held, iters, ppx=True, read_pi=False, **_):
    """A minibatch is the non-link stratum (m + 1 nodes) or a node's links,
    each half the time; a node's update reads its neighbours' rows (their ids
    are drawn, not read), reads and writes its phi row and writes its pi row;
    a minibatch edge reads its two new rows once more."""
    s = 2 if bf16 else 4
    links = 1.3 * degree + 1
    nodes = ((m + 1) + (links + 1)) / 2
    edges = (m + links) / 2
    work = dict(bytes=iters * (nodes * ((nns + 1) * K * s + K * (8 + s)) + 24 * K),
                flops=iters * (nodes * (nns + 1) * K * 4 + edges * K * 6 + nodes * K * 30))
    if ppx:
        pairs = 2 * max(4, int(held * n * degree * 0.6) // 2)
        work["bytes"] += pairs * (2 * K * s + 17)
        work["flops"] += pairs * K * 4
    if read_pi:
        work["bytes"] += n * K * (s + 4)
    return work


def work(case):
    kind = case["kind"]
    if kind == "chain":
        return chain_work(**case)
    if kind == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for a in batch_members(case):
            one = chain_work(iters=case["iters"], **a)
            total = {k: total[k] + one[k] for k in total}
        return total
    K = case["K"]
    s = 2 if case.get("bf16") else 8 if case.get("f64") else 4
    if kind == "init":
        cells = case["n"] * K
        return dict(bytes=cells * (4 + s + s + 4), flops=cells * 60)
    if kind == "heldout":
        rows = min(case["n"], 2 * case["pairs"])
        return dict(bytes=rows * K * s + case["pairs"] * 17 + 4 * K, flops=case["pairs"] * K * 4)
    pairs = case["n_src"] * case["per"]
    rows = min(case["n_nbr"], pairs)  # neighbour rows that pairs name
    return dict(bytes=s * K * (2 * case["n_src"] + rows + case["n_nbr"] + 6) + pairs * 17,
                flops=pairs * K * 8)


# -- 64-bit restatement ---------------------------------------------------------

M32 = np.uint64(0xffffffff)


def philox(x, y, z, w, seed, chain):
    """Philox4x32-10 blocks of the counters (arrays broadcast together) under
    the key (seed, chain): four uint64 arrays of 32-bit words."""
    x, y, z, w = (np.asarray(v, np.uint64) for v in np.broadcast_arrays(x, y, z, w))
    k0, k1 = seed & 0xffffffff, chain & 0xffffffff
    for _ in range(10):
        p, q = x * np.uint64(0xD2511F53), z * np.uint64(0xCD9E8D57)
        x, y, z, w = ((q >> np.uint64(32)) ^ y ^ np.uint64(k0), q & M32,
                      (p >> np.uint64(32)) ^ w ^ np.uint64(k1), p & M32)
        k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
    return x, y, z, w


def uniforms(tag, entity, step, t, below, key):
    """Draws t of a stream as integers in [0, below), below < 2^32: the high
    half of the 64-bit draw times below."""
    t = np.asarray(t, np.uint64)
    x, y, z, w = philox(t >> np.uint64(1), entity, step, tag, *key)
    odd = (t & np.uint64(1)).astype(bool)
    lo, hi = np.where(odd, z, x), np.where(odd, w, y)
    n = np.uint64(below)
    return ((hi * n + ((lo * n) >> np.uint64(32))) >> np.uint64(32)).astype(np.int64)


def normals(tag, entity, step, count, key):
    """Standard normals 0 .. count - 1 of the streams (a row per entity)."""
    entity = np.asarray(entity).reshape(-1, 1)
    words = philox(np.arange((count + 3) // 4), entity, step, tag, *key)
    u = [(v >> np.uint64(8)).astype(np.float64) for v in words]
    out = []
    for u1, u2 in ((u[0], u[1]), (u[2], u[3])):
        r = np.sqrt(-2.0 * np.log((u1 + 0.5) * 2.0 ** -24))
        out += [r * np.cos(2 * math.pi * u2 * 2.0 ** -24), r * np.sin(2 * math.pi * u2 * 2.0 ** -24)]
    return np.stack(out, -1).reshape(len(entity), -1)[:, :count]


def gammas(tag, entity, count, key):
    """Gamma(1, 1) draws 0 .. count - 1 of the streams (a row per entity) by
    Marsaglia and Tsang's rejection, an attempt per counter step."""
    entity = np.asarray(entity).reshape(-1, 1)
    e, idx = (v.reshape(-1) for v in np.broadcast_arrays(entity, np.arange(count)))
    out = np.zeros(e.shape)
    todo = np.arange(e.size)
    d = 1.0 - 1.0 / 3.0
    c = 1.0 / math.sqrt(9.0 * d)
    for attempt in range(64):
        x, y, z, _ = philox(idx[todo], e[todo], attempt, tag, *key)
        g = np.sqrt(-2.0 * np.log((x + 0.5) * 2.0 ** -32)) * np.cos(2 * math.pi * (y * 2.0 ** -32))
        v = 1.0 + c * g
        u = (z + 0.5) * 2.0 ** -32
        ok = v > 0
        v = np.where(ok, v, 1.0) ** 3
        ok &= (u < 1.0 - 0.0331 * g ** 4) | (np.log(u) < 0.5 * g * g + d * (1.0 - v + np.log(v)))
        out[todo[ok]] = d * v[ok]
        todo = todo[~ok]
        if not len(todo):
            break
    return out.reshape(len(entity), count)


def first_valid(draws, ok, want):
    """Per row, the first `want` valid draws without repeats; None where a row
    has too few."""
    order = np.argsort(np.where(ok, draws, -1 - np.arange(draws.shape[1])), axis=1, kind="stable")
    ranked = np.take_along_axis(draws, order, 1)
    okr = np.take_along_axis(ok, order, 1)
    new = okr.copy()
    new[:, 1:] &= ~(okr[:, :-1] & (ranked[:, 1:] == ranked[:, :-1]))
    keep = np.zeros_like(ok)
    np.put_along_axis(keep, order, new, 1)
    if (keep.sum(1) < want).any():
        return None
    keep &= np.cumsum(keep, 1) <= want
    return draws[keep].reshape(len(draws), want)


class ExactChain:
    """One chain in 64 bits: the draws of the sampler's streams (tags 1 to 8)
    and the literal update_phi, update_beta and perplexity sums."""

    def __init__(self, seed, n, K, m, nns, degree, held, chain=0, **_):
        self.n, self.K, self.m, self.nns = n, K, m, nns
        self.key = (seed & 0x7fffffff, chain)
        self.edges, self.held_out, self.test = make_graph(seed, n, degree, held)
        both = [np.concatenate([self.held_out[i], self.test[i]]).astype(np.int64) for i in (0, 1)]
        self.excluded = unique_keys(both[0], both[1], n)
        self.theta = gammas(8, 0, 2 * K, self.key).reshape(K, 2)
        self.beta = self.theta[:, 1] / self.theta.sum(1)
        self.phi = gammas(7, np.arange(n), K, self.key)
        self.pi = self.phi / self.phi.sum(1, keepdims=True)
        a, b = self.edges // n, self.edges % n
        src, dst = np.concatenate([a, b]), np.concatenate([b, a])
        order = np.lexsort((dst, src))
        self.col = dst[order]
        self.row = np.searchsorted(src[order], np.arange(n + 1))
        self.step_count, self.average_count = 1, 1
        self.ppx = np.zeros(len(self.held_out[0]))

    def keys(self, a, b):
        return np.minimum(a, b) * self.n + np.maximum(a, b)

    def minibatch(self, step):
        """(source, partners, y, scale) of an iteration's minibatch."""
        n, m = self.n, self.m
        if uniforms(1, 0, step, 0, 2, self.key) == 0:
            v = int(uniforms(2, 0, step, 0, n, self.key))
            count = m
            while True:
                count = 2 * count + 64
                u = uniforms(3, 0, step, np.arange(count), n, self.key)[None]
                k = self.keys(v, u)
                got = first_valid(u, (u != v) & ~is_in(self.edges, k) & ~is_in(self.excluded, k), m)
                if got is not None:
                    break
            scale = np.float32(n) * np.float32(n) / np.float32(m)
            scale = np.float32(float(scale) * (len(self.edges) / (n * (n - 1.0) / 2.0 - len(self.edges))))
            return v, got[0], 0, float(scale)
        attempt = 0
        while True:
            v = int(uniforms(2, 0, step, attempt, n, self.key))
            u = self.col[self.row[v]:self.row[v + 1]]
            u = u[~is_in(self.excluded, self.keys(v, u))]
            if len(u):
                return v, u, 1, float(n)
            attempt += 1

    def neighbours(self, step, nodes):
        want = self.nns + 1
        count = want
        while True:
            count = 2 * count + 32
            i = nodes[:, None]
            j = uniforms(4, i, step, np.arange(count)[None], self.n, self.key)
            k = self.keys(i, j)
            got = first_valid(j, (j != i) & ~is_in(self.excluded, k), want)
            if got is not None:
                return got, is_in(self.edges, self.keys(i, got))

    def step(self):
        n, K, t = self.n, self.K, self.step_count
        eps = float(np.float32(SCHEDULE[0] * (1.0 + t / SCHEDULE[1]) ** -SCHEDULE[2]))
        v, u, y, scale = self.minibatch(t)
        nodes = np.concatenate([[v], u])
        nbr, nbr_y = self.neighbours(t, nodes)
        alpha, nn, beta = 1.0 / K, n / self.nns, self.beta
        noise = normals(5, nodes, t, K, self.key)
        phi = self.phi[nodes]
        total = phi.sum(1, keepdims=True)
        p_i = phi / total
        grad = np.zeros_like(phi)
        for q in range(nbr.shape[1]):
            p_j, yy = self.pi[nbr[:, q]], nbr_y[:, q][:, None]
            e = np.where(yy, EPSILON, 1.0 - EPSILON)
            probs = p_i * (p_j * np.where(yy, beta, 1.0 - beta) + (1.0 - p_j) * e)
            grad += probs / probs.sum(1, keepdims=True) / phi - 1.0 / total
        new = np.maximum(np.abs(phi + eps / 2 * (alpha - phi + nn * grad) + np.sqrt(eps * phi) * noise), 1e-24)
        self.phi[nodes] = new
        self.pi[nodes] = new / new.sum(1, keepdims=True)
        f = self.pi[v] * self.pi[u]
        probs = f * (beta if y else 1.0 - beta)
        rest = (EPSILON if y else 1.0 - EPSILON) * (1.0 - f.sum(1))
        f = (probs / (probs.sum(1) + rest)[:, None]).sum(0)
        th = self.theta
        grads = np.stack([f * ((1 - y) / th[:, 0] - 1.0 / th.sum(1)), f * (y / th[:, 1] - 1.0 / th.sum(1))], 1)
        noise = normals(6, 0, t, 2 * K, self.key).reshape(K, 2)
        self.theta = np.maximum(np.abs(th + eps / 2 * (1.0 - th + scale * grads) + np.sqrt(eps * th) * noise), 1e-24)
        self.beta = self.theta[:, 1] / self.theta.sum(1)
        self.step_count += 1

    def perplexity(self):
        a, b, y = self.held_out
        like = pair_likelihood(torch.from_numpy(self.pi[a]), torch.from_numpy(self.pi[b]),
                               torch.from_numpy(self.beta), torch.from_numpy(y)).numpy()
        self.ppx = (self.ppx * (self.average_count - 1) + like) / self.average_count
        self.average_count += 1
        return -np.log(self.ppx).mean()


def pair_likelihood(pa, pb, beta, y):
    f = pa * pb
    y = y.bool()
    link = (f * beta).sum(1)
    other = (f * (1.0 - beta)).sum(1) + (1.0 - f.sum(1)) * (1.0 - EPSILON)
    return torch.where(y, link, other).clamp_min(1e-30)


def exact_chain(seed, case, iters):
    """The chain after `iters` iterations, or None where that is long."""
    # row elements that the neighbour loops touch, and the cells of the state
    if iters * (case["m"] + 20) * (case["nns"] + 1) * case["K"] > 6e8 or case["n"] * case["K"] > 4e6:
        return None
    chain = ExactChain(seed, **case)
    for _ in range(iters):
        chain.step()
    return chain


def exact(case, seed):
    kind = case["kind"]
    if kind == "chain":
        chain = exact_chain(seed, case, case["iters"])
        if chain is None:
            return None
        out = {"beta": chain.beta}
        if case["ppx"]:
            out["perplexity"] = chain.perplexity()
            out["held_out"] = chain.ppx
        if case["read_pi"]:
            out["pi"] = chain.pi
        return out
    if kind == "batch":
        return None  # several minutes: each of the chains, as above
    if kind == "init":
        key = (seed & 0x7fffffff, 0)
        theta = gammas(8, 0, 2 * case["K"], key).reshape(-1, 2)
        pi = []
        for r in range(0, case["n"], 2048):
            phi = gammas(7, np.arange(r, min(r + 2048, case["n"])), case["K"], key)
            pi.append(phi / phi.sum(1, keepdims=True))
        return {"pi": np.concatenate(pi), "beta": theta[:, 1] / theta.sum(1)}
    if kind == "heldout":
        pi, beta, a, b, y = make_heldout(case, seed)
        like = [pair_likelihood(pi[a[r:r + 8192].long(), :case["K"]].double(),
                                pi[b[r:r + 8192].long(), :case["K"]].double(), beta.double(),
                                y[r:r + 8192]) for r in range(0, case["pairs"], 8192)]
        like = torch.cat(like)
        return {"perplexity": float(-like.log().mean()), "held_out": like}
    phi, pi, theta, src, nbr, y = make_gradient(case, seed)
    leaves = [t.double().requires_grad_() for t in (phi, pi, theta)]
    grads = [torch.zeros_like(t) for t in leaves]
    loss = torch.zeros((), dtype=torch.float64, device="cuda")
    for r in range(0, len(src), 16384):  # in parts: a part's rows are gathered
        p, q, th = leaves
        s, yy = src[r:r + 16384], y[r:r + 16384].bool()
        beta = th[:, 1] / th.sum(1)
        rows = p[s]
        f = rows / rows.sum(1, keepdim=True) * q[nbr[r:r + 16384]]
        e = torch.full_like(yy, 1.0 - EPSILON, dtype=torch.float64).masked_fill(yy, EPSILON)
        prob = (f * (torch.where(yy[:, None], beta, 1.0 - beta) - e[:, None])).sum(1) + e
        part = prob.log().sum()
        for g, x in zip(grads, torch.autograd.grad(part, leaves)):
            g += x
        loss += part.detach()
    return {"loss": loss, "phi": grads[0], "pi": grads[1], "theta": grads[2]}
