"""GPU tests of the one-launch mini-batch sampler and of the one-CTA block-CSR helpers, at the sizes where their dispatch
changes: against the hop-by-hop operators (same counters, exact) and against torch."""
import numpy as np
import pytest
import torch

from conftest import make_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_seeds,fanouts,index,arrival", [
    (1, [3], torch.int64, False), (37, [15, 10, 5], torch.int32, False), (700, [4, 33], torch.int64, False),
    (3000, [10, 10, 5], torch.int64, False),      # large enough for the results to be copied out of the arena
    (300, [7, 5], torch.int64, True),
])
@pytest.mark.parametrize("replace", [False, True])
def test_blocks_in_one_launch_equal_the_hop_by_hop_operators(n_seeds, fanouts, index, arrival, replace):
    import fastgl
    indptr, indices = make_graph(20000, 14, seed=3, hub=4000)
    dev = torch.device("cuda", 0)
    ptr, src = torch.from_numpy(indptr).to(dev).to(index), torch.from_numpy(indices).to(dev)
    rng = np.random.default_rng(n_seeds)
    seeds = rng.choice(20000, size=n_seeds, replace=False).astype(np.int32)
    if n_seeds > 2:
        seeds[n_seeds // 2] = seeds[0]            # of two equal seeds the later position names the edges' destination
    cur = torch.from_numpy(seeds).to(dev)
    fastgl.set_sampling(arrival_order=arrival)
    try:
        nodes, blocks = fastgl.sample_blocks(src, ptr, cur, fanouts[::-1], replace=replace, rng_seed=5, rng_ctr=80)
    finally:
        fastgl.set_sampling(arrival_order=False)
    for hop, (fanout, (b_ptr, b_src, b_dst, n_src, n_dst)) in enumerate(zip(fanouts[::-1], blocks[::-1])):
        s, d, p, n_edges = fastgl.sample_node_csr(src, ptr, cur, fanout, replace=replace, rng_seed=5, rng_ctr=80 + hop)
        assert n_dst == cur.numel() and torch.equal(b_ptr, p) and b_src.numel() == n_edges
        global_src = s.clone()
        s, d, uniq = fastgl.transfer_edge_id(s, d, cur, n_dst, n_dst + n_edges, n_edges, n_edges)
        assert torch.equal(b_dst, d) and uniq.numel() == n_src
        if arrival:                               # the order of the new nodes is free: the next hop follows its own
            assert torch.equal(nodes[b_src.long()], global_src)
            cur = nodes[:n_src].contiguous()
        else:
            assert torch.equal(b_src, s)
            cur = uniq
    assert torch.equal(nodes, cur)


@pytest.mark.parametrize("n_seeds", [1024, 2000])
def test_a_bad_seed_is_reported_and_the_next_call_works(n_seeds):
    import fastgl
    indptr, indices = make_graph(5000, 10, seed=4)
    dev = torch.device("cuda", 0)
    ptr, src = torch.from_numpy(indptr).to(dev), torch.from_numpy(indices).to(dev)
    seeds = torch.arange(n_seeds, dtype=torch.int32, device=dev)
    good = fastgl.sample_blocks(src, ptr, seeds, [5, 5], rng_seed=1, rng_ctr=0)
    bad = seeds.clone()
    bad[17] = 5000
    with pytest.raises(RuntimeError, match="out of range"):
        fastgl.sample_blocks(src, ptr, bad, [5, 5], rng_seed=1, rng_ctr=0)
    again = fastgl.sample_blocks(src, ptr, seeds, [5, 5], rng_seed=1, rng_ctr=0)
    assert torch.equal(good[0], again[0]) and all(torch.equal(a[1], b[1]) for a, b in zip(good[1], again[1]))


@pytest.mark.parametrize("n", [0, 1, 16383, 16384, 16385, 32768, 32769, 100003])
def test_exclusive_sum_at_its_dispatch_sizes(n):
    import fastgl
    x = torch.randint(0, 9, (n,), dtype=torch.int32, device="cuda")
    want = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(x.long(), 0)])
    assert torch.equal(fastgl.exclusive_sum(x).long(), want)


@pytest.mark.parametrize("n_nodes,n_ids", [(1, 0), (1, 5000), (12288, 32768), (12289, 32768), (12288, 32769), (300, 77)])
def test_cal_deg_at_its_dispatch_sizes(n_nodes, n_ids):
    import fastgl
    ids = torch.randint(-3, n_nodes + 3, (n_ids,), dtype=torch.int32, device="cuda")
    inside = ids[(ids >= 0) & (ids < n_nodes)].long()
    assert torch.equal(fastgl.cal_deg(ids, n_nodes).long(), torch.bincount(inside, minlength=n_nodes))


@pytest.mark.parametrize("heads,width,n_dst,n_src,fanout", [(1, 10, 1, 1, 1), (8, 32, 700, 3000, 12), (3, 27, 65, 300, 70), (40, 4, 33, 90, 5),
                                                          (2, 512, 40, 100, 9)])
@pytest.mark.parametrize("slope", [0.2, 1.0])
def test_gat_attention_and_its_gradients_match_torch(heads, width, n_dst, n_src, fanout, slope):
    """float64 torch algebra; a difference is bounded by the rounding of sums of at most fanout * width float32 terms."""
    import fastgl
    from fastgl_b200.layers import edge_softmax
    rng = np.random.default_rng(heads)
    deg = rng.integers(0, fanout + 1, n_dst)
    deg[0] = fanout
    ptr = torch.from_numpy(np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)).cuda()
    src = torch.from_numpy(rng.integers(0, n_src, int(deg.sum())).astype(np.int32)).cuda()
    dst = torch.from_numpy(np.repeat(np.arange(n_dst), deg)).cuda()
    gen = torch.Generator("cuda").manual_seed(1)
    feat = torch.randn((n_src, heads * width), generator=gen, device="cuda")
    l, r = (torch.randn((1, heads, width), generator=gen, device="cuda") / width ** 0.5 for _ in range(2))
    dy = torch.randn((n_dst, heads * width), generator=gen, device="cuda")
    out, alpha, el, er = fastgl.gat_attention(ptr, src, feat, l, r, n_dst, heads, slope)
    grads = fastgl.gat_attention_backward(ptr, src, feat, l, r, el, er, alpha, dy, heads, slope)
    fastgl.check_status()
    f64, l64, r64 = (t.double().requires_grad_() for t in (feat, l, r))
    x = f64.view(n_src, heads, width)
    score = torch.nn.functional.leaky_relu((x * l64).sum(-1)[src.long()] + (x[:n_dst] * r64).sum(-1)[dst], slope)
    a64 = edge_softmax(score, dst, n_dst)
    want = torch.zeros((n_dst, heads, width), dtype=torch.float64, device="cuda").index_add_(0, dst, a64.unsqueeze(-1) * x[src.long()])
    has = torch.from_numpy(deg > 0).cuda()
    want = want.reshape(n_dst, -1)
    refs = torch.autograd.grad(want, (f64, l64, r64), dy.double())
    want = torch.where(has[:, None], want, feat[:n_dst].double())
    for got, ref in zip((out, *grads), (want, *refs)):
        assert got.shape == ref.shape
        assert float((got - ref).abs().max()) <= 1e-5 * max(1.0, float(ref.abs().max())) * max(1.0, (fanout * width) ** 0.5 / 8)


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (1, 1, 70), (5, 3, 64), (64, 32, 65), (65, 33, 1024), (100, 64, 20011), (602, 256, 3001), (256, 41, 1024),
                                   (13, 200, 4097)])
def test_weight_grad_matches_float64(m, n, k):
    """A running sum of k products of unit normals stays within 4 sqrt(k), and its k roundings of 2^-24 of that add up like
    sqrt(k): 2^-22 k (plus the products' own roundings, which count where k is small)."""
    import fastgl
    gen = torch.Generator("cuda").manual_seed(m)
    wide = torch.randn((k, m + 3), generator=gen, device="cuda")
    for x in (wide[:, :m], wide[:, 1: m + 1], wide[:, :m].contiguous()):
        dy = torch.randn((k, n), generator=gen, device="cuda")
        want = x.double().t() @ dy.double()
        got = fastgl.weight_grad(x, dy)
        assert float((got - want).abs().max()) <= 2.0 ** -22 * (k + 16)
        assert torch.equal(got, fastgl.weight_grad(x, dy))
