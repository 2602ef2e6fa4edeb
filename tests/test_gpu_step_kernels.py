"""Kernels of the training step that write a result in the operand form of the next product: the same values as the plain
kernel followed by ``split_tf32``, bit for bit; and the scatter that adds to its output."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fastgl():
    return pytest.importorskip("fastgl")


def block(n_dst, n_src, most, seed):
    g = torch.Generator().manual_seed(seed)
    deg = torch.randint(0, most + 1, (n_dst,), generator=g)
    deg[0], deg[-1] = 0, most
    ptr = torch.zeros(n_dst + 1, dtype=torch.int32)
    ptr[1:] = deg.cumsum(0)
    src = torch.randint(0, n_src, (int(ptr[-1]),), generator=g).int()
    return ptr.cuda(), src.cuda(), deg


def parts(fastgl, x):
    hi, lo = fastgl.split_tf32(x.contiguous())
    return [hi, lo, hi]


# widths: one vector, the last of each column-pass variant and the first of the next, a remainder
@pytest.mark.parametrize("dim,blocks", [(4, 3), (128, 2), (132, 3), (256, 3), (260, 2), (516, 3)])
def test_operand_form_of_the_forward(fastgl, dim, blocks):
    n_dst, pad, n_src = 45, 50, 97
    ptr, src, _ = block(n_dst, n_src, 37, dim)
    ptr = torch.cat([ptr, ptr.new_zeros(pad - n_dst)])      # rows beyond the real count are not read
    n_dev = torch.tensor([n_dst], dtype=torch.int32, device="cuda")
    x = torch.randn(n_src, dim, device="cuda")
    want = fastgl.aggregate(fastgl.AGG_MEAN, ptr, src, x, pad, zero_deg_passthrough=False, n_dst_dev=n_dev)
    for plain in (True, False):
        split = torch.full((pad, 3 * 2 * dim), 7.0, device="cuda")
        out = torch.empty(pad, 2 * dim, device="cuda")[:, dim:] if plain else None
        fastgl.aggregate_split(ptr, src, x, pad, split[:, dim:], 2 * dim, blocks, out=out, n_dst_dev=n_dev)
        y = x[:pad].clone()
        copy = torch.empty(pad, dim, device="cuda") if plain else None
        fastgl.bias_relu_dropout_(y, torch.randn(dim, device="cuda"), 0.5, rng_ctr=3, copy_out=copy, split=split, split_stride=2 * dim,
                                  blocks=blocks)
        assert not plain or (torch.equal(out, want) and torch.equal(copy, y))
        for b, (a, s) in enumerate(zip(parts(fastgl, want), parts(fastgl, y))):
            got = split[:, 2 * dim * b: 2 * dim * (b + 1)]
            if b < blocks:
                assert torch.equal(got[:, dim:], a) and torch.equal(got[:, :dim], s)
            else:
                assert bool((got == 7.0).all())


@pytest.mark.parametrize("classes", [1, 32, 47, 128])
def test_operand_form_of_the_gradients(fastgl, classes):
    rows, k, pitch = 37, 40, (classes + 3) // 4 * 4
    x, w, b = (torch.randn(*s, device="cuda") for s in ((rows, k), (k, classes), (classes,)))
    labels = torch.randint(0, classes, (rows,), device="cuda")
    split = torch.zeros(rows, 3 * pitch, device="cuda")
    loss, d = fastgl.linear_softmax_xent(x, w, b, labels, n_valid=rows - 3, split3=split, block_stride=pitch)
    loss0, d0 = fastgl.linear_softmax_xent(x, w, b, labels, n_valid=rows - 3)
    assert torch.equal(d, d0) and torch.equal(loss, loss0)
    for q, p in enumerate(parts(fastgl, d)):
        assert torch.equal(split[:, q * pitch: q * pitch + classes], p)
    # the ReLU backward: two blocks are the first two of three
    z = torch.randn(rows, classes, device="cuda")
    three, two = torch.zeros_like(split), torch.full_like(split, 7.0)
    fastgl.relu_dropout_backward_(d.clone(), out=z, p_drop=0.5, split3=three, block_stride=pitch)
    fastgl.relu_dropout_backward_(d.clone(), out=z, p_drop=0.5, split3=two, block_stride=pitch, blocks=2)
    for q in (0, 1):
        assert torch.equal(two[:, q * pitch: q * pitch + classes], three[:, q * pitch: q * pitch + classes])
    assert bool((two[:, 2 * pitch:] == 7.0).all())
    # several matrices in one launch
    outs = [(torch.zeros_like(t), torch.zeros_like(t)) for t in (x, w)]
    fastgl.split_tf32_many([(t, [(o[0], "hi"), (o[1], "lo")]) for t, o in zip((x, w), outs)])
    for t, o in zip((x, w), outs):
        p = parts(fastgl, t)
        assert torch.equal(o[0], p[0]) and torch.equal(o[1], p[1])


@pytest.mark.parametrize("mode", ["SUM", "MEAN"])
@pytest.mark.parametrize("dim,offset", [(1, 0), (6, 2), (64, 0), (64, 1), (300, 0)])
def test_scatter_that_adds(fastgl, mode, dim, offset):
    mode = getattr(fastgl, "AGG_" + mode)
    n_dst, n_src = 33, 70
    ptr, src, deg = block(n_dst, n_src, 40, dim)
    dy = torch.randn(n_dst, dim, device="cuda")
    own = torch.randn(n_dst, dim + offset, device="cuda")[:, offset:]     # offset 1 and 2: narrower vectors
    start = torch.randn(n_src, dim, device="cuda")
    for self_term in (None, own):
        got = fastgl.aggregate_backward(mode, ptr, src, dy, n_src, out=start.clone(), d_self=self_term, accumulate=True)
        want, size = start.double().cpu(), start.double().abs().cpu()
        w = (1.0 / deg.double().clamp(min=1)) if mode == fastgl.AGG_MEAN else torch.ones(n_dst, dtype=torch.float64)
        dst = torch.repeat_interleave(torch.arange(n_dst), deg)
        rows = dy.double().cpu()[dst] * w[dst, None]
        terms = torch.bincount(src.long().cpu(), minlength=n_src) + 2
        want.index_add_(0, src.long().cpu(), rows)
        size.index_add_(0, src.long().cpu(), rows.abs())
        if self_term is not None:
            want[:n_dst] += self_term.double().cpu()
            size[:n_dst] += self_term.double().abs().cpu()
        # t additions in any order, and the rounding of the weighted row: (t + 2) half-ulps of the sum of magnitudes
        bound = (terms[:, None] + 2) * 2.0 ** -24 * size
        assert bool(((got.double().cpu() - want).abs() <= bound).all())


# a padded launch: the rows from the real count on are left alone (forward) or become zero unread (backward)
@pytest.mark.parametrize("dim", [47, 256])       # scalar and vector kernels
@pytest.mark.parametrize("real", [0, 1, 37, 50])
def test_padding_rows_of_the_relu(fastgl, dim, real):
    rows = 50
    n = torch.tensor([real], dtype=torch.int32, device="cuda")
    y, dy = torch.randn(rows, dim, device="cuda"), torch.randn(rows, dim, device="cuda")
    want = fastgl.bias_relu_dropout_(y.clone(), None, 0.5, rng_ctr=5)
    copy = torch.full_like(y, 7.0)
    got = fastgl.bias_relu_dropout_(y.clone(), None, 0.5, rng_ctr=5, n_rows_dev=n, copy_out=copy)
    assert torch.equal(got[:real], want[:real]) and torch.equal(got[real:], y[real:])
    assert torch.equal(copy[:real], want[:real]) and bool((copy[real:] == 7.0).all())
    bias, bias0 = torch.zeros(dim, device="cuda"), torch.zeros(dim, device="cuda")
    ref = fastgl.relu_dropout_backward_(dy[:real].clone(), out=want[:real], p_drop=0.5, dbias=bias0) if real else dy[:0]
    poisoned, out = dy.clone(), want.clone()
    poisoned[real:] = out[real:] = float("nan")
    back = fastgl.relu_dropout_backward_(poisoned, out=out, p_drop=0.5, dbias=bias, n_rows_dev=n)
    assert torch.equal(back[:real], ref) and not bool(back[real:].any())
    # at most 50 terms, added in another order: 51 half-ulps of the sum of magnitudes
    assert bool(((bias - bias0).abs() <= 51 * 2.0 ** -24 * 2 * ref.abs().sum(0)).all())
