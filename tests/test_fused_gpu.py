"""The fused dense consumer (scores -> softmax / "+1" softmax / exp -> value product) on the GPU,
through the C ABI and the autograd module, against the CPU oracle and the reference-generated
golden vectors.  Tolerances (norm-wise): fp64 1e-12, fp32 1e-5.
"""
import numpy as np
import pytest

from conftest import assert_close

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = {np.float32: 1e-5, np.float64: 1e-12}
MODES = ["softmax", "softmax_plus_one", "exp"]

# (bs, n, h, w, wv); the fp32 cases with widths up to 128 take the tiled kernels (RAGGED: rows that end inside a slice of 32
# columns, filled by TMA and by element-wise copies, value rows of every padding), the others (and all fp64 cases) the generic ones
SHAPES = [(1, 1, 1, 1, 1), (2, 3, 4, 8, 8), (1, 9, 2, 7, 5), (2, 70, 3, 32, 32), (1, 130, 2, 64, 64),
          (1, 200, 2, 128, 128), (1, 64, 4, 96, 64), (2, 129, 2, 64, 128), (1, 257, 1, 32, 64), (1, 40, 3, 64, 48)]

RAGGED = [(2, 70, 3, 40, 24), (1, 130, 2, 33, 21), (1, 100, 2, 48, 40), (1, 200, 5, 100, 7), (1, 65, 1, 127, 128), (2, 66, 2, 64, 100),
          (1, 64, 3, 1, 64), (1, 33, 2, 129, 64)]


def _cabi():
    import l1attn_cabi
    return l1attn_cabi


def _rand(shape, dtype, seed, spread=1.0):
    rng = np.random.RandomState(seed)
    bs, n, h, w, wv = shape
    return ((spread * rng.standard_normal((bs, n, h, w))).astype(dtype),
            (spread * rng.standard_normal((bs, n, h, w))).astype(dtype),
            rng.standard_normal((bs, n, h, wv)).astype(dtype))


def _dev(a):
    return torch.from_numpy(a).cuda()


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES + RAGGED)
def test_fwd_vs_oracle(shape, dtype, mode):
    from oracle import oracle
    q, k, v = _rand(shape, dtype, sum(shape), spread=0.3)  # scores of order -1: weights of order 1/n
    vo = _cabi().dense_softmax_v_fwd(_dev(q), _dev(k), _dev(v), mode).cpu().numpy()
    ref = oracle.dense_softmax_v(q.astype(np.float64), k.astype(np.float64), v.astype(np.float64), mode)
    assert_close(vo, ref, TOL[dtype], "vo %s %s" % (shape, mode))


@pytest.mark.parametrize("mode", MODES)
def test_far_scores(mode):
    """All scores near -45: the plain softmax must still normalise (running maximum), the unshifted
    forms give tiny but correct weights."""
    from oracle import oracle
    shape = (1, 150, 2, 64, 64)
    q, k, v = _rand(shape, np.float32, 5)
    k = (k + 6.0).astype(np.float32)
    vo = _cabi().dense_softmax_v_fwd(_dev(q), _dev(k), _dev(v), mode).cpu().numpy()
    ref = oracle.dense_softmax_v(q.astype(np.float64), k.astype(np.float64), v.astype(np.float64), mode)
    assert np.isfinite(vo).all()
    # a score near -45 carries ~1e-5 of absolute fp32 rounding (64 terms), which exp() turns into the
    # same RELATIVE error of the weight: the bar for this case is 5e-5 in every mode
    assert_close(vo, ref, 5e-5, "far " + mode)


def test_golden_fixtures(golden):
    cabi = _cabi()
    g = golden["fused"]
    for name in g["names"]:
        q, k, v = g[name + "_q"], g[name + "_k"], g[name + "_v"]
        for mode in MODES:
            ref = g["%s_%s" % (name, mode)]
            vo64 = cabi.dense_softmax_v_fwd(_dev(q), _dev(k), _dev(v), mode).cpu().numpy()
            assert_close(vo64, ref, 1e-11 if name == "far" else 1e-12, "%s %s f64" % (name, mode))
            if name == "far":
                # scores near -320: exp() is below the fp32 range in the unshifted forms, and in the softmax
                # the ~1e-4 absolute fp32 rounding of such a score is a 1e-4 relative error of its weight;
                # test_far_scores covers the fp32 running maximum at a magnitude fp32 resolves
                continue
            vo32 = cabi.dense_softmax_v_fwd(_dev(q.astype(np.float32)), _dev(k.astype(np.float32)),
                                            _dev(v.astype(np.float32)), mode).cpu().numpy()
            assert_close(vo32, ref, 1e-5, "%s %s f32" % (name, mode))


def test_host_entry_point():
    from oracle import oracle
    q, k, v = _rand((2, 33, 2, 32, 32), np.float32, 3, spread=0.3)
    vo = _cabi().dense_softmax_v_fwd_host(q, k, v, "softmax")
    assert_close(vo, oracle.dense_softmax_v(q.astype(np.float64), k.astype(np.float64), v.astype(np.float64)), 1e-5, "host")


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("dims", [(2, 37, 3, 32, 32), (1, 150, 2, 64, 64), (1, 70, 2, 128, 128), (2, 66, 1, 64, 128),
                                  (1, 20, 2, 7, 5)] + RAGGED[:7])
def test_autograd_matches_the_unfused_chain(mode, dtype, dims):
    """Gradients of the fused module against torch autograd through the chain the reference's callers
    write (README.md:64-66), built here on pure-PyTorch scores."""
    import l1attn_fused_cuda
    torch.manual_seed(1)
    bs, n, h, w, wv = dims
    q = (0.3 * torch.randn(bs, n, h, w, dtype=dtype, device="cuda")).requires_grad_(True)
    k = (0.3 * torch.randn(bs, n, h, w, dtype=dtype, device="cuda")).requires_grad_(True)
    v = torch.randn(bs, n, h, wv, dtype=dtype, device="cuda", requires_grad=True)
    g = torch.randn(bs, n, h, wv, dtype=dtype, device="cuda")
    vo = l1attn_fused_cuda.L1AttnSoftmaxV(mode)(q, k, v)
    vo.backward(g)
    got = [vo.detach(), q.grad, k.grad, v.grad]

    q2, k2, v2 = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    x = -(q2[:, None] - k2[:, :, None]).abs().sum(-1) / w ** 0.5  # [b, s, t, h]
    if mode == "softmax":
        a = torch.softmax(x, 1)
    elif mode == "softmax_plus_one":
        a = torch.exp(x) / (1 + torch.exp(x).sum(1, keepdim=True))
    else:
        a = torch.exp(x)
    ref = torch.einsum("bsdh,bshw->bdhw", a, v2)
    ref.backward(g.double())
    tol = 1e-12 if dtype == torch.float64 else 1e-5
    for name, a_, b_ in zip(("vo", "dq", "dk", "dv"), got, (ref.detach(), q2.grad, k2.grad, v2.grad)):
        assert_close(a_.cpu().numpy(), b_.cpu().numpy(), tol, "%s %s" % (name, mode))


@pytest.mark.parametrize("dims", [(2, 70, 4, 32, 32), (1, 45, 3, 40, 24), (1, 90, 2, 33, 20), (2, 20, 2, 32, 32)])
@pytest.mark.parametrize("kind", ["equal_rows", "padded", "grid"])
def test_backward_with_equal_rows_and_ties(dims, kind):
    """Equal query and key rows (the distance has no slope in any column), padded tokens, and ties everywhere (more than
    the list holds), against torch's own chain in float64, whose |x| has slope 0 at 0."""
    import l1attn_fused_cuda
    torch.manual_seed(3)
    bs, n, h, w, wv = dims
    q, k = (0.3 * torch.randn(bs, n, h, w, device="cuda") for _ in range(2))
    if kind == "equal_rows":
        k[:, 3:9] = q[:, 5:11]
    elif kind == "padded":
        q[:, n - 7:], k[:, n - 7:] = 0, 0
        k[0, 2, 0, 1] = 0
    else:
        q, k = (q * 4).round() / 4, (k * 4).round() / 4
    v, g = torch.randn(bs, n, h, wv, device="cuda"), torch.randn(bs, n, h, wv, device="cuda")
    got = [t.clone().requires_grad_(True) for t in (q, k, v)]
    l1attn_fused_cuda.L1AttnSoftmaxV()(*got).backward(g)
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    x = -(ref[0][:, None] - ref[1][:, :, None]).abs().sum(-1) / w ** 0.5
    torch.einsum("bsdh,bshw->bdhw", torch.softmax(x, 1), ref[2]).backward(g.double())
    for name, a, b in zip(("dq", "dk", "dv"), got, ref):
        assert_close(a.grad.cpu().numpy(), b.grad.cpu().numpy(), 1e-5, name)


def test_backward_chunks_over_the_batch(monkeypatch):
    """The backward walks the batch in chunks; a chunk size of one item must give the same gradients."""
    import l1attn_fused_cuda
    torch.manual_seed(2)
    q, k, v = (torch.randn(3, 20, 2, 32, device="cuda", requires_grad=True) for _ in range(3))
    g = torch.randn(3, 20, 2, 32, device="cuda")
    l1attn_fused_cuda.L1AttnSoftmaxV()(q, k, v).backward(g)
    whole = [t.grad.clone() for t in (q, k, v)]
    for t in (q, k, v):
        t.grad = None
    monkeypatch.setattr(l1attn_fused_cuda, "_CHUNK_BYTES", 1)
    l1attn_fused_cuda.L1AttnSoftmaxV()(q, k, v).backward(g)
    for a, b in zip(whole, (q, k, v)):
        assert torch.equal(a, b.grad)


@pytest.mark.parametrize("value", [-np.inf, float(np.finfo(np.float32).min)])
@pytest.mark.parametrize("dims", [(1, 200, 2, 33, 21), (1, 200, 2, 64, 64), (2, 150, 1, 100, 7)])
def test_masked_keys(dims, value):
    """Keys at the type's lowest value or at infinity are infinitely far from every query (the distance overflows): they weigh nothing,
    also where whole tiles of them come first, and get no gradient."""
    import l1attn_fused_cuda
    torch.manual_seed(5)
    bs, n, h, w, wv = dims
    q, k, v, g = (torch.randn(bs, n, h, x, device="cuda") for x in (w, w, wv, wv))
    k[:, :130] = value
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = l1attn_fused_cuda.L1AttnSoftmaxV()(*leaves)
    out.backward(g)
    ref = [t.clone().double().requires_grad_(True) for t in (q, k[:, 130:], v[:, 130:])]
    x = -(ref[0][:, None] - ref[1][:, :, None]).abs().sum(-1) / w ** 0.5
    rout = torch.einsum("bsdh,bshw->bdhw", torch.softmax(x, 1), ref[2])
    rout.backward(g.double())
    for name, a, r in (("vo", out, rout), ("dq", leaves[0].grad, ref[0].grad), ("dk", leaves[1].grad[:, 130:], ref[1].grad),
                       ("dv", leaves[2].grad[:, 130:], ref[2].grad)):
        assert_close(a.detach().cpu().numpy(), r.detach().cpu().numpy(), 1e-5, name)
    assert not leaves[1].grad[:, :130].any() and not leaves[2].grad[:, :130].any()


@pytest.mark.parametrize("dims,step", [((18, 520, 1, 33, 33), 10), ((21, 600, 16, 64, 64), 11)])
def test_smaller_last_chunk(monkeypatch, dims, step):
    """A last chunk of fewer items splits its source rows over more ranges than the others: every item's gradients are what
    the item gives alone (the sums over ranges round differently)."""
    import l1attn_fused_cuda
    torch.manual_seed(4)
    bs, n, h, w, wv = dims
    q, k = (0.3 * torch.randn(bs, n, h, w, device="cuda") for _ in range(2))
    v, g = torch.randn(bs, n, h, wv, device="cuda"), torch.randn(bs, n, h, wv, device="cuda")
    monkeypatch.setattr(l1attn_fused_cuda, "_CHUNK_BYTES", step * n * n * h * 4)

    def gradients(sl):
        leaves = [t[sl].clone().requires_grad_(True) for t in (q, k, v)]
        l1attn_fused_cuda.L1AttnSoftmaxV()(*leaves).backward(g[sl])
        return [t.grad for t in leaves]

    whole = gradients(slice(None))
    for b in (0, step - 1, step, bs - 1):
        for name, x, r in zip(("dq", "dk", "dv"), whole, gradients(slice(b, b + 1))):
            assert_close(x[b:b + 1].cpu().numpy(), r.cpu().numpy(), 1e-5, name)


def test_module_argument_checks():
    import l1attn_fused_cuda
    q = torch.randn(1, 4, 2, 8, device="cuda")
    with pytest.raises(ValueError):
        l1attn_fused_cuda.L1AttnSoftmaxV("max")
    with pytest.raises(RuntimeError, match="must be a CUDA tensor"):
        l1attn_fused_cuda.L1AttnSoftmaxV()(q.cpu(), q, q)
    with pytest.raises(RuntimeError):
        l1attn_fused_cuda.L1AttnSoftmaxV()(q, q[:, :3], q)


def test_full_size_properties():
    """Benchmark shape [16, 1024, 16, 64]: with all-ones values the softmax weights of every row must
    sum to one; one batch item agrees with the unfused pipeline (library scores + torch softmax + einsum)."""
    cabi = _cabi()
    gen = torch.Generator(device="cuda").manual_seed(7)
    q = 0.3 * torch.randn(16, 1024, 16, 64, device="cuda", generator=gen)
    k = 0.3 * torch.randn(16, 1024, 16, 64, device="cuda", generator=gen)
    ones = torch.ones(16, 1024, 16, 64, device="cuda")
    vo = cabi.dense_softmax_v_fwd(q, k, ones, "softmax")
    assert float((vo - 1).abs().max()) < 1e-5
    v = torch.randn(16, 1024, 16, 64, device="cuda", generator=gen)
    vo = cabi.dense_softmax_v_fwd(q, k, v, "softmax")
    b = 5
    a = torch.softmax(cabi.dense_fwd(q[b:b + 1].contiguous(), k[b:b + 1].contiguous()), 1)
    ref = torch.einsum("bsdh,bshw->bdhw", a.double(), v[b:b + 1].double())
    assert_close(vo[b:b + 1].cpu().numpy(), ref.cpu().numpy(), 1e-5, "full size item")
    assert cabi.lib().l1attn_device_status() == 0
