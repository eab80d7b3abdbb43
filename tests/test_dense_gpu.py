"""Dense L1Attn forward/backward on the GPU, through the C ABI, against the CPU oracle.

Tolerances (norm-wise, see conftest.rel_err): fp64 1e-12, fp32 1e-5 -- the bars the task states.
"""
import numpy as np
import pytest

from conftest import PKG, assert_close

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = {np.float32: 1e-5, np.float64: 1e-12}

SHAPES = [(1, 1, 1, 1), (1, 16, 8, 64), (2, 5, 3, 7), (1, 9, 2, 33), (2, 17, 5, 16), (1, 33, 9, 65),
          (3, 70, 12, 32), (1, 130, 16, 64), (2, 64, 1, 128), (1, 3, 16, 7), (2, 40, 8, 97), (1, 65, 24, 64),
          (2, 150, 4, 64), (1, 140, 20, 48),   # (head counts that take the forward's four-head work items)
          (1, 300, 4, 32), (1, 600, 4, 32), (1, 1040, 4, 32), (1, 2050, 4, 32)]  # (few work items: the backward splits the source rows in 2, 4, 8 and 8)


def _cabi():
    import l1attn_cabi
    return l1attn_cabi


def _rand(shape, dtype, seed):
    rng = np.random.RandomState(seed)
    bs, n, h, w = shape
    return (rng.standard_normal(shape).astype(dtype), rng.standard_normal(shape).astype(dtype),
            rng.standard_normal((bs, n, n, h)).astype(dtype))


def _dev(a):
    return torch.from_numpy(a).cuda()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_fwd_bwd_vs_oracle(shape, dtype):
    from oracle import oracle
    cabi = _cabi()
    q, k, g = _rand(shape, dtype, hash(shape) % 1000)
    attn = cabi.dense_fwd(_dev(q), _dev(k)).cpu().numpy()
    dq, dk = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(g), _dev(q), _dev(k)))
    # the oracle runs in fp64 on the same (fp32-representable) inputs
    q64, k64, g64 = q.astype(np.float64), k.astype(np.float64), g.astype(np.float64)
    assert_close(attn, oracle.dense_fwd(q64, k64), TOL[dtype], "attn %s" % (shape,))
    rq, rk = oracle.dense_bwd(g64, q64, k64)
    assert_close(dq, rq, TOL[dtype], "dq %s" % (shape,))
    assert_close(dk, rk, TOL[dtype], "dk %s" % (shape,))


# rows that TMA cannot address: groups of 8, 4, 2 and 1 heads, last tiles and last 16-byte pieces of every fill, source rows
# that are split over several items; and 16-byte rows whose width ends inside a stage or whose heads come in groups of 2 and 1
RAGGED = [(2, 201, 6, 65), (1, 130, 3, 33), (1, 520, 1, 17), (1, 270, 2, 47), (1, 257, 5, 64), (1, 600, 3, 66), (2, 129, 8, 30),
          (1, 48, 9, 20), (2, 33, 7, 130), (1, 1040, 1, 7), (1, 513, 1, 48), (1, 300, 2, 36), (2, 70, 8, 40)]
# sets of at most 48 tokens: both sides of 16, 32 and 48, more than eight heads, widths on both sides of 32, few and many units
SMALL = [(3, 1, 2, 5), (5, 2, 9, 33), (4, 15, 3, 64), (4, 16, 8, 32), (3, 17, 8, 40), (2, 31, 5, 65), (2, 32, 17, 96),
         (3, 33, 2, 40), (2, 47, 9, 33), (2, 48, 8, 64), (2, 49, 3, 20), (75, 40, 8, 64)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", RAGGED + SMALL)
def test_ragged_and_small_vs_oracle(shape, dtype):
    test_fwd_bwd_vs_oracle(shape, dtype)


def test_golden_fixtures(golden):
    """Reference outputs (pure-PyTorch and compiled CPU extension) on seeded inputs, incl. the
    tie-heavy and zero-padded cases: sign(0) must be exactly 0."""
    cabi = _cabi()
    g = golden["dense"]
    for name in g["names"]:
        q, k, da = g[name + "_q"], g[name + "_k"], g[name + "_dattn"]
        attn = cabi.dense_fwd(_dev(q), _dev(k)).cpu().numpy()
        dq, dk = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(da), _dev(q), _dev(k)))
        for ref in ("py", "cpp"):
            if "%s_attn_%s" % (name, ref) not in g:
                continue
            assert_close(attn, g["%s_attn_%s" % (name, ref)], 1e-12, "%s attn vs %s" % (name, ref))
            assert_close(dq, g["%s_dq_%s" % (name, ref)], 1e-12, "%s dq vs %s" % (name, ref))
            assert_close(dk, g["%s_dk_%s" % (name, ref)], 1e-12, "%s dk vs %s" % (name, ref))
        # fp32 on the same inputs
        a32 = cabi.dense_fwd(_dev(q.astype(np.float32)), _dev(k.astype(np.float32))).cpu().numpy()
        assert_close(a32, g[name + "_attn_py"], 1e-5, name + " attn fp32")


def test_kat(golden):
    cabi = _cabi()
    g = golden["kat"]
    a = cabi.dense_fwd(_dev(g["f3_q"]), _dev(g["f3_k"])).cpu().numpy()
    expect = np.array([[-1, -1, 0, -.5], [0, -1, -1, -.5], [-1, 0, -1, -.5], [-.5, -.5, -.5, 0]], dtype=np.float32)
    assert np.array_equal(a[0, :, :, 0], expect)
    a1 = cabi.dense_fwd(_dev(g["f1_q"]), _dev(g["f1_k"])).cpu().numpy()
    assert_close(a1, g["f1_dense_attn"], 1e-6, "f1")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_ties_exact(dtype):
    """Inputs on a coarse grid: every difference and every sum is exact in fp32, so the GPU
    result must equal the oracle bit for bit up to the final scale multiply, and rows with
    q == k must contribute exactly nothing."""
    from oracle import oracle
    cabi = _cabi()
    rng = np.random.RandomState(5)
    shape = (2, 48, 8, 64)
    q = (np.round(rng.standard_normal(shape) * 2) / 2).astype(dtype)
    k = (np.round(rng.standard_normal(shape) * 2) / 2).astype(dtype)
    k[:, 40:] = q[:, 40:]  # identical rows
    q[:, 44:] = 0
    k[:, 44:] = 0  # zero padding
    g = np.round(rng.standard_normal((2, 48, 48, 8)) * 4).astype(dtype) / 4
    dq, dk = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(g), _dev(q), _dev(k)))
    rq, rk = oracle.dense_bwd(g.astype(np.float64), q.astype(np.float64), k.astype(np.float64))
    assert_close(dq, rq, 2e-7 if dtype == np.float32 else 1e-14, "dq ties")
    assert_close(dk, rk, 2e-7 if dtype == np.float32 else 1e-14, "dk ties")


@pytest.mark.parametrize("shape", [(2, 200, 8, 64), (1, 1040, 4, 32)])  # (the second: work items split their source rows)
@pytest.mark.parametrize("kind", ["sparse_ties", "padded", "q_is_k", "grid"])
def test_fast_backward_tie_handling(kind, shape):
    """fp32 shapes that take the compare-form backward (16-byte rows): a handful of planted ties, many
    zero-padded tokens (more candidates than the detector lists), q == k, and values on a coarse grid
    (ties everywhere).  The result must match the oracle as if every term had used sign(0) = 0."""
    from oracle import oracle
    cabi = _cabi()
    rng = np.random.RandomState(21)
    bs, n, nh, nw = shape
    q = rng.standard_normal(shape).astype(np.float32)
    k = rng.standard_normal(shape).astype(np.float32)
    if kind == "sparse_ties":
        for _ in range(7):
            b, t, s, h, w = (rng.randint(m) for m in (bs, n, n, nh, nw))
            k[b, s, h, w] = q[b, t, h, w]
        k[bs - 1, 5, 3, 7] = -0.0
        q[bs - 1, 9, 3, 7] = 0.0  # +0 == -0 is a tie too
    elif kind == "padded":
        q[:, n * 3 // 5:] = 0
        k[:, n * 9 // 20:] = 0
    elif kind == "q_is_k":
        k = q.copy()
    else:
        q, k = np.round(q * 2) / 2, np.round(k * 2) / 2
    g = rng.standard_normal((bs, n, n, nh)).astype(np.float32)
    dq, dk = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(g), _dev(q), _dev(k)))
    rq, rk = oracle.dense_bwd(g.astype(np.float64), q.astype(np.float64), k.astype(np.float64))
    assert_close(dq, rq, 1e-5, "dq " + kind)
    assert_close(dk, rk, 1e-5, "dk " + kind)
    # without scratch every tile takes the exact loop: same answer
    dq2, dk2 = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(g), _dev(q), _dev(k), scratch=None))
    assert_close(dq2, rq, 1e-5, "dq exact " + kind)
    assert_close(dk2, rk, 1e-5, "dk exact " + kind)


@pytest.mark.parametrize("shape", [(2, 90, 6, 33), (1, 300, 5, 20), (1, 540, 7, 9), (3, 24, 5, 36), (3, 16, 8, 32), (3, 45, 5, 36)])
@pytest.mark.parametrize("kind", ["sparse_ties", "padded", "q_is_k", "grid"])
def test_ragged_and_small_tie_handling(kind, shape):
    test_fast_backward_tie_handling(kind, shape)


def test_many_listed_ties_are_repaired():
    """A few zeros among the values of k rows and several hundred padded q rows: runs of listed ties on one element of d_k,
    close to as many as the list holds, on rows that stay on the fast path."""
    from oracle import oracle
    cabi = _cabi()
    q, k, g = _rand((1, 1000, 4, 32), np.float32, 35)
    q[:, 600:] = 0
    k[0, 7, 0, 3] = k[0, 8, 0, 3] = k[0, 9, 1, 31] = k[0, 500, 3, 0] = k[0, 501, 3, 5] = k[0, 650, 2, 16] = 0
    k[0, 700:] = 0  # (and padded k rows, so that the fast path drops pairs: 6 x 400 ties are left to the list)
    rq, rk = oracle.dense_bwd(g.astype(np.float64), q.astype(np.float64), k.astype(np.float64))
    dq, dk = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(g), _dev(q), _dev(k)))
    assert_close(dq, rq, 1e-5, "dq")
    assert_close(dk, rk, 1e-5, "dk")
    again = cabi.dense_bwd(_dev(g), _dev(q), _dev(k))
    assert np.array_equal(again[0].cpu().numpy(), dq) and np.array_equal(again[1].cpu().numpy(), dk)


@pytest.mark.parametrize("shape", [(2, 200, 8, 64), (1, 1040, 4, 32), (2, 90, 6, 33), (1, 540, 1, 20)])
def test_zero_rows_beside_zero_values(shape):
    """Padded tokens, and zeros among the values of other rows: those tie with the padded rows one by one, and with each
    other; a row that is zero but for its last column is not a padded one.  Non-finite gradients of padded pairs
    reach nothing."""
    from oracle import oracle
    cabi = _cabi()
    rng = np.random.RandomState(33)
    bs, n, nh, nw = shape
    q, k, g = _rand(shape, np.float32, 34)
    q[:, n - 5:], k[:, n - 9:] = 0, 0
    q[0, n - 5, 0, nw - 1], k[0, n - 9, 0, nw - 1] = 1e-30, -1e-30
    q[0, n - 4, 0, 0] = -0.0
    for x in (q, k):
        for _ in range(5):
            x[rng.randint(bs), rng.randint(n - 9), rng.randint(nh), rng.randint(nw)] = 0
    q[0, 3, nh - 1, 0] = k[0, 4, nh - 1, 0] = 0
    g2 = g.copy()
    g2[:, n - 8:, n - 4:] = np.nan
    g[:, n - 8:, n - 4:] = 0
    rq, rk = oracle.dense_bwd(g.astype(np.float64), q.astype(np.float64), k.astype(np.float64))
    for grad in (g, g2):
        dq, dk = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(grad), _dev(q), _dev(k)))
        assert_close(dq, rq, 1e-5, "dq")
        assert_close(dk, rk, 1e-5, "dk")


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 3e38])
@pytest.mark.parametrize("shape", [(2, 201, 6, 65), (1, 130, 3, 33), (1, 520, 1, 17), (1, 270, 2, 47), (1, 48, 9, 20)])
def test_ragged_rows_with_gradients_that_are_not_finite(shape, bad):
    """Infinities, NaN and sums that overflow give what the exact kernel gives, which takes the sign of every term (3e38 four
    times on one query and one source row, with both signs)."""
    cabi = _cabi()
    q, k, g = (_dev(a) for a in _rand(shape, np.float32, 38))
    b, n, h = shape[0] - 1, shape[1], shape[2] - 1
    if np.isfinite(bad):
        g[b, 3, 2:n:n // 4, h], g[b, 5:n:n // 4, n - 1, h] = bad, bad
        g[b, 3, 3, h] = -bad
    else:
        g[b, 3, n - 1, h] = bad
    got, want = cabi.dense_bwd(g, q, k), cabi.dense_bwd(g, q, k, scratch=None)
    for x, r in zip(got, want):
        assert torch.equal(x.nan_to_num(0.5, 2e38, -2e38), r.nan_to_num(0.5, 2e38, -2e38))
    assert not all(torch.isfinite(r).all() for r in want)


@pytest.mark.parametrize("shape", [(3, 12, 8, 32), (2, 30, 3, 33), (2, 45, 8, 64), (2, 70, 3, 33), (2, 130, 8, 64)])
def test_equal_infinities_are_ties(shape):
    """sign(inf - inf) is 0 in the reference (NaN compares as neither), in every kernel that fp32 takes with scratch."""
    from oracle import oracle
    cabi = _cabi()
    q, k, g = _rand(shape, np.float32, 40)
    n = shape[1]
    for b, h, w, x in ((0, 0, 0, np.inf), (1, 2, 31, -np.inf), (1, 1, 4, np.inf)):
        q[b, n - 2, h, w] = k[b, 3, h, w] = x
        q[b, 1, h, w] = -x
    with np.errstate(invalid="ignore"):
        rq, rk = oracle.dense_bwd(g.astype(np.float64), q.astype(np.float64), k.astype(np.float64))
    dq, dk = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(g), _dev(q), _dev(k)))
    assert_close(dq, rq, 1e-5, "dq")
    assert_close(dk, rk, 1e-5, "dk")


@pytest.mark.parametrize("mean", [0.0, 1.0])
@pytest.mark.parametrize("spread", [1.0, 0.3])
@pytest.mark.parametrize("shape", [(20, 64, 5, 33), (20, 100, 6, 33), (8, 201, 6, 65), (4, 333, 5, 33), (2, 1040, 1, 66)])
def test_ragged_rows_lose_no_precision(shape, spread, mean):
    """Sums of the gradients where q > k, of which half the sum of all is taken away, against one signed sum over all rows (the exact
    kernel): such a sum grows with the rows where the gradients have a mean and q lies in the middle of k.  Their errors are 0.1 to 1.06
    of its (a few percent of that is chance)."""
    cabi = _cabi()
    q, k, g = _rand(shape, np.float32, 39)
    q *= np.float32(spread)
    g = g if mean == 0 else (mean + 0.1 * g).astype(np.float32)
    t = [_dev(a) for a in (g, q, k)]
    exact = cabi.dense_bwd(*[x.double() for x in t])
    for x, s, e in zip(cabi.dense_bwd(*t), cabi.dense_bwd(*t, scratch=None), exact):
        err, of_sum = (float((y.double() - e).norm() / e.norm()) for y in (x, s))
        assert err <= 1.15 * of_sum, (err, of_sum)


@pytest.mark.parametrize("count", [1, 2, 7, 8, 9, 33])
def test_few_listed_ties_are_repaired(count):
    """Lists shorter than the repair's CTAs, and one more."""
    from oracle import oracle
    cabi = _cabi()
    q, k, g = _rand((1, 160, 4, 32), np.float32, 37)
    for i in range(count):
        k[0, 150 - i, i % 4, i % 32] = q[0, 3 * i, i % 4, i % 32]
    rq, rk = oracle.dense_bwd(g.astype(np.float64), q.astype(np.float64), k.astype(np.float64))
    for _ in range(20):
        dq, dk = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(g), _dev(q), _dev(k)))
        assert_close(dq, rq, 1e-5, "dq")
        assert_close(dk, rk, 1e-5, "dk")


def test_deterministic():
    cabi = _cabi()
    q, k, g = _rand((2, 96, 16, 64), np.float32, 11)
    a = [cabi.dense_bwd(_dev(g), _dev(q), _dev(k)) for _ in range(2)]
    assert torch.equal(a[0][0], a[1][0]) and torch.equal(a[0][1], a[1][1])
    f = [cabi.dense_fwd(_dev(q), _dev(k)) for _ in range(2)]
    assert torch.equal(f[0], f[1])


def test_host_buffers_with_a_smaller_last_group(monkeypatch):
    """The last group of batch items may need more scratch than the others (its source rows are split over more ranges)."""
    cabi = _cabi()
    monkeypatch.setenv("L1ATTN_HOST_GROUP", "10")
    q, k, g = _rand((18, 520, 1, 33), np.float32, 36)
    dq, dk = cabi.dense_bwd_host(g, q, k)
    for b in (0, 9, 10, 17):
        rq, rk = cabi.dense_bwd(_dev(g[b:b + 1]), _dev(q[b:b + 1]), _dev(k[b:b + 1]))
        assert_close(dq[b:b + 1], rq.cpu().numpy(), 1e-5, "dq")
        assert_close(dk[b:b + 1], rk.cpu().numpy(), 1e-5, "dk")
    assert cabi.lib().l1attn_host_release() == 0


def test_host_buffer_entry_points():
    from oracle import oracle
    cabi = _cabi()
    q, k, g = _rand((2, 37, 5, 24), np.float32, 3)
    attn = cabi.dense_fwd_host(q, k)
    dq, dk = cabi.dense_bwd_host(g, q, k)
    q64, k64, g64 = q.astype(np.float64), k.astype(np.float64), g.astype(np.float64)
    assert_close(attn, oracle.dense_fwd(q64, k64), 1e-5, "host attn")
    rq, rk = oracle.dense_bwd(g64, q64, k64)
    assert_close(dq, rq, 1e-5, "host dq")
    assert_close(dk, rk, 1e-5, "host dk")
    # asynchronous forms: forward and an independent backward enqueued together, several times over (the arena
    # has to grow and to be reused), results valid after the sync and equal to the synchronous ones
    for rep in range(3):
        attn2 = np.empty_like(attn)
        dq2, dk2 = np.empty_like(dq), np.empty_like(dk)
        cabi.dense_fwd_host(q, k, out=attn2, wait=False)
        cabi.dense_bwd_host(g, q, k, out=(dq2, dk2), wait=False)
        cabi.host_sync()
        assert np.array_equal(attn2, attn) and np.array_equal(dq2, dq) and np.array_equal(dk2, dk)
    assert cabi.lib().l1attn_host_release() == 0


def test_fp64_long_context_variant_full():
    """The float64 long-context variant [2,512,8,128], checked in full against the oracle at 1e-12."""
    from oracle import oracle
    cabi = _cabi()
    rng = np.random.RandomState(3001)
    shape = (2, 512, 8, 128)
    q, k = rng.standard_normal(shape), rng.standard_normal(shape)
    g = rng.standard_normal((2, 512, 512, 8))
    attn = cabi.dense_fwd(_dev(q), _dev(k)).cpu().numpy()
    dq, dk = (x.cpu().numpy() for x in cabi.dense_bwd(_dev(g), _dev(q), _dev(k)))
    assert_close(attn, oracle.dense_fwd(q, k), 1e-12, "attn")
    rq, rk = oracle.dense_bwd(g, q, k)
    assert_close(dq, rq, 1e-12, "dq")
    assert_close(dk, rk, 1e-12, "dk")


@pytest.mark.parametrize("shape", [(16, 1024, 16, 64), (2, 4096, 8, 128)])
def test_full_size_properties(shape):
    """The fp32 benchmark shapes [16,1024,16,64] and [2,4096,8,128], too large for the oracle: size-independent properties.
      * swapping q and k transposes the score matrix exactly (|q-k| is symmetric);
      * sampled (b, s, t) entries and sampled gradient rows match a float64 numpy evaluation;
      * the backward is linear in d_attn."""
    cabi = _cabi()
    bs, n, h, w = shape
    gen = torch.Generator(device="cuda").manual_seed(2000)
    q = torch.randn(shape, generator=gen, device="cuda")
    k = torch.randn(shape, generator=gen, device="cuda")
    attn = cabi.dense_fwd(q, k)
    attn_sw = cabi.dense_fwd(k, q)
    assert torch.equal(attn, attn_sw.transpose(1, 2))
    del attn_sw
    scale = -1.0 / np.sqrt(w)
    rng = np.random.RandomState(7)
    qh, kh = q.double().cpu().numpy(), k.double().cpu().numpy()
    for _ in range(64):
        b, s, t = rng.randint(bs), rng.randint(n), rng.randint(n)
        ref = scale * np.abs(qh[b, t] - kh[b, s]).sum(-1)
        assert_close(attn[b, s, t].cpu().numpy(), ref, 1e-5, "sample attn")
    g1 = torch.randn(attn.shape, generator=gen, device="cuda")
    dq1, dk1 = cabi.dense_bwd(g1, q, k)
    for _ in range(8):
        b, t = rng.randint(bs), rng.randint(n)
        sg = np.sign(qh[b, t][None] - kh[b])  # [s, h, w]
        ref = scale * (sg * g1[b, :, t].double().cpu().numpy()[:, :, None]).sum(0)
        assert_close(dq1[b, t].cpu().numpy(), ref, 1e-5, "sample dq")
        s = rng.randint(n)
        sg = np.sign(qh[b] - kh[b, s][None])  # [t, h, w]
        ref = -scale * (sg * g1[b, s].double().cpu().numpy()[:, :, None]).sum(0)
        assert_close(dk1[b, s].cpu().numpy(), ref, 1e-5, "sample dk")
    g2 = torch.randn(attn.shape, generator=gen, device="cuda")
    dq2, dk2 = cabi.dense_bwd(g2, q, k)
    g1.add_(g2)
    del g2
    dq3, dk3 = cabi.dense_bwd(g1, q, k)
    assert_close((dq1 + dq2).cpu().numpy(), dq3.cpu().numpy(), 1e-5, "linearity dq")
    assert_close((dk1 + dk2).cpu().numpy(), dk3.cpu().numpy(), 1e-5, "linearity dk")


def _offset_by_one(t):
    """A contiguous copy of t whose storage starts one element (4 bytes) past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    view = buf[1:].view(t.shape)
    view.copy_(t)
    assert view.is_contiguous() and view.data_ptr() % 16 == 4
    return view


def test_pointers_aligned_to_the_element_only():
    """The C ABI promises element alignment, not 16 bytes: tensors that start 4 bytes past a 16-byte
    boundary (a contiguous view with storage offset 1) must take the kernels without vector loads or
    tensor maps and give the aligned call's results -- dense forward/backward (with and without tie
    scratch), the fused consumer and the sparse operators."""
    import l1attn_fused_cuda
    cabi = _cabi()
    q, k, g = (torch.from_numpy(a).cuda() for a in _rand((2, 72, 8, 64), np.float32, 31))
    k[1, 7, 3, 5] = q[1, 9, 3, 5]  # one planted tie
    want_attn = cabi.dense_fwd(q, k)
    want = cabi.dense_bwd(g, q, k)
    qo, ko, go = _offset_by_one(q), _offset_by_one(k), _offset_by_one(g)
    out = _offset_by_one(torch.empty_like(want_attn))
    assert_close(cabi.dense_fwd(qo, ko, out=out).cpu().numpy(), want_attn.cpu().numpy(), 1e-6, "attn")
    for scratch in ("auto", None):
        outs = (_offset_by_one(torch.empty_like(q)), _offset_by_one(torch.empty_like(k)))
        got = cabi.dense_bwd(go, qo, ko, out=outs, scratch=scratch)
        for a, b in zip(got, want):
            assert_close(a.cpu().numpy(), b.cpu().numpy(), 1e-6, "gradients")
    # mixed: only q misaligned (the tie detector and the tensor-map path must both decline)
    got = cabi.dense_bwd(g, qo, k)
    for a, b in zip(got, want):
        assert_close(a.cpu().numpy(), b.cpu().numpy(), 1e-6, "gradients, q offset only")
    v = torch.randn(2, 72, 8, 64, device="cuda")
    want_vo = cabi.dense_softmax_v_fwd(0.3 * q, 0.3 * k, v)
    got_vo = cabi.dense_softmax_v_fwd(_offset_by_one(0.3 * q), _offset_by_one(0.3 * k), _offset_by_one(v),
                                      out=_offset_by_one(torch.empty_like(v)))
    assert_close(got_vo.cpu().numpy(), want_vo.cpu().numpy(), 1e-6, "fused vo")
    # sparse, through the C ABI with every float tensor offset
    from oracle import oracle
    rng = np.random.RandomState(4)
    co = np.stack([rng.randint(0, 72, 500), rng.randint(0, 72, 500)], 1)
    coo, dm, _ = oracle.expand_coo(co)
    ix = cabi.SparseIndex(torch.from_numpy(coo).cuda(), 72, dm)
    ix.check()
    qs, ks = 0.3 * q, 0.3 * k
    vo, attn = cabi.sparse_fwd(v, qs, ks, ix, True)
    grads = cabi.sparse_bwd(g[:, :, :64].contiguous().view(2, 72, 8, 64), v, qs, ks, ix, attn, True)
    dvo_o = _offset_by_one(g[:, :, :64].contiguous().view(2, 72, 8, 64))
    vo2, attn2 = cabi.sparse_fwd(_offset_by_one(v), _offset_by_one(qs), _offset_by_one(ks), ix, True,
                                 out=(_offset_by_one(torch.empty_like(vo)), _offset_by_one(torch.empty_like(attn))))
    assert_close(vo2.cpu().numpy(), vo.cpu().numpy(), 1e-6, "sparse vo")
    outs = (_offset_by_one(torch.empty_like(v)), None, _offset_by_one(torch.empty_like(q)), _offset_by_one(torch.empty_like(k)))
    grads2 = cabi.sparse_bwd(dvo_o, _offset_by_one(v), _offset_by_one(qs), _offset_by_one(ks), ix, attn2, True,
                             out=outs, scratch=_offset_by_one(torch.empty_like(attn)))
    for a, b in zip(grads2, grads):
        assert_close(a.cpu().numpy(), b.cpu().numpy(), 1e-6, "sparse gradients")
    torch.cuda.synchronize()
    assert cabi.lib().l1attn_device_status() == 0


def test_bounded_wait_gives_up_and_is_reported():
    """Every wait of the TMA kernels is bounded in time.  Here one warp waits (limit 3 ms) on a barrier that nothing
    completes: the wait gives up, the kernel returns, l1attn_device_status() reports the timeout exactly once, and
    the library keeps working.  Nothing faults and nothing hangs -- a wait that runs out is the whole test."""
    import time
    cabi = _cabi()
    lib = cabi.lib()
    torch.cuda.synchronize()
    assert lib.l1attn_device_status() == 0
    returned = torch.zeros(2, dtype=torch.int32, device="cuda")
    pinned = torch.zeros(16, dtype=torch.int32).pin_memory()
    t0 = time.time()
    assert lib.l1attn_test_wait_timeout(3000, returned.data_ptr(), None) == 0
    assert lib.l1attn_device_status_async(pinned.data_ptr(), None) == 0  # the no-sync way to learn of it
    torch.cuda.synchronize()
    assert time.time() - t0 < 30.0
    assert int(returned[0]) == 1, "the kernel must come back from the wait with `false`"
    assert int(pinned[0]) == 1
    # duration of one failed poll: the hot loops poll 2^18 times before they look at the clock, which must stay
    # in the range of a second
    ns_per_poll = 3e6 / max(1, int(returned[1]))
    print("failed mbarrier.try_wait poll: %.0f ns" % ns_per_poll)
    assert ns_per_poll < 20000
    assert lib.l1attn_device_status() == -7 and b"bounded wait" in lib.l1attn_strerror(-7)
    assert lib.l1attn_device_status() == 0  # cleared by the read
    assert lib.l1attn_test_wait_timeout(0, returned.data_ptr(), None) == -1  # limits outside 1 us .. 100 ms are refused
    q, k, g = (torch.from_numpy(a).cuda() for a in _rand((1, 64, 8, 64), np.float32, 2))
    a1 = cabi.dense_fwd(q, k)
    torch.cuda.synchronize()
    assert lib.l1attn_device_status() == 0 and torch.isfinite(a1).all()


def test_driver_raises_on_a_pending_timeout():
    """The pybind driver never synchronises; it looks at the error word in pinned memory and raises at the next
    call after a kernel gave up a wait."""
    import l1attn_cuda_drv
    cabi = _cabi()
    lib = cabi.lib()
    q = torch.randn(1, 32, 8, 64, device="cuda")
    l1attn_cuda_drv.forward(q, q)
    torch.cuda.synchronize()
    l1attn_cuda_drv.forward(q, q)  # nothing pending: fine
    returned = torch.zeros(2, dtype=torch.int32, device="cuda")
    assert lib.l1attn_test_wait_timeout(2000, returned.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="bounded wait"):
        l1attn_cuda_drv.forward(q, q)
    assert lib.l1attn_device_status() == 0  # the raise cleared it
    out = l1attn_cuda_drv.forward(q, q)[0]
    torch.cuda.synchronize()
    assert torch.isfinite(out).all()


def test_a_timeout_is_reported_once():
    """Whoever learns of a timeout first clears it for everyone: the status through the C ABI, then no error from the driver."""
    import l1attn_cuda_drv
    lib = _cabi().lib()
    q = torch.randn(1, 32, 8, 64, device="cuda")
    l1attn_cuda_drv.forward(q, q)  # (the host word exists from here on)
    returned = torch.zeros(2, dtype=torch.int32, device="cuda")
    assert lib.l1attn_test_wait_timeout(2000, returned.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert lib.l1attn_device_status() == -7
    l1attn_cuda_drv.forward(q, q)
    assert lib.l1attn_device_status() == 0


def test_a_timeout_before_the_first_driver_call_is_reported():
    """In a process of its own: the wait runs out before any driver call has set the host word up."""
    import subprocess
    import sys
    code = ("import torch, l1attn_cabi, l1attn_cuda_drv\n"
            "lib, q, r = l1attn_cabi.lib(), torch.randn(1, 32, 8, 64, device='cuda'), torch.zeros(2, dtype=torch.int32, device='cuda')\n"
            "assert lib.l1attn_test_wait_timeout(2000, r.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0\n"
            "torch.cuda.synchronize()\n"
            "try:\n    l1attn_cuda_drv.forward(q, q)\nexcept RuntimeError as e:\n    assert 'bounded wait' in str(e)\nelse:\n    raise SystemExit('not reported')\n"
            "l1attn_cuda_drv.forward(q, q)\n"
            "assert lib.l1attn_device_status() == 0\n")
    subprocess.run([sys.executable, "-c", code], check=True, cwd=PKG, timeout=300)
