"""The fused operator's 128-row kernels with the value products on the tensor cores (csrc/dense_softmax_v.cu): ragged ends of the tiles of 128
rows, 64 keys, 32 columns and 64 value columns, rows with and without TMA, masked keys, ties, and values that are not finite.  Every
test asserts that its sizes take the kernels it is about (148 (batch, head) pairs fill the GPU with 128-row CTAs)."""
import numpy as np
import pytest
import torch

from conftest import assert_close

pytestmark = pytest.mark.gpu
SHAPES = [(65, 64, 64), (100, 33, 21), (127, 32, 32), (128, 64, 33), (200, 17, 64), (256, 64, 64), (193, 48, 40), (128, 4, 1), (128, 64, 32)]
WIDE = [(128, 96, 64), (128, 65, 7), (200, 128, 32), (128, 97, 21)]  # (wider rows: the same CTAs without the tensor cores)
MODES = ["softmax", "softmax_plus_one", "exp"]
BS, HEADS = 37, 4


def _cabi():
    import l1attn_cabi
    return l1attn_cabi


def _assert_form(n, w, wv, forward=129, backward=129):
    form = _cabi().lib().l1attn_test_softmax_v_form
    assert (form(BS, n, HEADS, w, wv, 0), form(BS, n, HEADS, w, wv, 1)) == (forward, backward)


def _inputs(n, w, wv, seed=60):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(BS, n, HEADS, x, generator=gen, device="cuda") for x in (w, w, wv, wv)]


def _run(q, k, v, g, mode):
    """vo, dq, dk, dv in float32, and the float64 kernels' on the same values"""
    import l1attn_fused_cuda
    res = []
    for dt in (torch.float32, torch.float64):
        t = [x.to(dt).requires_grad_(True) for x in (q, k, v)]
        out = l1attn_fused_cuda.L1AttnSoftmaxV(mode)(*t)
        res.append([out.detach(), *torch.autograd.grad(out, t, g.to(dt))])
    return list(zip(("vo", "dq", "dk", "dv"), *res))


def _close(x, r, tol, name):
    assert_close(x.cpu().numpy(), r.cpu().numpy(), tol, name)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n,w,wv", SHAPES + WIDE)
def test_output_and_gradients(n, w, wv, mode):
    _assert_form(n, w, wv, *((128, 128) if w > 64 else (64, 129) if max(w, wv) <= 32 else (129, 129)))  # (narrow rows: the backward alone)
    # pieces hold the operands exactly; what is left are fp32 sums and the rounding of scores of about sqrt(w), which exp() makes relative
    for name, x, r in _run(*_inputs(n, w, wv), mode):
        _close(x, r, 1e-5, name)


@pytest.mark.parametrize("n,w,wv", [(65, 64, 64), (193, 48, 40), (200, 33, 21)])
def test_score_gradients_in_the_order_of_d_attn(n, w, wv):
    """The first half of the backward alone (l1attn_dense_softmax_v_bwd_dx): dx [b][s][t][h], equal rows among them."""
    _assert_form(n, w, wv)
    q, k, v, g = _inputs(n, w, wv)
    k[:, 3:9] = q[:, 5:11]
    res = []
    for dt in (torch.float32, torch.float64):
        a = [x.to(dt) for x in (q, k, v, g)]
        lse = torch.empty(q.shape[:3], dtype=dt, device="cuda")
        vo = _cabi().dense_softmax_v_fwd(*a[:3], lse=lse)
        dx, dv = torch.full((BS, n, n, HEADS), np.nan, dtype=dt, device="cuda"), torch.empty_like(a[2])
        _cabi().dense_softmax_v_bwd_dx(*a, lse, (vo * a[3]).sum(-1), dx, dv)
        res.append((lse, dx, dv))
    for name, x, r in zip(("lse", "dx", "dv"), *res):
        _close(x, r, 1e-5, name)


@pytest.mark.parametrize("value", [-np.inf, float(np.finfo(np.float32).min)])
@pytest.mark.parametrize("n,w,wv", [(200, 64, 64), (200, 33, 21)])
def test_masked_keys_in_front(n, w, wv, value):
    """Two whole tiles of keys that are infinitely far, and two keys more: they weigh nothing and get no gradient."""
    _assert_form(n, w, wv)
    q, k, v, g = _inputs(n, w, wv)
    k[:, :130] = value
    got = [x for _, x, _ in _run(q, k, v, g, "softmax")]
    ref = [t.double().requires_grad_(True) for t in (q, k[:, 130:], v[:, 130:])]
    out = []
    for b in range(BS):
        x = -(ref[0][b][None] - ref[1][b][:, None]).abs().sum(-1) / w ** 0.5
        out.append(torch.einsum("sdh,shw->dhw", torch.softmax(x, 0), ref[2][b]))
    out = torch.stack(out)
    grads = torch.autograd.grad(out, ref, g.double())
    for name, x, r in (("vo", got[0], out.detach()), ("dq", got[1], grads[0]), ("dk", got[2][:, 130:], grads[1]), ("dv", got[3][:, 130:], grads[2])):
        _close(x, r, 1e-5, name)
    assert not got[2][:, :130].any() and not got[3][:, :130].any()


@pytest.mark.parametrize("kind", ["equal_rows", "grid"])
def test_ties(kind):
    """Equal rows (their score has no slope) and ties everywhere, against torch's own chain in float64, whose |x| has slope 0 at 0."""
    n, w, wv = 100, 32, 40
    _assert_form(n, w, wv)
    q, k, v, g = _inputs(n, w, wv)
    if kind == "equal_rows":
        k[:, 3:9] = q[:, 5:11]
    else:
        q, k = (q * 4).round() / 4, (k * 4).round() / 4
    got = [x for _, x, _ in _run(q, k, v, g, "softmax")]
    for b in (0, 36):
        ref = [t[b].double().requires_grad_(True) for t in (q, k, v)]
        x = -(ref[0][None] - ref[1][:, None]).abs().sum(-1) / w ** 0.5
        out = torch.einsum("sdh,shw->dhw", torch.softmax(x, 0), ref[2])
        for name, x, r in zip(("vo", "dq", "dk", "dv"), got, (out.detach(), *torch.autograd.grad(out, ref, g[b].double()))):
            _close(x[b], r, 1e-5, name)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("where", ["v", "dvo", "both"])
@pytest.mark.parametrize("n,w,wv,bad", [(128, 64, 64, np.inf), (128, 64, 64, np.nan), (200, 33, 21, -np.inf), (193, 48, 32, np.inf)])
def test_values_that_are_not_finite(n, w, wv, bad, where, mode):
    """A value that is not finite has no pieces: what it reaches is what float64 says, of the same sign, and the others are as ever."""
    _assert_form(n, w, wv)
    q, k, v, g = _inputs(n, w, wv)
    if where != "dvo":
        v[3, n - 2, 2, 5] = bad
    if where != "v":
        g[5, 70, 1, wv - 1] = bad
    hit = torch.zeros(BS, 1, HEADS, 1, dtype=torch.bool, device="cuda")
    hit[3, 0, 2, 0], hit[5, 0, 1, 0] = where != "dvo", where != "v"
    for name, x, r in _run(q, k, v, g, mode):
        assert torch.isfinite(x[~hit.expand_as(x)]).all(), name
        assert torch.equal(x.isnan(), r.isnan()) and torch.equal(x.isposinf(), r.isposinf()) and torch.equal(x.isneginf(), r.isneginf()), name
        fine = x.isfinite()
        _close(x[fine], r[fine], 1e-5, name)


def _time(f):
    ends = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        ends.append(a.elapsed_time(b))
    return sorted(ends)[3]


def test_values_that_are_not_finite_cost_little():
    """One such value in every head's v and dvo: only its tiles pay, not the whole head (measured 1.0 to 1.3 times; a plain recomputation: 10 to 40)."""
    n, w, wv = 256, 64, 64
    _assert_form(n, w, wv)
    q, k, v, g = _inputs(n, w, wv)
    lse = torch.empty(q.shape[:3], device="cuda")
    vo = _cabi().dense_softmax_v_fwd(q, k, v, lse=lse)
    delta, dx, dv = (vo * g).sum(-1), torch.empty(BS, n, n, HEADS, device="cuda"), torch.empty_like(v)
    took = []
    for bad in (0.0, np.inf):
        v[:, 5, :, 3] += bad
        g[:, 70, :, 2] += bad
        took.append((_time(lambda: _cabi().dense_softmax_v_fwd(q, k, v, out=vo)), _time(lambda: _cabi().dense_softmax_v_bwd_dx(q, k, v, g, lse, delta, dx, dv))))
    assert took[1][0] < 3 * took[0][0] and took[1][1] < 3 * took[0][1], took


@pytest.mark.parametrize("n,w,wv", [(65, 64, 64), (200, 33, 21)])
def test_small_values(n, w, wv):
    """Values and gradients down to the smallest normal floats keep their 24 bits in the products (what is left are the roundings of scores and of
    subnormal outputs): v and dvo at 2^-119 one at a time, so that <v, dvo> does not leave the range."""
    _assert_form(n, w, wv)
    for i in (2, 3):
        t = _inputs(n, w, wv)
        t[i] *= 2.0 ** -119
        for name, x, r in _run(*t, "softmax"):
            _close(x, r, 1e-5, name)


@pytest.mark.parametrize("mode", ["softmax_plus_one", "exp"])
def test_small_weights(mode):
    """Scores of -84, unshifted: weights of 2^-121 keep their 24 bits.  q and k on a grid of 1/4 and a width of 64: scores without rounding, so the
    bound is that of exp() and of the sums alone."""
    n, w, wv = 100, 64, 64
    _assert_form(n, w, wv)
    q, k, v, g = _inputs(n, w, wv)
    q, k = (q.clamp(-3, 3) * 4).round() / 4, (k.clamp(-3, 3) * 4).round() / 4 + 10.5
    for name, x, r in _run(q, k, v, g, mode):
        if name in ("vo", "dv"):
            _close(x, r, 1e-6, name)


@pytest.mark.parametrize("mode", MODES)
def test_large_values(mode):
    """Values up to 1e36 beside ordinary ones stay in range, and each column keeps its precision."""
    n, w, wv = 128, 48, 40
    _assert_form(n, w, wv)
    q, k, v, g = _inputs(n, w, wv)
    v[..., 3] *= 1e36
    v[:, 5, :, 7] *= 1e20
    g[..., 3] = 0
    for name, x, r in _run(q, k, v, g, mode):
        for c in range(wv if name in ("vo", "dv") else 0):
            _close(x[..., c], r[..., c], 1e-5, (name, c))
        _close(x, r, 1e-5, name)


@pytest.mark.parametrize("n", [65, 128, 256])
def test_sums_of_one_sign(n):
    """The tensor core adds by truncation.  Of values of one sign the sums must not come out systematically small: on scores without rounding the
    mean relative error stays within half of what one truncated sum per tile gives (2^-24 x 3/4 or so, 4.5e-8)."""
    w, wv = 64, 64
    _assert_form(n, w, wv)
    q, k, v, g = _inputs(n, w, wv)
    q, k, v, g = (q * 4).round() / 4, (k * 4).round() / 4, v.abs() + 0.01, g.abs() + 0.01
    res = []
    for dt in (torch.float32, torch.float64):
        a = [x.to(dt) for x in (q, k, v, g)]
        lse = torch.empty(q.shape[:3], dtype=dt, device="cuda")
        vo = _cabi().dense_softmax_v_fwd(*a[:3], "exp", lse=lse)
        dx, dv = torch.empty((BS, n, n, HEADS), dtype=dt, device="cuda"), torch.empty_like(a[2])
        _cabi().dense_softmax_v_bwd_dx(*a, lse, torch.zeros_like(lse), dx, dv)
        res.append((vo, dx, dv))
    for name, x, r in zip(("vo", "dx", "dv"), *res):
        bias = float(((x.double() - r) / r).mean())
        assert abs(bias) < 2.25e-8, (name, bias)


def test_wait_that_counts_polls_gives_up_and_is_reported():
    """The wait of these kernels is bounded by its polls: 500 of them on a barrier that nothing completes, then the kernel returns and the
    status reports a timeout, once.  More polls than a hundred thousand are refused."""
    lib = _cabi().lib()
    torch.cuda.synchronize()
    assert lib.l1attn_device_status() == 0
    returned = torch.zeros(2, dtype=torch.int32, device="cuda")
    assert lib.l1attn_test_wait_polls(500, returned.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert returned.tolist() == [1, 500]
    assert lib.l1attn_device_status() == -7 and lib.l1attn_device_status() == 0
    assert lib.l1attn_test_wait_polls(0, returned.data_ptr(), None) == lib.l1attn_test_wait_polls(100001, returned.data_ptr(), None) == -1
