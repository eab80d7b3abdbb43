"""Performance cases: the calls that programs built on these operators make, as whole passes through the public modules.

Each case is a dict of plain values; `kind` says which operator it drives:

  dense    l1attn_cuda.L1Attn, scores and both gradients
  sparse   l1attn_sparse_cuda.L1AttnSparse / l1attn_sparse_bidi_cuda.L1AttnSparseBidi on a graph that is kept across
           passes, output and gradients, or (float16 / bfloat16 storage, as the operator offers it) the output alone
  graph    a graph that is new in every pass: SparseGraph (expandCoo and the edge index), attention, gradients
  fused    l1attn_fused_cuda.L1AttnSoftmaxV, output and gradients

`listed()` has the sizes of the repository's configurations and tests, `draw()` others of the same ranges.
"""
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "l1-attention_b200"))

import l1attn_cuda  # noqa: E402
import l1attn_fused_cuda  # noqa: E402
import l1attn_sparse_bidi_cuda  # noqa: E402
import l1attn_sparse_cuda  # noqa: E402

DTYPES = {"f32": torch.float32, "f64": torch.float64, "f16": torch.float16, "bf16": torch.bfloat16}
ELEMENT = {"f32": 4, "f64": 8, "f16": 2, "bf16": 2}


def dense(bs, n, h, w, dtype="f32", pad=False):
    return dict(kind="dense", bs=bs, n=n, h=h, w=w, dtype=dtype, pad=pad)


def sparse(bs, n, h, w, wv, fan, bidi=False, dtype="f32", softmax=True):
    return dict(kind="sparse", bs=bs, n=n, h=h, w=w, wv=wv, fan=fan, bidi=bidi, dtype=dtype, softmax=softmax)


def graph(bs, n, h, w, wv, fan):
    return dict(kind="graph", bs=bs, n=n, h=h, w=w, wv=wv, fan=fan, dtype="f32")


def fused(bs, n, h, w, wv, mode="softmax"):
    return dict(kind="fused", bs=bs, n=n, h=h, w=w, wv=wv, mode=mode, dtype="f32")


def listed():
    return [
        # a layer of a small model: the kernels are short, the calls around them count
        dict(dense(4, 128, 8, 64), name="dense_layer"),
        # many short sets, zero-padded to one length: padded query and key rows are equal in every column
        dict(dense(512, 16, 8, 32, pad=True), name="dense_sets"),
        # sizes off every multiple: odd token count and width (the width sweep 16 .. 128 has 33, 65 and 97), six heads
        dict(dense(48, 201, 6, 65), name="dense_odd"),
        # the configuration that the headline metric is quoted on
        dict(dense(16, 1024, 16, 64), name="dense_1024"),
        # long context
        dict(dense(2, 4096, 8, 128), name="dense_4096"),
        # float64, for checks at tight tolerances
        dict(dense(2, 512, 8, 128, dtype="f64"), name="dense_f64"),
        # one graph of 131072 edges, kept across steps
        dict(sparse(8, 4096, 8, 64, 64, 31), name="sparse_4096"),
        # a layer of the bidirectional transformer (d_model 256, 64 sequences of 256 tokens)
        dict(sparse(64, 256, 8, 32, 32, 16, bidi=True), name="sparse_bidi"),
        # inference with 16-bit storage
        dict(sparse(8, 4096, 8, 64, 64, 31, dtype="bf16"), name="sparse_bf16"),
        # another graph in every step, in-degrees of all sizes, ragged widths
        dict(graph(2, 3001, 6, 40, 24, 24), name="graph_new"),
        # dense attention without the score tensor, at the headline shape
        dict(fused(16, 1024, 16, 64, 64), name="fused_1024"),
        # the same with one more all-zero source row, at sizes off the usual multiples
        dict(fused(4, 333, 6, 48, 40, mode="softmax_plus_one"), name="fused_odd"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """One more case.  Batch sizes, token counts and edges per token over their logarithm, widths mostly of the usual
    multiples and sometimes odd; the batch shrinks until the case costs no more than the largest listed one."""
    kind = rng.choice(["dense", "dense", "dense", "sparse", "sparse", "graph", "fused"])
    h = rng.choice([1, 2, 3, 4, 5, 6, 8, 8, 8, 12, 16])
    w = rng.choice([16, 32, 32, 48, 64, 64, 64, 96, 128, rng.randint(8, 128)])
    if kind == "dense":
        c = dense(_log(rng, 1, 512), _log(rng, 16, 4096), h, w, dtype=rng.choice(["f32", "f32", "f32", "f64"]), pad=rng.random() < 0.3)
        most = 6e8 if c["dtype"] == "f64" else 8e9
        terms = c["n"] ** 2 * h * w
        c["n"] = c["n"] if terms <= most else int((most / (h * w)) ** 0.5)
    elif kind == "fused":
        wv = w if rng.random() < 0.7 else rng.choice([32, 64, 128, rng.randint(8, 128)])
        c = fused(_log(rng, 1, 64), _log(rng, 16, 2048), h, w, wv, mode=rng.choice(["softmax", "softmax", "softmax_plus_one", "exp"]))
        usual = w % 32 == 0 and wv in (32, 64, 128)
        most = 8e9 if usual else 4e8
        terms = c["n"] ** 2 * h * max(w, wv)
        c["n"] = c["n"] if terms <= most else int((most / (h * max(w, wv))) ** 0.5)
    else:
        wv = w if rng.random() < 0.7 else rng.choice([16, 32, 64, 128, rng.randint(8, 128)])
        n, fan = _log(rng, 64, 8192), _log(rng, 4, 48)
        if kind == "graph":
            c = graph(_log(rng, 1, 16), n, h, w, wv, fan)
        else:
            c = sparse(_log(rng, 1, 64), n, h, w, wv, fan, bidi=rng.random() < 0.5, dtype=rng.choice(["f32", "f32", "f32", "f64", "f16", "bf16"]),
                       softmax=rng.random() < 0.8)
        most = 4e8 if ELEMENT[c["dtype"]] < 8 else 1e8
    terms = {"dense": c["n"] ** 2, "fused": c["n"] ** 2}.get(c["kind"], c["n"] * (c.get("fan", 0) + 1)) * h * max(w, c.get("wv", 0))
    c["bs"] = max(1, min(c["bs"], int(most // max(1, terms))))
    return c


def _edges(case, gen, dev):
    """Rows (dst, src): every token's self edge and `fan` others per token, in random order.  The kept graph has `fan`
    distinct sources for every token; the graphs that come and go have in-degrees from none to twice `fan` and
    sources that are popular in different degrees."""
    n, fan = case["n"], case["fan"]
    tok = torch.arange(n, device=dev)
    if case["kind"] == "graph":
        half = torch.randint(0, 2 * fan + 1, (n // 2,), generator=gen, device=dev)
        deg = torch.cat([half, 2 * fan - half, tok.new_full((n % 2,), fan)])  # as many edges in every such graph
        dst = tok.repeat_interleave(deg)
        src = (torch.rand(dst.shape[0], generator=gen, device=dev) ** 1.5 * n).long().clamp_(max=n - 1)
    else:
        fan = min(fan, n - 1)
        dst = tok.repeat_interleave(fan)
        src = torch.rand(n, n, generator=gen, device=dev).fill_diagonal_(2).topk(fan, 1, largest=False).indices.reshape(-1)
    rows = torch.stack([torch.cat([tok, dst]), torch.cat([tok, src])], 1)
    return rows[torch.randperm(rows.shape[0], generator=gen, device=dev)]


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    bs, n, h, w = case["bs"], case["n"], case["h"], case["w"]
    wv = case.get("wv", w)

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=dev, dtype=torch.float64 if dt == torch.float64 else torch.float32).to(dt)

    st = {"case": case, "q": normal(bs, n, h, w), "k": normal(bs, n, h, w)}
    if case.get("pad"):
        length = torch.randint((n + 1) // 2, n + 1, (bs, 1), generator=gen, device=dev)
        keep = (torch.arange(n, device=dev)[None] < length)[:, :, None, None]
        st["q"], st["k"] = st["q"] * keep, st["k"] * keep
    if case["kind"] == "dense":
        st["module"], st["grad"] = l1attn_cuda.L1Attn(), normal(bs, n, n, h)
    else:
        st["v"], st["grad"] = normal(bs, n, h, wv), normal(bs, n, h, wv)
    if case["kind"] == "fused":
        st["module"] = l1attn_fused_cuda.L1AttnSoftmaxV(mode=case["mode"])
    elif case["kind"] == "graph":
        st["edges"] = _edges(case, gen, dev)
    elif case["kind"] == "sparse":
        st["module"] = l1attn_sparse_bidi_cuda.L1AttnSparseBidi() if case["bidi"] else l1attn_sparse_cuda.L1AttnSparse()
        st["coo"], st["dst_mxlen"], _ = l1attn_sparse_cuda.expandCoo(_edges(case, gen, dev))
        if case["bidi"]:
            st["vb"] = normal(bs, n, h, wv)
    if dt in (torch.float32, torch.float64):
        for name in ("q", "k", "v", "vb"):
            if name in st:
                st[name].requires_grad_(True)
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "dense":
        leaves = (st["q"], st["k"])
        out = st["module"](*leaves)
    elif case["kind"] == "fused":
        leaves = (st["q"], st["k"], st["v"])
        out = st["module"](*leaves)
    elif case["kind"] == "graph":
        leaves = (st["v"], st["q"], st["k"])
        g = l1attn_sparse_cuda.SparseGraph(st["edges"], device=st["edges"].device)
        out = g.attend(*leaves)
        return [out, *torch.autograd.grad(out, leaves, st["grad"]), g.coo, g.dst_mxlen, g.src_mxlen]
    else:
        leaves = (st["v"], st["vb"], st["q"], st["k"]) if case["bidi"] else (st["v"], st["q"], st["k"])
        out = st["module"](*leaves, st["coo"], st["dst_mxlen"], case["softmax"])
        if not out.requires_grad:
            return [out]
    return [out, *torch.autograd.grad(out, leaves, st["grad"])]


def work(case):
    """Every input read once, every output written once; an operation is an addition, a comparison or a multiplication."""
    es = ELEMENT[case["dtype"]]
    bs, n, h, w = case["bs"], case["n"], case["h"], case["w"]
    qk = bs * n * h * w
    if case["kind"] == "dense":
        pairs = bs * n * n * h
        # forward: subtract and add the absolute value; backward: compare and add to either gradient
        return {"bytes": es * (4 * qk + 2 * pairs), "flops": 5 * pairs * w}
    wv = case["wv"]
    val = bs * n * h * wv
    if case["kind"] == "fused":
        pairs = bs * n * n * h
        # scores, value product; backward: scores again, <v, dvo>, dv, both gradients of the scores
        return {"bytes": es * (4 * qk + 4 * val), "flops": pairs * ((2 + 2 + 3) * w + (2 + 2 + 2) * wv)}
    edges = n * (case["fan"] + 1)
    if case["dtype"] in ("f16", "bf16"):
        both = 2 if case["bidi"] else 1
        return {"bytes": es * (2 * qk + (1 + both) * val) + 16 * edges, "flops": bs * h * edges * (2 * w + 2 * both * wv)}
    both = 2 if case["kind"] == "sparse" and case["bidi"] else 1
    # graph: the edge list arrives as two int64 per row and leaves as four int32
    listing = 32 * edges if case["kind"] == "graph" else 16 * edges
    return {"bytes": es * (4 * qk + (2 + 2 * both) * val) + listing,
            "flops": bs * h * edges * ((2 + 4) * w + (2 + 4) * both * wv)}


def tolerance(case):
    """About four times what the operators differ by from themselves in float64 on the same values, over the listed cases
    and drawn ones (float32: 2.1e-6, at most 1.4e-5; bfloat16: 3.3e-3, at most 5.5e-2; float16: 3.1e-3 where weights are
    below its normal range, at most 1.6e-2; float64 has float32's figures times the ratio of their roundings).  Whole
    numbers (the expanded edge list) are equal."""
    if case["dtype"] == "f64":
        return {"rel": 2e-14, "max": 2e-13}
    if case["dtype"] == "bf16":
        return {"rel": 1.3e-2, "max": 2e-1}
    if case["dtype"] == "f16":
        return {"rel": 1.2e-2, "max": 6e-2}
    return {"rel": 1e-5, "max": 6e-5}


def _scores64(q, k):
    """[source, query, head] of one batch item; q, k [token, head, width] in float64."""
    step = max(1, (1 << 26) // q.numel())
    return torch.cat([(q[None] - k[s:s + step, None]).abs_().sum(-1) for s in range(0, k.shape[0], step)]) / -q.shape[-1] ** 0.5


def _gradients64(q, k, g):
    """Both gradients of _scores64 under g [source, query, head], with sign(0) = 0."""
    step = max(1, (1 << 26) // q.numel())
    dq, dk = torch.zeros_like(q), []
    for s in range(0, k.shape[0], step):
        terms = (q[None] - k[s:s + step, None]).sign_().mul_(g[s:s + step, :, :, None])
        dq += terms.sum(0)
        dk.append(terms.sum(1))
    scale = q.shape[-1] ** -0.5
    return dq * -scale, torch.cat(dk) * scale


def exact(case, seed):
    """What `run` returns for the inputs of this seed, in float64 from the definitions of the operators."""
    st = prepare(case, seed)
    q, k, v, vb, grad = (st[name].detach().double() if name in st else None for name in ("q", "k", "v", "vb", "grad"))
    bs, n = q.shape[:2]
    scale = -q.shape[-1] ** -0.5
    if case["kind"] == "dense":
        each = [(_scores64(q[b], k[b]), *_gradients64(q[b], k[b], grad[b])) for b in range(bs)]
        return [torch.stack(x) for x in zip(*each)]
    if case["kind"] == "fused":
        each = []
        for b in range(bs):
            x = _scores64(q[b], k[b])
            if case["mode"] == "softmax":
                p = x.softmax(0)
            else:
                p = x.exp()
                p = p / (1 + p.sum(0)) if case["mode"] == "softmax_plus_one" else p
            dp = torch.einsum("shc,thc->sth", v[b], grad[b])
            delta = 0 if case["mode"] == "exp" else (p * dp).sum(0)
            each.append((torch.einsum("sth,shc->thc", p, v[b]), *_gradients64(q[b], k[b], p * (dp - delta)), torch.einsum("sth,thc->shc", p, grad[b])))
        return [torch.stack(x) for x in zip(*each)]
    edges = st["edges"] if case["kind"] == "graph" else st["coo"][:, :2].long()
    dst, src = edges[:, 0], edges[:, 1]
    each = []
    for b in range(bs):
        diff = q[b][dst] - k[b][src]
        e = (diff.abs().sum(-1) * scale).exp()
        a = e / (1 + torch.zeros_like(q[b, :, :, 0]).index_add_(0, dst, e))[dst] if case.get("softmax", True) else e
        vo = torch.zeros_like(v[b]).index_add_(0, dst, a[..., None] * v[b][src])
        if case.get("bidi"):
            vo.index_add_(0, src, a[..., None] * vb[b][dst])
        if case["dtype"] in ("f16", "bf16"):
            each.append((vo,))
            continue
        da = (v[b][src] * grad[b][dst]).sum(-1)
        dv = torch.zeros_like(v[b]).index_add_(0, src, a[..., None] * grad[b][dst])
        dvb = ()
        if case.get("bidi"):
            da += (vb[b][dst] * grad[b][src]).sum(-1)
            dvb = (torch.zeros_like(v[b]).index_add_(0, dst, a[..., None] * grad[b][src]),)
        if case.get("softmax", True):
            da = da - torch.zeros_like(q[b, :, :, 0]).index_add_(0, dst, a * da)[dst]
        d = diff.sign_() * (a * da * scale)[..., None]
        each.append((vo, dv, *dvb, torch.zeros_like(q[b]).index_add_(0, dst, d), torch.zeros_like(k[b]).index_add_(0, src, -d)))
    out = [torch.stack(x) for x in zip(*each)]
    return out + [None, None, None] if case["kind"] == "graph" else out  # whole numbers: the expanded list and its lengths
