"""QuantLinear.forward's native path (PackedForward): the same answers as the general path, and the general path again
whenever the module's buffers are no longer those its copies were made from.  Decode attention at the edges of its sweep."""
import math
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def packed(K, N, bits, G, seed, bias=False, C=None):
    from cherryq_b200 import QuantLinear
    g = torch.Generator(device="cuda").manual_seed(seed)
    C = math.ceil(K / 64) // 8 * 8 if C is None else C
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.02).half()
    idx = torch.randperm(K, device="cuda", generator=g)[:C].int()
    b = torch.randn(N, device="cuda", generator=g).half() if bias else None
    lin = QuantLinear(bits, G, None, C / K, K, N, bias=bias).cuda()
    lin.pack(SimpleNamespace(weight=w, bias=b, cherry_indices=idx, group_size=G))
    return lin


def check(lin, x, dense, bias=None):
    ref = x.float() @ dense.float().T + (bias.float() if bias is not None else 0)
    y = lin(x)
    assert y.dtype == x.dtype and y.shape == x.shape[:-1] + (dense.shape[0],)
    assert float((y.float() - ref).abs().max() / ref.abs().max()) <= 2e-3         # fp16 output, as in the parity tests


@pytest.mark.parametrize("bits,bias", [(4, False), (3, True)])
def test_forward_follows_the_buffers(bits, bias):
    lin = packed(1024, 264, bits, 128, 1, bias)
    dense = lin.unpack()
    for shape in ((1024,), (1, 1024), (2, 3, 1024), (9, 1024), (40, 1024), (300, 1024)):
        x = torch.randn(shape, device="cuda").half()
        for _ in range(2):                                     # general path, then the native one
            check(lin, x, dense, lin.bias)
    assert lin._fast is not None
    x = torch.randn(2, 40, 1024, device="cuda").half()
    check(lin, x.transpose(0, 1), dense, lin.bias)             # not contiguous
    check(lin, x.float(), dense, lin.bias)                     # another type
    with pytest.raises(RuntimeError):
        lin(torch.randn(3, 1016, device="cuda").half())
    other = packed(1024, 264, bits, 128, 2, bias)
    for name in ("qweight", "scales", "cherry_weight", "cherry_indices"):
        setattr(lin, name, getattr(lin, name).clone())         # replaced, with tensors that keep a version
    check(lin, torch.randn(40, 1024, device="cuda").half(), dense, lin.bias)
    for name in ("qweight", "scales", "cherry_weight", "cherry_indices"):
        getattr(lin, name).copy_(getattr(other, name))         # written in place
    for m in (3, 40):
        check(lin, torch.randn(m, 1024, device="cuda").half(), other.unpack(), lin.bias)
    third = packed(1024, 264, bits, 128, 3, bias)
    lin.load_state_dict(third.state_dict())
    dense = third.unpack()
    for m in (3, 40):
        check(lin, torch.randn(m, 1024, device="cuda").half(), dense, lin.bias)
    lin.release_reference_buffers()
    for m in (3, 40, 3, 40):
        check(lin, torch.randn(m, 1024, device="cuda").half(), dense, lin.bias)
    lin.restore_reference_buffers()
    for m in (3, 40):
        check(lin, torch.randn(m, 1024, device="cuda").half(), dense, lin.bias)
    y = lin(torch.randn(3, 1024, device="cuda").half().requires_grad_())
    assert not y.requires_grad


def test_row_limits():
    import cherryq_b200
    limit = cherryq_b200.load_quant_cuda().RowLayer.row_limit
    for args, rows in (((4, 4096, 4096, 16, 128), 8), ((3, 8192, 28672, 32, 128), 8), ((4, 11008, 4096, 40, 128), 4),
                       ((3, 28672, 8192, 112, 128), 6), ((4, 28672, 8192, 112, 128), 4), ((3, 16384, 8192, 64, 128), 4),
                       ((3, 16384, 16384, 64, 128), 6), ((4, 4096, 4096, 256, 128), 0), ((4, 4096, 4096, 16, 64), 0)):
        assert limit(*args) == rows, args


@pytest.mark.parametrize("K,C", [(2048, 16), (9216, 40), (2048, 256)])     # row kernel, the same split along K, stream matvec
def test_kernel_does_not_depend_on_earlier_calls(K, C):
    """A prompt first, then decode batches: the bits of a layer that never saw the prompt, through every entry point."""
    from cherryq_b200.qlinear import forward_shared_input
    x = torch.randn(40, K, device="cuda").half()
    up = torch.randn(40, K, device="cuda").half()
    old = [packed(K, 264, 4, 128, s, C=C) for s in (1, 2)]
    for lin in old:
        lin(x)
        lin(x)
    limit = old[0]._row_limit()
    assert limit == {16: 8, 40: 4, 256: 0}[C]
    for m in (1, 2, 4, 5, 7, 8, 9, 16, 40):
        new = [packed(K, 264, 4, 128, s, C=C) for s in (1, 2)]
        ref = [lin(x[:m]) for lin in new]
        assert (new[0]._row is not None) == (m <= limit) and (new[0]._tile is not None) == (m > limit and m >= (1 if limit else 8))
        for _ in range(2):
            assert all(torch.equal(lin(x[:m]), r) for lin, r in zip(old, ref))
        assert all(torch.equal(a, b) for a, b in zip(forward_shared_input(old, x[:m]), ref))
        assert torch.equal(old[0].forward_swiglu(x[:m], up[:m]), new[0].forward_swiglu(x[:m], up[:m]))


@pytest.mark.parametrize("K,bits,G", [(2048, 4, 128), (1032, 3, 64), (9216, 3, 128)])      # whole rows, a ragged group, split along K
@pytest.mark.parametrize("m,with_delta", [(1, True), (1, False), (4, True), (5, True)])
def test_norm_in_front_of_a_shared_input(K, bits, G, m, with_delta):
    """The norm kernel and the layers' own forward against both in one launch (up to four rows)."""
    import cherryq_b200
    from cherryq_b200.qlinear import forward_normed_input
    qc = cherryq_b200.load_quant_cuda()
    lins = [packed(K, n, bits, G, s) for s, n in ((1, 264), (2, 520))]
    h = torch.randn(m, K, device="cuda").half() * 3
    delta = torch.randn(m, K, device="cuda").half() if with_delta else None
    w = (torch.randn(K, device="cuda") * 0.1 + 1).half()
    outs, total = forward_normed_input(lins, h, delta, w, 1e-5)
    if with_delta:
        y, want = qc.rmsnorm(h, delta, w, 1e-5, True)
    else:
        y, want = qc.rmsnorm(h, None, w, 1e-5, False)[0], h
    assert torch.equal(total, want)
    for lin, out in zip(lins, outs):
        ref = lin(y).float()
        # the sum of squares is added in another order: a few of the norm's values move by one fp16 step
        assert float((out.float() - ref).norm()) <= 3e-4 * float(ref.norm()) and out.shape == (m, lin.out_features)


@pytest.mark.parametrize("K,bits,G", [(2048, 4, 128), (1032, 3, 64), (9216, 3, 128)])
@pytest.mark.parametrize("m", [1, 2, 3, 4])
def test_row_kernel_with_the_norm_in_front(K, bits, G, m):
    """The operator itself, for all the rows that it takes."""
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()
    lins = [packed(K, n, bits, G, s) for s, n in ((1, 264), (2, 520))]
    h, delta = torch.randn(m, K, device="cuda").half() * 3, torch.randn(m, K, device="cuda").half()
    w = (torch.randn(K, device="cuda") * 0.1 + 1).half()
    buf = torch.empty(m, 784, dtype=torch.float16, device="cuda")
    outs = list(buf.split([264, 520], dim=1))
    total = qc.row_layers_matvec_norm([l.row_layer(m) for l in lins], h, delta, w, 1e-5, outs)
    y, want = qc.rmsnorm(h, delta, w, 1e-5, True)
    assert torch.equal(total, want)
    for lin, out in zip(lins, outs):
        ref = lin(y).float()
        assert float((out.float() - ref).norm()) <= 3e-4 * float(ref.norm())           # as in test_norm_in_front_of_a_shared_input


@pytest.mark.parametrize("bits,G", [(4, 128), (3, 64)])
@pytest.mark.parametrize("shape", [(9,), (2, 16), (33,)])
def test_shared_input_beyond_the_row_kernel(bits, G, shape):
    """One launch of the GEMM for the layers equals their own forward, bias included; a hook is still called."""
    from cherryq_b200.qlinear import forward_shared_input
    K = 1032
    lins = [packed(K, N, bits, G, N + i, i == 1, 16) for i, N in enumerate((520, 136, 136))]
    x = torch.randn(*shape, K, device="cuda").half()
    want = [l(x) for l in lins]
    got = forward_shared_input(lins, x)
    assert all(a.shape == b.shape and torch.equal(a, b) for a, b in zip(got, want))
    seen = []
    handle = lins[2].register_forward_hook(lambda m, a, o: seen.append(o))
    got = forward_shared_input(lins, x)
    handle.remove()
    assert len(seen) == 1 and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("m", [9, 32])
def test_shared_input_keeps_a_forward_set_on_the_instance(m):
    from cherryq_b200.qlinear import forward_shared_input
    lins = [packed(1032, N, 4, 128, N, False, 16) for N in (520, 136)]
    x = torch.randn(m, 1032, device="cuda").half()
    want = [lins[0](x), lins[1](x) + 1]
    own = lins[1].forward
    lins[1].forward = lambda x: own(x) + 1
    assert all(torch.equal(a, b) for a, b in zip(forward_shared_input(lins, x), want))


@pytest.mark.parametrize("m,C", [(9, 16), (40, 16), (3, 256)])
def test_swiglu_beyond_the_row_kernel_is_the_torch_expression(m, C):
    """Rows above the row kernel's limit and layers it does not take: silu in fp32, not the fast exponential.  Every fp16
    gate value, infinities and NaN among them."""
    lin = packed(2048, 264, 4, 128, 3, C=C)
    gate = torch.arange(65536, device="cuda").to(torch.int16).view(torch.float16)
    act = torch.nn.functional.silu(gate.float()).half() * torch.ones_like(gate)
    import cherryq_b200
    got = cherryq_b200.load_quant_cuda().silu_mul(gate, torch.ones_like(gate), True)
    assert torch.equal(got.isnan(), act.isnan()) and torch.equal(got.nan_to_num(7.0), act.nan_to_num(7.0))
    gate, up = (torch.randn(m, 2048, device="cuda").half() * 3 for _ in range(2))
    assert torch.equal(lin.forward_swiglu(gate, up), lin(torch.nn.functional.silu(gate.float()).half() * up))


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("H,KV,max_seq,at", [(4, 4, 2300, (0, 255, 256, 2299)), (8, 2, 600, (1, 511, 512, 599)), (3, 3, 40, (0, 7, 38, 39))])
def test_attention_sweep_edges(D, H, KV, max_seq, at):
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()
    g = torch.Generator(device="cuda").manual_seed(D + H)
    B = len(at)
    q = torch.randn(B, H, D, device="cuda", generator=g).half()
    k, v = (torch.randn(B, max_seq, KV, D, device="cuda", generator=g).half() for _ in range(2))
    for b, p in enumerate(at):                                 # nothing past the position takes part
        k[b, p + 1:] = float("nan")
        v[b, p + 1:] = float("nan")
    pos = torch.tensor(at, device="cuda")
    out = qc.attn_decode(q, k, v, pos).view(B, H, D)
    for b, p in enumerate(at):
        kk = k[b, :p + 1].float().repeat_interleave(H // KV, dim=1)
        vv = v[b, :p + 1].float().repeat_interleave(H // KV, dim=1)
        s = torch.einsum("hd,phd->hp", q[b].float(), kk) / math.sqrt(D)
        ref = torch.einsum("hp,phd->hd", s.softmax(-1), vv)
        assert float((out[b].float() - ref).abs().max()) <= 4e-3     # fp16 output of values near 1, fast exponentials


@pytest.mark.parametrize("H,KV", [(4, 4), (8, 2)])
@pytest.mark.parametrize("D,max_seq,at,bad", [(128, 300, 5, 3), (64, 300, 299, 299), (256, 300, 0, 0), (128, 700, 699, 300), (32, 300, 5, 3)])
def test_attention_keeps_nan_scores(D, H, KV, max_seq, at, bad):
    """A key of NaN makes its head's output NaN, as a softmax does, wherever it falls among the lanes and ranges; one of
    -infinity has no weight."""
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()
    q = torch.rand(1, H, D, device="cuda").half() + 0.1
    k, v = (torch.randn(1, max_seq, KV, D, device="cuda").half() for _ in range(2))
    pos = torch.tensor([at], device="cuda")
    k[0, bad, 0] = float("nan")
    out = qc.attn_decode(q, k, v, pos).view(H, D)
    assert out[:H // KV].isnan().all() and out[H // KV:].isfinite().all()
    if at:
        k[0, bad, 0] = float("-inf")
        out = qc.attn_decode(q, k, v, pos).view(H, D)
        keep = [p for p in range(at + 1) if p != bad]
        s = torch.einsum("hd,pd->hp", q[0, :H // KV].float(), k[0, keep, 0].float()) / math.sqrt(D)
        ref = s.softmax(-1) @ v[0, keep, 0].float()
        assert float((out[:H // KV].float() - ref).abs().max()) <= 4e-3


def test_attention_calls_of_different_sizes_share_a_workspace():
    """Many heads after few: what the earlier calls left in the workspace is not taken for counters.  Also a call that is
    first made under capture, and a graph that is replayed after the workspace has grown."""
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()

    def case(B, H, D, max_seq, at):
        g = torch.Generator(device="cuda").manual_seed(B + H + D)
        q = torch.randn(B, H, D, device="cuda", generator=g).half()
        k, v = (torch.randn(B, max_seq, H, D, device="cuda", generator=g).half() for _ in range(2))
        s = torch.einsum("bhd,bphd->bhp", q.float(), k[:, :at + 1].float()) / math.sqrt(D)
        ref = torch.einsum("bhp,bphd->bhd", s.softmax(-1), v[:, :at + 1].float()).half()
        return (q, k, v, torch.full((B,), at, device="cuda")), ref

    def right(out, ref):
        assert float((out.view_as(ref) - ref).abs().max()) <= 4e-3         # as in test_attention_sweep_edges

    first, ref_first = case(1, 8, 128, 1024, 1000)
    qc.attn_decode(*first)
    stream = torch.cuda.Stream()
    graph, inner = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    late, ref_late = case(7, 40, 64, 4096, 4000)
    with torch.cuda.stream(stream):
        stream.wait_stream(torch.cuda.default_stream())
        with torch.cuda.graph(graph, stream=stream):
            out_first = qc.attn_decode(*first)
        with torch.cuda.graph(inner, stream=stream):
            out_late = qc.attn_decode(*late)
    torch.cuda.synchronize()
    for B, H, D, max_seq, at in ((1, 40, 128, 4096, 4000), (4, 40, 128, 512, 300), (8, 16, 64, 1024, 1000), (2, 8, 256, 700, 650),
                                 (8, 32, 64, 600, 599), (3, 5, 32, 2000, 1999)):
        args, ref = case(B, H, D, max_seq, at)
        for _ in range(2):
            right(qc.attn_decode(*args), ref)
        for gr, out, want in ((graph, out_first, ref_first), (inner, out_late, ref_late)):
            out.fill_(float("nan"))
            gr.replay()
            right(out, want)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,max_seq", [(1, 37, 1024), (1, 38, 1024), (4, 16, 2300), (8, 32, 512), (16, 37, 1024), (20, 37, 1024),
                                         (21, 36, 1030)])
def test_attention_on_both_sides_of_the_dispatch(D, B, H, max_seq):
    """Heads up to and beyond a CTA per SM, four and five CTAs per SM (148 SMs), at the first and last positions."""
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()
    g = torch.Generator(device="cuda").manual_seed(H)
    q = torch.randn(B, H, D, device="cuda", generator=g).half()
    k, v = (torch.randn(B, max_seq, H, D, device="cuda", generator=g).half() for _ in range(2))
    at = [0, max_seq - 1, 255, 256, max_seq // 2]
    pos = torch.tensor([at[b % 5] for b in range(B)], device="cuda")
    for p in (pos, torch.full_like(pos, max_seq - 1)):
        out = qc.attn_decode(q, k, v, p).view(B, H, D)
        for b in {0, 1 % B, 2 % B, B - 1}:
            n = int(p[b]) + 1
            s = torch.einsum("hd,phd->hp", q[b].float(), k[b, :n].float()) / math.sqrt(D)
            ref = torch.einsum("hp,phd->hd", s.softmax(-1), v[b, :n].float())
            assert float((out[b].float() - ref).abs().max()) <= 4e-3         # as in test_attention_sweep_edges


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,KV,max_seq", [(5, 8, 1, 193), (5, 6, 2, 700), (20, 64, 8, 400), (1, 64, 8, 4100), (5, 40, 40, 300),
                                            (9, 50, 50, 500)])
def test_attention_on_tensor_cores(D, B, H, KV, max_seq):
    """Turns of 16 positions a warp (64 and 192 a CTA), one to eight heads per KV head, one and several ranges, CTAs of 4 and
    12 warps.  Weights beside the largest that an 11-bit weight would lose, and infinite values: of weight 0 and not."""
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()
    g = torch.Generator(device="cuda").manual_seed(H + max_seq)
    G = H // KV
    q = torch.randn(B, H, D, device="cuda", generator=g).half()
    k, v = (torch.randn(B, max_seq, KV, D, device="cuda", generator=g).half() for _ in range(2))
    at = [0, 15, 16, 63, 64, 191, 192, max_seq - 1, max_seq // 2]
    pos = torch.tensor([min(at[b % 9], max_seq - 1) for b in range(B)], device="cuda")
    v[:, 1:, 0] *= 0.02
    v[:, 0, 0] = 300.                                           # one large value: the others show in the last bits
    k[:, 0, 0] *= 0.5

    def reference(b, vv):
        n = int(pos[b]) + 1
        s = torch.einsum("gd,pd->gp", q[b, :G].double(), k[b, :n, 0].double()) / math.sqrt(D)
        return s.softmax(-1) @ vv[b, :n, 0].double()
    out = qc.attn_decode(q, k, v, pos).view(B, H, D)
    for b in range(B):
        ref = reference(b, v)
        # half an fp16 step of the result, and 2^-16 for the exponentials and fp32 sums
        assert bool(((out[b, :G].double() - ref).abs() <= (2.0 ** -11 + 2.0 ** -16) * ref.abs() + 1e-6).all())
    v[:, 0, 0, 1], v[:, 0, 0, 2] = float("inf"), float("-inf")
    out = qc.attn_decode(q, k, v, pos).view(B, H, D)
    assert bool((out[:, :G, 1] == float("inf")).all() and (out[:, :G, 2] == float("-inf")).all())
    assert bool(out[:, :G, 3:].isfinite().all() and out[:, :G, 0].isfinite().all() and out[:, G:].isfinite().all())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,KV,n", [(1, 32, 32, 40), (1, 32, 32, 300), (2, 8, 1, 193), (1, 8, 8, 1100), (20, 64, 8, 400)])
def test_attention_keeps_nan_where_the_weights_are_zero(D, B, H, KV, n):
    """One position takes all the weight (2^-400 is left for each other one).  Zero times a NaN or infinite value is NaN, a NaN score
    makes its head NaN: of positions in the same turn, in other warps and in other ranges."""
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()
    g = torch.Generator(device="cuda").manual_seed(n)
    q = torch.randn(B, H, D, device="cuda", generator=g).half() * 0.1
    k, v = (torch.randn(B, n, KV, D, device="cuda", generator=g).half() * 0.1 for _ in range(2))
    q[:, :, 0] = 60
    k[:, :, :, 0] = 0
    at = torch.full((B,), n - 1, device="cuda")
    for top in (0, n - 1):
        keys = k.clone()
        keys[:, top, :, 0] = 60                                     # score 3600 / sqrt(D)
        for other in (1, 9, n // 2, n - 2):
            values = v.clone()
            values[:, other, 0, 1], values[:, other, 0, 2] = float("nan"), float("inf")
            out = qc.attn_decode(q, keys, values, at).view(B, KV, H // KV, D)
            assert bool(out[:, 0, :, 1:3].isnan().all() and out[:, 0, :, 3:].isfinite().all() and out[:, 1:].isfinite().all())
            bad = keys.clone()
            bad[:, other, 0, 5] = float("nan")
            out = qc.attn_decode(q, bad, v, at).view(B, KV, H // KV, D)
            assert bool(out[:, 0].isnan().all() and out[:, 1:].isfinite().all())


@pytest.mark.parametrize("H,KV", [(32, 32), (64, 8)])
@pytest.mark.parametrize("B,n", [(4, 1100), (2, 4096)])
def test_attention_is_as_exact_as_fp32_sums(H, KV, B, n):
    """Outputs that are not the correctly rounded ones, of peaked scores (deviation 4): an error of e before the last rounding
    turns a share of about e / 2^-10.5 of the fp16 results.  fp32 sums leave 1e-6 (scores of up to 20, each rounded a few
    times by 2^-24 of itself), which is 1.5e-3 of the outputs, give or take 1e-4 at these numbers; bound 2e-3.  (Sums left to
    the tensor cores, which cut off: 2.1e-3 to 3.4e-3.)"""
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()
    D, G, wrong, total = 128, H // KV, 0, 0
    g = torch.Generator(device="cuda").manual_seed(H + n)
    for _ in range(12):
        q = (torch.randn(B, H, D, device="cuda", generator=g) * 4).half()
        k, v = (torch.randn(B, n, KV, D, device="cuda", generator=g).half() for _ in range(2))
        v += 0.5
        out = qc.attn_decode(q, k, v, torch.full((B,), n - 1, device="cuda")).view(B, KV, G, D)
        for b in range(B):
            s = torch.einsum("hgd,phd->hgp", q[b].view(KV, G, D).double(), k[b].double()) / math.sqrt(D)
            ref = torch.einsum("hgp,phd->hgd", s.softmax(-1), v[b].double())
            wrong += int((out[b] != ref.half()).sum())
            total += ref.numel()
    assert wrong <= 2e-3 * total


@pytest.mark.parametrize("B,H,KV,D,max_seq", [(3, 4, 4, 128, 40), (2, 8, 1, 64, 700), (17, 64, 8, 128, 400), (2, 8, 2, 256, 40), (3, 6, 6, 32, 300)])
def test_attention_step_is_rotation_cache_write_and_attention(B, H, KV, D, max_seq):
    """One launch and the two kernels, at the first and last positions of ranges and caches and at positions outside, which
    read and write nothing of the new token."""
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()
    g = torch.Generator(device="cuda").manual_seed(B + D)
    at = [0, max_seq - 1, 15, 16, -1, max_seq, 63, 64]
    pos = torch.tensor([at[b % 8] for b in range(B)], device="cuda")
    q = torch.randn(B, H, D, device="cuda", generator=g).half()
    k, v = (torch.randn(B, KV, D, device="cuda", generator=g).half() for _ in range(2))
    caches = [torch.randn(B, max_seq, KV, D, device="cuda", generator=g).half() for _ in range(2)]
    ang = torch.outer(torch.arange(max_seq, device="cuda", dtype=torch.float32), torch.rand(D // 2, device="cuda", generator=g))
    cos, sin = ang.cos(), ang.sin()
    q1, k1, mine = q.clone(), k.clone(), [c.clone() for c in caches]
    out = qc.attn_decode_step(q1, k1, v, cos, sin, pos, *mine)
    qc.rope_cache(q, k, v, cos, sin, pos, *caches)
    want = qc.attn_decode(q, caches[0], caches[1], pos)
    assert torch.equal(mine[1], caches[1])
    # (a rotation may contract its products otherwise: one step of fp16)
    assert float((mine[0].float() - caches[0].float()).abs().max()) <= 4e-3
    changed = (mine[0] != caches[0]).any(-1).any(-1)
    assert int(changed.sum()) <= B and not bool(changed[pos < 0].any()) and not bool(changed[pos >= max_seq].any())
    assert float((out.float() - want.float()).abs().max()) <= 4e-3           # as in test_attention_sweep_edges


@pytest.mark.parametrize("m,C", [(1, 16), (40, 16), (3, 256)])     # row kernel, GEMM, stream matvec
def test_copies_dropped_while_another_stream_uses_them(m, C):
    """The block of a dropped copy is not given out before the launches that read it have finished, and is afterwards."""
    lin = packed(2048, 520, 4, 128, 1, C=C)
    x = torch.randn(m, 2048, device="cuda").half()
    want = lin(x)
    blob = (lin._row or lin._tile or lin._prepared).blob
    ptr, size = blob.data_ptr(), blob.numel()
    del blob
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(400_000_000)                             # about 0.2 s
        y = lin(x)
    lin._drop_copies()
    held = [torch.empty(size, dtype=torch.uint8, device="cuda").fill_(0xFF) for _ in range(4)]
    assert not side.query(), "the test must look while the launch is pending"
    assert all(t.data_ptr() != ptr for t in held)
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    del held
    torch.cuda.empty_cache()
    later = [torch.empty(size, dtype=torch.uint8, device="cuda") for _ in range(8)]
    assert len(later) == 8 and torch.equal(lin(x), want)


@pytest.mark.parametrize("m,C", [(1, 16), (40, 16), (3, 256)])
def test_first_call_is_refused_under_capture(m, C):
    """A captured re-pack would run with the graph only; the refusal leaves the capture and the layer usable."""
    lin = packed(2048, 264, 4, 128, 2, C=C)
    x = torch.randn(m, 2048, device="cuda").half()
    dense = lin.unpack()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        z = x + 1
        with pytest.raises(RuntimeError, match="before the capture"):
            lin(x)
    graph.replay()
    assert torch.equal(z, x + 1)
    check(lin, x, dense)
    with torch.cuda.graph(graph := torch.cuda.CUDAGraph()):
        y = lin(x)
    graph.replay()
    assert torch.equal(y, lin(x))


@pytest.mark.parametrize("m,C", [(1, 16), (40, 16), (3, 256)])     # row kernel, GEMM, stream matvec
@pytest.mark.parametrize("name", ["qweight", "scales", "cherry_weight"])
def test_buffers_of_the_wrong_size_are_refused(m, C, name):
    lin = packed(2048, 264, 4, 128, 3, C=C)
    setattr(lin, name, getattr(lin, name)[:-2].clone())
    with pytest.raises(RuntimeError, match=name):
        lin(torch.zeros(m, 2048, device="cuda").half())


@pytest.mark.parametrize("m", [1, 40])
def test_forward_of_modules_with_parameters_and_of_copies(m):
    """A reference buffer turned into a parameter, a deep copy made after a call: the same answers."""
    import copy
    lin = packed(1024, 264, 4, 128, 4)
    x = torch.randn(m, 1024, device="cuda").half()
    want = lin(x)
    other = copy.deepcopy(lin)
    assert torch.equal(other(x), want) and torch.equal(other(x), want)
    lin.qweight = torch.nn.Parameter(lin.qweight.clone(), requires_grad=False)
    for _ in range(3):
        assert torch.equal(lin(x), want)
    lin.qweight = torch.nn.Parameter(torch.zeros_like(lin.qweight), requires_grad=False)
    assert not torch.equal(lin(x), want)
