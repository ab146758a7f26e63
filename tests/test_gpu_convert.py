"""The one-pass conversion kernels against the numpy oracle and the torch expressions they replace, byte for byte, at the
edges of their tiles: rows that are not a multiple of 64, columns that are not a multiple of 128, groups of one chunk, of
several and of a whole row, octets with cherry columns and group boundaries inside."""
import numpy as np
import pytest

from oracle import cherryq_oracle as O
from test_gpu_parity import dev, gpu_pack, gpu_unpack, ptr

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cabi():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cherryq_b200 import _cabi
    _cabi.lib()
    return _cabi


def layer(K, N, C, dtype, seed):
    rng = np.random.default_rng(seed)
    w = (rng.normal(size=(N, K)) * 0.02).astype(dtype)
    idx = rng.permutation(K)[:C]
    if C:
        idx[:min(C, 8)] = np.arange(min(C, 8)) + 8                 # a whole octet of cherries
        idx = np.unique(idx)
        idx = np.concatenate([idx, np.setdiff1d(np.arange(K), idx)[:C - len(idx)]])
        w[:, idx] = (rng.normal(size=(N, C)) * 0.2).astype(dtype)
        idx = rng.permutation(idx)
    w[0] = 0                                                       # the smallest scale
    w[1] = np.asarray(0.5 * np.sign(w[1].astype(np.float32) + 1e-9), dtype)     # quotients on the code boundaries
    w[2, ::3] = np.asarray(6e-8, dtype)                            # subnormal in fp16
    w[3] *= np.asarray(1000, dtype)
    return w, idx


@pytest.mark.parametrize("dtype", [np.float16, np.float32])
@pytest.mark.parametrize("K,N,bits,G,C", [
    (8, 8, 4, 128, 0), (136, 72, 3, 64, 8), (1024, 64, 4, 128, 8), (1032, 136, 3, 128, 16), (1040, 56, 4, 256, 24),
    (2048, 200, 3, 2048, 8), (512, 64, 4, 96, 16), (4096, 128, 3, 64, 128), (640, 8, 4, 640, 200)])
def test_pack_and_unpack(cabi, K, N, bits, G, C, dtype):
    w, idx = layer(K, N, C, dtype, K + N)
    ref = O.pack(w, idx, bits, G)
    got = gpu_pack(cabi, w, idx, bits, G)
    for key in ("qweight", "scales", "cherry_weight", "cherry_indices"):
        assert np.array_equal(got[key].view(np.uint8), ref[key].view(np.uint8)), key
    dense = O.unpack(ref["qweight"], ref["scales"], ref["cherry_weight"], ref["cherry_indices"], bits, G, K)
    assert np.array_equal(gpu_unpack(cabi, ref, bits, K, G).view(np.uint16), dense.view(np.uint16))


@pytest.mark.parametrize("dtype", [np.float16, np.float32])
@pytest.mark.parametrize("K,N,G,C", [(1040, 2056, 1040, 16), (1040, 200, 1040, 16), (520, 4104, 520, 0), (520, 1000, 520, 0),
                                     (1552, 1544, 512, 8)])
def test_pack_of_long_groups(cabi, K, N, G, C, dtype):
    """Groups of several chunks, on both sides of the rule between the one-pass kernel and the general pair."""
    w, idx = layer(K, N, C, dtype, K + N)
    ref = O.pack(w, idx, 3, G)
    got = gpu_pack(cabi, w, idx, 3, G)
    for key in ("qweight", "scales", "cherry_weight", "cherry_indices"):
        assert np.array_equal(got[key].view(np.uint8), ref[key].view(np.uint8)), key


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("K,N,G,C", [(264, 72, 1, 24), (264, 72, 4, 24), (264, 8, 12, 16), (520, 136, 20, 64), (1032, 64, 24, 1016),
                                     (128, 64, 64, 120)])
def test_pack_and_unpack_of_narrow_groups_and_many_cherries(cabi, K, N, G, C, bits):
    """Octets with several cherry columns, with group boundaries among them, with no code at all; groups inside an octet."""
    w, idx = layer(K, N, C, np.float16, K + G)
    ref = O.pack(w, idx, bits, G)
    got = gpu_pack(cabi, w, idx, bits, G)
    for key in ("qweight", "scales", "cherry_weight", "cherry_indices"):
        assert np.array_equal(got[key].view(np.uint8), ref[key].view(np.uint8)), key
    dense = O.unpack(ref["qweight"], ref["scales"], ref["cherry_weight"], ref["cherry_indices"], bits, G, K)
    assert np.array_equal(gpu_unpack(cabi, ref, bits, K, G).view(np.uint16), dense.view(np.uint16))


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("K,N,bits,G,C", [(1032, 12296, 4, 128, 16), (1160, 10856, 3, 64, 8), (4096, 3080, 3, 128, 2056),
                                          (2048, 6152, 4, 128, 520)])
def test_pack_of_large_matrices(cabi, K, N, bits, G, C, offset):
    """From 12 million fp16 weights on: rows that end inside a warp's 32, columns inside a block's 128, cherry columns among
    32 columns and so many that a block's columns do not fit the tile; weights and codes off their alignment."""
    w, idx = layer(K, N, C, np.float16, K + N)
    if C == 520:
        idx = np.concatenate([np.arange(1000, 1500), np.arange(2028, 2048)])            # side by side, and at the end
    ref = O.pack(w, idx, bits, G)
    wd = torch.zeros(N * K + offset, dtype=torch.float16, device="cuda")
    wd[offset:] = dev(w).flatten()
    q = torch.zeros(ref["qweight"].size + offset, dtype=torch.uint8, device="cuda")
    t = [dev(np.zeros_like(ref[k])) for k in ("scales", "cherry_weight", "cherry_indices")]
    cabi.check(cabi.lib().cq_pack(wd.data_ptr() + 2 * offset, 0, ptr(dev(idx.astype(np.int32))), bits, K, N, C, G,
                                  q.data_ptr() + offset, *[ptr(a) for a in t], None, None), "pack")
    torch.cuda.synchronize()
    assert np.array_equal(q[offset:].cpu().numpy(), ref["qweight"].ravel())
    for a, key in zip(t, ("scales", "cherry_weight", "cherry_indices")):
        assert np.array_equal(a.cpu().numpy().view(np.uint8), ref[key].view(np.uint8)), key


@pytest.mark.parametrize("K,N,bits,G,C", [(1032, 12296, 4, 128, 8), (8192, 1544, 4, 64, 128), (2064, 12296, 3, 128, 64)])
def test_pack_of_large_matrices_into_unaligned_codes(cabi, K, N, bits, G, C):
    """On the kernel whose warps go down the rows, up to a cherry column in 128, in 64 of wide layers, in 32 of larger ones."""
    w, idx = layer(K, N, C, np.float16, K + N)
    ref = O.pack(w, idx, bits, G)
    q = torch.zeros(ref["qweight"].size + 1, dtype=torch.uint8, device="cuda")
    t = [dev(np.zeros_like(ref[k])) for k in ("scales", "cherry_weight", "cherry_indices")]
    wd, idd = dev(w), dev(idx.astype(np.int32))
    cabi.check(cabi.lib().cq_pack(ptr(wd), 0, ptr(idd), bits, K, N, C, G, q.data_ptr() + 1,
                                  *[ptr(a) for a in t], None, None), "pack")
    torch.cuda.synchronize()
    assert np.array_equal(q[1:].cpu().numpy(), ref["qweight"].ravel())
    for a, key in zip(t, ("scales", "cherry_weight", "cherry_indices")):
        assert np.array_equal(a.cpu().numpy().view(np.uint8), ref[key].view(np.uint8)), key


@pytest.mark.parametrize("N,G,dtype", [(64, 128, np.float16), (64, 128, np.float32), (64, 12, np.float16), (400, 128, np.float16)])
def test_cherry_columns_beyond_32767(cabi, N, G, dtype):
    """The indices are 16-bit words: as signed numbers the upper half of a layer's columns would be negative.  All pack kernels,
    both unpack kernels, and the row and GEMM kernels on the layer."""
    from types import SimpleNamespace
    from cherryq_b200 import QuantLinear
    K, C = 33024, 8
    rng = np.random.default_rng(N + G)
    idx = rng.permutation([0, 100, 32766, 32767, 32768, 32769, 33000, K - 1])
    w = (rng.normal(size=(N, K)) * 0.02).astype(dtype)
    ref = O.pack(w, idx, 4, G)
    got = gpu_pack(cabi, w, idx, 4, G)
    for key in ("qweight", "scales", "cherry_weight", "cherry_indices"):
        assert np.array_equal(got[key].view(np.uint8), ref[key].view(np.uint8)), key
    columns = ref["cherry_indices"].view(np.uint16).astype(np.int32)
    dense = O.unpack(ref["qweight"], ref["scales"], ref["cherry_weight"], columns, 4, G, K)
    assert np.array_equal(gpu_unpack(cabi, ref, 4, K, G).view(np.uint16), dense.view(np.uint16))
    if dtype == np.float16 and G == 128:
        lin = QuantLinear(4, G, None, C / K, K, N, bias=False).cuda()
        lin.pack(SimpleNamespace(weight=dev(w), bias=None, cherry_indices=dev(idx.astype(np.int32)), group_size=G))
        for m in (1, 40):
            x = torch.randn(m, K, device="cuda").half()
            want = x.double() @ dev(dense).double().T
            assert float((lin(x).double() - want).abs().max() / want.abs().max()) <= 2e-3       # fp16 output, as in the parity tests


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("K,N,bits,G,C", [(904, 13928, 3, 1, 8), (1032, 12232, 4, 4, 24), (1160, 10856, 3, 12, 32),
                                          (2048, 6152, 4, 96, 64), (1024, 12296, 3, 64, 0)])
def test_unpack_going_down_the_rows(cabi, K, N, bits, G, C, offset):
    """From 12 million weights on, eight and more blocks of columns, few cherry columns: octets with one inside, with group boundaries, of groups narrower
    than an octet; rows that end inside a tile; codes and outputs off their alignment."""
    w, idx = layer(K, N, C, np.float16, K + G)
    ref = O.pack(w, idx, bits, G)
    t = [dev(ref[k]) for k in ("scales", "cherry_weight", "cherry_indices")]
    q = torch.zeros(ref["qweight"].size + offset, dtype=torch.uint8, device="cuda")
    q[offset:] = dev(ref["qweight"]).flatten()
    out = torch.zeros(N * K + offset, dtype=torch.float16, device="cuda")
    cabi.check(cabi.lib().cq_unpack_dense(q.data_ptr() + offset, *[ptr(a) for a in t], bits, K, N, C, G,
                                          out.data_ptr() + 2 * offset, None), "unpack")
    dense = O.unpack(ref["qweight"], ref["scales"], ref["cherry_weight"], ref["cherry_indices"], bits, G, K)
    assert np.array_equal(out[offset:].cpu().numpy().view(np.uint16), dense.view(np.uint16).ravel())


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("K,N,bits,G,C", [(1032, 24416, 4, 12, 16), (1160, 21704, 3, 96, 24), (2056, 12256, 4, 64, 40), (1032, 24416, 3, 8, 8),
                                          (1024, 24584, 3, 64, 0)])
def test_unpack_of_the_largest_matrices(cabi, K, N, bits, G, C, offset):
    """From 25 million weights on the blocks go down the rows: the edges of test_unpack_going_down_the_rows."""
    test_unpack_going_down_the_rows(cabi, K, N, bits, G, C, offset)


def test_unpack_into_unaligned_buffers(cabi):
    K, N, bits, G, C = 264, 72, 3, 128, 8
    w, idx = layer(K, N, C, np.float16, 5)
    ref = O.pack(w, idx, bits, G)
    t = [dev(ref[k]) for k in ("scales", "cherry_weight", "cherry_indices")]
    q = torch.zeros(ref["qweight"].size + 1, dtype=torch.uint8, device="cuda")
    q[1:] = dev(ref["qweight"]).flatten()
    out = torch.zeros(N * K + 1, dtype=torch.float16, device="cuda")
    cabi.check(cabi.lib().cq_unpack_dense(q.data_ptr() + 1, *[ptr(a) for a in t], bits, K, N, C, G, out.data_ptr() + 2, None), "unpack")
    dense = O.unpack(ref["qweight"], ref["scales"], ref["cherry_weight"], ref["cherry_indices"], bits, G, K)
    assert np.array_equal(out[1:].cpu().numpy().view(np.uint16), dense.view(np.uint16).ravel())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("K,N,bits,G,C", [(128, 3, 4, 128, 8), (264, 5, 3, 64, 16), (1032, 9, 4, 100, 40), (4096, 6, 2, 128, 16),
                                         (2312, 7, 4, 4096, 8)])
def test_fake_quantised_weight(pkg, K, N, bits, G, C, dtype):
    """The kernel's weight and gradient equal the torch expressions', infinite and NaN weights included."""
    from cherryq_b200 import cherry_linear as CL
    w, idx = layer(K, max(N, 4), C, np.float32, K + bits)
    w[3, 5], w[2, 70] = np.inf, np.nan
    lin = CL.QuantLinear(K, w.shape[0], w_bits=bits, group_size=G, cherryq=True, cherry_fraction=C / K).cuda().to(dtype).train()
    lin.weight.data.copy_(dev(w))
    lin.register_cherry_indices(dev(idx.astype(np.int32)))
    assert lin._one_pass(lin.weight)
    got = lin._adjust_weight(lin.weight), lin._adjust_weight(lin.weight, ste=False)
    lin._one_pass = lambda weight: False
    ref = lin._adjust_weight(lin.weight), lin._adjust_weight(lin.weight, ste=False)
    for a, b in zip(got, ref):
        assert a.dtype == b.dtype and torch.equal(a.isnan(), b.isnan())
        assert torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0))
    g = torch.randn_like(lin.weight)
    got[0].backward(g)
    assert torch.equal(lin.weight.grad, g)


@pytest.mark.parametrize("K,N,G,C,M", [(136, 4, 64, 8, 1), (256, 9, 128, 8, 3), (1160, 264, 64, 16, 8), (2048, 520, 256, 8, 9),
                                       (4096, 256, 128, 72, 33), (256, 12, 256, 0, 17)])
def test_fp32_operator(cabi, K, N, G, C, M):
    """vecquant3matmul_cherryq with fp32 activations: exact integer sums, so only the fixed point of x (2^-30 of the power of
    two at the largest of a group's columns, 128 at most), the conversion of a sum and a few fp32 additions round: 1e-6 of the result's norm is four times
    that.  An infinite activation gives the same infinities and NaN as the plain sum."""
    rng = np.random.default_rng(K + M)
    _, idx = layer(K, 8, C, np.float32, K)
    idx = np.sort(idx).astype(np.int32)
    Kc = K - C
    u = rng.integers(0, 8, size=(Kc, N))
    q = O.pack_codes(u.astype(np.uint8), 3)
    s = (rng.random(((Kc + G - 1) // G, N)) * 0.1).astype(np.float32)
    cw = rng.normal(size=(C, N)).astype(np.float32)
    x = rng.normal(size=(M, K)).astype(np.float32)
    x[:, ::7] *= 1e-3
    x[0] *= 1e-30        # steps of x below the smallest normal number (fp32 atomics flush sums below 2^-126: 1e-8 of these)
    base = rng.normal(size=(M, N)).astype(np.float32) * (x.std(axis=1, keepdims=True))
    dense = np.zeros((K, N))
    dense[idx] = cw
    dense[O.normal_columns(K, idx)] = (u - 3.5) * np.repeat(s, G, axis=0)[:Kc].astype(np.float64)

    def run(x):
        out = dev(base.copy())
        t = [dev(a) for a in (x, q, cw, idx, s)]
        cabi.check(cabi.lib().cq_vecquant3matmul_cherryq(ptr(t[0]), ptr(t[1]), ptr(t[2]), ptr(t[3]), ptr(t[4]), ptr(out), M, K,
                                                         q.shape[0], N, C, G, 0, 0, None), "fp32 operator")
        torch.cuda.synchronize()
        return out.cpu().numpy().astype(np.float64)

    ref = x.astype(np.float64) @ dense + base
    y = run(x)
    err = np.linalg.norm(y - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() <= 1e-6, err
    x[M - 1, K // 2 + 1] = np.inf
    with np.errstate(invalid="ignore"):
        ref = x.astype(np.float64) @ dense + base
    y = run(x)
    assert np.array_equal(np.isinf(y), np.isinf(ref)) and np.array_equal(np.sign(y[np.isinf(y)]), np.sign(ref[np.isinf(ref)]))
    assert np.array_equal(np.isnan(y), np.isnan(ref))


@pytest.mark.parametrize("K,N,G,C,M", [(2176, 20008, 64, 40, 3), (2176, 20008, 128, 8, 16), (1024, 516, 128, 8, 9)])
def test_fp32_operator_of_wide_layers(cabi, K, N, G, C, M):
    """Several blocks of 512 columns, the last one short; cherry columns shared by all parts of K, in the last one alone, and
    in parts of their own.  Bound as in test_fp32_operator."""
    test_fp32_operator(cabi, K, N, G, C, M)


@pytest.mark.parametrize("K,N,G,C,M", [(2048, 5632, 128, 512, 9), (2048, 5632, 64, 256, 1), (1024, 516, 128, 72, 16)])
def test_fp32_operator_with_many_cherry_columns(cabi, K, N, G, C, M):
    """Shared by the main parts although SMs are left, and in parts of their own, four at a time and what remains of them.  Bound
    as in test_fp32_operator."""
    test_fp32_operator(cabi, K, N, G, C, M)


@pytest.mark.parametrize("K,N,C,M,ratio", [(1024, 264, 8, 9, 1e4), (2120, 40, 24, 3, 1e4), (1024, 264, 8, 17, 1e-5)])
def test_fp32_operator_groups_of_unlike_magnitudes(cabi, K, N, C, M, ratio):
    """Groups of 64 columns whose activations are `ratio` times their neighbours' and whose scales as much smaller: the
    products have one magnitude, and those of each group keep their own bits.  Bound as in test_fp32_operator.  A NaN in
    one group reaches every output of its row and no other row."""
    rng = np.random.default_rng(K + M)
    idx = np.sort(rng.permutation(K)[:C]).astype(np.int32)
    Kc = K - C
    u = rng.integers(0, 8, size=(Kc, N))
    q = O.pack_codes(u.astype(np.uint8), 3)
    big = np.arange((Kc + 63) // 64) % 2 == 0
    s = ((rng.random((len(big), N)) + 0.1) * np.where(big, 1 / ratio, 1.0)[:, None]).astype(np.float32)
    cw = rng.normal(size=(C, N)).astype(np.float32)
    x = rng.normal(size=(M, K)).astype(np.float32)
    cols = O.normal_columns(K, idx)
    x[:, cols] *= np.repeat(np.where(big, ratio, 1.0), 64)[:Kc].astype(np.float32)
    dense = np.zeros((K, N))
    dense[idx] = cw
    dense[cols] = (u - 3.5) * np.repeat(s, 64, axis=0)[:Kc].astype(np.float64)

    def run(x):
        out = torch.zeros(M, N, device="cuda")
        t = [dev(a) for a in (x, q, cw, idx, s)]
        cabi.check(cabi.lib().cq_vecquant3matmul_cherryq(ptr(t[0]), ptr(t[1]), ptr(t[2]), ptr(t[3]), ptr(t[4]), ptr(out), M, K,
                                                         q.shape[0], N, C, 64, 0, 0, None), "fp32 operator")
        torch.cuda.synchronize()
        return out.cpu().numpy().astype(np.float64)

    ref = x.astype(np.float64) @ dense
    y = run(x)
    err = np.linalg.norm(y - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() <= 1e-6, err
    x[M - 1, cols[70]] = np.nan
    z = run(x)
    assert np.isnan(z[M - 1]).all()
    assert np.linalg.norm(z[:M - 1] - ref[:M - 1]) <= 1e-6 * np.linalg.norm(ref[:M - 1])


def test_fake_quantised_weight_under_transforms(pkg):
    """torch.func over the training layer takes the torch expressions: the values and gradients of the layer by itself."""
    from cherryq_b200 import cherry_linear as CL
    K, N, C = 264, 24, 16
    w, idx = layer(K, N, C, np.float32, 3)
    lin = CL.QuantLinear(K, N, w_bits=4, group_size=64, cherryq=True, cherry_fraction=C / K).cuda().train()
    lin.register_cherry_indices(dev(idx.astype(np.int32)))
    w = dev(w)
    x = torch.randn(3, K, device="cuda")

    def loss(w, x):
        return torch.func.functional_call(lin, {"weight": w}, (x,)).square().sum()

    def plain(w, x):
        w = w.clone().requires_grad_()
        y = loss(w, x)
        return y.detach(), torch.autograd.grad(y, w)[0]

    # fp32 sums in another order: 1e-5 of the norm is over ten times K * 2^-24
    def same(a, b):
        assert float((a - b).norm() / b.norm()) <= 1e-5

    value, grad = plain(w, x)
    same(torch.func.grad(loss)(w, x), grad)
    same(torch.func.vmap(torch.func.grad(loss), (None, 0))(w, x), torch.stack([plain(w, r)[1] for r in x]))
    t = torch.randn_like(w)
    v, tangent = torch.func.jvp(lambda w: loss(w, x), (w,), (t,))
    same(v, value)
    same(tangent, (grad * t).sum())
    ws = torch.stack([w, 2 * w])
    same(torch.func.vmap(loss, (0, None))(ws, x), torch.stack([plain(v, x)[0] for v in ws]))
