"""GPU parity tests of the prefill GEMM (tcgen05 tensor cores, weights dequantised into tensor
memory) through the C ABI and through the drop-in `quant_cuda` ops, against the reference's dense
mode: x . unpack()^T with the fp16 weights of `unpack()` (golden fixtures / numpy oracle)."""
import ctypes as C

import numpy as np
import pytest

from conftest import golden_cases, load_golden
from oracle import cherryq_oracle as O
from test_gpu_parity import Prepared, dev, make_case, ptr, rel_err
from test_gpu_tile import TilePrepared

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# fp16 inputs, exact fp16 weights of unpack(), fp32 accumulation in the tensor core, one fp16 store:
# the error against the fp64 product is the store's rounding (2^-11 relative per element)
GEMM_TOL = 1e-3


@pytest.fixture(scope="module")
def cabi():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cherryq_b200 import _cabi
    _cabi.lib()
    return _cabi


@pytest.fixture(scope="module")
def qc():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import cherryq_b200
    return cherryq_b200.load_quant_cuda()


def gemm(cabi, p, x, y=None, accumulate=False):
    lib = cabi.lib()
    xd = dev(x) if isinstance(x, np.ndarray) else x
    M = xd.shape[0]
    ws = torch.empty(lib.cq_tlayer_gemm_workspace_bytes(C.byref(p.L), M), dtype=torch.uint8, device="cuda")
    if y is None:
        y = torch.full((M, p.L.N), float("nan"), dtype=torch.float16, device="cuda")
    cabi.check(lib.cq_tlayer_gemm(C.byref(p.L), ptr(xd), p.L.K, ptr(y), p.L.N, M, int(accumulate), ptr(ws),
                                  ptr(p.status), None), "gemm")
    torch.cuda.synchronize()
    assert int(p.status.item()) == 0, f"a device-side wait timed out (status {int(p.status.item())})"
    return y


@pytest.mark.parametrize("name", golden_cases())
@pytest.mark.parametrize("M", [32, 45, 130])
def test_gemm_on_golden_layers(cabi, name, M):
    g = load_golden(name)
    p = TilePrepared(cabi, g["qweight"], g["scales"], g["cherry_weight"], g["cherry_indices"], g["bits"], g["K"], g["G"])
    x = np.random.default_rng(M).normal(size=(M, int(g["K"]))).astype(np.float16)
    y = gemm(cabi, p, x).cpu().numpy()
    assert np.isfinite(y).all()
    ref = x.astype(np.float64) @ g["dense"].astype(np.float64).T          # dense = the reference's unpack()
    assert rel_err(y, ref) <= GEMM_TOL
    y2 = gemm(cabi, p, x).cpu().numpy()
    assert np.array_equal(y.view(np.uint16), y2.view(np.uint16))


@pytest.mark.parametrize("K,N,bits,M", [(4096, 11008, 4, 256), (4096, 11008, 3, 200), (11008, 4096, 4, 128),
                                         (4096, 4096, 3, 33), (4096, 4096, 4, 520)])
def test_gemm_llama7b_shapes(cabi, K, N, bits, M):
    w, idx, pk, dense = make_case(K, N, bits, 128, seed=K + N + bits)
    p = TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], bits, K, 128)
    x = torch.randn(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).half()
    y = gemm(cabi, p, x)
    ref = x.float() @ dev(dense).float().T                                 # fp32 matmul of the dequantised weights
    err = float((y.float() - ref).abs().max() / ref.abs().max())
    assert err <= 2e-3, err


@pytest.mark.parametrize("K,N,bits,G,frac,M", [
    (256, 24, 4, 128, 1 / 16, 40),       # N not a multiple of 16, one row tile mostly empty
    (640, 136, 3, 64, 1 / 32, 64),       # 64-wide groups, two row tiles, second one 8 rows
    (384, 16, 4, -1, 1 / 24, 32),        # one group per row
    (1024, 264, 3, 128, 0.0, 100),       # no cherries
    (512, 128, 4, 256, 0.25, 129),       # 128 cherry columns = 8 cherry items
])
def test_gemm_edge_shapes(cabi, K, N, bits, G, frac, M):
    w, idx = O.make_layer(K, N, bits, K if G == -1 else G, frac, 3, np.float16)
    pk = O.pack(w, idx, bits, K if G == -1 else G)
    dense = O.unpack(pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], bits, K if G == -1 else G, K)
    p = TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], bits, K, G)
    x = np.random.default_rng(7).normal(size=(M, K)).astype(np.float16)
    y = gemm(cabi, p, x).cpu().numpy()
    ref = x.astype(np.float64) @ dense.astype(np.float64).T
    assert rel_err(y, ref) <= GEMM_TOL


def test_gemm_accumulates_like_the_reference(cabi):
    g = load_golden("k256_n32_b4_g128_f16")
    p = TilePrepared(cabi, g["qweight"], g["scales"], g["cherry_weight"], g["cherry_indices"], 4, g["K"], g["G"])
    rng = np.random.default_rng(0)
    x = rng.normal(size=(48, int(g["K"]))).astype(np.float16)
    base = rng.normal(size=(48, int(g["N"]))).astype(np.float16)
    y = gemm(cabi, p, x, y=dev(base.copy()), accumulate=True).cpu().numpy()
    ref = x.astype(np.float64) @ g["dense"].astype(np.float64).T + base.astype(np.float64)
    assert rel_err(y, ref) <= GEMM_TOL


def test_gemm_equals_the_matvec_path(cabi):
    """The same layer and activations through the decode kernel (16 rows at a time) and the GEMM."""
    w, idx, pk, dense = make_case(2048, 512, 4, 128, seed=9)
    p = TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], 4, 2048, 128)
    x = np.random.default_rng(2).normal(size=(64, 2048)).astype(np.float16)
    a = gemm(cabi, p, x).float()
    b = Prepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], 4, 2048, 128).matvec(x).float()
    assert float((a - b).abs().max() / b.abs().max()) <= 2e-3


@pytest.mark.parametrize("bits", [4, 3])
def test_quant_cuda_ops_route_large_batches_to_the_gemm(qc, bits):
    K, N, G, M = 1024, 384, 128, 96
    w, idx, pk, dense = make_case(K, N, bits, G, seed=bits)
    t = [dev(pk[k]) for k in ("qweight", "cherry_weight", "cherry_indices", "scales")]
    x = torch.randn(M, K, device="cuda").half()
    base = torch.randn(M, N, device="cuda").half()
    out = base.clone()
    if bits == 4:
        qc.vecquant4matmul_cherryq(x, t[0], t[1], t[2], t[3], out, G)
    else:
        qc.vecquant3matmul_cherryq(x, t[0], t[1], t[2], t[3], out, G, True)
    torch.cuda.synchronize()
    qc.poll()
    ref = x.float() @ dev(dense).float().T + base.float()
    assert float((out.float() - ref).abs().max() / ref.abs().max()) <= 2e-3
    # the decode path on a slice of the same rows agrees
    out2 = base[:8].clone()
    if bits == 4:
        qc.vecquant4matmul_cherryq(x[:8].contiguous(), t[0], t[1], t[2], t[3], out2, G)
    else:
        qc.vecquant3matmul_cherryq(x[:8].contiguous(), t[0], t[1], t[2], t[3], out2, G, True)
    torch.cuda.synchronize()
    assert float((out2.float() - out[:8].float()).abs().max() / ref.abs().max()) <= 2e-3


@pytest.mark.parametrize("K,N,bits,G,M", [
    (512, 392, 3, 128, 1), (1024, 136, 4, 128, 31), (2048, 1024, 3, 64, 33), (384, 4096, 4, 128, 127), (8192, 1024, 3, 128, 257),
    (2048, 2440, 4, 256, 513), (1024, 9600, 3, 128, 300), (256, 40, 4, 128, 2049)])
def test_gemm_block_tile_and_run_edges(cabi, K, N, bits, G, M):
    """Token blocks that end inside a step of 32, an odd number of row tiles (the pair's second CTA repeats one), calls of
    whole units and calls whose units are all cut into runs; twelve calls back to back on one workspace give the same bits."""
    w, idx, pk, dense = make_case(K, N, bits, G, seed=K + M)
    p = TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], bits, K, G)
    x = torch.randn(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).half()
    y = gemm(cabi, p, x)
    ref = x.float() @ dev(dense).float().T                                 # fp32 matmul of the dequantised weights
    err = float((y.float() - ref).abs().max() / ref.abs().max())
    assert err <= 2e-3, err                                                # as in test_gemm_llama7b_shapes
    lib = cabi.lib()
    ws = torch.empty(lib.cq_tlayer_gemm_workspace_bytes(C.byref(p.L), M), dtype=torch.uint8, device="cuda")
    outs = [torch.full_like(y, float("nan")) for _ in range(12)]
    for o in outs:
        cabi.check(lib.cq_tlayer_gemm(C.byref(p.L), ptr(x), K, ptr(o), N, M, 0, ptr(ws), ptr(p.status), None), "gemm")
    torch.cuda.synchronize()
    assert int(p.status.item()) == 0
    assert all(torch.equal(o, y) for o in outs)


def test_gemm_accumulates_and_strides_unaligned(cabi):
    """Outputs at a 2-byte aligned address with an odd row stride, whole units, added to what is there."""
    K, N, M = 1024, 264, 70
    w, idx, pk, dense = make_case(K, N, 4, 128, seed=2)
    p = TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], 4, K, 128)
    lib = cabi.lib()
    xb = torch.randn(M * (K + 1) + 1, device="cuda").half()
    yb = torch.randn(M * (N + 3) + 1, device="cuda").half()
    x, base = xb[1:].view(M, K + 1)[:, :K], yb[1:].view(M, N + 3).clone()
    ws = torch.empty(lib.cq_tlayer_gemm_workspace_bytes(C.byref(p.L), M), dtype=torch.uint8, device="cuda")
    cabi.check(lib.cq_tlayer_gemm(C.byref(p.L), xb.data_ptr() + 2, K + 1, yb.data_ptr() + 2, N + 3, M, 1, ptr(ws), ptr(p.status), None), "gemm")
    torch.cuda.synchronize()
    ref = x.float() @ dev(dense).float().T + base[:, :N].float()
    got = yb[1:].view(M, N + 3)
    assert float((got[:, :N].float() - ref).abs().max() / ref.abs().max()) <= 2e-3
    assert torch.equal(got[:, N:], base[:, N:])


@pytest.mark.parametrize("M", [70, 9599])
def test_gemm_units_cut_into_runs(cabi, M):
    """On 148 SMs: 70 rows are two units of 33 items, both cut; 9599 rows are 74 whole units and two cut ones in one call.
    Plain, several times, and added to outputs at a 2-byte aligned address with an odd row stride."""
    K, N = 4096, 264
    w, idx, pk, dense = make_case(K, N, 3, 128, seed=3)
    p = TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], 3, K, 128)
    x = torch.randn(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).half()
    ref = x.float() @ dev(dense).float().T
    y = gemm(cabi, p, x)
    assert float((y.float() - ref).abs().max() / ref.abs().max()) <= 2e-3          # as in test_gemm_llama7b_shapes
    for _ in range(4):
        assert torch.equal(gemm(cabi, p, x), y)
    yb = torch.randn(M * (N + 3) + 1, device="cuda").half()
    base = yb[1:].view(M, N + 3).clone()
    ws = torch.empty(cabi.lib().cq_tlayer_gemm_workspace_bytes(C.byref(p.L), M), dtype=torch.uint8, device="cuda")
    cabi.check(cabi.lib().cq_tlayer_gemm(C.byref(p.L), ptr(x), K, yb.data_ptr() + 2, N + 3, M, 1, ptr(ws), ptr(p.status), None), "gemm")
    torch.cuda.synchronize()
    got, want = yb[1:].view(M, N + 3), ref + base[:, :N].float()
    assert float((got[:, :N].float() - want).abs().max() / want.abs().max()) <= 2e-3
    assert torch.equal(got[:, N:], base[:, N:]) and int(p.status.item()) == 0


@pytest.mark.parametrize("K", [128, 256, 384, 512, 640, 896])
def test_gemm_every_fourth_item_of_a_group(cabi, K):
    """Units of 1 to 8 items (a decode group takes every fourth, counted over the units): 20 token blocks x 5 pairs of row
    tiles are whole units and cut ones in one call of 148 SMs."""
    N, M = 1160, 5000
    w, idx, pk, dense = make_case(K, N, 4, 128, seed=K)
    p = TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], 4, K, 128)
    x = torch.randn(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(K)).half()
    ref = x.float() @ dev(dense).float().T
    y = gemm(cabi, p, x)
    assert float((y.float() - ref).abs().max() / ref.abs().max()) <= 2e-3          # as in test_gemm_llama7b_shapes
    assert torch.equal(gemm(cabi, p, x), y)


@pytest.mark.parametrize("widths", [(264, 8), (1024, 4096, 136), (2440, 128, 128, 9600)])
@pytest.mark.parametrize("M,offset", [(1, 0), (45, 1), (300, 0), (2049, 0)])
def test_gemm_of_layers_together_is_the_separate_calls(cabi, widths, M, offset):
    """Layers with fewer, as many and more units than clusters in one launch: the same bits as one by one, also added to
    outputs off their alignment."""
    lib, K, bits, G = cabi.lib(), 1160, 3, 64
    ps = []
    for i, N in enumerate(widths):
        _, _, pk, _ = make_case(K, N, bits, G, seed=N + i)
        ps.append(TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], bits, K, G))
    n, g = len(ps), torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=g).half()
    base = [torch.randn(M * N + offset, device="cuda", generator=g).half() for N in widths]
    want = []
    for p, b, N in zip(ps, base, widths):
        y = b.clone()[offset:].view(M, N)
        ws = torch.empty(lib.cq_tlayer_gemm_workspace_bytes(C.byref(p.L), M), dtype=torch.uint8, device="cuda")
        cabi.check(lib.cq_tlayer_gemm(C.byref(p.L), ptr(x), K, y.data_ptr(), N, M, 1, ptr(ws), ptr(p.status), None), "gemm")
        want.append(y)
    bufs = [b.clone() for b in base]
    ws = torch.empty(lib.cq_tlayers_gemm_workspace_bytes(C.byref(ps[0].L), n, M), dtype=torch.uint8, device="cuda")
    ls = (C.POINTER(type(ps[0].L)) * n)(*[C.pointer(p.L) for p in ps])
    ys = (C.c_void_p * n)(*[b.data_ptr() + 2 * offset for b in bufs])
    lds = (C.c_int32 * n)(*widths)
    cabi.check(lib.cq_tlayers_gemm(ls, n, ptr(x), K, ys, lds, None, M, 1, ptr(ws), ptr(ps[0].status), None), "gemm")
    torch.cuda.synchronize()
    assert all(int(p.status.item()) == 0 for p in ps)
    for w, b, N in zip(want, bufs, widths):
        assert torch.equal(b[offset:].view(M, N), w)


@pytest.mark.parametrize("N,M", [(8, 9), (136, 45), (2440, 300), (9600, 2049)])
def test_gemm_adds_the_bias_to_the_rounded_outputs(cabi, N, M):
    """Whole units and cut ones, the last rows of a tile; infinite and large biases: the bits of the addition afterwards."""
    lib, K = cabi.lib(), 1160
    _, _, pk, _ = make_case(K, N, 3, 64, seed=N)
    p = TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], 3, K, 64)
    x = torch.randn(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).half()
    buf = torch.randn(N + 1, device="cuda").half()
    bias = buf[1:]                                                          # two bytes off
    bias[2], bias[N - 1] = float("inf"), 60000.0
    y = torch.empty(M, N, dtype=torch.float16, device="cuda")
    ws = torch.empty(lib.cq_tlayers_gemm_workspace_bytes(C.byref(p.L), 1, M), dtype=torch.uint8, device="cuda")
    args = [(C.POINTER(type(p.L)) * 1)(C.pointer(p.L)), 1, ptr(x), K, (C.c_void_p * 1)(y.data_ptr()), (C.c_int32 * 1)(N),
            (C.c_void_p * 1)(bias.data_ptr())]
    cabi.check(lib.cq_tlayers_gemm(*args, M, 0, ptr(ws), ptr(p.status), None), "gemm")
    assert lib.cq_tlayers_gemm(*args, M, 1, ptr(ws), ptr(p.status), None) == 1          # not with accumulate
    torch.cuda.synchronize()
    assert int(p.status.item()) == 0
    assert torch.equal(y, gemm(cabi, p, x) + bias)


@pytest.mark.parametrize("M,offset", [(9, 1), (45, 0), (300, 0), (2049, 1)])
def test_gemm_of_layers_together_adds_each_bias(cabi, M, offset):
    """Layers with whole and with cut units in one launch, every second one with a bias (two bytes off): the bits of the
    separate calls and the addition afterwards, into outputs on and off their alignment."""
    lib, K, bits, G = cabi.lib(), 1160, 3, 64
    widths = (2440, 8, 9600, 136)
    ps = []
    for N in widths:
        _, _, pk, _ = make_case(K, N, bits, G, seed=N)
        ps.append(TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], bits, K, G))
    n = len(ps)
    x = torch.randn(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).half()
    biases = [torch.randn(N + 1, device="cuda").half()[1:] if i % 2 == 0 else None for i, N in enumerate(widths)]
    biases[0][3], biases[2][9599] = float("-inf"), 60000.0
    bufs = [torch.empty(M * N + offset, dtype=torch.float16, device="cuda") for N in widths]
    ws = torch.empty(lib.cq_tlayers_gemm_workspace_bytes(C.byref(ps[0].L), n, M), dtype=torch.uint8, device="cuda")
    ls = (C.POINTER(type(ps[0].L)) * n)(*[C.pointer(p.L) for p in ps])
    ys = (C.c_void_p * n)(*[b.data_ptr() + 2 * offset for b in bufs])
    bs = (C.c_void_p * n)(*[None if b is None else b.data_ptr() for b in biases])
    cabi.check(lib.cq_tlayers_gemm(ls, n, ptr(x), K, ys, (C.c_int32 * n)(*widths), bs, M, 0, ptr(ws), ptr(ps[0].status), None), "gemm")
    torch.cuda.synchronize()
    assert all(int(p.status.item()) == 0 for p in ps)
    for p, buf, b, N in zip(ps, bufs, biases, widths):
        want = gemm(cabi, p, x)
        assert torch.equal(buf[offset:].view(M, N), want if b is None else want + b)


@pytest.mark.parametrize("bits,G", [(3, 64), (3, 128), (4, 128), (4, 256)])
def test_gemm_weights_are_unpacked_exactly_at_every_scale(cabi, bits, G):
    """Rows of the identity read the dequantised weights back: bit for bit unpack()'s, with scales from the smallest
    subnormal to where the largest code reaches fp16's range."""
    K, N = 1024, 264
    w, idx, pk, dense = make_case(K, N, bits, G, seed=bits + G)
    rng = np.random.default_rng(G)
    scales = np.exp2(rng.uniform(-24, 13, size=pk["scales"].shape)).astype(np.float16)
    scales[:, :4] = np.float16(2.0 ** -24)
    dense = O.unpack(pk["qweight"], scales, pk["cherry_weight"], pk["cherry_indices"], bits, G, K)
    p = TilePrepared(cabi, pk["qweight"], scales, pk["cherry_weight"], pk["cherry_indices"], bits, K, G)
    y = gemm(cabi, p, torch.eye(K, device="cuda").half())
    assert torch.equal(y.T, dev(dense))


@pytest.mark.parametrize("M", [16, 300])
def test_gemm_behind_a_kernel_that_waits_for_long(cabi, M):
    """Programmatic launches let the GEMM start while an exchange two kernels before it still waits, here for a rank that
    does not exist and 1.5 s long: longer than the GEMM's own waits may last, which only begin afterwards."""
    import cherryq_b200
    qc = cherryq_b200.load_quant_cuda()
    lib = cabi.lib()
    K, N = 2048, 1024
    w, idx, pk, dense = make_case(K, N, 4, 128, seed=M)
    p = TilePrepared(cabi, pk["qweight"], pk["scales"], pk["cherry_weight"], pk["cherry_indices"], 4, K, 128)
    h = torch.randn(M, K, device="cuda").half()
    ones = torch.ones(K, dtype=torch.float16, device="cuda")
    want = gemm(cabi, p, qc.rmsnorm(h, None, ones, 1e-5, False)[0])
    region = C.c_void_p()
    cabi.check(lib.cq_peer_region_create(1 << 20, C.byref(region)), "create")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    x = torch.randn(1, 256, device="cuda").half()
    out = torch.zeros(1, 512, dtype=torch.float16, device="cuda")
    y = torch.zeros_like(want)
    ws = torch.empty(lib.cq_tlayer_gemm_workspace_bytes(C.byref(p.L), M), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    regions = (C.c_void_p * 2)(region.value, region.value)
    cabi.check(lib.cq_peer_allgather(regions, 2, 0, 1 << 20, ptr(x), ptr(out), 1, 256, 1500, ptr(status), stream), "exchange")
    xn = qc.rmsnorm(h, None, ones, 1e-5, False)[0]
    cabi.check(lib.cq_tlayer_gemm(C.byref(p.L), ptr(xn), K, ptr(y), N, M, 0, ptr(ws), ptr(p.status), stream), "gemm")
    torch.cuda.synchronize()
    cabi.check(lib.cq_peer_region_destroy(region), "destroy")
    assert int(status.item()) & 8                                  # the exchange ran into its limit
    assert int(p.status.item()) == 0
    assert torch.equal(y, want)
