"""When QuantLinear forgets its re-packed copies: host logic, with stand-ins for the copies."""
import pytest

torch = pytest.importorskip("torch")

NAMES = ("qweight", "scales", "cherry_weight", "cherry_indices")


def layer():
    from cherryq_b200 import QuantLinear
    lin = QuantLinear(4, 128, None, 1 / 64, 1024, 264, bias=False)
    lin._sync_key()
    lin._row = lin._tile = "copy"
    return lin


def test_copies_follow_storages_and_versions():
    lin = layer()
    lin._sync_key()
    assert lin._tile == "copy"
    lin.scales.add_(1)                                             # written in place
    lin._sync_key()
    assert lin._row is None and lin._tile is None
    lin._tile = "copy"
    lin.qweight = lin.qweight.clone()                              # replaced, the old one still alive
    lin._sync_key()
    assert lin._tile is None


@pytest.mark.parametrize("name", NAMES)
def test_copies_go_with_a_buffer_replaced_at_the_same_address(name):
    """The allocator hands the freed block to the next tensor of the size; its version is 0 like the old one's."""
    for _ in range(50):
        lin = layer()
        old = getattr(lin, name)
        ptr, shape, dtype = old.data_ptr(), old.shape, old.dtype
        del old
        setattr(lin, name, None)
        setattr(lin, name, torch.empty(shape, dtype=dtype))
        if getattr(lin, name).data_ptr() == ptr and getattr(lin, name)._version == 0:
            break
    else:
        pytest.skip("the allocator did not hand the freed block back")
    lin._sync_key()
    assert lin._row is None and lin._tile is None


def test_copy_and_pickle_leave_the_copies_behind():
    """A module that has answered calls copies and pickles like one that has not; a released one is refused."""
    import copy
    import io
    lin = layer()
    lin._fast = lin._prepared = lock = __import__("threading").Lock()          # not to be pickled, like a copy on the GPU
    lin.scales.fill_(2)
    buf = io.BytesIO()
    torch.save(lin, buf)
    buf.seek(0)
    for other in (copy.deepcopy(lin), copy.copy(lin), torch.load(buf, weights_only=False)):
        assert all(torch.equal(getattr(other, n), getattr(lin, n)) for n in NAMES)
        assert other._row is other._tile is other._fast is other._prepared is other._prepared_key is None
        other._sync_key()
    assert lin._tile == "copy" and lin._fast is lock
    lin._prepared_key = "released"
    with pytest.raises(TypeError):
        copy.deepcopy(lin)


def _wrapped_call(kind, lin, monkeypatch):
    """Something that a call of the layer runs besides QuantLinear.forward; returns what takes it away again."""
    from cherryq_b200 import QuantLinear
    if kind == "instance forward":                                 # as device-placement wrappers and adapters set it
        own = lin.forward
        lin.forward = lambda x: own(x) + 1
    elif kind == "instance _forward":
        own = lin._forward
        lin._forward = lambda x: own(x) + 1
    elif kind == "class forward":
        own = QuantLinear.forward
        monkeypatch.setattr(QuantLinear, "forward", lambda self, x: own(self, x) + 1)
    elif kind == "subclass call":
        lin.__class__ = type("Sub", (QuantLinear,), {"__call__": lambda self, x: QuantLinear.__call__(self, x) + 1})
    elif kind == "hook":
        return lin.register_forward_hook(lambda m, a, o: o + 1).remove
    elif kind == "compiled":
        lin._compiled_call_impl = lambda x: x
    else:
        register = getattr(torch.nn.modules.module, kind)
        return register(lambda *a: None).remove
    return lambda: None


@pytest.mark.parametrize("kind", ["instance forward", "instance _forward", "class forward", "subclass call", "hook", "compiled",
                                  "register_module_forward_hook", "register_module_forward_pre_hook",
                                  "register_module_full_backward_hook"])
def test_layers_that_share_an_input_keep_their_own_calls(kind, monkeypatch):
    """One launch stands for the calls of several layers only where each call is QuantLinear.forward and nothing else."""
    from types import SimpleNamespace
    from cherryq_b200 import QuantLinear, qlinear
    monkeypatch.setattr(QuantLinear, "_row_limit", lambda self: 8)
    monkeypatch.setattr(QuantLinear, "tile_layer", lambda self: "copy")
    x = SimpleNamespace(is_cuda=True, dtype=torch.float16, shape=(16, 1024))
    lins = [layer(), layer()]
    assert qlinear._tile_copies(lins, x, 16) == ["copy", "copy"]
    remove = _wrapped_call(kind, lins[1], monkeypatch)
    try:
        assert qlinear._tile_copies(lins, x, 16) is None
    finally:
        remove()


@pytest.mark.parametrize("rows", [1, 2, 4, 5])
def test_the_norm_rides_in_the_launch_for_one_row(rows, monkeypatch):
    """For more rows the norm kernel in front of the layers is the faster way."""
    from types import SimpleNamespace
    from cherryq_b200 import qlinear
    lins = [layer(), layer()]
    for lin in lins:
        lin.row_layer = lambda n=1: "copy"
    calls = []

    def rmsnorm(h, delta, weight, eps, with_sum):
        calls.append("norm")
        return h, h

    def matvec(*args):
        calls.append("layers")

    def matvec_norm(rls, h, *args):
        calls.append("layers with the norm")
        return h
    fake = SimpleNamespace(rmsnorm=rmsnorm, row_layers_matvec=matvec, row_layers_matvec_norm=matvec_norm)
    monkeypatch.setattr(qlinear, "load_quant_cuda", lambda: fake)
    h, w = torch.ones(rows, 1024, dtype=torch.float16), torch.ones(1024, dtype=torch.float16)
    outs, total = qlinear.forward_normed_input(lins, h, h.clone(), w, 1e-5)
    assert calls == (["layers with the norm"] if rows == 1 else ["norm", "layers"])
    assert [o.shape for o in outs] == [(rows, 264)] * 2 and total is h


def test_layers_that_share_an_input_are_looked_at_once(monkeypatch):
    """The host's part of a call beyond the row kernel's limit: each layer's buffers are compared once, the first one's once
    more for the row kernel."""
    from types import SimpleNamespace
    from cherryq_b200 import QuantLinear, qlinear
    looks = []
    own = QuantLinear._sync_key
    monkeypatch.setattr(QuantLinear, "_sync_key", lambda self: (looks.append(self), own(self)))
    monkeypatch.setattr(qlinear, "_gemm_together", lambda layers, tls, x, rows: tls)
    lins = [layer(), layer(), layer()]
    for lin in lins:
        lin._row_rows = 8
    looks.clear()
    x = SimpleNamespace(is_cuda=True, dtype=torch.float16, shape=(16, 1024), numel=lambda: 16 * 1024)
    assert qlinear.forward_shared_input(lins, x) == ["copy"] * 3
    assert [sum(l is lin for l in looks) for lin in lins] == [2, 1, 1]
