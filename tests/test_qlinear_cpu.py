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
