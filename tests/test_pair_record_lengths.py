"""Boxes, extents and slab offsets of a wrong length are refused as the
general path refuses them, also where their lengths make up a record's sum
(checked without a device)."""
import pytest

torch = pytest.importorskip("torch")

BOX = (0, 0, 0, 6, 4, 3, 1, 1, 1)


@pytest.fixture()
def T(monkeypatch):
    try:
        from carpet_b200 import transfer
    except ImportError as e:
        pytest.skip(str(e))
    transfer.general = []
    monkeypatch.setattr(transfer, "lib", type("L", (), dict(
        cgx_transfer=staticmethod(lambda *a: transfer.general.append(a) or 0),
        cgx_transfer_pair=staticmethod(lambda *a: pytest.fail("packed"))))())
    return transfer


@pytest.mark.parametrize("dbox,sbox,slab", [(BOX[:8], BOX + (1,), None), (BOX + (1,), BOX[:8], None),
                                            (BOX + (1,), BOX, (0, 0)), (BOX[:8], BOX, (0, 0, 0, 0))])
def test_lengths_that_make_up_the_sum(T, dbox, sbox, slab):
    d = T.Data(BOX, device="cpu")
    with pytest.raises((IndexError, ValueError)):
        T.transfer_data(d, [d], [0.0], dbox, sbox, 0.0, 1, 0, slab_offset=slab, stream=1)
    with pytest.raises((IndexError, ValueError)):
        T.copy_data(d, d, dbox, sbox, slab_offset=slab, stream=1)
    assert not T.general


def test_an_extent_that_makes_up_the_sum(T):
    d, e = T.Data(BOX, device="cpu"), T.Data(BOX, device="cpu")
    e.extent = list(BOX) + [1]
    for dst, src in ((e, d), (d, e)):
        with pytest.raises(ValueError):
            T.transfer_data(dst, [src], [0.0], BOX[:8], BOX, 0.0, 1, 0, stream=1)
    assert not T.general


def test_iterators_reach_the_general_path_whole(T):
    d = T.Data(BOX, device="cpu")
    T.transfer_data(d, [d], [0.0], iter(BOX), map(int, BOX), 0.0, 1, 0, stream=1)
    (args,) = T.general
    assert tuple(args[6]) == BOX and tuple(args[7]) == BOX
