"""The mask bits of waypoints and targets (lib.waypoint_bits) against one widened mask at a time."""
import numpy as np
import pytest

from fdt_b200 import lib


def _mask(seed, *shape):
    return (np.random.default_rng(seed).random(shape) > 0.5).astype(np.float32)


def _reference(masks):
    bits = np.zeros(np.shape(masks[0]), np.uint32)
    for w, m in enumerate(masks):
        bits |= (np.asarray(m) != 0).astype(np.uint32) << np.uint32(w)
    return bits.view(np.int32)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("shapes", [[(3, 4, 5)], [(3, 4, 5), (5,)], [()]], ids=["equal", "broadcast", "scalars"])
def test_bits_equal_one_mask_at_a_time(n, shapes):
    masks = [_mask(i, *shapes[i % len(shapes)]) for i in range(n)]
    got, want = lib.waypoint_bits(masks), _reference(masks)
    assert got.shape == want.shape and got.dtype == want.dtype and got.flags.c_contiguous
    assert np.array_equal(got, want)


@pytest.mark.parametrize("position", [0, 1, 7, 8, 9, 16])
def test_first_mask_gives_the_shape(position):
    """A mask that broadcasts to the first one's shape is taken at every position, and a larger one refused."""
    small, large = [_mask(i, 3, 4, 5) for i in range(17)], [_mask(i, 1, 4, 5) for i in range(17)]
    small[max(position, 1)] = _mask(99, 5)
    assert np.array_equal(lib.waypoint_bits(small), _reference(small))
    large[max(position, 1)] = _mask(99, 3, 4, 5)
    with pytest.raises(ValueError):
        lib.waypoint_bits(large)


def test_fortran_order_gives_a_contiguous_volume():
    masks = [np.asfortranarray(_mask(i, 3, 4, 5)) for i in range(9)]
    got = lib.waypoint_bits(masks)
    assert got.flags.c_contiguous and np.array_equal(got, _reference(masks))
