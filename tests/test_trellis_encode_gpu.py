"""The converter's trellis tile encoder on the GPU (euhedral_b200_trellis_encode_tiles) against the reference encoder's
golden tiles and against the CPU restatement that those tiles pin."""

import numpy as np
import pytest

from euhedral_b200 import library
from oracle import oracle_c as OC
from oracle import oracle_np as O
from tests.gpu_util import Device

pytestmark = pytest.mark.gpu

RATES = [(32, 2, 0), (40, 2, 0xAAAA), (48, 3, 0), (56, 3, 0xAAAA), (64, 4, 0), (80, 5, 0), (96, 6, 0)]


@pytest.fixture(scope="module")
def dev():
    device = Device()
    yield device
    assert device.gpu.take_device_error() == 0
    device.release()


def encode(dev, tiles, w, need=None, offset=0):
    lib = dev.gpu.lib
    count = tiles.shape[0]
    need = need or lib.euhedral_b200_trellis_encode_scratch_bytes(count, w)
    d_t, d_s, d_h = dev.put(np.ascontiguousarray(tiles, dtype=np.float32)), dev.empty(count * 512), dev.empty(offset + need + 64)
    d_v, d_w = dev.empty(count * 1024), dev.empty(count * w * 2)
    with dev.submit():
        assert lib.euhedral_b200_trellis_encode_tiles(d_t.data_ptr(), count, w, d_s.data_ptr(), d_v.data_ptr(), d_w.data_ptr(), d_h.data_ptr() + offset, need) == 0
    guard = dev.get(d_h[offset + need:], np.uint8, (64,))
    assert np.all(guard == 0xA5) and np.all(dev.get(d_h, np.uint8, (offset,)) == 0xA5)   # nothing beyond the scratch
    encode.decoded, encode.words = dev.get(d_v, np.float32, (count, 256)), dev.get(d_w, np.int16, (count, w))
    return dev.get(d_s, np.uint16, (count, 256))


@pytest.mark.parametrize("w,ka,mask", RATES)
def test_golden_tiles(dev, golden, w, ka, mask):
    g = golden("trellis")
    states = encode(dev, g["tiles_in"], w)
    assert np.array_equal(states, g[f"tiles_{w}_idx"])
    packed = O.trellis_pack_states(states, ka, mask)
    assert np.array_equal(packed, g[f"tiles_{w}_packed"])
    assert np.array_equal(encode.words, packed)       # the library's own packing and values
    assert np.array_equal(encode.decoded.astype(np.float16).view(np.uint16), g[f"tiles_{w}_out"].view(np.uint16))
    assert np.array_equal(O.trellis_decode_tiles(packed, w).view(np.uint16), g[f"tiles_{w}_out"].view(np.uint16))


@pytest.mark.parametrize("w,ka,mask", [(48, 3, 0), (40, 2, 0xAAAA)])
def test_more_tiles_than_ctas_against_the_cpu_restatement(dev, w, ka, mask):
    """Every CTA encodes several tiles in turn (its history slab and cost rows are reused); scaled and shifted inputs."""
    rng = np.random.default_rng(w)
    count = 4 * dev.gpu.multiprocessor_count() + 3
    tiles = (rng.standard_normal((count, 256)) * rng.uniform(0.2, 1.5, (count, 1))).astype(np.float32)
    tiles[0] = 0.0
    tiles[1, ::7] = 4.0
    expect, _ = OC.trellis_encode_tiles(tiles[:24], ka, mask)
    states = encode(dev, tiles, w)
    assert np.array_equal(states[:24], expect)
    again = encode(dev, tiles[count - 8:], w)     # the same tiles at other places of the list: the same states
    assert np.array_equal(again, states[count - 8:])


@pytest.mark.parametrize("w,ka,mask", RATES)
@pytest.mark.parametrize("extra", [0, 1, 2])
def test_tiles_in_flight_against_the_cpu_restatement(dev, w, ka, mask, extra):
    """One tile alone, as many as CTAs and a few more (a CTA with one tile beside CTAs with two): the states of the whole tiles, tiles of
    equal weights (every cost ties), weights beyond FP16 (infinite costs) and no weight at all among them."""
    rng = np.random.default_rng(100 * w + extra)
    count = [1, dev.gpu.multiprocessor_count() + 2, 2 * dev.gpu.multiprocessor_count() + 3][extra]
    tiles = rng.standard_normal((count, 256)).astype(np.float32)
    if count > 1:
        tiles[1] = 0.25
        tiles[-1, 100:140] = 1e6
        tiles[-2] = 0.0
        tiles[-3, 5] = -70000.0
    states = encode(dev, tiles, w)
    for part in (slice(0, 4), slice(-4, None)):
        expect, _ = OC.trellis_encode_tiles(tiles[part], ka, mask)
        assert np.array_equal(states[part], expect)


@pytest.mark.parametrize("w,ka,mask", RATES)
def test_weights_that_are_not_numbers_against_the_cpu_restatement(dev, w, ka, mask):
    """A NaN weight's costs win no comparison: its position and those behind it take the lowest predecessors. At either end of each pass,
    at even and odd positions, NaN of both signs, beside an infinite weight, in a whole tile."""
    rng = np.random.default_rng(w)
    at = [0, 1, 2, 3, 126, 127, 128, 129, 254, 255]
    tiles = rng.standard_normal((len(at) + 4, 256)).astype(np.float32)
    tiles[np.arange(len(at)), at] = np.nan
    tiles[len(at), 0], tiles[len(at), 128] = -np.nan, np.nan
    tiles[len(at) + 1, 0], tiles[len(at) + 1, 1] = np.nan, -np.inf
    tiles[len(at) + 2, 0], tiles[len(at) + 2, 2] = np.inf, np.nan
    tiles[len(at) + 3] = np.nan
    expect, _ = OC.trellis_encode_tiles(tiles, ka, mask)
    assert np.array_equal(encode(dev, tiles, w), expect)


@pytest.mark.parametrize("w,ka,mask", RATES)
@pytest.mark.parametrize("offset", [4, 8, 12])
def test_scratch_at_any_multiple_of_four(dev, w, ka, mask, offset):
    """The scratch need not lie on the boundary of the kernels' widest stores; what is used of it stays inside."""
    rng = np.random.default_rng(w + offset)
    tiles = rng.standard_normal((3, 256)).astype(np.float32)
    expect, _ = OC.trellis_encode_tiles(tiles, ka, mask)
    assert np.array_equal(encode(dev, tiles, w, offset=offset), expect)


@pytest.mark.parametrize("w,ka,mask", [(32, 2, 0), (40, 2, 0xAAAA)])
@pytest.mark.parametrize("count", [1, 2, 150, 299])
def test_two_bits_in_a_slab_an_sm(dev, w, ka, mask, count):
    """At 2 and 2.5 bits a scratch of one slab of 4 MB for each SM will do (half as many CTAs), also at an odd address; less is refused."""
    rng = np.random.default_rng(w + count)
    tiles = rng.standard_normal((count, 256)).astype(np.float32)
    least = min(count, dev.gpu.multiprocessor_count()) << 22
    expect = encode(dev, tiles, w)
    assert np.array_equal(encode(dev, tiles, w, need=least), expect)
    assert np.array_equal(encode(dev, tiles, w, need=least, offset=8), expect)
    assert np.array_equal(encode(dev, tiles, w, need=least + 100), expect)
    ends = np.r_[0:1, count - 1:count]
    assert np.array_equal(expect[ends], OC.trellis_encode_tiles(tiles[ends], ka, mask)[0])
    d_t, d_s, d_h = dev.put(tiles), dev.empty(count * 512), dev.empty(least)
    with dev.submit():
        assert dev.gpu.lib.euhedral_b200_trellis_encode_tiles(d_t.data_ptr(), count, w, d_s.data_ptr(), 0, 0, d_h.data_ptr(), least - 1) == library.SIZE_OVERFLOW


def test_status_codes(dev):
    lib = dev.gpu.lib
    tiles = dev.put(np.zeros((2, 256), dtype=np.float32))
    out, scratch = dev.empty(1024), dev.empty(1 << 20)
    with dev.submit():
        assert lib.euhedral_b200_trellis_encode_tiles(tiles.data_ptr(), 2, 72, out.data_ptr(), 0, 0, scratch.data_ptr(), 1 << 20) == library.ROUTE_UNAVAILABLE
        assert lib.euhedral_b200_trellis_encode_tiles(tiles.data_ptr(), 2, 48, out.data_ptr(), 0, 0, scratch.data_ptr(), 1024) == library.SIZE_OVERFLOW
        assert lib.euhedral_b200_trellis_encode_tiles(0, 2, 48, out.data_ptr(), 0, 0, scratch.data_ptr(), 1 << 20) == library.INVALID_ARGUMENT
    assert lib.euhedral_b200_trellis_encode_scratch_bytes(2, 48) == 2 * 256 * 8192
