"""Q3G64_F16S decode GEMV through the C ABI against the oracle (modelled on native/tests/test_q3_kernels.py)."""

import numpy as np
import pytest

from euhedral_b200 import layouts, library, sharding
from oracle import oracle_c as OC
from oracle import oracle_np as O
from tests.gpu_util import Device, max_relative_error, random_x

pytestmark = pytest.mark.gpu

SHAPES = [(1024, 16), (1024, 64), (5120, 96), (17408, 32), (5120, 1024), (128, 16), (2560, 192)]  # (K, N)


@pytest.fixture(scope="module")
def dev():
    device = Device()
    yield device
    assert device.gpu.take_device_error() == 0
    device.release()


def random_tensor(rng, n, k):
    """Random codes and edge FP16 scales (zero, subnormal, large, negative), as the reference's kernel test does
    (native/tests/test_q3_kernels.py:25,121-133)."""
    codes = rng.integers(-4, 4, size=(n, k)).astype(np.int8)
    groups = k // 64
    scales = (rng.standard_normal((n, groups)) * 0.01).astype(np.float16)
    scales[0, 0] = 0.0
    scales[-1, -1] = np.float16(6.0e-8)
    scales[n // 2, groups // 2] = np.float16(-3.5)
    scales[1 % n, 0] = np.float16(1000.0)
    blob = np.frombuffer(O.q3_assemble(codes, scales, n, k), dtype=np.uint8).copy()
    return blob, O.q3_dense(blob.tobytes(), n, k)


def run(dev, x_bits, blob, n, k, reference=False, **select):
    rows = x_bits.shape[0]
    d_x, d_w, d_y = dev.put(x_bits), dev.put(blob), dev.empty(rows * n * 2)
    with dev.submit(**select) as gpu:
        call = gpu.linear_q3_reference_bf16 if reference else gpu.linear_q3_bf16
        call(d_x.data_ptr(), d_w.data_ptr(), d_y.data_ptr(), rows, k, n, blob.size)
    return dev.get(d_y, np.uint16, (rows, n))


def close_to(got_bits, expect):
    got = O.bf16_to_f32(got_bits).astype(np.float64)
    bound = np.abs(expect) * 2.0 ** -7 + np.max(np.abs(expect)) * 1e-3
    return np.all(np.abs(got - expect) <= bound) and max_relative_error(got, expect) <= 2e-3 + 2.0 ** -8


@pytest.mark.parametrize("k,n", SHAPES)
def test_decode_matches_float64(dev, k, n):
    rng = np.random.default_rng(k * 17 + n)
    blob, dense = random_tensor(rng, n, k)
    for rows in (1, 2, 3, 4, 5, 8):
        x = random_x(rng, rows, k)
        assert close_to(run(dev, x, blob, n, k), O.linear_f64(x, dense)), (rows, k, n)


def test_quantized_gaussian_weights(dev):
    rng = np.random.default_rng(0xE1)
    k, n = 5120, 256
    weights = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    blob = OC.q3_quantize(weights)
    x = random_x(rng, 3, k)
    assert close_to(run(dev, x, blob, n, k), O.linear_f64(x, O.q3_dense(blob.tobytes(), n, k)))


@pytest.mark.parametrize("k,n", SHAPES)
def test_rows_are_bitwise_the_one_row_call(dev, k, n):
    rng = np.random.default_rng(k + 3 * n)
    blob, _ = random_tensor(rng, n, k)
    x = random_x(rng, 8, k)
    single = np.concatenate([run(dev, x[r:r + 1], blob, n, k) for r in range(8)])
    for rows in (3, 8):
        assert np.array_equal(run(dev, x[:rows], blob, n, k), single[:rows])
    many = random_x(rng, 32, k)
    grouped = run(dev, many, blob, n, k, row_exact=True)   # without it, more than 8 rows take the prefill route
    for r in (0, 7, 8, 31):
        assert np.array_equal(grouped[r], run(dev, many[r:r + 1], blob, n, k)[0])


def test_scalar_kernel_and_exact_numerics(dev):
    rng = np.random.default_rng(12)
    k, n = 1024, 32
    blob, dense = random_tensor(rng, n, k)
    x = random_x(rng, 2, k)
    reference = run(dev, x, blob, n, k, reference=True)
    assert np.array_equal(reference, O.q3_linear_scalar_kernel(x, blob.tobytes(), n, k))
    dev.gpu.select_exact_numerics(True)
    try:
        assert np.array_equal(run(dev, x, blob, n, k), reference)
    finally:
        dev.gpu.select_exact_numerics(False)
    # K % 128 != 0: no decode kernel, the scalar kernel runs (K is padded to 128 in the layout)
    k2, n2 = 200, 16
    weights = (rng.standard_normal((n2, k2)) * 0.02).astype(np.float32)
    blob2 = OC.q3_quantize(weights)
    x2 = random_x(rng, 2, k2)
    assert np.array_equal(run(dev, x2, blob2, n2, k2), O.q3_linear_scalar_kernel(x2, blob2.tobytes(), n2, k2))


def test_status_codes(dev):
    lib = library.load()
    k, n = 1024, 16
    blob, _ = random_tensor(np.random.default_rng(2), n, k)
    d_x, d_w, d_y = dev.put(random_x(np.random.default_rng(3), 1, k)), dev.put(blob), dev.empty(n * 2)
    call = lib.euhedral_cuda_linear_q3_bf16
    assert call(None, d_w.data_ptr(), d_y.data_ptr(), 1, k, n, blob.size) == library.INVALID_ARGUMENT
    assert call(d_x.data_ptr(), d_w.data_ptr(), d_y.data_ptr(), 1, k, n, 0) == library.INVALID_ARGUMENT
    assert call(d_x.data_ptr(), d_w.data_ptr(), d_y.data_ptr(), 1, k, n, blob.size + 2) == library.FORMAT_MISMATCH
    assert call(d_x.data_ptr(), d_w.data_ptr(), d_y.data_ptr(), 1, k, n, blob.size) == library.SUCCESS


def test_row_shards_equal_the_whole(dev):
    rng = np.random.default_rng(8)
    k, n = 5120, 1024
    blob, _ = random_tensor(rng, n, k)
    x = random_x(rng, 3, k)
    whole = run(dev, x, blob, n, k)
    for shards in (2, 8):
        parts = [run(dev, x, sharding.q3_rows(blob, n, k, s * n // shards, n // shards), n // shards, k) for s in range(shards)]
        assert np.array_equal(np.concatenate(parts, axis=1), whole)


# The last two are the fused objects the reference's converter emits and its host calls as one tensor: query_key_value
# (5120 + 1024 + 1024 rows) and gate_up (2 x 17408 rows), tools/euhedral_artifacts/trellis.py:128-146.
@pytest.mark.parametrize("n,k", [(17408, 5120), (5120, 17408), (1024, 5120), (5120, 5120), (7168, 5120), (34816, 5120)])
def test_model_shapes(dev, n, k):
    rng = np.random.default_rng(0xE1)
    weights = (rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02))
    blob = OC.q3_quantize(weights)
    for rows in (1, 3, 4, 5):
        x = random_x(np.random.default_rng(0xA0 + rows), rows, k)
        got = O.bf16_to_f32(run(dev, x, blob, n, k)).astype(np.float64)
        expect = OC.q3_linear(x, blob, n, k).astype(np.float64)
        assert max_relative_error(got, expect) <= 2e-3 + 2.0 ** -8


# Shapes that take every launch geometry of the decode kernel: tall tensors on the persistent grid (several tiles per warp
# in turn, a last cluster with a short share, an odd tile count), one K slice (no cluster) on the persistent grid, two K
# slices, an odd number of chunks per slice, few rows of tiles.
GRID_SHAPES = [(17424, 5120), (40000, 1024), (3088, 2048), (2000, 1536), (5120, 17408), (48, 4352), (9232, 8192)]  # (N, K)


@pytest.mark.parametrize("n,k", GRID_SHAPES)
def test_launch_geometries(dev, n, k):
    plan = library.decode_plan("q3", 5, k, n)
    assert plan["ctas"] % plan["k_slices"] == 0
    rng = np.random.default_rng(n * 31 + k)
    weights = rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02)
    blob = OC.q3_quantize(weights)
    for rows in (1, 2, 5, 8):
        x = random_x(np.random.default_rng(0xB0 + rows), rows, k)
        got_bits = run(dev, x, blob, n, k)
        got = O.bf16_to_f32(got_bits).astype(np.float64)
        expect = OC.q3_linear(x, blob, n, k).astype(np.float64)
        assert max_relative_error(got, expect) <= 2e-3 + 2.0 ** -8, (rows, n, k)
        if rows == 5:   # every row of the call is the one-row call, bit for bit
            for r in (0, 4):
                assert np.array_equal(run(dev, x[r:r + 1], blob, n, k)[0], got_bits[r])



def slot_chunks(rows, k, n):
    """(chunks of a ring slot, of a piece) of the decode launch: the one choice of warps, slot and depth whose shared memory is the plan's."""
    plan = library.decode_plan("q3", rows, k, n)
    split, team, piece = plan["k_slices"], plan["pieces"], plan["piece_chunks"]
    tiles, widest = n // 16, -(-(k // 128) // split)
    span = min(tiles, -(-tiles // (plan["ctas"] // split)) + 1)
    owned = -(-span // split) + 1 if split > 1 else 0
    found = set()
    for warps in (16, 8, 4, 2, 1):
        for box in {piece, min(piece, 3)}:
            for depth in (3, 2):
                partials = layouts.align_up(rows * (widest * 256 + 64) + widest * 128, 128)
                slots = layouts.align_up(partials + warps * 1024 + owned * split * 512, 128)
                if warps >= team and slots + warps * depth * (16 * box * 48 + 16 * 48 + 8) == plan["shared_bytes"]:
                    found.add(box)
    assert len(found) == 1
    return found.pop(), piece


# Against one-row calls, whose slots hold whole pieces, at the row counts where the rows leave no room for whole ones at some K: even and
# odd cuts, one slice and several, scale planes that TMA takes and that it does not.
@pytest.mark.parametrize("n,k", [(48, 5120), (272, 4224), (4800, 4736), (64, 6016), (32, 8192), (336, 12416), (16, 17408)])
@pytest.mark.parametrize("rows", [6, 7, 8, 24])
def test_rows_in_parted_rings_equal_one_row_calls(dev, n, k, rows):
    rng = np.random.default_rng(n + k + rows)
    blob, _ = random_tensor(rng, n, k)
    x = random_x(rng, rows, k)
    got = run(dev, x, blob, n, k)
    for r in {0, rows // 2, rows - 1}:
        assert np.array_equal(run(dev, x[r:r + 1], blob, n, k)[0], got[r]), r


# Slots of parts, of pieces of five chunks and of four. Among those of four are pieces of three, whose second slot brings nothing that is
# decoded. Scale planes that TMA takes (K a multiple of 512) and that it does not.
@pytest.mark.parametrize("rows,n,k,piece", [(8, 48, 5120, 5), (7, 4800, 5120, 5), (8, 4800, 4736, 5), (8, 32768, 16384, 4), (8, 32768, 14336, 4),
                                            (8, 32768, 14080, 4), (7, 32768, 16000, 4), (8, 24576, 16000, 4)])
def test_slots_of_parts_equal_one_row_calls(dev, rows, n, k, piece):
    assert slot_chunks(rows, k, n) == (3, piece)
    assert slot_chunks(1, k, n) == (piece, piece)
    rng = np.random.default_rng(n + k + rows)
    size, scales = layouts.q3_byte_size(n, k), layouts.q3_scale_offset(n, k)
    blob = rng.integers(0, 256, size, dtype=np.uint8)
    blob[scales:scales + n * k // 32].view(np.float16)[:] = (rng.standard_normal(n * k // 64, dtype=np.float32) * 0.01).astype(np.float16)
    x = random_x(rng, rows, k)
    d_x, d_w, d_y = dev.put(x), dev.put(blob), dev.empty(rows * n * 2)
    with dev.submit() as gpu:
        gpu.linear_q3_bf16(d_x.data_ptr(), d_w.data_ptr(), d_y.data_ptr(), rows, k, n, size)
    got = dev.get(d_y, np.uint16, (rows, n))
    for r in (0, rows // 2, rows - 1):
        with dev.submit() as gpu:
            gpu.linear_q3_bf16(d_x.data_ptr() + r * k * 2, d_w.data_ptr(), d_y.data_ptr(), 1, k, n, size)
        assert np.array_equal(dev.get(d_y, np.uint16, (1, n))[0], got[r]), r
    dev.release()   # some of the weights are large


# Calls of one row, of eight and of nine (eight and one) on the same weight want maps of both kinds of slots, as members of a group too.
@pytest.mark.parametrize("k", [5120, 4736])
def test_a_weight_called_with_changing_row_counts(dev, k):
    rng = np.random.default_rng(k)
    shapes = [1024, 512, 48]
    blobs = [random_tensor(rng, n, k)[0] for n in shapes]
    weights = [dev.put(blob) for blob in blobs]
    x = random_x(rng, 9, k)
    d_x, d_y = dev.put(x), [dev.empty(9 * n * 2) for n in shapes]
    single = [np.concatenate([run(dev, x[r:r + 1], blob, n, k) for r in range(9)]) for n, blob in zip(shapes, blobs)]
    assert slot_chunks(8, k, sum(shapes))[0] == 3 and slot_chunks(1, k, sum(shapes))[0] == 5
    for rows in (1, 8, 9, 1, 7, 2, 8):
        if rows <= 8:
            with dev.submit() as gpu:
                assert gpu.linear_group_bf16("q3", [d_x.data_ptr()] * 3, [w.data_ptr() for w in weights], [y.data_ptr() for y in d_y], rows, k, shapes,
                                             [b.size for b in blobs]) is not False
            for n, y, expect in zip(shapes, d_y, single):
                assert np.array_equal(dev.get(y, np.uint16, (rows, n)), expect[:rows]), (rows, n)
        for n, w, blob, y, expect in zip(shapes, weights, blobs, d_y, single):
            with dev.submit() as gpu:
                gpu.linear_q3_bf16(d_x.data_ptr(), w.data_ptr(), y.data_ptr(), rows, k, n, blob.size)
            assert np.array_equal(dev.get(y, np.uint16, (rows, n)), expect[:rows]), (rows, n)


def test_every_fp16_scale_pattern(dev):
    """The FP16 group scale reaches the sum as its exact FP32 value for every finite bit pattern, subnormals and both
    zeros included (the reference pins its conversion over all 65,536 patterns, native/tests/test_q3_conversion.py:18-41;
    NaN payloads are the scalar oracle's business only, native/src/q3/contiguous.cuh:16-20). One row per pattern: a single
    code 1 under that scale against x = 1, so the output is bf16(f32(scale)) - on the decode kernel and on the scalar one
    (the scale -0 gives +0: every sum starts at +0)."""
    n, k = 65536, 128
    patterns = np.arange(n, dtype=np.uint16)
    finite = ((patterns >> 10) & 31) != 31
    codes = np.zeros((n, k), dtype=np.int8)
    codes[:, 0] = 1
    scales = np.zeros((n, 2), dtype=np.float16)
    scales[:, 0] = np.where(finite, patterns, 0).astype(np.uint16).view(np.float16)
    blob = np.frombuffer(O.q3_assemble(codes, scales, n, k), dtype=np.uint8).copy()
    x = np.zeros((1, k), dtype=np.uint16)
    x[0, 0] = 0x3F80   # 1.0
    expect = O.bf16_bits(scales[:, 0].astype(np.float32))
    expect[0x8000] = 0   # a sum that starts at +0 stays +0 when -0 is added
    for reference in (False, True):
        got = run(dev, x, blob, n, k, reference=reference)[0]
        wrong = np.flatnonzero(finite & (got != expect))
        assert wrong.size == 0, (reference, wrong.size, [(hex(int(i)), hex(int(got[i])), hex(int(expect[i]))) for i in wrong[:12]])
